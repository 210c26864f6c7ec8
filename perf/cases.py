"""Performance cases of the search engine: the searches its users run, through
the public entry points, on synthetic genomes with the statistics of the
benchmark's (41% GC with a drift of +-10% per 100 kbp, N runs, a few other
IUPAC bytes, several records).

The outputs are the rows (bytes) or hit keys a search returns.  The path does
no floating-point work: `work` counts the bytes it cannot do without, and
leaves `flops` at zero (the integer pipe's share is in the design notes).
"""
import ctypes
import importlib
import math

import numpy as np
import torch

P = importlib.import_module("cas-offinder_gb300")

# PAM (written as in the input file's pattern), spacer length, PAM in front.
PAMS = {"NGG": (20, False), "NRG": (20, False), "NNGRRT": (21, False), "NNAGAAW": (20, False),
        "NNNNGMTT": (24, False), "TTTV": (23, True)}
IUPAC = {"A": "A", "C": "C", "G": "G", "T": "T", "R": "AG", "Y": "CT", "K": "GT", "M": "AC", "W": "AT", "S": "CG",
         "H": "ACT", "B": "CGT", "V": "ACG", "D": "AGT", "N": "ACGT"}
CODE = "TCAG"  # plane code hi * 2 + lo of a base


def listed():
    return [
        # A caller with its own device memory searches one 1 Mbp chunk for one
        # compare string: the smallest call, a handful of short launches.
        {"name": "chunk_static", "kind": "static", "n": (1 << 20) - 37, "pam": "NGG", "mm": 4},
        # A bacterial-size genome (10 Mbp), a new four-guide input file per search.
        {"name": "small_genome", "kind": "input", "n": 10_000_000, "records": 4, "pam": "NGG", "guides": 4, "mm": 4,
         "dna": 0, "rna": 0},
        # One guide against a whole human-size genome, no bulges: what a guide
        # design page asks for, a new input file each time.
        {"name": "one_guide", "kind": "input", "n": 3_100_000_023, "records": 24, "pam": "NGG", "guides": 1, "mm": 3,
         "dna": 0, "rna": 0},
        # The headline search: 4 guides, NRG, DNA bulge 2, RNA bulge 1, 5
        # mismatches, whole genome, the same input searched again.
        {"name": "plain", "kind": "repeat", "n": 3_100_000_023, "records": 24, "pam": "NRG", "guides": 4, "mm": 5,
         "dna": 2, "rna": 1},
        # A genome in page-locked host memory, uploaded and searched in one call.
        {"name": "from_host", "kind": "planes", "n": 801_000_007, "records": 8, "pam": "NGG", "guides": 10, "mm": 4,
         "dna": 1, "rna": 0},
        # A batch of single-guide input files of mixed spacer lengths, PAMs,
        # limits and bulges with some degenerate codes, in one search.
        {"name": "batch_mixed", "kind": "batch", "n": 400_000_003, "records": 6, "files": 96, "mm_lo": 3, "mm_hi": 6,
         "dna_hi": 2, "rna_hi": 1},
        # Four PAM families (5' and 3', degenerate), 256 guides each, bulges 1/1.
        {"name": "pam_sets", "kind": "sets", "n": 800_000_011, "records": 8, "guides": 256, "mm": 4, "dna": 1, "rna": 1},
        # A burst of small requests to a server that keeps the genome resident.
        {"name": "served_burst", "kind": "served", "n": 250_000_001, "records": 5, "requests": 48, "guides_hi": 8,
         "mm_hi": 6, "dna_hi": 2, "rna_hi": 1},
        # A CRISPR library screen: 1,000 guides, no bulges, rows streamed to
        # the caller and counted into the summary table.
        {"name": "library", "kind": "stream", "n": 1_000_000_003, "records": 12, "pam": "NGG", "guides": 1000, "mm": 4,
         "dna": 0, "rna": 0},
        # Paired TALEN-style targets (20 + 12 + 20 nt, every start a candidate).
        {"name": "long_pairs", "kind": "long", "n": 30_000_001, "records": 3, "half": 20, "gap": 12, "guides": 3, "mm": 8},
    ]


# ------------------------------------------------------------------ ranges
def _variants(spacer, dna, rna):
    return (1 + dna * spacer if dna else 1) + sum(spacer + 1 - i for i in range(1, rna + 1))


def _density(pam):
    d = 1.0
    for c in pam:
        d *= len(IUPAC[c]) / 4.0
    return 2.0 * d


def _pass_rate(positions, mm):
    return sum(math.comb(positions, k) * 0.75 ** k * 0.25 ** (positions - k) for k in range(min(mm, positions) + 1))


def _expected(case):
    """(variant tests, output bytes) expected of one pass."""
    n, kind = case["n"], case["kind"]

    def of(pam, spacer, guides, mm, dna, rna):
        cand, v = n * _density(pam), guides * _variants(spacer, dna, rna)
        per = 2 * len(pam) + 2 * spacer + 50
        hits = sum(cand * guides * _pass_rate(spacer - (i if i < 0 else 0), mm) for i in range(dna * spacer + 1))
        hits += sum((spacer + 1 - i) * cand * guides * _pass_rate(spacer - i, mm) for i in range(1, rna + 1))
        return cand * v, hits * per

    if kind == "static":
        return n * _density(case["pam"]), 8.0 * 1024
    if kind == "long":
        return n * 2.0 * case["guides"] * 8, n * 2.0 * case["guides"] * _pass_rate(2 * case["half"], case["mm"]) * 180
    if kind == "sets":
        parts = [of(p, s, case["guides"], case["mm"], case["dna"], case["rna"]) for p, s in
                 (("NNGRRT", 21), ("NNNNGMTT", 24), ("NNAGAAW", 20), ("TTTV", 23))]
    elif kind in ("batch", "served"):
        # Mean over the uniform mix of limits, bulges and PAMs.
        parts, count = [], case["files"] if kind == "batch" else case["requests"]
        guides = 1.0 if kind == "batch" else (case["guides_hi"] - 1) / max(math.log(case["guides_hi"]), 0.7) + 0.5
        lo = case.get("mm_lo", 2)
        mix = [(p, m, d, r) for p in ("NGG", "NRG") for m in range(lo, case["mm_hi"] + 1)
               for d in range(case["dna_hi"] + 1) for r in range(case["rna_hi"] + 1)]
        for p, m, d, r in mix:
            t, b = of(p, 21, guides * count / len(mix), m, d, r)
            parts.append((t, b))
    else:
        parts = [of(case["pam"], PAMS[case["pam"]][0], case["guides"], case["mm"], case["dna"], case["rna"])]
    return sum(p[0] for p in parts), sum(p[1] for p in parts)


# Largest expected work of a drawn case: below that of the largest listed one.
MAX_TESTS, MAX_BYTES = 1.0e11, 7.0e7


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "input", "input", "repeat", "planes", "batch", "sets", "served", "stream", "long"])
    case = {"kind": kind}
    if kind == "static":
        return {"kind": kind, "n": _log_int(rng, 20_000, 1 << 21), "pam": rng.choice(sorted(PAMS)), "mm": rng.randint(2, 6)}
    top = {"input": 3.1e9, "repeat": 3.1e9, "planes": 1.0e9, "batch": 6e8, "sets": 1.0e9, "served": 4e8, "stream": 1.5e9,
           "long": 6e7}[kind]
    low = {"input": 2e6, "repeat": 2e7, "long": 1e6}.get(kind, top / 20)
    case["n"] = _log_int(rng, low, top)
    case["records"] = rng.randint(1, 24)
    if kind in ("input", "repeat", "planes"):
        case.update(pam=rng.choice(sorted(PAMS)), guides=_log_int(rng, 1, 24), mm=rng.randint(2, 6), dna=rng.randint(0, 2),
                    rna=rng.randint(0, 2))
    elif kind == "stream":
        case.update(pam=rng.choice(["NGG", "NNGRRT", "TTTV"]), guides=_log_int(rng, 100, 2000), mm=rng.randint(2, 4), dna=0,
                    rna=0)
    elif kind == "batch":
        case.update(files=_log_int(rng, 8, 200), mm_lo=rng.randint(2, 3), mm_hi=rng.randint(4, 6), dna_hi=rng.randint(0, 2),
                    rna_hi=rng.randint(0, 1))
    elif kind == "sets":
        case.update(guides=_log_int(rng, 16, 300), mm=rng.randint(3, 5), dna=rng.randint(0, 1), rna=rng.randint(0, 1))
    elif kind == "served":
        case.update(requests=_log_int(rng, 4, 64), guides_hi=_log_int(rng, 1, 32), mm_hi=rng.randint(3, 6),
                    dna_hi=rng.randint(0, 2), rna_hi=rng.randint(0, 1))
    else:
        case.update(half=rng.randint(15, 20), gap=rng.randint(9, 24), guides=rng.randint(1, 6), mm=rng.randint(5, 10))
    tests, nbytes = _expected(case)
    over = max(tests / MAX_TESTS, nbytes / MAX_BYTES)
    if over > 1:
        case["n"] = max(100_003, int(case["n"] / over))
    return case


def work(case):
    """Planes read once (0.375 bytes per position) and rows written once."""
    return {"bytes": 0.375 * case["n"] + _expected(case)[1], "flops": 0.0}


# ------------------------------------------------------------------ inputs
def _planes(n, records, seed):
    """Random genome planes on the GPU: (hi, lo, ot) int32 tensors, record
    starts, exception positions and bytes."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    words = (n + 31) // 32
    W = words + 4

    def rnd():
        return torch.randint(-2 ** 31, 2 ** 31, (W,), dtype=torch.int32, device=dev, generator=gen)

    # lo = C or G: probability 41% +- 10% per window of 100 kbp, in 1/256 steps,
    # built from random words one binary digit at a time; hi is a fair bit.
    gc = torch.from_numpy(((0.41 + 0.10 * rng.uniform(-1, 1, W // 3125 + 1)) * 256).astype(np.int32)).to(dev)
    gc = gc.repeat_interleave(3125)[:W]
    hi, lo = rnd(), torch.zeros(W, dtype=torch.int32, device=dev)
    for j in range(8):
        r, m = rnd(), -((gc >> j) & 1)
        lo = (lo & r) | (m & (lo | r))
    del gc, r, m
    # Runs of N (5% of positions, 1% in genomes below 50 Mbp), then a few
    # other bytes, the separators and the words past the end.
    frac, most = (0.05, 100_000) if n >= 50_000_000 else (0.01, 10_000)
    most = max(2, min(most, n // 50))
    least = max(1, min(most // 100, 1000))
    k = int(frac * n / (0.5 * (least + most)))
    a = rng.integers(0, n, k)
    b = np.minimum(a + rng.integers(least, most + 1, k), n)
    delta = torch.zeros(W + 1, dtype=torch.int32, device=dev)
    aw, bw = (a + 31) // 32, b // 32  # whole words of N
    whole = aw < bw
    one = torch.ones(int(whole.sum()), dtype=torch.int32, device=dev)
    delta.index_add_(0, torch.from_numpy(aw[whole]).to(dev), one)
    delta.index_add_(0, torch.from_numpy(bw[whole]).to(dev), -one)
    ot = -(delta.cumsum(0)[:W] > 0).to(torch.int32)
    # Ragged ends of the runs, separators, exceptions: single words on the host.
    edge = {}

    def mark(w, mask, h, l):
        o = edge.setdefault(int(w), [0, 0, 0, 0])  # mask, hi, lo of marked bits
        o[1] = (o[1] & ~mask) | (mask if h else 0)
        o[2] = (o[2] & ~mask) | (mask if l else 0)
        o[0] |= mask

    full = 0xFFFFFFFF
    for s, e in zip(a.tolist(), b.tolist()):
        if s // 32 == (e - 1) // 32 and e > s:
            mark(s // 32, ((1 << (e - s)) - 1) << (s % 32), 0, 0)
            continue
        if s % 32:
            mark(s // 32, (full << (s % 32)) & full, 0, 0)
        if e % 32:
            mark(e // 32, (1 << (e % 32)) - 1, 0, 0)
    exc_pos = np.unique(rng.integers(0, n, n // 50_000_000 + 1)).astype(np.uint64)
    lens = np.exp(rng.uniform(0.0, 1.67, records))
    starts = np.concatenate(([0], np.floor(np.cumsum(lens / lens.sum())[:-1] * n).astype(np.int64))) if records > 1 else \
        np.zeros(1, np.int64)
    exc_pos = exc_pos[~np.isin(exc_pos.astype(np.int64), starts[1:] - 1)]
    exc_byte = rng.choice(np.frombuffer(b"MRKY", np.uint8), exc_pos.size)
    for p in exc_pos.tolist():
        mark(p // 32, 1 << (p % 32), 1, 0)
    for s in starts[1:].tolist():
        mark((s - 1) // 32, 1 << ((s - 1) % 32), 0, 1)
    if n % 32:
        mark(n // 32, (full << (n % 32)) & full, 0, 1)
    for w in range(words, W):
        mark(w, full, 0, 1)
    hi &= ~ot
    lo &= ~ot
    at = torch.tensor(list(edge), dtype=torch.int64, device=dev)
    m, h, l = (torch.from_numpy(np.array([e[i] for e in edge.values()], np.uint32).view(np.int32)).to(dev) for i in (0, 1, 2))
    hi[at] = (hi[at] & ~m) | h
    lo[at] = (lo[at] & ~m) | l
    ot[at] |= m
    return hi, lo, ot, starts, exc_pos, exc_byte, rng


def _host(t):
    """Page-locked host copy of a device tensor, as uint32."""
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy().view(np.uint32)


def _sites(rng, planes, n, pattern, count):
    """`count` genome windows that match `pattern` on the forward strand."""
    hi, lo, ot = planes
    L, out = len(pattern), []
    allowed = np.array([[b in IUPAC[c] for b in CODE] for c in pattern])
    while len(out) < count:
        p = rng.integers(0, n - L, 4096)
        pos = p[:, None] + np.arange(L)[None, :]
        w, b = pos >> 5, (pos & 31).astype(np.uint32)
        code = ((hi[w] >> b) & 1) * 2 + ((lo[w] >> b) & 1)
        ok = allowed[np.arange(L)[None, :], code].all(1) & ~((ot[w] >> b) & 1).any(1)
        out += ["".join(CODE[c] for c in row) for row in code[ok][:count - len(out)]]
    return out


def _guides(rng, planes, n, pam, spacer, pam5, count, iupac=0.0):
    """Guides of real targets: spacers next to a PAM of the genome, as the
    input file writes them (N over the PAM)."""
    pattern = pam + "N" * spacer if pam5 else "N" * spacer + pam
    out = []
    for s in _sites(rng, planes, n, pattern, count):
        sp = s[len(pam):] if pam5 else s[:spacer]
        if iupac:
            sp = "".join(rng.choice(list("RYKMWSBDHV")) if rng.random() < iupac else c for c in sp)
        out.append("N" * len(pam) + sp if pam5 else sp + "N" * len(pam))
    return pattern, out


def _text(pattern, dna, rna, guides, mms):
    head = pattern + (f" {dna} {rna}" if dna or rna else "")
    return "\n".join(["resident", head] + [f"{g} {m}" for g, m in zip(guides, mms)]) + "\n"


def _log_uniform(rng, hi):
    return max(1, int(round(math.exp(rng.uniform(0.0, math.log(hi)))))) if hi > 1 else 1


class State:
    """What a program holds between searches: the engine with its resident
    genome, its server, its input files."""

    def __init__(self, kind):
        self.kind, self.engine, self.server = kind, None, None

    def __del__(self):
        if self.server is not None:
            self.server.stop()
        if self.engine is not None:
            self.engine.close()


def _static(case, seed):
    """A chunk in device memory with some sites close to the guide."""
    n, (spacer, pam5) = case["n"], PAMS[case["pam"]]
    hi, lo, ot, _, _, _, rng = _planes(n, 1, seed)
    h = [_host(x) for x in (hi, lo, ot)]
    pattern, guides = _guides(rng, h, n, case["pam"], spacer, pam5, 1)
    site = _sites(rng, h, n, pattern, 1)[0]
    guide, L = guides[0], len(pattern)
    for p in rng.integers(0, n - L, max(1, n // 40_000)).tolist():
        bases = [g if g != "N" else s for g, s in zip(guide, site)]
        for k in rng.choice([i for i, g in enumerate(guide) if g != "N"], rng.integers(0, case["mm"] + 1), replace=False):
            bases[k] = CODE[rng.integers(0, 4)]
        for k, c in enumerate(bases):
            w, b, code = (p + k) >> 5, np.uint32(1 << ((p + k) & 31)), CODE.index(c)
            for plane, bit in ((h[0], code >> 1), (h[1], code & 1), (h[2], 0)):
                plane[w] = (plane[w] | b) if bit else (plane[w] & ~b)
    s = State("static")
    s.planes = [torch.from_numpy(x.view(np.int32)).cuda() for x in h]
    s.hits = torch.full((1024,), 2 ** 63 - 1, dtype=torch.int64, device="cuda")
    s.count = torch.zeros(1, dtype=torch.int64, device="cuda")
    s.args = (n, pattern.encode(), guide.encode(), L, case["mm"])
    return s


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "static":
        return _static(case, seed)
    hi, lo, ot, starts, exc_pos, exc_byte, rng = _planes(n, case["records"], seed)
    h = [_host(x) for x in (hi, lo, ot)]
    del hi, lo, ot
    names = [f"chr{i + 1}" for i in range(len(starts))]
    s = State(kind)
    s.rows = torch.zeros(int(3.5 * _expected(case)[1]) + (4 << 20), dtype=torch.uint8)
    s.engine = P.CasOFFinder(0)
    genome = (*h, n, exc_pos, exc_byte, names, starts.tolist())
    if kind == "planes":
        s.genome = genome
    else:
        s.engine.load_genome_planes(*genome)
    if kind in ("input", "repeat", "planes", "stream"):
        spacer, pam5 = PAMS[case["pam"]]
        pattern, guides = _guides(rng, h, n, case["pam"], spacer, pam5, case["guides"])
        s.text = _text(pattern, case["dna"], case["rna"], guides, [case["mm"]] * len(guides))
        if kind in ("repeat", "planes"):
            s.engine.readInputFile(s.text)
        elif kind == "stream":
            s.engine.set_summary(True)
            s.summary = torch.zeros(case["guides"] * (case["mm"] + 1) * 100, dtype=torch.uint8)
    elif kind == "sets":
        for pam in ("NNGRRT", "NNNNGMTT", "NNAGAAW", "TTTV"):
            spacer, pam5 = PAMS[pam]
            pattern, guides = _guides(rng, h, n, pam, spacer, pam5, case["guides"])
            s.engine.batch_add_input(_text(pattern, case["dna"], case["rna"], guides, [case["mm"]] * len(guides)))
    elif kind == "batch":
        for _ in range(case["files"]):
            spacer, pam = int(rng.integers(20, 25)), str(rng.choice(["NGG", "NRG"]))
            pattern, guides = _guides(rng, h, n, pam, spacer, False, 1, iupac=0.02)
            s.engine.batch_add_input(_text(pattern, int(rng.integers(0, case["dna_hi"] + 1)),
                                           int(rng.integers(0, case["rna_hi"] + 1)), guides,
                                           [int(rng.integers(case["mm_lo"], case["mm_hi"] + 1))]))
    elif kind == "served":
        s.texts = []
        for _ in range(case["requests"]):
            pam = str(rng.choice(["NGG", "NRG", "NNGRRT", "TTTV"]))
            spacer, pam5 = PAMS[pam]
            pattern, guides = _guides(rng, h, n, pam, spacer, pam5, _log_uniform(rng, case["guides_hi"]))
            s.texts.append(_text(pattern, int(rng.integers(0, case["dna_hi"] + 1)), int(rng.integers(0, case["rna_hi"] + 1)),
                                 guides, [int(m) for m in rng.integers(2, case["mm_hi"] + 1, len(guides))]))
        s.server = P.Server(s.engine)
    else:
        half, gap = case["half"], case["gap"]
        L = 2 * half + gap
        guides = [g[:half] + "N" * gap + g[half + gap:] for g in _sites(rng, h, n, "N" * L, case["guides"])]
        s.text = _text("N" * L, 0, 0, guides, [case["mm"]] * len(guides))
    return s


def _keep(s, rows, at=0):
    """The rows of a search at (address, length) copied into the caller's own
    buffer behind the `at` bytes it holds, as a program keeps them past the
    engine's next search: the buffer and the bytes in it."""
    addr, n = rows
    if n:
        src = np.frombuffer((ctypes.c_uint8 * n).from_address(addr), np.uint8)
        s.rows[at:at + n].copy_(torch.from_numpy(src))
    return s.rows, at + n


def run(s):
    if s.kind == "static":
        n, pattern, guide, L, mm = s.args
        st = P.lib().cof_search_chunk_static(*(ctypes.c_void_p(x.data_ptr()) for x in s.planes), n, pattern, guide, L, mm,
                                             ctypes.c_void_p(s.hits.data_ptr()), s.hits.numel(),
                                             ctypes.c_void_p(s.count.data_ptr()),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != P.COF_OK:
            raise P.CofError(st, "cof_search_chunk_static")
        # Hits come in no particular order: the caller sorts its buffer.
        return torch.sort(s.hits).values, s.count
    if s.kind in ("input", "long"):
        s.engine.readInputFile(s.text)
        return _keep(s, s.engine.search_view())
    if s.kind == "planes":
        return _keep(s, s.engine.search_planes_view(*s.genome))
    if s.kind == "stream":
        s.engine.readInputFile(s.text)
        at, table = 0, s.summary.numpy()

        def write(data):
            nonlocal at
            s.rows.numpy()[at:at + len(data)] = np.frombuffer(data, np.uint8)
            at += len(data)

        s.engine.search_stream(write)
        summary = s.engine.summary()
        table[:len(summary)] = np.frombuffer(summary, np.uint8)
        return s.rows, at, s.summary
    if s.kind == "served":
        at = 0
        for t in [s.server.submit(t) for t in s.texts]:
            addr, n, _ = s.server.wait_view(t)
            _, at = _keep(s, (addr, n), at)
            s.server.release(t)
        return s.rows, at
    return _keep(s, s.engine.search_view())
