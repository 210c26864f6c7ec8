"""The table screen's plan (host logic, no GPU): every compare variant sits in
one class, and the bound summed over the runs rules out no window that a
direct count against the mismatch rule accepts, whatever the partition."""
import random

import numpy as np
import pytest

from cases import random_guides

BASES = "TCAG"  # plane code hi * 2 + lo
CLASSES = {c: sum((b not in s) << i for i, b in enumerate(BASES)) | 16 * (c in BASES) for c, s in {
    "A": "A", "C": "C", "G": "G", "T": "T", "R": "AG", "Y": "CT", "K": "GT", "M": "AC", "W": "AT", "S": "CG",
    "H": "ACT", "B": "CGT", "V": "ACG", "D": "AGT", "N": BASES}.items()}

SPECS = [("N" * 21 + "GG", 0, 0, [4], 0.0, 4), ("N" * 21 + "RG", 2, 1, [5], 0.0, 4), ("N" * 24 + "NRG", 2, 1, [3, 6, 8], 0.05, 3),
         ("TTTV" + "N" * 23, 1, 1, [0, 4], 0.0, 5), ("N" * 20 + "NAG", 1, 2, [15], 0.0, 2), ("N" * 9 + "NGG", 0, 0, [2], 0.0, 2),
         ("N" * 29 + "NRG", 0, 0, [6], 0.1, 3), ("N" * 45 + "NGG", 2, 1, [9], 0.02, 2), ("N" * 59 + "NGG", 2, 2, [12, 7], 0.0, 2),
         ("N" * 20 + "NGG", 0, 0, [3, 4], 0.0, 150)]


@pytest.mark.parametrize("spec", SPECS, ids=[str(i) for i in range(len(SPECS))])
def test_bound_rules_out_no_hit(P, built, spec):
    pattern, dna, rna, mms, iupac, count = spec
    rng, pam5 = random.Random(str(spec)), pattern[0] != "N"
    core = pattern.rstrip("N") if pam5 else pattern.lstrip("N")
    guides = random_guides(rng, count, len(pattern) - len(core), core, pam5, iupac)
    text = "g\n" + pattern + (f" {dna} {rna}" if dna or rna else "") + "\n" + "".join(
        f"{g} {mms[i % len(mms)]}\n" for i, g in enumerate(guides))
    planned = 0
    for level in range(9):
        s = P.screen_plan(text, level)
        if s is None:
            continue
        planned += 1
        L, rec = s["L"], s["records"]
        top = 1 << (s["bits"] - 1)
        assert sum(s["cap"][:s["K"]]) < 2 * top and sum(s["cap"][:s["K"]]) >= top
        assert sorted(int(r[5]) >> 4 for r in rec) == list(range(s["variants"]))
        # Class masks per record and position, bits T C A G other.
        cls = np.zeros((len(rec), L), np.uint8)
        for k in range(L):
            i = k >= 32
            for b, w in enumerate((8, 9, 10, 11, 6) if i else (0, 1, 2, 3, 4)):
                cls[:, k] |= (((rec[:, w] >> np.uint32(k & 31)) & 1) << b).astype(np.uint8)
        if not dna and not rna and count <= 8:
            assert sorted(map(bytes, cls)) == sorted({bytes(CLASSES[c] for c in g) for g in guides})
        limit = (rec[:, 5] & 15).astype(int)
        # Windows: random, and spelled from variants with up to limit + 2 changes.
        win = np.array([[rng.randrange(4) for _ in range(L)] for _ in range(120)])
        for w in win[:100]:
            v = rng.randrange(len(rec))
            ok = [[b for b in range(4) if not cls[v, k] >> b & 1] for k in range(L)]
            w[:] = [rng.choice(o) for o in ok]
            for k in rng.sample(range(L), min(L, rng.randint(0, int(limit[v]) + 2))):
                w[k] = rng.randrange(4)
        other = np.zeros_like(win, bool)
        for w in other[::5]:
            w[[rng.randrange(L) for _ in range(rng.randint(1, 3))]] = True
        bits = np.where(other, 4, win)
        first = s["first"]
        for w, o, code in zip(win, other, bits):
            direct = ((cls >> code[None, :].astype(np.uint8)) & 1).sum(1)
            hits = set(np.flatnonzero(direct <= limit).tolist())
            low = (cls >> w[None, :].astype(np.uint8)) & 1  # what the tables see: other bytes read as bases
            seen = set()
            for word in range(s["words"]):
                total = 0
                for k in range(s["K"]):
                    a, q, entry = s["a"][k], s["q"][k], 0
                    for c in range(s["fields"]):
                        v0, v1 = first[word, c], first[word, c + 1]
                        d = low[v0:v1, a:a + q].sum(1).astype(int) + (top - 1 - limit[v0:v1] if k == 0 else 0)
                        entry |= min([s["cap"][k], *d.tolist()]) << (c * s["bits"])
                    total += entry
                assert total < 1 << 32
                for c in range(s["fields"]):
                    if not total >> (c * s["bits"]) & top or (s["degenerate"] and o.any()):
                        seen.update(range(first[word, c], first[word, c + 1]))
            assert hits <= seen, (level, hits - seen)
    assert planned
