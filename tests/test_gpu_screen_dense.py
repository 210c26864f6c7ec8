"""The table screen where candidates crowd: more than 320 of one strand in
2,048 starts (the scanning kernel stages them in rounds), and more passing
candidates in one warp's share than its list has room for (they are counted on
the spot).  Rows against the oracle's; that the branches are reached follows
from the genome, the lists' sizes and the shares."""
import random
import re

import pytest

import cases

pytestmark = pytest.mark.gpu

G = "G" * 20
# Records: runs in which nearly every start is a candidate and a hit, broken
# by N, other bytes and record ends, next to ordinary sequence.
RUNS = ["G" * 5000 + "N" * 30 + "GA" * 2000 + "C" * 3000 + "R" + "C" * 1500, "AGG" * 2100 + "TC" * 1700, "G" * 23, "C" * 2500]


def write(tmp, P, runs, pattern, guides, limit, bulges=""):
    seqs = [bytes(r.encode()) + bytes(P.synth_record(9, i, 9001)) for i, r in enumerate(runs)]
    gpath = str(tmp / "genome.fa")
    cases.write_genome(gpath, "fasta", [f"r{i}" for i in range(len(seqs))], seqs)
    inp = str(tmp / "input.txt")
    with open(inp, "w") as f:
        f.write(gpath + "\n" + pattern + bulges + "\n" + "".join(f"{g} {limit}\n" for g in guides))
    return inp, b";".join(seqs)


def starts_per_unit(genome, pam):
    """Most starts per 2,048 whose window, 20 bytes and `pam`, holds a PAM."""
    counts = {}
    for m in re.finditer(b"(?=[^;]{20}%s)" % pam, genome):
        counts[m.start() // 2048] = counts.get(m.start() // 2048, 0) + 1
    return max(counts.values())


def spelled(k, n):
    rng = random.Random(n)
    return ["".join(rng.choice("ACGT") for _ in range(n)) for _ in range(k)]


def check(P, oracle, inp, tmp):
    out = str(tmp / "ora.tsv")
    assert cases.run_cli(oracle, inp, out, threads=8).returncode == 0
    want = open(out, "rb").read()
    with P.CasOFFinder(0) as eng:
        eng.read_input_path(inp)
        eng.load_genome_file(eng.chrdir)
        assert P.HEADER.encode() + eng.search() == want
        return eng.schedule(), eng.last_hit_count()[0]


@pytest.mark.parametrize("pam, core, guides, limit", [
    ("NGG", b"[ACGTNR]GG", [G, "GA" * 10, "ACGTTGCAACGGTCATGCAT", "AGG" * 6 + "AG"], 4),
    ("NRG", b"[ACGTNR][AG]G", ["R" * 20, "GA" * 10, "C" * 20], 3),
], ids=["NGG", "NRG"])
def test_dense_units_of_the_scanning_screen(pam, core, guides, limit, P, built, oracle, tmp_path):
    inp, genome = write(tmp_path, P, RUNS, "N" * 20 + pam, [g + "NNN" for g in guides], limit)
    assert starts_per_unit(genome, core) > 320
    schedule, hits = check(P, oracle, inp, tmp_path)
    assert " screen scanning " in schedule, schedule
    # Units of 2,048 starts that are all hits: a warp takes a whole unit, and
    # 2^18 items shared out over 24 warps an SM leave room for 71 of them.
    assert hits > 4096


@pytest.mark.parametrize("pattern, guides, limit", [
    ("N" * 23, [G + "GGG"] + spelled(12, 23), 3),
    ("N" * 24, ["GR" * 12] + spelled(12, 24), 2),
    ("N" * 46, ["G" * 46] + spelled(12, 46), 5),
], ids=["three runs", "degenerate", "two words"])
def test_full_lists_of_the_queue_screen(pattern, guides, limit, P, built, oracle, tmp_path):
    inp, genome = write(tmp_path, P, RUNS, pattern, guides, limit)
    schedule, hits = check(P, oracle, inp, tmp_path)
    assert " screen " in schedule and "scanning" not in schedule, schedule
    # A warp takes 64 candidates at a time, all of them hits here and there;
    # 2^18 items shared out over 32 warps an SM leave room for 53.
    assert hits > 4096
