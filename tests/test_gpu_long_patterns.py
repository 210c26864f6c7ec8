"""Variants of more than 32 counted positions, where the choice between the
table screen and the popcount comparer depends on the genome's size: the rows
equal the oracle's on both sides of the line, and a handle whose genome
crosses it chooses anew."""
import random

import pytest

import cases

pytestmark = pytest.mark.gpu


def spelled(seed, k, shape):
    rng = random.Random(seed)
    return ["".join(rng.choice("ACGT") if c == "x" else "N" for c in shape) for _ in range(k)]


@pytest.mark.parametrize("pattern, shape, k, mm", [
    ("N" * 52, "x" * 20 + "N" * 12 + "x" * 20, 9, 10),
    ("N" * 46, "x" * 17 + "N" * 12 + "x" * 17, 33, 7),
    ("N" * 40 + "NRG", "x" * 40 + "NNN", 100, [9, 12]),
])
def test_genome_size_changes_the_choice(pattern, shape, k, mm, P, built, oracle, tmp_path):
    guides = spelled(k, k, shape)
    seen = []
    with P.CasOFFinder(0) as eng:
        want = {}
        for n in (50_000, 5_000_000, 50_000):
            if n not in want:
                tmp = tmp_path / str(n)
                tmp.mkdir()
                inp, _ = cases.make_case(str(tmp), seed=n + k, lens=[n - 9000, 8999], pattern=pattern, mm=mm, guides=guides,
                                         per_guide=12, n_frac=0.02)
                out = str(tmp / "ora.tsv")
                assert cases.run_cli(oracle, inp, out, threads=8).returncode == 0
                want[n] = inp, open(out, "rb").read()
                assert len(cases.rows_of(want[n][1])) > k
            inp, rows = want[n]
            if not seen:  # one input for all genomes
                eng.read_input_path(inp)
            eng.load_genome_file(open(inp).readline().strip())
            assert P.HEADER.encode() + eng.search() == rows
            assert P.HEADER.encode() + eng.search() == rows
            seen.append(eng.comparer_info()["kind"])
    assert seen == ["popcount", "screen", "popcount"]
