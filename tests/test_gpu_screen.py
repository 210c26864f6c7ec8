"""The table screen on the GPU against the oracle and the other comparers, at
the forms where it can go wrong: three and four runs, one- and two-word
windows, 4- and 5-bit fields, degenerate codes next to non-base bytes, limits
0 to 15, several table words, every start a candidate, a short spacer, and
candidate counts around a warp's and a CTA's share; and the direct count for
inputs of a few variants."""
import pytest

import cases

pytestmark = pytest.mark.gpu

SPECS = [
    dict(seed=301, lens=[90000, 40000], pattern="N" * 21 + "RG", dna=2, rna=1, mm=5, per_guide=40),
    dict(seed=302, lens=[60000, 3000], pattern="N" * 24 + "NRG", dna=2, rna=1, mm=[3, 6, 8], iupac_frac=0.05,
         per_guide=30, sprinkle_chars="MRKYSWn", n_frac=0.05),
    dict(seed=303, lens=[80000], pattern="TTTV" + "N" * 23, dna=1, rna=1, mm=[0, 4], n_guides=40, per_guide=8),
    dict(seed=304, lens=[50000], pattern="N" * 20 + "NAG", dna=1, rna=2, mm=[2, 15], per_guide=10, n_guides=2),
    dict(seed=305, lens=[70000], pattern="N" * 9 + "NGG", mm=2, per_guide=30, n_guides=9),
    dict(seed=306, lens=[40000], pattern="N" * 45 + "NGG", dna=2, rna=1, mm=[4, 5], per_guide=30, iupac_frac=0.02,
         sprinkle_chars="MRKY"),
    dict(seed=307, lens=[30001], pattern="N" * 52, mm=[8, 10], n_guides=70, per_guide=2, n_frac=0.2),
    dict(seed=308, lens=[150000], pattern="N" * 20 + "NGG", mm=[3, 4], n_guides=600, per_guide=2),
    dict(seed=309, lens=[33], pattern="N" * 20 + "NGG", mm=6, n_guides=9, per_guide=1),
    dict(seed=310, lens=[2000, 500], pattern="N" * 32, mm=6, n_guides=40, per_guide=2, iupac_frac=0.1, n_frac=0.3),
]
DIRECT = [
    dict(seed=321, lens=[65536 - 22, 4096], pattern="N" * 22 + "R", mm=4, n_guides=1, per_guide=60, iupac_frac=0.05,
         sprinkle_chars="MRKYSWn", n_frac=0.05),
    dict(seed=322, lens=[20000, 30, 2047], pattern="N" * 52, mm=[8, 60], n_guides=2, per_guide=20, n_frac=0.1),
    dict(seed=323, lens=[50000], pattern="N" * 32, mm=[0, 31], n_guides=2, per_guide=20, iupac_frac=0.2),
    dict(seed=324, lens=[40000, 64], pattern="N" * 61 + "NGG", mm=[20, 3], n_guides=2, per_guide=20),
    dict(seed=325, lens=[22], pattern="N" * 20 + "NGG", mm=20, n_guides=1, per_guide=0),
    dict(seed=326, lens=[23], pattern="N" * 23, mm=20, n_guides=1, per_guide=0),
    dict(seed=327, lens=[90001], pattern="TTTV" + "N" * 20, mm=[5, 18], n_guides=8, per_guide=10),
]


@pytest.mark.parametrize("spec", SPECS + DIRECT, ids=[str(c["seed"]) for c in SPECS + DIRECT])
def test_screen_matches_oracle(spec, P, built, oracle, tmp_path):
    inp, _ = cases.make_case(str(tmp_path), **spec)
    a = str(tmp_path / "ora.tsv")
    assert cases.run_cli(oracle, inp, a, threads=4).returncode == 0
    want = open(a, "rb").read()
    with P.CasOFFinder(0) as eng:
        eng.read_input_path(inp)
        eng.load_genome_file(eng.chrdir)
        for kind in (0, 2, 1, 0):
            eng.set_comparer(kind)
            assert P.HEADER.encode() + eng.search() == want, f"comparer {kind}"
            if kind == 0 and spec["seed"] not in (304, 321, 327):
                assert eng.comparer_info()["kind"] == ("direct" if spec in DIRECT else "screen")
            if kind == 2:
                assert eng.comparer_info()["kind"] in ("popcount", "bit-sliced")
