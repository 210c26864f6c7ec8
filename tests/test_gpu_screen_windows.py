"""Screens of many words look the queue's extracted windows up (windows_kernel):
the rows equal the oracle's for one- and two-word windows, three and four runs,
degenerate guides and windows with non-base bytes, and queue lengths at the
edges of a warp's share."""
import re

import pytest

import cases

pytestmark = pytest.mark.gpu

SPECS = [
    dict(seed=401, lens=[60000, 40000], pattern="N" * 20 + "NGG", dna=1, mm=[3, 6], n_guides=120, per_guide=4),
    dict(seed=402, lens=[50000, 129], pattern="N" * 24 + "NRG", dna=1, rna=1, mm=[4, 6], n_guides=80, per_guide=4,
         iupac_frac=0.05, sprinkle_chars="MRKYSWn", n_frac=0.05),
    dict(seed=403, lens=[40000], pattern="N" * 45 + "NGG", dna=1, mm=[5, 8], n_guides=80, per_guide=3, iupac_frac=0.03,
         sprinkle_chars="MRKY", n_frac=0.1),
    dict(seed=404, lens=[30000, 31], pattern="TTTV" + "N" * 30, dna=1, mm=[5, 7], n_guides=90, per_guide=3),
    dict(seed=405, lens=[23], pattern="N" * 20 + "NGG", dna=1, mm=[4, 5], n_guides=150, per_guide=0),
]


@pytest.mark.parametrize("spec", SPECS, ids=[str(s["seed"]) for s in SPECS])
def test_windows_match_oracle(spec, P, built, oracle, tmp_path):
    inp, _ = cases.make_case(str(tmp_path), **spec)
    out = str(tmp_path / "ora.tsv")
    assert cases.run_cli(oracle, inp, out, threads=4).returncode == 0
    want = open(out, "rb").read()
    with P.CasOFFinder(0) as eng:
        eng.read_input_path(inp)
        eng.load_genome_file(eng.chrdir)
        assert P.HEADER.encode() + eng.search() == want
        words = [int(w) for w in re.findall(r"screen (?!scanning).*? words=(\d+)", eng.schedule())]
        assert words and max(words) >= 8, eng.schedule()
