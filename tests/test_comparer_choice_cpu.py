"""Which comparer a pattern group gets (host logic, no GPU), at inputs whose
measured times are far enough apart to say which it should be."""
import random

import pytest


def text(spacers, pam, guides, mm, bulges="", seed=1):
    """An input file: `spacers` = lengths of the spelled parts with 12 N between."""
    rng = random.Random(seed)
    part = lambda f: ("N" * 12).join(f(n) for n in spacers)
    lines = [part(lambda n: "".join(rng.choice("ACGT") for _ in range(n))) + "N" * len(pam) + f" {mm}" for _ in range(guides)]
    return "g\n" + part(lambda n: "N" * n) + pam + bulges + "\n" + "\n".join(lines) + "\n"


# More than 32 counted positions: the alternative is the popcount comparer
# (150 Mbp or, all-N pairs, 30 Mbp; ms with the screen / without).
@pytest.mark.parametrize("spec, kind", [
    (((20, 20), "", 9, 8), "screen"),  # 0.78 / 3.07
    (((20, 20), "", 9, 10), "screen"),  # 1.43 / 3.07
    (((20, 20), "", 32, 8), "screen"),  # 1.58 / 3.07
    (((20, 20), "", 100, 8), "screen"),  # 3.09 / 6.98
    (((20, 20), "", 100, 14), "popcount"),
    (((17, 17), "", 32, 6), "screen"),  # 1.41 / 3.07
    (((40,), "NGG", 32, 12), "screen"),  # 0.58 / 0.92
    (((40,), "NGG", 100, 12), "screen"),  # 1.05 / 2.14
    (((40,), "NGG", 1000, 9), "screen"),  # 2.32 / 14.8
    (((40,), "NGG", 100, 16), "popcount"),  # limits above 15 have no screen
])
def test_long_patterns_compare_with_the_popcount_comparer(P, built, spec, kind):
    assert P.comparer_plan(text(*spec), 30_000_000)["kind"] == kind


# Up to 8 variants the direct count is compared with the comparer that runs
# where no screen can (limits above 15, spellings of fewer than 9 positions;
# ms on 50 Mbp, direct / counted).
@pytest.mark.parametrize("spec, kind", [
    (((32,), "NNGRRT", 8, 16), "bit-sliced"),  # 0.338 / 0.063
    (((25,), "NNAGAAW", 8, 16), "bit-sliced"),  # 0.283 / 0.069
    (((8,), "NNGRRT", 8, 1), "bit-sliced"),  # 0.111 / 0.050
    (((28,), "NGG", 8, 16), "bit-sliced"),  # 0.546 / 0.363
    (((40,), "NNGRRT", 8, 16), "popcount"),  # 0.406 / 0.109
    (((40,), "NGG", 8, 20), "popcount"),  # 0.404 / 0.321
    (((40,), "NGG", 4, 20), "direct"),  # 0.211 / 0.316
    (((8,), "NGG", 1, 1), "direct"),  # 0.031 / 0.100
    (((21,), "NNGRRT", 1, 16), "direct"),  # 0.133 / 0.711: two of three candidates are hits
    (((20,), "NGG", 8, 16), "direct"),  # 2.77 / 3.75
    (((20, 20), "", 8, 16), "direct"),
])
def test_direct_count_is_compared_where_no_screen_can_run(P, built, spec, kind):
    assert P.comparer_plan(text(*spec))["kind"] == kind


# Where the whole count is short, only a screen far ahead is taken.
@pytest.mark.parametrize("spec, kind", [
    (((40,), "NGG", 100, 12), "popcount"),  # 41 / 26 us on 100 kbp
    (((40,), "NGG", 1000, 15), "popcount"),  # 285 / 67 us
    (((20, 20), "", 100, 8), "popcount"),  # 73 / 60 us
    (((40,), "NGG", 20, 8, " 1 1"), "screen"),  # 35 / 88 us
])
def test_long_patterns_on_short_genomes(P, built, spec, kind):
    assert P.comparer_plan(text(*spec), 100_000)["kind"] == kind
