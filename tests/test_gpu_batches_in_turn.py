"""A batch takes over the previous one's device buffers and captured passes:
searches of different batches in turn give the rows of a fresh engine each."""
import random

import pytest

pytestmark = pytest.mark.gpu


def guides(rng, k, n, pam, mm):
    return "".join("".join(rng.choice("ACGT") for _ in range(n)) + "N" * pam + f" {mm}\n" for _ in range(k))


@pytest.mark.parametrize("autotune", [False, True])
def test_batches_in_turn(P, built, autotune):
    rng = random.Random(29)
    recs = [bytes(rng.choice(b"ACGTACGTN") for _ in range(n)) for n in (700_001, 33)]
    text, starts = P.reference_text(recs)
    inputs = {
        "few": "x\n" + "N" * 20 + "NGG\n" + guides(rng, 3, 20, 3, 6),
        "few_too": "x\n" + "N" * 20 + "NGG\n" + guides(rng, 3, 20, 3, 6),  # same shape, other guides
        "bulges": "x\n" + "N" * 20 + "NRG 2 1\n" + guides(rng, 3, 20, 3, 5),
        "many": "x\n" + "N" * 18 + "NGG\n" + guides(rng, 400, 18, 3, 4),
        "high": "x\n" + "N" * 20 + "NGG\n" + guides(rng, 40, 20, 3, 9),
        "direct": "x\n" + "N" * 23 + "\n" + guides(rng, 2, 23, 0, 9),
        "long": "x\n" + "N" * 45 + "NGG\n" + guides(rng, 2, 45, 3, 22),
    }
    batches = [["few"], ["few_too"], ["many"], ["few"], ["bulges", "few", "direct"], ["high"], ["direct"], ["long", "many"],
               ["bulges"], ["few_too", "bulges"], ["few"], ["few"]]

    def rows(eng, batch):
        eng.batch_clear()
        for name in batch:
            eng.batch_add_input(inputs[name])
        return eng.search()

    fresh = {}
    for batch in batches:
        with P.CasOFFinder(0) as eng:
            eng.set_autotune(False)
            eng.load_genome_text(bytes(text), ["a", "b"], starts)
            fresh[tuple(batch)] = rows(eng, batch)
    assert all(fresh.values())
    with P.CasOFFinder(0) as eng:
        eng.set_autotune(autotune)
        eng.load_genome_text(bytes(text), ["a", "b"], starts)
        for i, batch in enumerate(batches):
            assert rows(eng, batch) == fresh[tuple(batch)], (i, batch)
