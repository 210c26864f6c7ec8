"""The candidates and variant tests a profiled search reports: the same for
every comparer, and exact where one pass over the genome counts more than
2^32 of them."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_planes(P, torch, n, seed):
    """Planes of n random bases (P.pack_text's layout past the end)."""
    W = P.plane_words(n)
    planes = torch.randint(-2 ** 31, 2 ** 31 - 1, (3, W), dtype=torch.int32,
                           generator=torch.Generator().manual_seed(seed)).numpy().view(np.uint32)
    planes[2] = 0
    end = P.pack_text(b"A" * (32 + n % 32))
    for p in range(3):
        planes[p, n // 32 + 1 if n % 32 else n // 32:] = end[p][2 if n % 32 else 1:]
        if n % 32:
            keep = np.uint32((1 << n % 32) - 1)
            planes[p, n // 32] = (planes[p, n // 32] & keep) | (end[p][1] & ~keep)
    return planes


def profiled(eng):
    eng.set_profiling(True)
    eng.reset_stats()
    rows = eng.search()
    got = eng.kernel_stats("finder.candidates")["units"], eng.kernel_stats("comparer.tests")["units"]
    eng.set_profiling(False)
    return rows, got


def test_counts_agree_between_comparers(P, built):
    torch = pytest.importorskip("torch")
    n = (1 << 26) + 4321  # two segments
    rng = random.Random(5)
    planes = random_planes(P, torch, n, 11)
    spacer = ["".join(rng.choice("ACGT") for _ in range(20)) for _ in range(3)]
    batch = ["x\n" + "N" * 20 + pam + "\n" + "".join(f"{s}{'N' * len(pam)} 3\n" for s in spacer)
             for pam in ("NGG", "NNN", "RG")]
    with P.CasOFFinder(0) as eng:
        eng.load_genome_planes(planes[0], planes[1], planes[2], n, None, None, ["c"], [0])
        for t in batch:
            eng.batch_add_input(t)
        seen = []
        for kind in (0, 2, 1):
            eng.set_comparer(kind)
            seen.append(profiled(eng))
            if kind == 0:
                assert " direct" in eng.schedule() and " screen scanning" in eng.schedule(), eng.schedule()
        assert seen[0] == seen[1] == seen[2]


def test_one_pass_counts_past_32_bits(P, built):
    torch = pytest.importorskip("torch")
    n = 2_200_000_011
    planes = random_planes(P, torch, n, 12)
    with P.CasOFFinder(0) as eng:
        eng.load_genome_planes(planes[0], planes[1], planes[2], n, None, None, ["c"], [0])
        eng.readInputFile("x\n" + "N" * 23 + "\n" + "ACGTTGCAACGGTCATGCATGCA 0\n" + "TTGACCATGGACCATTGCAGGAC 1\n")
        _, (candidates, tests) = profiled(eng)
        assert eng.comparer_info()["kind"] == "direct"
        assert candidates == 2 * (n - 22) > 1 << 32
        assert tests == 2 * candidates
