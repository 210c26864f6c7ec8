"""Device memory of the table screens: buffers that only their speed depends
on are held where a screen uses them."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MiB = 1 << 20


def random_genome(P, torch, n, seed):
    """Planes of n random bases (P.pack_text's layout past the end)."""
    W = P.plane_words(n)
    planes = torch.randint(-2 ** 31, 2 ** 31 - 1, (3, W), dtype=torch.int32,
                           generator=torch.Generator().manual_seed(seed)).numpy().view(np.uint32)
    planes[2] = 0
    assert n % 32 == 0
    for p, words in enumerate(P.pack_text(b"A" * 32)[:3]):
        planes[p, n // 32:] = words[1:]
    return planes[0], planes[1], planes[2], n, None, None, ["c"], [0]


def guides(rng, k, mm):
    return "".join("".join(rng.choice("ACGT") for _ in range(20)) + f"NNN {mm}\n" for _ in range(k))


def test_timing_partitions_holds_no_unused_buffers(P, built):
    """A search whose partitions all scan the planes with one table word needs
    neither a candidate queue (512 MiB) nor a queue's windows (1 GiB)."""
    torch = pytest.importorskip("torch")
    genome = random_genome(P, torch, 3 << 26, 1)
    rng = random.Random(3)
    with P.CasOFFinder(0) as eng:
        eng.load_genome_text(b"ACGT" * 100, ["c"], [0])
        eng.readInputFile("x\n" + "N" * 20 + "NRG 2 1\n" + guides(rng, 4, 3))
        eng.search()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        eng.load_genome_planes(*genome)
        eng.readInputFile("x\n" + "N" * 20 + "NRG 2 1\n" + guides(rng, 4, 3))
        assert eng.search()
        schedule = eng.schedule()
        assert " screen scanning " in schedule and schedule.count("us]") == 2, schedule
        held = (free - torch.cuda.mem_get_info()[0]) / MiB
        # The list of what passes (512 MiB), planes, hits and tables.
        assert held < 800, held
