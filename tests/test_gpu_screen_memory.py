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


class Ballast:
    """Device memory taken so that `room` bytes are left free."""

    def __init__(self, torch, room):
        self.torch = torch
        self.block = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.block = None
        self.torch.cuda.empty_cache()


# A search that leaves a list of 512 MiB and both queues behind, and one whose
# hits and rows take about 400 MB.
def few(rng):
    return ["x\n" + "N" * 20 + "NGG\n" + guides(rng, 4, 3), "x\n" + "N" * 23 + "\n" + guides(rng, 20, 2)]


def many(rng):
    return "x\n" + "N" * 20 + "NGG\n" + guides(rng, 9, 10)


def test_search_takes_the_lists_memory_back(P, built):
    """Where memory is short, hits and rows come before the screens' buffers, and
    later searches do not try for larger ones until a genome is loaded."""
    torch = pytest.importorskip("torch")
    genome = random_genome(P, torch, 3 << 26, 1)
    rng = random.Random(4)
    texts, rich = few(rng), many(rng)
    with P.CasOFFinder(0) as eng:
        eng.load_genome_planes(*genome)
        eng.readInputFile(rich)
        want = eng.search()
        assert eng.last_hit_count()[0] > 2_500_000
    with P.CasOFFinder(0) as eng:
        eng.load_genome_planes(*genome)
        for t in texts:
            eng.batch_add_input(t)
        rows = eng.search()
        assert "screen scanning" in eng.schedule()
        with Ballast(torch, 256 * MiB):
            eng.readInputFile(rich)
            assert eng.search() == want
            assert eng.search() == want
        free = torch.cuda.mem_get_info()[0]
        eng.batch_clear()
        for t in texts:
            eng.batch_add_input(t)
        for _ in range(2):
            assert eng.search() == rows
            assert free - torch.cuda.mem_get_info()[0] < 64 * MiB
        eng.load_genome_planes(*genome)
        assert eng.search() == rows
        assert free - torch.cuda.mem_get_info()[0] > 400 * MiB


def test_server_takes_the_lists_memory_back(P, built):
    """The same for a server, whose rows are formatted on another thread."""
    torch = pytest.importorskip("torch")
    genome = random_genome(P, torch, 3 << 26, 1)
    rng = random.Random(4)
    texts, rich = few(rng), many(rng)
    want = []
    with P.CasOFFinder(0) as eng:
        eng.load_genome_planes(*genome)
        for t in texts + [rich]:
            eng.readInputFile(t)
            want.append(eng.search())
    with P.CasOFFinder(0) as eng:
        eng.load_genome_planes(*genome)
        with P.Server(eng) as srv:
            for t, w in zip(texts, want):
                assert srv.wait(srv.submit(t))[0] == w
            torch.cuda.synchronize()
            with Ballast(torch, 256 * MiB):
                for t, w in ((rich, want[2]), (texts[0], want[0]), (rich, want[2])):
                    assert srv.wait(srv.submit(t))[0] == w
