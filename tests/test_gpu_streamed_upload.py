"""Searches under a streamed upload (scans chunk by chunk as the copies arrive,
finders segment by segment) give the rows of the resident genome's search."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEG = 1 << 26


@pytest.mark.parametrize("n", [1, 22, 5000, SEG // 2 + 70, SEG + 3, 5 * SEG // 2 - 40, 7 * SEG + 1])
def test_streamed_upload(P, built, n):
    torch = pytest.importorskip("torch")
    W = P.plane_words(n)
    rng = random.Random(n)
    planes = torch.randint(-2 ** 31, 2 ** 31 - 1, (3, W), dtype=torch.int32, generator=torch.Generator().manual_seed(n))
    planes[2] = 0
    host = planes.numpy().view(np.uint32)
    if n % 32:
        host[:, n // 32] &= (1 << n % 32) - 1
    host[:, (n + 31) // 32:] = 0
    pos = np.arange(n, 32 * W)  # past the genome: other bytes, as P.pack_text leaves them
    empty = P.pack_text(b"A" * min(n, 100))[2]
    if (empty[-1] >> 31) & 1:
        np.bitwise_or.at(host[2], pos // 32, np.uint32(1) << (pos % 32).astype(np.uint32))
    site = "GATTACAGATTACCAGGCAT"

    def put(at):  # the site with its PAM, across the ends of chunks and segments
        for k, c in enumerate(site + "TGG"):
            code = "TCAG".index(c)
            w, b = (at + k) // 32, np.uint32(1 << (at + k) % 32)
            for p, bit in ((0, code >> 1), (1, code & 1)):
                host[p, w] = host[p, w] | b if bit else host[p, w] & ~b

    ends = {32 * (SEG // 64) * k for k in range(1, n // (SEG // 2) + 1)} | {n}
    for e in ends:
        for at in (e - 70, e - 23 - 20):
            if 0 <= at and at + 23 <= n:
                put(at)
    g = ["".join(rng.choice("ACGT") for _ in range(20)) + "NNN" for _ in range(2)]
    batch = ["x\n" + "N" * 20 + "NGG\n" + site + "NNN 3\n" + f"{g[0]} 4\n",  # scanned
             "x\n" + "N" * 23 + "\n" + site + "NNN 2\n",  # counted at every start
             "x\n" + "N" * 20 + "NNG 1 1\n" + f"{g[0]} 2\n{g[1]} 4\n"]  # queued
    names, starts = ["c"], [0]
    with P.CasOFFinder(0) as eng:
        eng.set_autotune(False)
        eng.load_genome_planes(host[0], host[1], host[2], n, None, None, names, starts)
        eng.batch_clear()
        for t in batch[:2]:
            eng.batch_add_input(t)
        for extra in (None, batch[2] if n < 3 * SEG else None):
            if extra:
                eng.batch_add_input(extra)
            want = eng.search()
            assert n < 200 or want.count(b"\n") >= 2 * len([e for e in ends if e >= 70])
            pinned = torch.empty(3 * W, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32).reshape(3, W)
            pinned[:] = host
            for src in (pinned, host):
                for profiled in (False, True):
                    eng.set_profiling(profiled)
                    got = P._bytes_at(*eng.search_planes_view(src[0], src[1], src[2], n, None, None, names, starts))
                    eng.set_profiling(False)
                    assert got == want
            assert eng.search() == want
