"""Searches with few hits are sorted and written without the host knowing their
count; at the edges of that path (hits, text size, jobs) the rows equal those
of the general path, which profiled searches take."""
import random

import pytest

pytestmark = pytest.mark.gpu

SITE = "GATTACAGATTACCAGGCAT"


@pytest.mark.parametrize("hits,name_len", [(0, 4), (1, 4), (33, 4), (1024, 40), (2047, 4), (2048, 4), (2049, 4), (2048, 900)])
def test_few_hits_match_general_path(P, built, hits, name_len):
    rng = random.Random(hits)
    unit = len(SITE) + 3
    recs = [bytearray(rng.choice(b"ACT") for _ in range(unit * (hits // 2 + 3))) for _ in range(2)]
    for i in range(hits):
        at = unit * (i // 2 + 1)
        recs[i % 2][at:at + unit] = (SITE + "TGG").encode()
    text, starts = P.reference_text(recs)
    names = [c * name_len for c in "ab"]
    job = "x\n" + "N" * 20 + "NGG\n" + SITE + "NNN 0\n"
    other = "x\n" + "N" * 20 + "NGG 1 0\n" + SITE + "NNN 1\n"  # bulge rows: several per hit
    with P.CasOFFinder(0) as eng:
        eng.load_genome_text(bytes(text), names, starts)
        eng.set_summary(True)

        def both(load):
            out = []
            for profiled in (False, True):
                load()
                eng.set_profiling(profiled)
                rows = eng.search()
                out.append((rows, eng.last_hit_count(), [eng.job_rows(j) for j in range(eng.batch_size())],
                            [eng.job_summary(j) for j in range(eng.batch_size())]))
                parts = []
                eng.search_stream(parts.append)
                assert b"".join(parts) == rows
            eng.set_profiling(False)
            assert out[0] == out[1]
            return out[0]

        got = both(lambda: eng.readInputFile(job))
        assert got[1][0] == hits and got[0].count(b"\n") == hits
        if hits <= 1024:
            def load():
                eng.batch_clear()
                for j in range(5):
                    eng.batch_add_input(other if j % 2 else job)
            both(load)
