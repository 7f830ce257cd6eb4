"""The recount of many words by the transform of their counts, over plans of
one to three strip sweeps and several parts, against the oracle; and it works
in the memory that the engine holds: the device's free memory does not change
while recounts run."""
import threading

import numpy as np
import pytest

from coldcase_gb300.lns import TransformEngine

pytestmark = pytest.mark.gpu


# one tile; one strip sweep; two with one part and with several; three
@pytest.mark.parametrize("q,n,R,m", [(5, 4, 2, 40000), (7, 6, 2, 200000), (16, 4, 2, 100000), (7, 8, 2, 250000),
                                     (4, 12, 2, 400000), (3, 14, 1, 400000), (9, 7, 3, 100000), (2, 16, 3, 60000), (9, 8, 3, 55000)])
def test_recount_of_many_words(covlib, q, n, R, m):
    from oracle import pyoracle as po
    idx = np.random.default_rng(q + n).integers(0, q ** n, m)
    want = po.cover_count(TransformEngine.index_word(_Cell(q, n), idx), q, n, R)
    e = TransformEngine(q, n, R)
    try:
        e.recount(idx[:3])
        e.gain_map()
        m0 = e.map()
        for _ in range(2):
            e.recount(idx)
            assert (e.cnt() == want).all()
        assert (e.map() == m0).all()             # a recount leaves the last map
        e.recount(idx[:3])
        e.gain_map()
        assert (e.map() == m0).all()
    finally:
        e.close()


class _Cell:
    def __init__(self, q, n):
        self.q, self.pw = q, np.array([q ** (n - 1 - j) for j in range(n)], dtype=np.int64)


def test_recount_allocates_nothing(covlib):
    import torch
    q, n, R = 8, 8, 3                            # 67 MB of word counts
    idx = np.random.default_rng(1).integers(0, q ** n, 200000)
    e = TransformEngine(q, n, R)
    try:
        e.recount(idx)
        torch.cuda.synchronize()
        free = [torch.cuda.mem_get_info()[0]]
        done = threading.Event()

        def watch():
            while not done.is_set():
                free.append(torch.cuda.mem_get_info()[0])

        t = threading.Thread(target=watch)
        t.start()
        try:
            for _ in range(100):
                e.recount(idx)
        finally:
            done.set()
            t.join()
        assert len(free) > 50 and min(free) == free[0]
    finally:
        e.close()
