"""The coverage count by tiles (marks on the middle digits, row and column
sums of each block of the last two) against the oracle's ball marking: every
alphabet with its own kernel and the generic one, words of one to a few
digits, every radius, the empty code, repeats, an output at any 2-byte
alignment, tiles of both sizes; and the engine's state build on the same
tiles (counts and private counts of a fresh instance)."""
import ctypes

import numpy as np
import pytest

from coldcase_gb300 import lib as L
from coldcase_gb300.engine import Pool
from coldcase_gb300.workloads import uniform_code

pytestmark = pytest.mark.gpu

CASES = [(q, n, R, m) for q, n, m in ((2, 1, 3), (7, 1, 2), (16, 2, 5), (5, 2, 4), (3, 3, 4), (8, 3, 9), (2, 13, 40),
                                      (3, 8, 50), (4, 6, 60), (5, 6, 70), (6, 5, 30), (7, 5, 33), (8, 5, 21),
                                      (9, 4, 25), (13, 3, 17))
         for R in sorted({0, 1, 2, 3, n}) if R <= n] + [(7, 6, 2, 0), (7, 6, 4, 30000), (6, 7, 3, 9000), (9, 5, 2, 40000)]


@pytest.mark.parametrize("q,n,R,m", CASES)
def test_count_equals_oracle(covlib, q, n, R, m):
    import torch
    from oracle import pyoracle as po
    code = uniform_code(q, n, m, 7 * q + n + R)
    if m > 2:
        code[1] = code[0]
    N = q ** n
    want = po.cover_count(code, q, n, R) if m else np.zeros(N, dtype=np.uint16)
    dev = torch.from_numpy(np.ascontiguousarray(code)).cuda() if m else None
    buf = torch.zeros(N + 8, dtype=torch.int16, device="cuda")
    for off in (0, 1, 2):
        buf.fill_(-7)
        L.check(covlib.cov_count_dev(q, n, R, dev.data_ptr() if m else None, m,
                                     ctypes.c_void_p(buf.data_ptr() + 2 * off), None))
        torch.cuda.synchronize()
        got = buf.cpu().numpy()
        assert (got[off:off + N].view(np.uint16) == want).all(), off
        assert (got[:off] == -7).all() and (got[off + N:] == -7).all()


@pytest.mark.parametrize("q,n,R,m", [(2, 1, 0, 1), (3, 2, 1, 3), (5, 2, 2, 4), (16, 2, 1, 9), (2, 12, 3, 40), (3, 7, 2, 60),
                                     (5, 5, 2, 30), (6, 5, 3, 12), (7, 5, 1, 900), (8, 4, 2, 25), (11, 3, 1, 200),
                                     (7, 4, 1, 20000)])
def test_state_build_equals_oracle(covlib, q, n, R, m):
    from oracle import pyoracle as po
    code = uniform_code(q, n, m, 3 * q + n + R)
    want = po.cover_count(code, q, n, R)
    words = np.stack(np.unravel_index(np.arange(q ** n), (q,) * n), 1).astype(np.uint8)
    with Pool(1, cluster=1) as pool:
        s = pool.add(q, n, R, m, code=code, seed=1)
        assert (pool.cnt(s) == want).all()
        assert pool.status(s)["uncovered"] == int((want == 0).sum())
        # P[k] = (words at distance R that only k covers, how many of them differ from it at each position)
        P = np.zeros((m, n + 1), dtype=np.int64)
        once = np.flatnonzero(want == 1)
        for x in once[:: max(1, len(once) // 4000)] if m > 1000 else once:
            d = (code != words[x][None, :])
            k = np.flatnonzero(d.sum(1) <= R)
            assert len(k) == 1
            if d[k[0]].sum() == R:
                P[k[0], 0] += 1
                P[k[0], 1:] += d[k[0]]
        if m <= 1000:
            assert (pool.private(s) == P).all()
        else:
            assert (pool.private(s) >= P).all()
