"""Private counts of a fresh instance at radius 1 for codes longer than one
list chunk of the state build (4096 codewords) that leave many words covered
once: equal to the counts made here from every such word's only coverer."""
import numpy as np
import pytest

from coldcase_gb300.engine import Pool
from coldcase_gb300.workloads import uniform_code

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,n,m", [(7, 6, 6000), (6, 7, 9000), (8, 5, 4097), (5, 8, 12300), (11, 5, 8192), (2, 16, 8000)])
def test_private_counts_of_long_codes(covlib, q, n, m):
    code = uniform_code(q, n, m, q + n)
    code[7] = code[m - 1]                                  # a codeword twice covers nothing alone
    N = q ** n
    pw = q ** np.arange(n - 1, -1, -1, dtype=np.int64)
    at = code.astype(np.int64) @ pw
    times = np.bincount(at, minlength=N)
    who = np.full(N, -1, dtype=np.int64)
    who[at] = np.arange(m)
    x = np.arange(N, dtype=np.int64)
    cnt = times.copy()
    near = []                                              # (position, words' neighbours in that position)
    for j in range(n):
        d = x // pw[j] % q
        for v in range(1, q):
            y = x + ((d + v) % q - d) * pw[j]
            cnt += times[y]
            near.append((j, y))
    P = np.zeros((m, n + 1), dtype=np.int64)
    for j, y in near:                                      # once covered, by a codeword that differs at j
        k = who[y[(cnt == 1) & (times[y] == 1)]]
        np.add.at(P[:, 0], k, 1)
        np.add.at(P[:, 1 + j], k, 1)
    assert P[:, 0].sum() > 1000
    with Pool(1, cluster=1) as pool:
        s = pool.add(q, n, 1, m, code=code, seed=1)
        assert (pool.cnt(s) == cnt).all()
        assert (pool.private(s) == P).all()
