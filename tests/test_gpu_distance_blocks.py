"""The distance transform on blocks of two digits (q = 5..8) against the
oracle: tiles of two digits up to the largest, one tile and many, codewords
kept in registers and not, distances up to the word length, repeated
codewords and digits outside the alphabet."""
import ctypes

import numpy as np
import pytest

from coldcase_gb300 import lib as L
from coldcase_gb300.workloads import uniform_code

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,n,m", [(5, 2, 1), (5, 3, 2), (5, 9, 1), (5, 10, 300), (6, 2, 3), (6, 4, 1), (6, 8, 9000),
                                   (6, 9, 40), (7, 3, 1), (7, 8, 1), (7, 8, 2100), (7, 8, 9000), (8, 2, 1), (8, 4, 2),
                                   (8, 7, 1), (8, 7, 3000), (8, 8, 20000)])
def test_blocks_equal_oracle(covlib, q, n, m):
    import torch
    from oracle import pyoracle as po
    code = uniform_code(q, n, m, 3 * q + n)
    if m > 3:
        code[m // 2] = code[0]
    want = po.linemin(code, q, n, threads=8)
    sent = np.concatenate([code, np.full((1, n), q, dtype=np.uint8)])      # no word of the space: ignored
    dev = torch.from_numpy(sent).cuda()
    N = q ** n
    buf = torch.zeros(N + 64, dtype=torch.uint8, device="cuda")
    for off in (0, 16, 5):
        buf.fill_(255)
        for count in (m + 1, m):
            L.check(covlib.cov_mindist_dev(q, n, dev.data_ptr(), count, ctypes.c_void_p(buf.data_ptr() + off), None))
            torch.cuda.synchronize()
            got = buf.cpu().numpy()
            assert (got[off:off + N] == want).all()
            assert (got[:off] == 255).all() and (got[off + N:] == 255).all()
