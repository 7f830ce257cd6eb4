"""The distance transform of a device code with digits outside the alphabet:
such a codeword is no word of the space and is ignored, whichever of its
digits is outside, in every form (blocks, lines and sweeps) and with the
allocating and the static scratch."""
import ctypes

import numpy as np
import pytest

from coldcase_gb300 import lib as L
from coldcase_gb300.workloads import uniform_code

pytestmark = pytest.mark.gpu


# blocks (q = 5..8), lines, and sweeps (many codewords)
@pytest.mark.parametrize("q,n,m", [(5, 7, 3), (8, 6, 4), (3, 9, 4), (10, 5, 5), (16, 4, 3),
                                   (8, 6, 60000), (4, 8, 60000), (2, 12, 60000), (11, 5, 60000)])
def test_codewords_outside_the_alphabet_are_ignored(covlib, q, n, m):
    import torch
    from oracle import pyoracle as po
    code = uniform_code(q, n, m, 11 * q + n)
    # a digit outside at each position in turn, the least and the largest one
    # among them: sums below q^n and past it
    bad = np.zeros((4 * n, n), dtype=np.uint8)
    for j in range(n):
        bad[4 * j:4 * j + 4] = code[j % m]
        bad[4 * j:4 * j + 4, j] = (q, q + 1, 2 * q, 255)
    want = po.linemin(code, q, n, threads=8)
    dev = torch.from_numpy(np.concatenate([bad[:2 * n], code, bad[2 * n:]])).cuda()
    only = torch.from_numpy(bad).cuda()
    N = q ** n
    buf = torch.empty(N, dtype=torch.uint8, device="cuda")
    for fn in (covlib.cov_mindist_dev, covlib.cov_mindist_dev_static):
        for d_code, count, expect in ((dev, m + 4 * n, want), (only, 4 * n, np.full(N, n + 1, dtype=np.uint8))):
            buf.fill_(255)
            L.check(fn(q, n, d_code.data_ptr(), count, ctypes.c_void_p(buf.data_ptr()), None))
            torch.cuda.synchronize()
            assert (buf.cpu().numpy() == expect).all(), fn
