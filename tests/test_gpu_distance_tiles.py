"""The distance transform by tiles from the code alone (few codewords) and by
sweeps (many), against the oracle: every alphabet, one tile and many, tiles
whose rows start at any byte, an unaligned destination, repeated codewords,
the empty code, and sizes on either side of the rule between the two."""
import ctypes

import numpy as np
import pytest

from coldcase_gb300 import lib as L
from coldcase_gb300 import verify
from coldcase_gb300.workloads import uniform_code

pytestmark = pytest.mark.gpu

CASES = [(q, n, m) for q, n in ((2, 16), (2, 9), (3, 9), (3, 3), (4, 8), (5, 7), (6, 6), (7, 7), (8, 5), (8, 7),
                                (9, 5), (10, 5), (11, 4), (13, 4), (16, 5), (16, 2), (7, 1), (2, 1))
         for m in (1, 37, 900)] + [(7, 7, 9000), (8, 6, 60000), (6, 7, 4097), (3, 13, 200), (7, 8, 0), (8, 3, 0)]


@pytest.mark.parametrize("q,n,m", CASES)
def test_distance_equals_oracle(covlib, q, n, m):
    import torch
    from oracle import pyoracle as po
    code = uniform_code(q, n, m, 5 * q + n)
    if m > 2:
        code[1] = code[0]
    N = q ** n
    want = po.linemin(code, q, n, threads=8) if m else np.full(N, n + 1, dtype=np.uint8)
    hist = np.bincount(want, minlength=n + 2)
    dist, h, rad = verify.mindist(code, q, n)
    assert (dist == want).all() and (h == hist).all() and rad == int(want.max())
    _, h2, rad2 = verify.mindist(code, q, n, want_dist=False)
    assert (h2 == hist).all() and rad2 == rad
    buf = torch.zeros(N + 16, dtype=torch.uint8, device="cuda")
    dev = torch.from_numpy(np.ascontiguousarray(code)).cuda() if m else None
    ptr = dev.data_ptr() if m else None
    for off in (0, 1, 4, 6):                     # any alignment of the destination, nothing written outside it
        for fn in (covlib.cov_mindist_dev, covlib.cov_mindist_dev_static):
            buf.fill_(255)
            L.check(fn(q, n, ptr, m, ctypes.c_void_p(buf.data_ptr() + off), None))
            torch.cuda.synchronize()
            got = buf.cpu().numpy()
            assert (got[off:off + N] == want).all(), (off, fn)
            assert (got[:off] == 255).all() and (got[off + N:] == 255).all()
