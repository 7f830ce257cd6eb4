"""What the verification calls' scratch pool keeps is given back when the
library runs short of device memory."""
import numpy as np
import pytest

from coldcase_gb300 import verify
from coldcase_gb300.engine import Pool
from coldcase_gb300.lib import CovError
from coldcase_gb300.workloads import uniform_code

pytestmark = pytest.mark.gpu


def test_kept_scratch_is_given_back(covlib):
    import torch
    code = uniform_code(6, 6, 41, 1)
    want = verify.mindist(code, 6, 6)[0]
    with Pool(1, cluster=1) as pool:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        record = 72                                   # bytes of a kept move record
        with pytest.raises(CovError):                 # more records than the device has memory for
            pool.add(4, 6, 1, 300, seed=1, trace=1, trace_cap=2 * torch.cuda.mem_get_info()[1] // record)
        assert torch.cuda.mem_get_info()[0] >= before + (32 << 20)      # a pool reserves 32 MB at least
        s = pool.add(4, 6, 1, 300, seed=1)            # the pool of searches still works
        pool.run(10)
        assert pool.status(s)["it"] == 10
    assert (verify.mindist(code, 6, 6)[0] == want).all()
