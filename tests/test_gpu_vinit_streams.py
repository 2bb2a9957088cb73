"""The start index right after a refresh that another stream has not run yet."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('lookup', ['product', 'hash'])
def test_vinit_beside_a_pending_refresh(lookup):
    rng = np.random.default_rng(5)
    wl = W.jw_workload('streams', 8, 3, 40, 40, 2)
    ham = rq.PauliSumXZ.from_xz(wl.x, wl.z, wl.coeffs, 16, force_real=True, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(wl.states, 16), (1, 2), lookup=lookup)
    before = op.vinit()
    side = torch.cuda.Stream()
    for c in (-wl.coeffs, rng.standard_normal(wl.coeffs.shape[0])):
        ham.set_coeffs(torch.as_tensor(c))
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)      # about 0.1 s before the refresh runs
            op.refresh()
        got = op.vinit()
        side.synchronize()
        want = int(op.diagonal(0).argmin())
        assert got == want != before
        before = want
