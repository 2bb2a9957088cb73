"""FP32 slab copies on a device without room for them: the layout change fails with an error, the
operator keeps working, and a later attempt with room is complete."""
import numpy as np
import pytest
import torch

import rqutils_b200 as rq
from rqutils_b200 import _lib

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _fill_device(leave):
    """Tensors that take the device's free memory down to about ``leave`` bytes."""
    hold = []
    for step in (1024 * MIB, 64 * MIB):
        while True:
            free, _ = torch.cuda.mem_get_info()
            if free < leave + step:
                break
            try:
                hold.append(torch.empty((free - leave) // step * step, dtype=torch.uint8,
                                        device='cuda'))
            except torch.OutOfMemoryError:      # less in one piece: smaller ones
                break
    return hold


def test_fp32_slabs_without_memory():
    # No group on the high half: the high slabs are empty and the low ones take 1 GB.
    rng = np.random.default_rng(1)
    n, nh, nl = 34, 1 << 16, 128
    hi = np.sort(rng.choice(1 << 17, size=nh, replace=False)).astype(np.uint64)
    states = ((hi[:, None] << np.uint64(17)) | np.arange(nl, dtype=np.uint64)[None, :]).reshape(-1)
    x = np.arange(32, dtype=np.uint64)
    z = rng.integers(0, 1 << 34, size=32, dtype=np.uint64) & ~x      # no Y: real elements
    ham = rq.PauliSumXZ.from_xz(x, z, rng.standard_normal(32), n, force_real=True, padded=True)
    op = rq.SQDOperator(ham, rq.Subspace.from_u64(states, n), cache_strategy=(1, 2))
    v = torch.randn(op.size, dtype=torch.float32, device='cuda')
    ref = op.matvec(v)
    op.set_layout(0, 'product')
    _lib.trim_memory()
    torch.cuda.empty_cache()
    hold = _fill_device(256 * MIB)
    try:
        with pytest.raises(_lib.SQDError):
            op.set_layout(1, 'product')
    finally:
        del hold
        torch.cuda.empty_cache()
    assert op.get_layout(1) == 'csr' and torch.equal(op.matvec(v), ref)
    op.set_layout(1, 'product')
    # 32 products a row in another order, each sum within 32 ulps of the largest row
    assert (op.matvec(v) - ref).abs().max() <= 64 * 2.0 ** -23 * ref.abs().max()
