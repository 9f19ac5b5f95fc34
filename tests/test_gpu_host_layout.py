"""Host transfers: pinned memory (converted by the kernel that reads or writes it
over the link), pageable memory (through a staging buffer) and the asynchronous
pair give the same bits, for both host types and precisions, whole and single
fields, aligned and unaligned buffers, and odd boxes."""
import numpy as np
import pytest
import torch

from muram_main_gb300 import gpumhd

pytestmark = pytest.mark.gpu


def _buffer(n, dtype, pinned, offset):
    """n values starting `offset` values into an allocation."""
    t = torch.zeros(n + offset + 4, dtype=dtype)
    if pinned:
        t = t.pin_memory()
    return t[offset : offset + n]


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(4, 4, 4), (13, 7, 5), (30, 9, 11), (33, 18, 6)])
def test_pinned_pageable_and_async_transfers_agree(gpu_lib, precision, dtype, shape):
    g = gpumhd.MuramGPU(gpumhd.default_params(*shape, precision=precision))
    nodes = int(np.prod(g.shape))
    npt = np.float32 if dtype == torch.float32 else np.float64
    rng = np.random.default_rng(sum(shape) + precision)
    for field, nf in ((gpumhd.FIELD_U, 8), (gpumhd.FIELD_PHI, 1)):
        data = torch.from_numpy(rng.standard_normal(nodes * nf)).to(dtype)
        want = data.float().to(dtype) if precision == 32 else data
        for pinned, offset in ((True, 0), (True, 1), (False, 0), (False, 3)):
            src, dst = _buffer(nodes * nf, dtype, pinned, offset), _buffer(nodes * nf, dtype, pinned, offset)
            src.copy_(data)
            g.upload_ptr(field, src.data_ptr(), npt)
            g.download_ptr(field, dst.data_ptr(), npt)
            assert torch.equal(dst, want), (field, pinned, offset)
            g.upload_ptr(field, torch.zeros_like(src).data_ptr(), npt)
            g.upload_ptr_async(field, src.data_ptr(), npt)
            dst.zero_()
            g.download_ptr_async(field, dst.data_ptr(), npt)
            g.synchronize()
            assert torch.equal(dst, want), (field, pinned, offset, "async")
    g.close()
