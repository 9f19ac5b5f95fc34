"""Asynchronous transfers do move the data: the field is cleared and found zero
before each asynchronous upload, and the cleared host buffer is kept until the
copies are done."""
import numpy as np
import pytest
import torch

from muram_main_gb300 import gpumhd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("offset", [0, 1])
def test_async_upload_after_a_cleared_field(gpu_lib, precision, dtype, pinned, offset):
    npt = np.float32 if dtype == torch.float32 else np.float64
    for shape in ((4, 4, 4), (30, 9, 11), (33, 18, 6)):
        g = gpumhd.MuramGPU(gpumhd.default_params(*shape, precision=precision))
        nodes = int(np.prod(g.shape))
        rng = np.random.default_rng(sum(shape))
        for field, nf in ((gpumhd.FIELD_U, 8), (gpumhd.FIELD_PHI, 1)):
            data = torch.from_numpy(rng.standard_normal(nodes * nf)).to(dtype)
            want = data.float().to(dtype) if precision == 32 else data
            bufs = [torch.zeros(nodes * nf + 4, dtype=dtype) for _ in range(3)]
            if pinned:
                bufs = [b.pin_memory() for b in bufs]
            zero, src, dst = (b[offset : offset + nodes * nf] for b in bufs)
            src.copy_(data)
            g.upload_ptr(field, zero.data_ptr(), npt)
            dst.fill_(7.0)
            g.download_ptr(field, dst.data_ptr(), npt)
            assert torch.equal(dst, zero), (shape, field)
            g.upload_ptr_async(field, src.data_ptr(), npt)
            g.download_ptr_async(field, dst.data_ptr(), npt)
            g.synchronize()
            assert torch.equal(dst, want), (shape, field)
        g.close()
