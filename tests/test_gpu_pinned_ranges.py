"""Host transfers from parts of pinned memory: allocated pinned, or registered
with the driver, at the start, inside and up to the end of the piece."""
import numpy as np
import pytest
import torch

from muram_main_gb300 import gpumhd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("registered", [False, True])
@pytest.mark.parametrize("precision", [32, 64])
def test_transfers_within_a_pinned_piece(gpu_lib, registered, precision):
    g = gpumhd.MuramGPU(gpumhd.default_params(33, 18, 6, precision=precision))
    n = int(np.prod(g.shape)) * 8
    page, bytes_ = 4096, 3 * n * 8
    if registered:
        raw = np.zeros(bytes_ + 2 * page, dtype=np.uint8)
        at = (-raw.ctypes.data) % page
        size = (bytes_ + page - 1) // page * page
        ptr = raw.ctypes.data + at
        assert int(torch.cuda.cudart().cudaHostRegister(ptr, size, 0)) == 0
        whole = raw[at : at + bytes_].view(np.float64)
    else:
        keep = torch.zeros(3 * n, dtype=torch.float64).pin_memory()
        whole = keep.numpy()
    try:
        data = np.random.default_rng(4).standard_normal(n).astype(np.float32).astype(np.float64)
        for offset in (0, 2, 1001, 2 * n):
            src, dst = whole[offset : offset + n], whole[:n] if offset == 2 * n else whole[2 * n :]
            src[:] = data
            g.upload_ptr(gpumhd.FIELD_U, src.ctypes.data, np.float64)
            if offset < n:
                dst[:] = 0.0
            g.download_ptr(gpumhd.FIELD_U, dst.ctypes.data, np.float64)
            assert np.array_equal(dst, data), offset
    finally:
        g.synchronize()
        g.close()
        if registered:
            assert int(torch.cuda.cudart().cudaHostUnregister(ptr)) == 0
