"""FP32 TVD sweeps (paired arithmetic, interface logarithms) against the FP64 ones.

One TVDlimit call on the same float32 state in both precisions, at the sizes
where the kernels' tiling can go wrong: x around multiples of the 28 cells a
warp updates, y and z around the chunk lengths.  A state with density steps of
a factor three takes the logarithm's general path.  A sweep changes a value by
less than its size with a relative error of a few float roundings: three sweeps
stay below 2e-6 of the field's maximum."""
import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd, initial

pytestmark = pytest.mark.gpu


def _tvd(U, shape, precision, closed, dt):
    nx, ny, nz = shape
    kw = dict(periodic_x=0, grav=2.74e4) if closed else {}
    g = gpumhd.MuramGPU(gpumhd.default_params(nx, ny, nz, 1.6e6 if closed else 3.2e6, precision=precision, **kw),
                        eos_path=H.EOS_SMALL)
    g.upload_state(U)
    g.ConsToPrim()
    if dt is None:
        dt = 0.8 * g.MHD_Residual()
    g.upload_state(U)
    g.TVDlimit(dt)
    out = H.interior(g.download_state())
    g.close()
    return out, dt


@pytest.mark.parametrize("shape", [(4, 4, 4), (27, 9, 33), (28, 32, 8), (29, 31, 34), (56, 17, 16), (57, 40, 65)])
@pytest.mark.parametrize("closed", [False, True])
@pytest.mark.parametrize("steps", [False, True])
def test_tvdlimit_fp32_matches_fp64(gpu_lib, shape, closed, steps):
    tab = initial.EosTable(H.EOS_SMALL)
    box = initial.stratified_box if closed else initial.periodic_box
    U = box(tab, *shape, seed=sum(shape)).astype(np.float32).astype(np.float64)
    if steps:
        i, j, k = (np.arange(n) for n in U.shape[:0:-1])
        U[:5] *= np.where(((i // 5)[None, None, :] + (j // 3)[None, :, None] + (k // 4)[:, None, None]) % 3 == 0, 3.0, 1.0)
        U = U.astype(np.float32).astype(np.float64)
    ref, dt = _tvd(U, shape, 64, closed, None)
    got, _ = _tvd(U, shape, 32, closed, dt)
    e = H.rel_linf(got, ref)
    assert np.all(e <= 2e-6), e


@pytest.mark.parametrize("shape", [(4, 4, 4), (16, 12, 8), (33, 20, 12)])
def test_default_launch_shapes_keep_results(gpu_lib, shape):
    """Small boxes march one-plane stage chunks and two-cell TVD chunks by
    themselves; whole-box chunks give the same bits."""
    out = []
    for zc, td in ((0, 0), (shape[2], 64)):
        tab = initial.EosTable(H.EOS_SMALL)
        g = gpumhd.MuramGPU(gpumhd.default_params(*shape, 3.2e6), eos_path=H.EOS_SMALL)
        g.upload_state(initial.periodic_box(tab, *shape, seed=9))
        g.set_tuning(zc, td)
        g.run_steps(3)
        out.append(g.download_state())
        g.close()
    assert np.array_equal(out[0], out[1])
