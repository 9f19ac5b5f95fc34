"""Paths that form the same values give the same bits."""
import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd, initial

pytestmark = pytest.mark.gpu

BOXES = [((24, 16, 16), False, {}), ((29, 9, 33), True, {}), ((64, 40, 36), True, {}),
         ((24, 16, 16), False, dict(CFL_tvd=0.3)), ((29, 9, 33), True, dict(eta=1e10)),
         ((16, 12, 8), False, dict(spitzer=0.5))]


def _box(shape, closed, precision, kw):
    tab = initial.EosTable(H.EOS_SMALL)
    U = (initial.stratified_box if closed else initial.periodic_box)(tab, *shape, seed=3)
    kw = dict(kw, **(dict(periodic_x=0, grav=2.74e4) if closed else {}))
    p = gpumhd.default_params(*shape, 1.6e6 if closed else 3.2e6, precision=precision, **kw)
    g = gpumhd.MuramGPU(p, eos_path=H.EOS_SMALL)
    g.upload_state(U)
    return g


@pytest.mark.parametrize("box", range(len(BOXES)))
def test_fp64_routines_and_fused_steps(gpu_lib, box):
    """FP64: the routines in ComputeSolution's order and the fused steps, whose
    kernels share every formula, give the same bits."""
    shape, closed, kw = BOXES[box]
    a, b = _box(shape, closed, 64, kw), _box(shape, closed, 64, kw)
    a.exchange_grid(True)
    dts = [a.step_reference_order()[0] for _ in range(3)]
    assert list(b.run_steps(3)) == dts
    assert np.array_equal(H.interior(a.download_state()), H.interior(b.download_state()))
    a.close()
    b.close()
