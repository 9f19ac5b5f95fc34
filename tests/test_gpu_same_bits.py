"""Paths that form the same values give the same bits."""
import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd, initial

pytestmark = pytest.mark.gpu

BOXES = [((24, 16, 16), False, {}), ((29, 9, 33), True, {}), ((64, 40, 36), True, {}),
         ((24, 16, 16), False, dict(CFL_tvd=0.3)), ((29, 9, 33), True, dict(eta=1e10)),
         ((16, 12, 8), False, dict(spitzer=0.5)),
         ((24, 16, 16), False, dict(divB_switch=1, divB_itmax=4, divB_err=0.2)),
         ((24, 16, 16), False, dict(va_adjust=1.0)),
         ((30, 9, 33), True, dict(xbnd=1, bnd_bcrit=1e3, bnd_eps_top=0.0)),
         ((30, 9, 33), True, dict(xbnd=1, bnd_bcrit=1e3, bnd_eps_top=0.0, spitzer=0.5, divB_switch=1, divB_itmax=4,
                                  divB_err=0.2))]


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


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("rho_log", [1.0, 0.0])
@pytest.mark.parametrize("shape,closed", [((24, 16, 16), False), ((29, 9, 33), True), ((64, 40, 36), True)])
def test_diagnostics_leave_the_state_alone(gpu_lib, precision, rho_log, shape, closed):
    """An output step's diagnostics, asked for or not: the same state."""
    kw = dict(tvd=[1.0e-11, rho_log, 10.0, 0.2, 1.0, 1.0, 1.0, 1.0, 0.75, 100.0])
    out = []
    for on in (False, True):
        g = _box(shape, closed, precision, kw)
        g.exchange_grid(True)
        for _ in range(2):
            g.step_reference_order(diagnostics=on)
        out.append(g.download_state())
        g.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("closed", [False, True])
def test_fp32_diagnostics_near_fp64(gpu_lib, closed):
    """TVDlimit's diagnostics (the last five arrays and tvar6) of the FP32 sweeps
    against the FP64 ones on a box with viscous and resistive heating off the
    vertical boundary (tvd[5] = 0.4): 1e-4 of each array's L2 norm (1e-2 for the
    Boris energy tvar6), the bar of the diagnostics' own test."""
    shape = (29, 9, 33)
    kw = dict(tvd=[1.0e-11, 1.0, 10.0, 0.2, 1.0, 0.4, 1.0, 1.0, 0.75, 100.0], tvd_h_bnd=[0.2, 0.25])
    got = {}
    for precision in (64, 32):
        g = _box(shape, closed, precision, kw)
        g.exchange_grid(True)
        g.step_reference_order(diagnostics=True)
        got[precision] = g.download_diagnostics()
        g.close()
    floor = 1e-6 * np.sqrt(np.sum(got[64][0] ** 2))
    for q, name in enumerate(gpumhd.DIAG_NAMES):
        ref = got[64][q]
        e = np.sqrt(np.sum((got[32][q] - ref) ** 2)) / max(np.sqrt(np.sum(ref ** 2)), floor)
        print(name, f"{e:.2e}")
        assert e <= (1e-2 if name == "tvar6" else 1e-4), (name, e)
