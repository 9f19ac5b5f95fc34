"""Compensated FP32 runs repeat bit for bit.

A ghost row of the x and y sweeps reads the rounding remainder of the interior
cell it images; that cell's own thread, in another block of the same launch,
replaces it.  The sweeps therefore read one array of remainders and write
another, and no run depends on which block came first."""
import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho_log", [1.0, 0.0])
@pytest.mark.parametrize("cfl_tvd", [0.95, 0.3])  # one TVD pass per step, two half passes
@pytest.mark.parametrize("shape,closed", [((16, 12, 8), False), ((61, 40, 36), True)])
def test_compensated_runs_repeat(gpu_lib, shape, closed, cfl_tvd, rho_log):
    tab = initial.EosTable(H.EOS_SMALL)
    U = (initial.stratified_box if closed else initial.periodic_box)(tab, *shape, seed=12)
    kw = dict(periodic_x=0, grav=2.74e4) if closed else {}
    tvd = [1.0e-11, rho_log, 10.0, 0.2, 1.0, 1.0, 1.0, 1.0, 0.75, 100.0]
    out = []
    for capture in (True, True, False):
        p = gpumhd.default_params(*shape, 1.6e6 if closed else 3.2e6, precision=32, compensated=1, CFL_tvd=cfl_tvd,
                                  tvd=tvd, **kw)
        g = gpumhd.MuramGPU(p, eos_path=H.EOS_SMALL)
        g.upload_state(U)
        g.run_steps(12, capture=capture)
        assert g.step_info()[3] == (1 if cfl_tvd < 0.8 else 0)
        out.append(g.download_state())
        g.close()
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
