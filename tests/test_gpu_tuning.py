"""Launch shapes carried from one context to another.

What gpumhd_get_tuning reports after the autotuner, given to
gpumhd_set_tuning of a second context, launches the same shapes: its TVD
sweeps take the same time.  (On this box a sweep with 32 cells per thread
takes more than twice the time of one with the launcher's own short chunks,
so shapes that differ show; the bound leaves 30 % for the spread of the
smallest of five measurements.)"""
import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd, initial

pytestmark = pytest.mark.gpu


def _box(precision):
    tab = initial.EosTable(H.EOS_SMALL)
    g = gpumhd.MuramGPU(gpumhd.default_params(64, 64, 64, 3.2e6, precision=precision), eos_path=H.EOS_SMALL)
    g.upload_state(initial.periodic_box(tab, 64, 64, 64, seed=2))
    g.run_steps(2)
    return g


def _sweeps(g):
    """The y and z sweeps' times, ms: the smallest of five measurements."""
    return np.min([list(g.profile_steps(4).values())[6:8] for _ in range(5)], axis=0)


@pytest.mark.parametrize("precision", [64, 32])
def test_tuning_carries_over(gpu_lib, precision):
    a, b = _box(precision), _box(precision)
    a.autotune(trial_steps=3)
    t = a.tuning()
    b.set_tuning(t["stage_zchunk"], t["tvd_chunk"])
    assert b.tuning()["tvd_chunk"] == t["tvd_chunk"] and b.tuning()["stage_zchunk"] == t["stage_zchunk"]
    ta, tb = _sweeps(a), _sweeps(b)
    print(f"FP{precision} tuning {t}: y, z sweeps {ta} ms, carried over {tb} ms")
    a.close()
    b.close()
    assert np.all(ta <= 1.3 * tb) and np.all(tb <= 1.3 * ta), (ta, tb)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("shape,closed", [((16, 12, 8), False), ((29, 35, 34), True)])
def test_chunk_lengths_keep_results(gpu_lib, precision, shape, closed):
    """An ensemble takes a TVD chunk as it is: lengths from one cell to the whole
    pencil, odd ones among them, give the bits of the box alone."""
    tab = initial.EosTable(H.EOS_SMALL)
    U = (initial.stratified_box if closed else initial.periodic_box)(tab, *shape, seed=6)
    kw = dict(periodic_x=0, grav=2.74e4) if closed else {}
    out = []
    for td in (None, 1, 2, 3, 5, 16, 64):
        p = gpumhd.default_params(*shape, 1.6e6 if closed else 3.2e6, precision=precision, **kw)
        g = gpumhd.MuramGPU(p, eos_path=H.EOS_SMALL)
        g.upload_state(U)
        if td is None:
            g.run_steps(3)
        else:
            g.set_tuning(0, td)
            e = gpumhd.MuramEnsemble([g])
            e.run_steps(3)
            e.close()
        out.append(g.download_state())
        g.close()
    assert all(np.array_equal(out[0], o) for o in out[1:]), [float(np.max(np.abs(o - out[0]))) for o in out[1:]]
