"""TVDlimit away from its default physics: small optical depth (tau0 <= 1e-5,
where cells faster than CME_thresh times the fast speed lose the diffusivity
of density, energy and velocity but keep the field's), the diffusion
coefficients and the boundary slopes.

FP64 against the oracle (relative L-infinity <= 1e-12 per field, the FP64
bar), FP32 against FP64 on the same float32 state (2e-6 of the field's largest
value: three sweeps of a few float roundings each)."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd, initial

pytestmark = pytest.mark.gpu

TVD = [1.0e-11, 1.0, 10.0, 0.2, 1.0, 1.0, 1.0, 1.0, 0.75, 100.0]  # the defaults
BND = dict(tvd_h_bnd=[0.2, 0.25])  # boundary profiles several cells deep
CASES = {
    "mach": dict(tau0=0.0, thresh=True),
    "mach_no_log": dict(tau0=0.0, thresh=True, tvd={1: 0.0}),
    "thin": dict(tau0=0.0),
    "coeff": dict(BND, tvd_coeff=[0.9, 0.7, 0.8, 0.6], tvd_visc_bnd=[0.5, 0.8], tvd_eta_bnd=[0.75, 0.4]),
    "slopes": dict(BND, tvd_visc_bnd=[1.6, 1.3], tvd_eta_bnd=[1.2, 1.7]),
    "visc_slope": dict(BND, tvd_visc_bnd=[1.0, 1.5]),
    "eta_slope": dict(BND, tvd_eta_bnd=[1.5, 1.0]),
    "profiles": dict(BND, tvd_h=[1.5, 2.0, 1.2, 0.8], tvd_cs=[0.5, 0.2, 0.3, 0.1], tvd={5: 0.4, 6: 0.7, 7: 1.4}),
    "no_hyperdiffusion": dict(tvd={4: 0.0}),
    "no_speed_limit": dict(tvd={8: 0.0}),
    "no_log": dict(tvd={1: 0.0}),
}


def _box(shape, closed):
    tab = initial.EosTable(H.EOS_SMALL)
    U = (initial.stratified_box if closed else initial.periodic_box)(tab, *shape, seed=sum(shape))
    return U.astype(np.float32).astype(np.float64)


class _Oracle:
    def __init__(self, kw, shape, U, closed):
        from oracle import oracle as O
        self.L = O.lib()
        dx = 1.6e6 if closed else 3.2e6
        self.p = O.make_params(*shape, dx, periodic_x=not closed, **kw)
        self.p.va_adjust = 0.0
        eos = O.Eos(H.EOS_SMALL)
        self.U, prim = U.copy(), U.copy()
        aux = np.zeros((5,) + U.shape[1:])
        self.L.mo_cons_to_prim(C.byref(self.p), eos.ptr, prim, *aux)
        self.L.mo_adjust_valf_max(C.byref(self.p), prim, aux[0], np.zeros(5))
        self.dt = 0.8 * self.L.mo_mhd_residual(C.byref(self.p), prim, aux[0], np.zeros_like(U))
        self.p.dt = self.dt
        self.prim, self.pres = prim, aux[0]

    def tvd(self):
        out = self.U.copy()
        self.L.mo_tvdlimit(C.byref(self.p), out, self.pres, self.dt)
        return out


def _mach_threshold(o):
    """A threshold that about half of the cells pass, and none so closely that
    a rounding decides (the oracle's result is the same on either side)."""
    d, v, B = o.prim[0], o.prim[1:4], o.prim[5:8]
    ratio = np.sqrt(np.sum(v ** 2, 0) / (np.sum(B ** 2, 0) / d + 5.0 / 3.0 * o.pres / d))
    for q in np.linspace(0.5, 0.6, 21):
        t = float(np.quantile(H.interior(ratio[None])[0], q))
        got = []
        for f in (1 - 1e-5, 1.0, 1 + 1e-5):
            o.p.tvd[9] = t * f
            got.append(o.tvd())
        # a threshold moved by 1e-5 changes nothing but which cells it catches
        if np.array_equal(got[0], got[1]) and np.array_equal(got[1], got[2]):
            return t
    raise AssertionError("no threshold clear of every cell")


@pytest.mark.parametrize("shape,closed", [((24, 16, 16), False), ((29, 9, 33), True)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_tvdlimit_options(gpu_lib, name, shape, closed):
    kw = dict(CASES[name])
    tvd = list(TVD)
    for i, x in kw.pop("tvd", {}).items():
        tvd[i] = x
    kw["tvd"] = tvd
    thresh = kw.pop("thresh", False)
    if closed:
        kw["grav"] = 2.74e4
    U = _box(shape, closed)
    o = _Oracle(kw, shape, U, closed)
    if thresh:
        kw["tvd"][9] = o.p.tvd[9] = _mach_threshold(o)
    ref = o.tvd()
    got = {}
    for precision in (64, 32):
        p = gpumhd.default_params(*shape, 1.6e6 if closed else 3.2e6, precision=precision,
                                  periodic_x=0 if closed else 1, **kw)
        g = gpumhd.MuramGPU(p, eos_path=H.EOS_SMALL)
        g.upload_state(U)
        g.upload_field(gpumhd.FIELD_PRES, o.pres)
        g.TVDlimit(o.dt)
        got[precision] = H.interior(g.download_state())
        g.close()
    e = H.rel_linf(got[64], H.interior(ref))
    print(f"{name} {shape}: FP64 against the oracle {np.array2string(e, precision=2)}")
    assert np.all(e <= 1e-12), e
    e = H.rel_linf(got[32], got[64])
    print(f"{name} {shape}: FP32 against FP64 {np.array2string(e, precision=2)}")
    assert np.all(e <= 2e-6), e


def test_fused_steps_above_the_mach_threshold(gpu_lib):
    """Five fused FP64 steps with tau0 = 0 and a threshold that half of the
    cells pass, against the oracle."""
    from oracle import oracle as O
    shape = (24, 16, 16)
    U = _box(shape, False)
    o = _Oracle(dict(tau0=0.0), shape, U, False)
    tvd = list(TVD)
    tvd[9] = _mach_threshold(o)
    st = O.State(O.make_params(*shape, 3.2e6, tau0=0.0, tvd=tvd), U)
    dts = [x[0] for x in st.step(O.Eos(H.EOS_SMALL), 5)]
    g = gpumhd.MuramGPU(gpumhd.default_params(*shape, 3.2e6, tau0=0.0, tvd=tvd), eos_path=H.EOS_SMALL)
    g.upload_state(U)
    assert np.allclose(g.run_steps(5), dts, rtol=1e-12, atol=0)
    e = H.rel_linf(g.download_state(), st.U)
    g.close()
    assert np.all(e <= 1e-12), e


def test_adjoint_above_the_mach_threshold(gpu_lib):
    """The gradient of the top layers' B_x^2 after three steps with tau0 = 0,
    projected on random directions, against central differences of the forward
    steps; the field keeps its diffusivity in the fast cells in both."""
    nx, ny, nz, steps = 16, 12, 8, 3
    tab = initial.EosTable(H.EOS_SMALL)
    U0 = initial.periodic_box(tab, nx, ny, nz, seed=41)
    # diffusivities that depend on the cell's Alfven speed, through the Boris factor
    kw = dict(tau0=0.0, tvd_h=[2.0, 2.0, 1.0, 2.0], va_max=1.5e5, tvd=list(TVD))
    kw["tvd"][9] = _mach_threshold(_Oracle(kw, (nx, ny, nz), U0, False))
    g = gpumhd.MuramGPU(gpumhd.default_params(nx, ny, nz, 3.2e6, **kw), eos_path=H.EOS_SMALL)
    g.upload_state(U0)
    dt = 0.6 * float(g.run_steps(1)[0])
    g.close()
    g = gpumhd.MuramGPU(gpumhd.default_params(nx, ny, nz, 3.2e6, autostep=0, dt=dt, **kw),
                        eos_path=H.EOS_SMALL)
    mask = np.random.default_rng(7).uniform(0.0, 1.0, (nz, ny, 8))

    def after(U):
        g.upload_state(U)
        g.run_steps(steps)
        return g.download_state()

    UT = after(U0)
    lam = np.zeros_like(UT)
    lam[5, 2:-2, 2:-2, -10:-2] = 2.0 * mask * UT[5, 2:-2, 2:-2, -10:-2]
    g.upload_state(U0)
    grad = g.adjoint(steps, lam, checkpoint_every=2)
    rng = np.random.default_rng(3)
    scale = np.sqrt(np.mean(U0[:, 2:-2, 2:-2, 2:-2] ** 2, axis=(1, 2, 3)))
    errs = []
    for _ in range(6):
        v = np.zeros_like(U0)
        v[:, 2:-2, 2:-2, 2:-2] = rng.standard_normal(U0[:, 2:-2, 2:-2, 2:-2].shape) * scale[:, None, None, None]
        v = initial.fill_ghosts(v, periodic_x=True)
        J = [float(np.sum(mask * after(U0 + s * 1e-8 * v)[5, 2:-2, 2:-2, -10:-2] ** 2)) for s in (1, -1)]
        fd = (J[0] - J[1]) / 2e-8
        errs.append(abs(float(np.sum(grad * v)) - fd) / abs(fd))
    g.close()
    print("adjoint vs central differences, relative errors:", np.array2string(np.array(errs), precision=2))
    assert np.median(errs) < 1e-6 and max(errs) < 1e-5, errs
