"""The adjoint takes the forward's branch where a floor is met exactly.

In a uniform box nothing moves: every stage and sweep gives the state back, and
the energy floors of Tcheck and TVDlimit,
    eps_min rho + |M|^2 / (2 rho),
formed in two ways, are compared with an energy that equals one of them to the
bit.  The forward keeps the energy (it is not below the floor), so the total
energy's gradient with respect to each cell's energy is 1.  A reverse pass that
rounds the floor differently finds it above the energy in the states chosen
here and returns 0."""
from fractions import Fraction as F
import math

import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd

EPS_MIN = 2.0e12


def fma(a, b, c):
    return float(F(a) * F(b) + F(c))


def floors(d, m, fused):
    """(TVDlimit's floor, Tcheck's floor) of a cell, products and sums rounded
    once (as the kernels do) or separately."""
    mad = fma if fused else lambda a, b, c: a * b + c
    k = mad(m[2], m[2], mad(m[1], m[1], m[0] * m[0]))
    vv = math.sqrt(k) / d
    return mad(EPS_MIN, d, 0.5 * k / d), mad(EPS_MIN, d, 0.5 * d * vv * vv)


def tie_states(which, count):
    """(density, momentum, energy): energy on floor `which`, not below the other
    one, and below its separately rounded value."""
    rng = np.random.default_rng(17 + which)
    out = []
    while len(out) < count:
        d = float(3e-7 * rng.uniform(0.5, 2.0))
        m = [float(d * x) for x in rng.normal(0.0, 1e5, 3)]
        once, apart = floors(d, m, True), floors(d, m, False)
        e = once[which]
        if once[1 - which] <= e < apart[which]:
            out.append((d, m, e))
    return out


def test_tie_states_exist():
    for which in (0, 1):
        for d, m, e in tie_states(which, 4):
            assert floors(d, m, True)[which] == e < floors(d, m, False)[which]


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1], ids=["TVDlimit", "Tcheck"])
def test_floor_met_exactly(gpu_lib, which):
    n = 6
    for d, m, e in tie_states(which, 4):
        U = np.empty((8, n + 4, n + 4, n + 4))
        for q, x in enumerate([d, *m, e, 20.0, -10.0, 5.0]):
            U[q] = x
        p = gpumhd.default_params(n, n, n, 3.2e6, autostep=0, dt=0.5)
        p.tchk[0] = EPS_MIN
        g = gpumhd.MuramGPU(p, eos_path=H.EOS_SMALL)
        g.upload_state(U)
        g.run_steps(2)
        assert np.array_equal(g.download_state(), U)  # nothing moves, no floor acts
        lam = np.zeros_like(U)
        lam[4, 2:-2, 2:-2, 2:-2] = 1.0
        g.upload_state(U)
        grad = g.adjoint(2, lam)
        g.close()
        assert np.allclose(H.interior(grad)[4], 1.0, rtol=0, atol=1e-9), H.interior(grad)[4].ravel()[:4]
