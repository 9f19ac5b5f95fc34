"""FP64 rounding against extended precision.

The oracle's source is compiled once more with `long double` in place of
`double` (80 bits on x86-64, 128 on AArch64; the parameters, the step control
and the EOS file stay as they are), and both the FP64 GPU steps and the plain
oracle are measured against it.  The GPU's sums are fused where that saves a
rounding and its logarithms and exponentials are its own, so its bits are not
the oracle's; its errors have to be no larger than the plain double
arithmetic's, up to a fifth for the chance in a field's accumulated
roundings."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

import helpers as H
from muram_main_gb300 import gpumhd, initial
from oracle import oracle as O

LD = np.longdouble


@pytest.fixture(scope="module")
def extended(tmp_path_factory):
    if np.finfo(LD).nmant <= 52:
        pytest.skip("long double is no wider than double here")
    d = tmp_path_factory.mktemp("extended")
    wide = lambda s: re.sub(r"\bdouble\b", "long double", s)
    src, hdr = (open(os.path.join(O.HERE, f)).read() for f in ("muram_oracle.c", "muram_oracle.h"))
    at = hdr.index("} mo_params")  # the parameters are doubles, and pointers to them
    (d / "muram_oracle.h").write_text(hdr[:at] + wide(hdr[at:]).replace("int nz, long double dx", "int nz, double dx"))
    at = src.index("\nvoid mo_save_cons(")  # before it: parameters and the EOS file, which stay as they are
    src = re.sub(r"static inline double sm.*", lambda m: wide(m.group()), src[:at]) + re.sub(
        r"long double(\* \w+ = p->)", r"double\1", wide(src[at:]))
    (d / "muram_oracle.c").write_text(src)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-std=c11", "-include", "tgmath.h", "-fPIC", "-shared", "-o",
                    str(d / "x.so"), str(d / "muram_oracle.c"), "-lm"], check=True)
    L = C.CDLL(str(d / "x.so"))
    L.mo_eos_load.restype = C.c_void_p
    L.mo_eos_load.argtypes = [C.c_char_p]
    return L


def _extended_steps(L, p, U, steps):
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    U = np.ascontiguousarray(U, dtype=LD).copy()
    U0, R, aux = np.zeros_like(U), np.zeros_like(U), np.zeros((5,) + U.shape[1:], dtype=LD)
    field = [np.zeros(U.shape[1:], dtype=LD) for _ in range(6)]  # phi, divB, sflx, sflx0, Rflx, BgradT
    fields = (C.c_void_p * 6)(*[f.ctypes.data for f in field])
    eos = C.c_void_p(L.mo_eos_load(H.EOS_SMALL.encode()))
    assert eos
    L.mo_boundaries(C.byref(p), ptr(U))
    for _ in range(steps):
        assert L.mo_step_ex(C.byref(p), eos, ptr(U), ptr(U0), ptr(R), ptr(aux), fields) == 0
    return U


def _errors(A, E):
    """Relative L2 per field over the interior."""
    A, E = H.interior(np.asarray(A, dtype=LD)), H.interior(E)
    return np.array([float(np.sqrt(((a - e) ** 2).sum() / (e ** 2).sum())) for a, e in zip(A, E)])


BOXES = [((64, 12, 10), True, 2), ((20, 16, 12), False, 5)]


def test_oracle_in_extended_precision_is_near_the_oracle(extended):
    shape, closed, steps = (20, 16, 12), False, 2
    U = initial.periodic_box(initial.EosTable(H.EOS_SMALL), *shape, seed=6)
    E = _extended_steps(extended, O.make_params(*shape, 3.2e6), U, steps)
    st = O.State(O.make_params(*shape, 3.2e6), U)
    st.step(O.Eos(H.EOS_SMALL), steps)
    e = _errors(st.U, E)
    assert np.all(e > 0) and np.all(e <= 1e-13), e


@pytest.mark.gpu
@pytest.mark.parametrize("box", range(len(BOXES)))
def test_fp64_is_no_less_exact_than_plain_doubles(gpu_lib, extended, box):
    shape, closed, steps = BOXES[box]
    tab = initial.EosTable(H.EOS_SMALL)
    U = (initial.stratified_box if closed else initial.periodic_box)(tab, *shape, seed=5 + box)
    dx, grav = (1.6e6, 2.74e4) if closed else (3.2e6, 0.0)
    params = lambda: O.make_params(*shape, dx, periodic_x=not closed, grav=grav)
    E = _extended_steps(extended, params(), U, steps)
    st = O.State(params(), U)
    st.step(O.Eos(H.EOS_SMALL), steps)
    g = gpumhd.MuramGPU(gpumhd.default_params(*shape, dx, periodic_x=0 if closed else 1, grav=grav),
                        eos_path=H.EOS_SMALL)
    g.upload_state(U)
    g.run_steps(steps)
    gpu, plain = _errors(g.download_state(), E), _errors(st.U, E)
    g.close()
    print(f"{shape}, {steps} steps: relative L2 from extended precision, GPU {np.array2string(gpu, precision=2)}, "
          f"plain doubles {np.array2string(plain, precision=2)}")
    assert np.all(gpu <= 1.2 * plain), (gpu, plain)
