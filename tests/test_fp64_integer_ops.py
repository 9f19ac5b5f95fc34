"""FP64 operations on the integer pipe (gpumhd_i64.cuh), compiled for the host.

Division, square root, comparisons and conversions must give the host's own
IEEE results bit for bit, whatever the seed's rounding (the GPU's approximate
reciprocal and root are within 2^-21; the host seed is skewed by as much);
log and exp stay within 0.51 and 0.62 ulp, so within one ulp of the C
library's."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
static float skew = 1.0f;
#define I64_SEED_SKEW(r) ((r) * skew)
#include "gpumhd_i64.cuh"
using namespace i64f;
extern "C" void set_skew(float s) { skew = s; }
#define UN(name, f) extern "C" void name(long n, const double* a, const double*, double* o) { for (long i = 0; i < n; i++) o[i] = f(a[i]); }
#define BIN(name, f) extern "C" void name(long n, const double* a, const double* b, double* o) { for (long i = 0; i < n; i++) o[i] = f(a[i], b[i]); }
BIN(t_div, div) BIN(t_max, max2) BIN(t_min, min2) BIN(t_fmax, fmax2) BIN(t_lt, (double)lt)
UN(t_sqrt, sqrt_) UN(t_log, log_) UN(t_exp, exp_) UN(t_half, half) UN(t_quarter, quarter) UN(t_trunc, (double)trunc_pos)
extern "C" void t_float(long n, const double* a, const double*, double* o) { for (long i = 0; i < n; i++) o[i] = from_float((float)a[i]); }
"""


@pytest.fixture(scope="module")
def ops(tmp_path_factory):
    d = tmp_path_factory.mktemp("i64")
    src, lib = d / "i64.cpp", d / "i64.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "muram_main_gb300", "csrc"), str(src), "-o", str(lib)], check=True)
    L = C.CDLL(str(lib))

    def call(name, a, b=None):
        a = np.ascontiguousarray(a, np.float64)
        b = a if b is None else np.ascontiguousarray(b, np.float64)
        o = np.empty_like(a)
        p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))
        getattr(L, name)(C.c_long(a.size), p(a), p(b), p(o))
        return o

    call.skew = lambda s: L.set_skew(C.c_float(s))
    return call


def _values(seed, n=200000):
    """Mantissas of every length and next to 1 and 2, the whole exponent range, and the special values."""
    rng = np.random.default_rng(seed)
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    keep = rng.integers(0, 53, n).astype(np.uint64)
    kind = rng.integers(0, 4, n)
    ones = np.uint64((1 << 52) - 1)
    m = np.where(kind == 1, m & (ones << keep) & ones, np.where(kind == 2, ones - (m & np.uint64(7)), np.where(
        kind == 3, m & np.uint64(7), m)))
    e = np.where(rng.random(n) < 0.5, rng.integers(900, 1150, n), rng.integers(0, 2047, n)).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64)
    x = ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308, 1.0, -1.0,
                        2.0, 0.5, np.finfo(float).max, np.nextafter(1, 0), np.nextafter(2, 0), 1e-100])
    x[: special.size ** 2] = np.repeat(special, special.size)
    y = rng.permutation(x)
    y[: special.size ** 2] = np.tile(special, special.size)
    return x, y


def _same_bits(a, b):
    return np.all((a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b)))


@pytest.mark.parametrize("skew", [1.0, 1 + 4e-7, 1 - 4e-7])
def test_division_and_root_are_correctly_rounded(ops, skew):
    ops.skew(skew)
    with np.errstate(all="ignore"):
        for seed in range(3):
            a, b = _values(seed)
            assert _same_bits(ops("t_div", a, b), a / b)
            assert _same_bits(ops("t_sqrt", a), np.sqrt(a))
            sq = a * a
            assert _same_bits(ops("t_sqrt", sq), np.sqrt(sq))
    ops.skew(1.0)


def test_comparisons_scalings_and_conversions(ops):
    with np.errstate(all="ignore"):
        a, b = _values(7)
        zeros = (a == 0) & (b == 0)  # -0 orders before +0 there
        for name, want in (("t_max", np.where(a < b, b, a)), ("t_min", np.where(b < a, b, a)), ("t_fmax", np.fmax(a, b)),
                           ("t_lt", (a < b).astype(float))):
            got = ops(name, a, b)
            assert _same_bits(got[~zeros], want[~zeros]), name
            if name != "t_lt":
                assert np.all(got[zeros] == 0)
        assert _same_bits(ops("t_half", a), 0.5 * a)
        assert _same_bits(ops("t_quarter", a), 0.25 * a)
        assert _same_bits(ops("t_float", a), a.astype(np.float32).astype(np.float64))
        t = np.where((a >= 1) & (a < 2.0 ** 31), np.trunc(a), 0.0)
        assert np.array_equal(ops("t_trunc", a), t)


def test_log_and_exp_within_an_ulp(ops):
    rng = np.random.default_rng(3)
    with np.errstate(all="ignore"):
        x = np.abs(_values(11)[0])
        x[::3] = np.exp(rng.uniform(-40, 40, x[::3].size))
        x[::7] = rng.uniform(0.5, 1.5, x[::7].size)
        got, want = ops("t_log", x), np.log(x)
        ok = np.isfinite(want)
        assert np.all(np.abs(got - want)[ok] <= np.spacing(np.abs(want[ok])))
        assert _same_bits(got[~ok], want[~ok])
        x = _values(13)[0]
        x[::2] = rng.uniform(-745, 710, x[::2].size)
        x[::3] = rng.uniform(-2, 2, x[::3].size)
        got, want = ops("t_exp", x), np.exp(x)
        ok = np.isfinite(want)
        assert np.all(np.abs(got - want)[ok] <= np.spacing(want[ok]))
        assert _same_bits(got[~ok], want[~ok])
