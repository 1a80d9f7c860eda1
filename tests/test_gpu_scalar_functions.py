"""The short reciprocals, square roots and rotation tangents of hc_scalar.cuh against
extended precision, over the ranges that they are declared for (normal and positive;
a reciprocal's result normal too), with the ends of the range, powers of two and their
neighbours among the inputs.

Bounds.  FP64: an FP32 seed is within 2^-21 (the seed functions' documented errors and the
truncated argument's 2^-23), a third-order step leaves its cube, 2^-63 times a constant
below 1, and the last FMA rounds to half a unit: 0.51 ulp of the result is 2^-52.9 relative at
most, and 2^-52 is asserted.  FP32: one Newton step leaves 1.5 times the square of 2^-21.5, the
products round once each to 2^-24 of a term that is itself the small correction: 2^-23 asserted for the
reciprocal, 2^-22.5 for the root, whose x y^2 rounds twice.  Tangents only bring an inner
product down (they are computed from FP32 values in both precisions): 2^-18 relative of
the exact tangent, sign included."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
EXT = np.longdouble


@pytest.fixture(scope="module")
def scalar(hc, tmp_path_factory):
    from hcore_gb300 import build

    so = str(tmp_path_factory.mktemp("scalar") / "scalar_functions.so")
    subprocess.run([build.nvcc()] + build._flags() + ["-shared", "-cudart", "static", "-o", so,
                                                      os.path.join(HERE, "scalar_functions.cu")], check=True)
    lib = C.CDLL(so)

    def call(what, *args):
        args = [np.ascontiguousarray(a) for a in args]
        args += [np.ones_like(args[0])] * (3 - len(args))
        f, t = (lib.scalar_f64, C.c_double) if args[0].dtype == np.float64 else (lib.scalar_f32, C.c_float)
        out = np.empty_like(args[0])
        ptr = [a.ctypes.data_as(C.POINTER(t)) for a in args + [out]]
        assert f(what, len(out), *ptr) == 0
        return out

    return call


def _inputs(dt, lo, hi, n=200000):
    """n values of exponents lo .. hi, then every power of two there and its neighbours"""
    rng = np.random.default_rng(9)
    x = np.ldexp(1 + rng.random(n).astype(dt), rng.integers(lo, hi, n)).astype(dt)
    p = np.ldexp(dt(1), np.arange(lo, hi + 1)).astype(dt)
    x = np.concatenate([x, p, np.nextafter(p[1:], dt(0)), np.nextafter(p[:-1], dt(np.inf))])
    return x[np.isfinite(x)]


@pytest.mark.parametrize("dt,lo,hi,bound", [(np.float64, -1022, 1021, 2.0 ** -52), (np.float32, -126, 125, 2.0 ** -23)])
def test_reciprocal(scalar, dt, lo, hi, bound):
    x = _inputs(dt, lo, hi)
    got, one = scalar(0, x).astype(EXT), EXT(1)
    assert float(np.abs(got * x.astype(EXT) - one).max()) <= bound


@pytest.mark.parametrize("dt,lo,hi,bound", [(np.float64, -1022, 1023, 2.0 ** -52),
                                            (np.float32, -126, 127, 2.0 ** -22.5)])
def test_reciprocal_square_root(scalar, dt, lo, hi, bound):
    x = _inputs(dt, lo, hi)
    got = scalar(1, x).astype(EXT)
    assert float(np.abs(got * np.sqrt(x.astype(EXT)) - EXT(1)).max()) <= bound


@pytest.mark.parametrize("dt,span", [(np.float64, 300), (np.float32, 30)])
def test_tangent(scalar, dt, span):
    rng = np.random.default_rng(8)
    n = 100000
    app = (10.0 ** rng.uniform(-span / 10, span / 10, n)).astype(dt)
    aqq = np.where(rng.random(n) < 0.2, app, app * (10.0 ** rng.uniform(-3, 3, n))).astype(dt)
    apq = (np.sqrt(app.astype(float) * aqq) * 10.0 ** rng.uniform(-5, 0, n) * rng.choice([-1, 1], n)).astype(dt)
    w, v = aqq.astype(EXT) - app.astype(EXT), 2 * apq.astype(EXT)
    w = (aqq - app).astype(dt).astype(EXT)   # (the difference as the kernels round it)
    want = np.abs(v) / (np.abs(w) + np.sqrt(w * w + v * v)) * np.where((w < 0) != (v < 0), -1, 1)
    got = scalar(2, app, aqq, apq).astype(EXT)
    assert (np.sign(got) == np.sign(want)).all()
    assert float(np.abs(got / want - 1).max()) <= 2.0 ** -18
