"""The fixed-point quaternions of the FP64 integer powers (qj_fxmath.h) built
for the host, against 300-bit values.  Relative to the exact result's norm: a
product loses at most 2^-55 (four truncated halves of at least 2^58), a
difference that fx_near passes 2^-53, the conversion back 2^-53."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quijibo_gb300", "csrc")

SOURCE = """
#include "qj_fxmath.h"
static void put(fx_quat r, double* o, int* e) {
  o[0] = (double)r.w; o[1] = (double)r.x; o[2] = (double)r.y; o[3] = (double)r.z; *e = r.e - 62; }
static fx_quat get(const double* q) { return fx_quat_of(q[0], q[1], q[2], q[3]); }
void product(const double* q, const int* pw, long n, double* o, int* e) {
  fx_quat r = get(q);
  for (long i = 0; i < n; i++) {
    fx_quat b = get(q + 4 * i), t = b;
    if (pw[i] > 1) t = fx_qsq(b);
    for (int k = 2; k < pw[i]; k++) t = fx_qmul(t, b);
    r = i ? fx_qmul(r, t) : t;
  }
  put(r, o, e);
}
int difference(const double* a, const double* b, double* o, int* e) {
  fx_quat x = get(a), y = get(b), d = fx_qsub(x, y);
  put(d, o, e);
  return fx_near(d, x, y);
}
double scaled(double v, int k) { return fx_scale(v, k); }
"""


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    d = tmp_path_factory.mktemp("fxq")
    (d / "fx.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o",
                    str(d / "fx.so"), str(d / "fx.c"), "-lm"], check=True)
    lib = ctypes.CDLL(str(d / "fx.so"))
    lib.scaled.restype = ctypes.c_double
    lib.scaled.argtypes = [ctypes.c_double, ctypes.c_int]
    return lib


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _mul(a, b):
    return [a[0] * b[0] - a[1] * b[1] - a[2] * b[2] - a[3] * b[3],
            a[0] * b[1] + a[1] * b[0] + a[2] * b[3] - a[3] * b[2],
            a[0] * b[2] - a[1] * b[3] + a[2] * b[0] + a[3] * b[1],
            a[0] * b[3] + a[1] * b[2] - a[2] * b[1] + a[3] * b[0]]


def _exact(q):
    return [mpmath.mpf(float(v)) for v in q]


def _norm(q):
    return mpmath.sqrt(sum(v * v for v in q))


def _off(o, e, exact):
    got = [mpmath.ldexp(mpmath.mpf(float(v)), int(e)) for v in o]
    return _norm([a - b for a, b in zip(got, exact)]) / _norm(exact)


@pytest.mark.parametrize("n", [1, 2, 24, 48])
@pytest.mark.parametrize("kind", ["even", "scales", "sparse", "extreme"])
def test_products(fx, n, kind):
    rng = np.random.RandomState(n)
    out, e = np.empty(4), ctypes.c_int()
    with mpmath.workprec(300):
        for _ in range(40):
            q = rng.uniform(-1, 1, (n, 4))
            if kind == "scales":
                q *= 10.0 ** rng.uniform(-6, 6, (n, 1))
            elif kind == "sparse":
                q *= (rng.uniform(size=(n, 4)) < 0.4) * 10.0 ** rng.uniform(-25, 0, (n, 4))
                q[np.abs(q).sum(1) == 0, rng.randint(4)] = -1.0
            elif kind == "extreme":  # powers of two: the ends of the mantissa's range
                q = rng.choice([-1.0, 1.0, np.nextafter(1, 0), -np.nextafter(2, 0)], (n, 4))
            q = np.ascontiguousarray(q)
            pw = rng.randint(1, 5, n).astype(np.int32)
            fx.product(_p(q), _p(pw), ctypes.c_long(n), _p(out), ctypes.byref(e))
            want, products = None, int(pw.sum()) - 1
            for i in range(n):
                for _ in range(pw[i]):
                    want = _exact(q[i]) if want is None else _mul(want, _exact(q[i]))
            # a power's earlier products count once for each later factor's place
            assert _off(out, e.value, want) <= products * 2.0 ** -55 + n * 5 * 2.0 ** -60 + 2.0 ** -53


def test_zero_factor_gives_zero(fx):
    q = np.array([[1.0, -2.0, 0.5, 0.0], [0.0, -0.0, 0.0, 0.0], [-3.0, 1.0, 1.0, 1.0]])
    out, e = np.empty(4), ctypes.c_int()
    fx.product(_p(q), _p(np.array([2, 3, 1], np.int32)), ctypes.c_long(3), _p(out), ctypes.byref(e))
    assert not out.any()


@pytest.mark.parametrize("bits", [0, 3, 5, 6, 7, 12, 40, 70])
def test_differences(fx, bits):
    rng = np.random.RandomState(bits)
    out, e = np.empty(4), ctypes.c_int()
    with mpmath.workprec(300):
        for _ in range(400):
            a = rng.uniform(-1, 1, 4) * 2.0 ** rng.randint(-8, 8) * 10.0 ** rng.uniform(-9, 0, 4)
            d = rng.uniform(-1, 1, 4)
            b = a + d * np.abs(a).max() / np.abs(d).max() * 2.0 ** -bits
            near = fx.difference(_p(a), _p(b), _p(out), ctypes.byref(e))
            want = [x - y for x, y in zip(_exact(a), _exact(b))]
            if near:
                assert _norm(want) < 2.0 ** -4 * max(np.abs(a).max(), np.abs(b).max())
            else:
                assert _off(out, e.value, want) <= 2.0 ** -53 + 2.0 ** -53
            if bits >= 8:
                assert near


@pytest.mark.parametrize("v,k,want", [
    (1.5, 3, 12.0), (-1.5, -3, -0.1875), (0.0, 900, 0.0), (-0.0, -900, -0.0), (1.0, 1024, np.inf),
    (-1.0, 5000, -np.inf), (1.0, -1022, 2.0 ** -1022), (1.0, -1023, 0.0), (np.inf, -5, np.inf),
    (np.nan, 2, np.nan), (1.75, 1023, 1.75 * 2.0 ** 1023)])
def test_scale(fx, v, k, want):
    got = fx.scaled(v, k)
    assert np.array_equal(got, want, equal_nan=True) and np.signbit(got) == np.signbit(want)
