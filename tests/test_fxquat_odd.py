"""What the fixed-point quaternion products (qj_fxmath.h) keep of FP64's: sign
symmetry, exact cancellation of conjugates, and `odd` where a component would
have fewer bits than in FP64.  Built for the host."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quijibo_gb300", "csrc")

SOURCE = """
#include "qj_fxmath.h"
static void put(fx_quat r, long long* o) {
  o[0] = r.w; o[1] = r.x; o[2] = r.y; o[3] = r.z; o[4] = r.e; o[5] = r.odd; }
static fx_quat get(const double* q) { return fx_quat_of(q[0], q[1], q[2], q[3]); }
void product(const double* q, long n, long long* o) {
  fx_quat r = get(q);
  for (long i = 1; i < n; i++) r = fx_qmul(r, get(q + 4 * i));
  put(r, o);
}
void power(const double* q, long n, long long* o) {
  fx_quat b = get(q), r = fx_qsq(b);
  for (long i = 2; i < n; i++) r = fx_qpower(r, b);
  put(r, o);
}
void beside(const double* roots, const double* q, long n, long long* o) {
  int top = -1100;
  for (long i = 0; i < n; i++) {
    const double* r = roots + 4 * i;
    if (fx_top(r[0], r[1], r[2], r[3]) > top) top = fx_top(r[0], r[1], r[2], r[3]);
  }
  const int map = fx_beside_of((const double(*)[4])roots, (int)n, top), t = fx_top(q[0], q[1], q[2], q[3]);
  o[5] = map && fx_beside(map, q[1], q[2], q[3], t > top ? t : top);
}
void difference(const double* a, const double* b, long long* o) { put(fx_qsub(get(a), get(b)), o); }
"""


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    d = tmp_path_factory.mktemp("fxo")
    (d / "fx.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o",
                    str(d / "fx.so"), str(d / "fx.c"), "-lm"], check=True)
    lib = ctypes.CDLL(str(d / "fx.so"))

    def call(name, *args):
        o = np.empty(6, np.int64)
        ptr = [np.ascontiguousarray(a, float) for a in args if not isinstance(a, int)]
        rest = [ctypes.c_long(a) for a in args if isinstance(a, int)]
        getattr(lib, name)(*[a.ctypes.data_as(ctypes.c_void_p) for a in ptr], *rest,
                           o.ctypes.data_as(ctypes.c_void_p))
        return o[:4], int(o[4]), int(o[5])
    return call


CONJ = np.array([1, -1, -1, -1])
TURNS = [np.array([1, 1, -1, -1]), np.array([1, -1, 1, -1]), np.array([1, -1, -1, 1])]


def _factors(rng, n, kind):
    q = rng.uniform(-1, 1, (n, 4))
    if kind == "scales":
        q *= 10.0 ** rng.uniform(-12, 0, (n, 4))
    elif kind == "plane":
        q[:, 2:] *= 10.0 ** rng.uniform(-25, -1)
    elif kind == "axis":
        q[:, 1:] *= 10.0 ** rng.uniform(-25, -1)
    elif kind == "twos":
        q = rng.choice([-1.0, 1.0, 0.5, -2.0, 0.0], (n, 4))
        q[:, rng.randint(4)] = -1.0
    return q


@pytest.mark.parametrize("kind", ["even", "scales", "plane", "axis", "twos"])
def test_mirror_images_have_the_same_bits(fx, kind):
    rng = np.random.RandomState(1)
    for _ in range(300):
        q = _factors(rng, 5, kind)
        calls = [("product", q, 5), ("power", q[0], 2), ("power", q[0], 3), ("difference", q[0], q[1])]
        for s in TURNS:  # turns by half about an axis: (ab)' = a'b'
            for name, *args in calls:
                v, e, odd = fx(name, *args)
                w, we, wo = fx(name, *[t if isinstance(t, int) else t * s for t in args])
                assert (w * s == v).all() and (we, wo) == (e, odd)
        # (ab)* = b* a*; the square is a function of the scalar and one vector
        v, e, odd = fx("product", q[:2], 2)
        w, we, wo = fx("product", q[1::-1] * CONJ, 2)
        assert (w * CONJ == v).all() and (we, wo) == (e, odd)
        assert (fx("power", q[0] * CONJ, 2)[0] * CONJ == fx("power", q[0], 2)[0]).all()
        assert (-fx("difference", -q[0], -q[1])[0] == fx("difference", q[0], q[1])[0]).all()


@pytest.mark.parametrize("kind", ["even", "scales", "plane", "twos"])
def test_conjugate_factors_cancel(fx, kind):
    rng = np.random.RandomState(2)
    for _ in range(300):
        q = _factors(rng, 1, kind)[0]
        v, _, odd = fx("product", np.stack([q, q * CONJ]), 2)
        assert not v[1:].any() and v[0] > 0 and (odd or not q[1:].any())


@pytest.mark.parametrize("kind", ["even", "scales", "plane", "axis", "twos"])
def test_components_are_kept_or_marked(fx, kind):
    """A component's terms are cut by less than a unit each and its factors by
    one before: 12 units.  Unmarked, the largest term has 2^44 of them."""
    rng = np.random.RandomState(3)
    marked = 0
    with mpmath.workprec(300):
        for _ in range(400):
            a, b = _factors(rng, 2, kind)
            v, e, odd = fx("product", np.stack([a, b]), 2)
            marked += odd
            if odd:
                continue
            a, b = [[mpmath.mpf(float(t)) for t in q] for q in (a, b)]
            terms = [[a[0] * b[0], -a[1] * b[1], -a[2] * b[2], -a[3] * b[3]],
                     [a[0] * b[1], a[1] * b[0], a[2] * b[3], -a[3] * b[2]],
                     [a[0] * b[2], -a[1] * b[3], a[2] * b[0], a[3] * b[1]],
                     [a[0] * b[3], a[1] * b[2], -a[2] * b[1], a[3] * b[0]]]
            for c in range(4):
                got = mpmath.ldexp(int(v[c]), e - 62)
                assert abs(got - sum(terms[c])) <= 12 * mpmath.mpf(2) ** -44 * max(abs(t) for t in terms[c])
    assert marked <= 4 if kind == "even" else True


def test_a_tiny_component_is_marked(fx):
    for tiny in (1e-17, 5e-324, -1e-300):
        assert fx("product", [[1.0, tiny, 0.0, 0.0]], 1)[2]
        assert fx("difference", [1.0, 0.5, tiny, 0.0], [0.25, 1.0, 0.0, 0.0])[2] & 4
    assert not fx("product", [[1.0, 0.0, 0.0, 0.0], [0.5, 0.0, 0.0, 0.0]], 2)[2]
    assert not fx("product", [[1.0, 0.5, 0.0, 0.0], [0.5, 0.25, 0.0, 0.0]], 2)[2]


@pytest.mark.parametrize("roots,near,not_near", [
    ("axis", [[1, 1e-3, 0.3, 0.3], [0.1, 1e-17, 0, 0], [2.0, 1e-3, 1e-3, 1e-3]],
     [[1, 0, 0.3, 0.3], [1, 0, 0, 0], [1, 0.1, -0.1, 0.1]]),
    ("plane", [[1, 0.3, 1e-3, 0], [0.2, 0.3, 1e-17, -1e-4]],
     [[1, 0.3, 0, 0], [1, 0.3, 1e-3, 0.5], [1, 0, 0.1, 0.1]]),
    ("almost", [[1, 0.3, 0, 0], [1, 0.3, 1e-3, 0]], [[1, 0.3, 0.2, 0.1]]),
    ("flat", [], [[1, 0.3, 0.2, 0], [1, 0.3, 0.2, 1e-9], [1, 0, 0, 0]]),
    ("any", [], [[1, 0.3, 1e-9, 0], [1, 1e-9, 1e-9, 1e-9]])])
def test_beside_the_roots_axis_or_plane(fx, roots, near, not_near):
    r = np.random.RandomState(4).uniform(-1.2, 1.2, (9, 4))
    r[:, {"axis": slice(1, 4), "plane": slice(2, 4), "almost": slice(2, 4), "flat": slice(3, 4),
          "any": slice(0, 0)}[roots]] *= 1e-6 if roots == "almost" else 0.0
    for q in near:
        assert fx("beside", r, q, 9)[2]
    for q in not_near:
        assert not fx("beside", r, q, 9)[2]
