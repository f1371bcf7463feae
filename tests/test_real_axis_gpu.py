"""Points on the real axis of maps with conjugate roots.  The products of
conjugate factors cancel exactly there in FP64, and the orbits stay on the
axis; a vector part of one rounding takes them off it, to another value."""
import numpy as np
import pytest

from quijibo_gb300 import lib
from quijibo_gb300.rootsets import Grid, RootSet

pytestmark = pytest.mark.gpu
LINE = Grid((65, 1, 1))  # cell centres with y = z = 0


def conjugate_map(seed, nb):
    """One pair and one real root (and nb of the same below), a pair's roots
    in turn, as fitted real polynomials have them."""
    rng = np.random.RandomState(seed)

    def side():
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        a, b, c = rng.uniform(-1, 1, 3)
        return np.array([[a, *(b * u)], [a, *(-b * u)], [c, 0, 0, 0]])

    top, bottom = side(), side()[:nb]
    return RootSet(top_roots=top, top_powers=np.ones(3), bottom_roots=bottom,
                   bottom_powers=np.ones(nb), scale=1.3)


def _mul(a, b):
    w = ((a[0] * b[0] - a[1] * b[1]) - b[2] * a[2]) - a[3] * b[3]
    x = ((a[2] * b[3] - a[3] * b[2]) + b[0] * a[1]) + a[0] * b[1]
    y = ((a[3] * b[1] - a[1] * b[3]) + b[0] * a[2]) + a[0] * b[2]
    z = ((a[1] * b[2] - a[2] * b[1]) + b[0] * a[3]) + a[0] * b[3]
    return np.stack([w, x, y, z])


def _div(a, b):
    inv = 1.0 / (((b[0] * b[0] + b[1] * b[1]) + b[2] * b[2]) + b[3] * b[3])
    return _mul(a, np.stack([b[0] * inv, -b[1] * inv, -b[2] * inv, -b[3] * inv]))


def _field(rs, q, max_it, escape, lagrange):
    """log|q_N| with exponents 1 and every product in the reference's order
    and rounding (QUATERNION.cpp:154-182, RATIONAL_4D.cpp:27-73)."""
    top, bottom = rs.top_roots[:, :, None], rs.bottom_roots[:, :, None]
    q = q.copy()

    def mag(v):
        return np.sqrt(((v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]) + v[3] * v[3])

    for _ in range(max_it):
        live = mag(q) < escape
        p = q[:, live]
        if lagrange and len(bottom):
            r = np.zeros_like(p)
            r[0] = 1.0
            for k in range(len(top)):
                r = _mul(r, p - top[k])
                if k < len(bottom):
                    r = _div(r, p - bottom[k])
        else:
            r = p - top[0]
            for k in range(1, len(top)):
                r = _mul(r, p - top[k])
            if len(bottom):
                b = p - bottom[0]
                for k in range(1, len(bottom)):
                    b = _mul(b, p - bottom[k])
                r = _div(r, b)
        q[:, live] = r * rs.scale
    return np.log(mag(q))


def _start(g):
    x, y, z = (np.array([(-0.5 * w + i * (w / n)) + (w / n) * 0.5 for i in range(n)])
               for n, w in zip(g.res, g.lengths))
    z, y, x = np.meshgrid(z, y, x, indexing="ij")
    return np.stack([x.ravel(), y.ravel(), z.ravel(), np.full(x.size, g.slice)])


def _integer_form(ctx, rs, g, max_it, lagrange):
    h = ctx.upload(rs)
    it = ctx.iter_params(max_it, 2.0, precision=lib.QJG_FP32_REFINE, rel_tol=1e-30,
                         refine_pow=lib.QJG_REFINE_INT, lagrange=lagrange)
    f, _, st = ctx.field_host(h, g, it)
    ctx.free(h)
    assert st["refined"] == f.size
    return f.ravel()


def _assert_same(f, want):
    """The logarithm's own rounding: the device's within 1 ulp, numpy's too."""
    assert (np.abs(f - want) <= 2 * np.spacing(np.abs(want))).all()


@pytest.mark.parametrize("max_it", [1, 40])
@pytest.mark.parametrize("seed,nb", [(0, 0), (100, 0), (112, 0), (1, 1), (3, 3), (32, 3), (65, 3)])
def test_integer_powers_in_the_lagrange_order(ctx, seed, nb, max_it):
    rs = conjugate_map(seed, nb)
    _assert_same(_integer_form(ctx, rs, LINE, max_it, True),
                 _field(rs, _start(LINE), max_it, 2.0, True))


@pytest.mark.parametrize("max_it", [1, 40])
@pytest.mark.parametrize("seed,nb", [(0, 0), (100, 0), (112, 0), (1, 1), (3, 3), (32, 3), (65, 3)])
def test_integer_powers(ctx, seed, nb, max_it):
    rs = conjugate_map(seed, nb)
    f, want = _integer_form(ctx, rs, LINE, max_it, False), _field(rs, _start(LINE), max_it, 2.0, False)
    if nb == 1:  # half a pair below: off the axis from the first step, no exact cancellation
        assert (np.abs(f - want) <= 1e-9 * (1 + np.abs(want))).all()
    else:
        _assert_same(f, want)


def _assert_polar_forms(ctx, oracle, rs, g):
    """One last-bit change in every power leaves these fields within 1e-6;
    a vector part of 2^-61 changes the sign of up to two thirds of them."""
    o = oracle.field(rs, g, 40, 2.0)["field"]
    h = ctx.upload(rs)
    for it in (ctx.iter_params(40, 2.0),
               ctx.iter_params(40, 2.0, precision=lib.QJG_FP32_REFINE, rel_tol=1e-30)):
        f = ctx.field_host(h, g, it)[0]
        assert np.array_equal(f > 0, o > 0)
        assert (np.abs(f - o) <= 1e-6 * (1 + np.abs(o))).all()
    ctx.free(h)


@pytest.mark.parametrize("seed,nb", [(11, 0), (13, 0), (18, 0), (19, 0), (1, 3), (14, 3), (16, 3), (18, 3), (32, 3)])
def test_polar_powers(ctx, oracle, seed, nb):
    _assert_polar_forms(ctx, oracle, conjugate_map(seed, nb), LINE)


@pytest.mark.parametrize("g", [Grid((33, 1, 1)), Grid((21, 21, 21))])
@pytest.mark.parametrize("c", [-0.6, -1.2])
def test_cubic(ctx, oracle, c, g):
    """q^3 + c, the pair before the real root; on the odd cube the axis cells
    have y and z a rounding off 0."""
    z = np.roots([1, 0, 0, c])
    pair, real = z[z.imag > 1e-9][0], z[abs(z.imag) < 1e-9][0].real
    top = [[pair.real, pair.imag, 0, 0], [pair.real, -pair.imag, 0, 0], [real, 0, 0, 0]]
    _assert_polar_forms(ctx, oracle, RootSet(top_roots=np.array(top), top_powers=np.ones(3)), g)


@pytest.mark.parametrize("form", ["polar", "integer"])
@pytest.mark.parametrize("nt,nb", [(5, 0), (6, 3)])
def test_mirror_images_have_the_same_bits(ctx, nt, nb, form):
    """Roots on the real axis: the map commutes with every reflection that
    keeps it; the cells of a 16^3 grid are each other's mirror images."""
    rng = np.random.RandomState(nt)
    roots = np.zeros((nt + nb, 4))
    roots[:, 0] = rng.uniform(-1.2, 1.2, nt + nb)
    powers = rng.uniform(0.5, 2, nt + nb) if form == "polar" else rng.choice([1.0, 2.0, 3.0], nt + nb)
    rs = RootSet(top_roots=roots[:nt], top_powers=powers[:nt], bottom_roots=roots[nt:],
                 bottom_powers=powers[nt:], scale=0.7)
    g = Grid((16, 16, 16))
    if form == "integer":
        f = _integer_form(ctx, rs, g, 25, False).reshape(16, 16, 16)
    else:
        h = ctx.upload(rs)
        f = ctx.field_host(h, g, ctx.iter_params(25, 2.0))[0]
        ctx.free(h)
    bits = f.view(np.uint64)
    assert np.array_equal(bits, bits[:, ::-1]) and np.array_equal(bits, bits[::-1])
