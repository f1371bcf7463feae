"""Orbits that settle on cycles of known period (q^2 + c near the centre of a
period-2, 3 or 6 component) and the counters that show they are cut short."""
import numpy as np
import pytest

from quijibo_gb300 import lib
from quijibo_gb300.rootsets import Grid, RootSet
from test_orbit_period_gpu import settling_map

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# c whose critical orbit 0 -> c -> c^2 + c ... returns after p steps
CENTRES = {2: -1.0 + 0j, 3: -0.12256116687665362 + 0.7448617666197442j,
           6: 0.3890068405697712 + 0.2158506508724438j}
PERIODS = [2, 3, 6]


def cycle(c, p):
    z = 0j
    for _ in range(600 * p):
        z = z * z + c
    out = [z]
    for _ in range(p - 1):
        out.append(out[-1] ** 2 + c)
    return np.array(out)


def cycle_map(p, rate):
    """q^2 + c as (q - r)(q + r), in the (w, x) plane, whose attracting p-cycle
    contracts by `rate`: small rates settle early."""
    a, b = 0.0, 0.003 if p == 6 else 0.02
    while np.abs(np.prod(2 * cycle(CENTRES[p] + 1j * b, p))) < rate:
        b *= 1.25
    for _ in range(60):
        t = 0.5 * (a + b)
        a, b = (t, b) if np.abs(np.prod(2 * cycle(CENTRES[p] + 1j * t, p))) < rate else (a, t)
    r = np.sqrt(-(CENTRES[p] + 1j * a))
    return RootSet(top_roots=np.array([[r.real, r.imag, 0, 0], [-r.real, -r.imag, 0, 0]]),
                   top_powers=np.ones(2))


PLANE = Grid((61, 61, 1))  # cells with y = z = 0


@pytest.mark.parametrize("p", PERIODS)
def test_the_maps_have_these_periods(p):
    r = complex(*cycle_map(p, 0.02).top_roots[0, :2])
    z = cycle(-r * r, p)
    assert abs(z[-1] ** 2 - r * r - z[0]) < 1e-12 and abs(abs(np.prod(2 * z)) - 0.02) < 1e-6
    assert min(abs(z[0] - z[k]) for k in range(1, p)) > 1e-2 and np.abs(z).max() < 1.9


# every remainder of the steps left, modulo 6
@pytest.mark.parametrize("max_it", range(54, 60))
@pytest.mark.parametrize("p", PERIODS)
@pytest.mark.parametrize("precision,de", [(lib.QJG_FP32, True), (lib.QJG_FP32, False),
                                          (lib.QJG_FP32_REFINE, True)])
def test_fp32_orbits_on_cycles_are_cut_short(ctx, p, max_it, precision, de):
    h = ctx.upload(cycle_map(p, 0.02))
    it = ctx.iter_params(max_it, 2.0, precision=precision, want_de=de, refine_pow=lib.QJG_REFINE_INT)
    out = []
    try:
        for pairs in (True, False):
            lib.set_field32_pairs(pairs)
            out.append((*ctx.field_host(h, PLANE, it, de=de), ctx.field_applied()))
    finally:
        lib.set_field32_pairs(True)
        ctx.free(h)
    (fa, da, sa, na), (fb, db, sb, nb) = out
    assert np.array_equal(fa.view(np.uint64), fb.view(np.uint64))
    if de:
        assert np.array_equal(da.view(np.uint32), db.view(np.uint32))
    # the cycle has p points: an orbit that is cut short came back after a
    # multiple of p steps; the one-voxel kernel applies the map to the end
    assert 0 < na < sa["voxel_iters"] and nb == sb["voxel_iters"] == sa["voxel_iters"]


@pytest.mark.parametrize("max_it", range(96, 102))
@pytest.mark.parametrize("p", PERIODS)
@pytest.mark.parametrize("refine_pow", [lib.QJG_REFINE_INT, lib.QJG_REFINE_POW])
def test_fp64_orbits_on_cycles_equal_the_full_loop(ctx, p, max_it, refine_pow):
    """With the distance estimate only period 1 ends early: the full loop."""
    h = ctx.upload(cycle_map(p, 0.02))
    f, g = [ctx.field_host(h, PLANE, ctx.iter_params(
        max_it, 2.0, precision=lib.QJG_FP32_REFINE, rel_tol=1e-30, refine_pow=refine_pow, want_de=de),
        de=de) for de in (False, True)]
    ctx.free(h)
    assert np.array_equal(f[0].view(np.uint64), g[0].view(np.uint64))
    assert f[2]["refined_iters"] == g[2]["refined_iters"] and f[2]["refined"] == f[0].size


def test_counts_of_one_call(ctx):
    """Reading a call's counters again changes nothing; short caps leave
    nothing to cut; a mesh counts its slabs' planes once each."""
    rs, g = settling_map(0, 16, 8), Grid((35, 22, 9))
    h = ctx.upload(rs)
    it = ctx.iter_params(40, 2.0, precision=lib.QJG_FP32)
    field = torch.empty(g.n_voxels, dtype=torch.float64, device="cuda")
    ctx.field(h, g, it, field.data_ptr())
    a = ctx.stats(), ctx.field_applied()
    b = ctx.stats(), ctx.field_applied()
    assert a == b and 0 < a[1] < a[0]["voxel_iters"]
    ctx.field_host(h, g, it)
    assert ctx.field_applied() == a[1]
    cap = 3 * g.n_voxels
    v = torch.empty(3 * cap, dtype=torch.float64, device="cuda")
    t = torch.empty(6 * cap, dtype=torch.int32, device="cuda")
    for slab in (0, 2):
        _, st = ctx.mesh_stream(h, g, it, d_verts64=v.data_ptr(), vert_cap=cap, d_tris=t.data_ptr(),
                                tri_cap=2 * cap, slab_nz=slab)
        assert ctx.field_applied() == a[1] and st["field"]["voxel_iters"] == a[0]["voxel_iters"]
    for max_it in (1, 3):
        _, _, st = ctx.field_host(h, g, ctx.iter_params(max_it, 2.0, precision=lib.QJG_FP32))
        assert ctx.field_applied() == st["voxel_iters"]
    ctx.field_host(h, g, ctx.iter_params(4, 2.0))
    assert ctx.field_applied() == 0  # no bulk pass
    ctx.free(h)


@pytest.mark.parametrize("max_it", [60, 61])
def test_meshes_of_a_cycle(ctx, max_it):
    """The FP32-first bisection's decisions are the FP64 form's.  The 2-cycle
    in a plane through the real axis at no special angle; it attracts from
    all sides, and its orbits settle in every component."""
    rs = cycle_map(2, 0.02)
    rs.top_roots[:, 1:] = rs.top_roots[:, 1:2] * np.array([0.48, 0.6, 0.64])
    h, g = ctx.upload(rs), Grid((28, 26, 24))
    it = ctx.iter_params(max_it, 2.0, precision=lib.QJG_FP32)
    st = ctx.field_host(h, g, it)[2]
    assert ctx.field_applied() < 0.9 * st["voxel_iters"]
    cap = 5 * g.n_voxels
    out = []
    for precision in (lib.QJG_FP64, lib.QJG_FP32_REFINE):
        v = torch.zeros(3 * cap, dtype=torch.float64, device="cuda")
        t = torch.zeros(3 * cap, dtype=torch.int32, device="cuda")
        _, st = ctx.mesh_stream(h, g, ctx.iter_params(max_it, 2.0, precision=precision, rel_tol=1e-6),
                                d_verts64=v.data_ptr(), vert_cap=cap, d_tris=t.data_ptr(), tri_cap=cap)
        out.append((st["n_verts"], st["n_tris"], v.cpu().numpy(), t.cpu().numpy()))
    ctx.free(h)
    assert st["map_evals_fp32"] > 0 and out[0][0] > 0 and out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][3], out[1][3]) and np.array_equal(out[0][2], out[1][2])


# ------------------------------------------------------------ fitting energy

def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", torch.float64)


def _energy(ctx, rs, xyz, max_it, precision):
    """Energy, gradient (d_sat = 0: settled samples have one), applications
    and orbit lengths."""
    P, X, T = _dev(lib.params_of(rs)), _dev(xyz), _dev(np.zeros(len(xyz)))
    args = (P.data_ptr(), rs.n_top, rs.n_bottom, len(xyz), X.data_ptr(), T.data_ptr(), max_it, 2.0)
    iters = torch.zeros(len(xyz), dtype=torch.int32, device="cuda")
    ctx.energy(*args, precision=precision, d_iters=iters.data_ptr(), d_sat=0.0)
    grad = torch.empty_like(P)
    e = ctx.energy(*args, precision=precision, d_grad=grad.data_ptr(), d_sat=0.0)
    return e, grad.cpu().numpy(), ctx.energy_last_work()[0], int(iters.sum())


SAMPLES = np.array([[0.02, 0.01, 0.0], [-0.03, 0.02, 0.0], [0.01, -0.04, 0.0]])


@pytest.mark.parametrize("p,rate,max_it", [(2, 0.1, 120), (2, 0.1, 121), (3, 0.02, 90), (3, 0.02, 91),
                                           (3, 0.02, 92), (6, 0.02, 91), (6, 0.02, 93), (6, 0.02, 95)])
def test_fp64_gradient_on_cycles(ctx, p, rate, max_it):
    """Central difference along the gradient: as test_gradient_of_settled_samples,
    with |d log E| below 1e4 and h = 1e-8."""
    rs = cycle_map(p, rate)
    e, g, applied, iters = _energy(ctx, rs, SAMPLES, max_it, lib.QJG_FP64)
    assert np.isfinite(e) and np.isfinite(g).all() and applied < iters
    u, params = g / np.linalg.norm(g), lib.params_of(rs)
    P, X, T = _dev(params), _dev(SAMPLES), _dev(np.zeros(len(SAMPLES)))

    def at(h):
        q = P + h * _dev(u)
        return ctx.energy(q.data_ptr(), 2, 0, len(SAMPLES), X.data_ptr(), T.data_ptr(), max_it, 2.0,
                          precision=lib.QJG_FP64, d_sat=0.0)

    h = 1e-8
    fd = (at(h) - at(-h)) / (2 * h)
    assert abs(np.linalg.norm(g) - fd) <= 1e-3 * abs(fd)


# d stays in FP32's range (d^2 below 1e30)
@pytest.mark.parametrize("p,rate,max_it", [(2, 0.3, 44), (2, 0.3, 45), (3, 0.1, 43), (3, 0.1, 44),
                                           (3, 0.1, 45), (6, 0.05, 45), (6, 0.05, 47), (6, 0.05, 49)])
def test_fp32_gradient_on_cycles(ctx, p, rate, max_it):
    """FP32 and the batch entry against FP64."""
    rs = cycle_map(p, rate)
    e64, g64, _, _ = _energy(ctx, rs, SAMPLES, max_it, lib.QJG_FP64)
    e32, g32, applied, iters = _energy(ctx, rs, SAMPLES, max_it, lib.QJG_FP32)
    assert applied < iters and e64 < 1e30
    assert np.linalg.norm(g32 - g64) <= 1e-2 * np.linalg.norm(g64)
    P, X, T = _dev(lib.params_of(rs)), _dev(SAMPLES), _dev(np.zeros(len(SAMPLES)))
    grads = [torch.empty_like(P) for _ in range(2)]
    es = ctx.energy_batch([dict(d_params=P.data_ptr(), n_top=2, n_bot=0, n=len(SAMPLES),
                                d_xyz=X.data_ptr(), d_target=T.data_ptr(), max_it=max_it, escape=2.0,
                                d_sat=0.0, d_grad=g.data_ptr()) for g in grads])
    for e, g in zip(es, grads):
        assert abs(e - e32) <= 1e-6 * abs(e32)
        assert np.linalg.norm(g.cpu().numpy() - g32) <= 1e-5 * np.linalg.norm(g32)


# --------------------------------------- caps about the line of the watch

@pytest.mark.parametrize("max_it", [5, 6, 8, 9])
@pytest.mark.parametrize("nt,nb", [(8, 0), (16, 8), (48, 24), (24, 8), (23, 8)])
@pytest.mark.parametrize("de", [False, True])
def test_caps_about_the_watch(ctx, nt, nb, max_it, de):
    """Below 9 applications (6 with 32 roots or more) nothing is watched:
    every orbit is applied to its end, with the same values."""
    h, g = ctx.upload(settling_map(nt, nt, nb)), Grid((35, 22, 5))
    it = ctx.iter_params(max_it, 2.0, precision=lib.QJG_FP32, want_de=de)
    out = []
    try:
        for pairs in (True, False):
            lib.set_field32_pairs(pairs)
            out.append((*ctx.field_host(h, g, it, de=de), ctx.field_applied()))
    finally:
        lib.set_field32_pairs(True)
        ctx.free(h)
    (fa, da, sa, na), (fb, db, sb, _) = out
    assert np.array_equal(fa.view(np.uint64), fb.view(np.uint64))
    if de:
        assert np.array_equal(da.view(np.uint32), db.view(np.uint32))
    assert sa["voxel_iters"] == sb["voxel_iters"] >= na
    if max_it < (6 if nt + nb >= 32 else 9):
        assert na == sa["voxel_iters"]
