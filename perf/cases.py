"""What this library's users have it do, as measurable cases.

Each case is one call (or, for the set-up a program keeps, one call on a kept
map) of the Python bindings of the C ABI: the escape-time field, the meshers,
the optimizer's objective and the fitting energy.  Sizes, root counts,
exponents and iteration caps are those of the repository's workloads
(quijibo_gb300/rootsets.py, samples.py), its serving mix, its tests and the
toothOptimizer levels; the inputs are drawn from the seed alone.
"""
import math

import numpy as np
import torch

from quijibo_gb300 import lib
from quijibo_gb300.rootsets import Grid, RootSet

_CTX = None


def _ctx():
    """The one context a program keeps for its device."""
    global _CTX
    if _CTX is None:
        _CTX = lib.Context(0)
    return _CTX


class _Map:
    """A resident root set, freed with its owner."""

    def __init__(self, rs):
        self.handle = _ctx().upload(rs)

    def __del__(self):
        try:
            _CTX.free(self.handle)
        except Exception:
            pass


# ------------------------------------------------------------------- cases

def listed():
    return [
        # a serving request at the small end: the latency of one field call
        {"name": "field_small", "kind": "field", "x": 32, "y": 32, "z": 32, "nt": 12, "nb": 4,
         "exps": "12", "max_it": 20, "precision": "fp32refine", "rel_tol": 1e-6, "de": False,
         "lagrange": False, "rotated": False, "deep": False},
        # the headline workload: the precision form at 512^3, 16 / 8 roots.
        # "deep": maps whose inside settles far from the surface, as the
        # benchmark's do; the others are any maps that bound a shape
        {"name": "field_512", "kind": "field", "x": 512, "y": 512, "z": 512, "nt": 16, "nb": 8,
         "exps": "12", "max_it": 40, "precision": "fp32refine", "rel_tol": 1e-6, "de": False,
         "lagrange": False, "rotated": False, "deep": True},
        # an odd grid, rotated as the reference's viewers place it, root counts
        # of no particular size, with the distance estimate for a renderer;
        # the server's default of the band rule alone
        {"name": "field_odd_de", "kind": "field", "x": 203, "y": 171, "z": 139, "nt": 23, "nb": 11,
         "exps": "123", "max_it": 30, "precision": "fp32refine", "rel_tol": 0.0, "de": True,
         "lagrange": False, "rotated": True, "deep": False},
        # the large map (48 / 24 roots, 60 iterations): four slices' worth of
        # the 2200^3 grid, one step of a slab-streaming program
        {"name": "field_large_slab", "kind": "field", "x": 2200, "y": 2200, "z": 4, "nt": 48,
         "nb": 24, "exps": "12", "max_it": 60, "precision": "fp32refine", "rel_tol": 1e-6,
         "de": False, "lagrange": False, "rotated": False, "deep": True},
        # an optimized shape (its exponents are no integers) in the precision form
        {"name": "field_fitted", "kind": "field", "x": 128, "y": 128, "z": 128, "nt": 12, "nb": 6,
         "exps": "real", "max_it": 20, "precision": "fp32refine", "rel_tol": 0.0, "de": False,
         "lagrange": False, "rotated": False, "deep": False},
        # the same shape's field as the reference computes it: plain FP64
        {"name": "field_fp64", "kind": "field", "x": 64, "y": 64, "z": 64, "nt": 12, "nb": 6,
         "exps": "real", "max_it": 20, "precision": "fp64", "rel_tol": 0.0, "de": False,
         "lagrange": False, "rotated": False, "deep": False},
        # a mesh request: streaming marching cubes in the precision form
        {"name": "mesh_128", "kind": "mesh", "res": 128, "nt": 16, "nb": 8, "exps": "12",
         "max_it": 40, "precision": "fp32refine", "rel_tol": 1e-6, "deep": False},
        # bunnyMarchingCubes3D's run: the streaming mesher in plain FP64
        {"name": "mesh_fp64", "kind": "mesh", "res": 48, "nt": 12, "nb": 6, "exps": "real",
         "max_it": 20, "precision": "fp64", "rel_tol": 0.0, "deep": False},
        # marching cubes of a stored field (linear edges), a field larger than L2
        {"name": "mesh_stored", "kind": "stored", "x": 400, "y": 384, "z": 320},
        # toothOptimizer's objective at its finest and its coarsest level
        {"name": "objective_97", "kind": "objective", "res": 97, "target": 64, "nt": 12, "nb": 6},
        {"name": "objective_25", "kind": "objective", "res": 25, "target": 64, "nt": 12, "nb": 6},
        # one gradient of the fitting energy at the differentiation workload's size
        {"name": "energy_200k", "kind": "energy", "n": 200_000, "nt": 64, "nb": 16, "max_it": 30,
         "precision": "fp32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field", "field", "field", "field", "fp64", "mesh", "mesh", "stored",
                       "objective", "objective", "energy", "energy"])
    nt = _log_int(rng, 4, 48)
    nb = rng.choice([0, max(1, nt // 3), max(1, nt // 2)])
    if kind in ("field", "fp64"):
        fp64 = kind == "fp64"
        edge = _log_int(rng, 24, 72 if fp64 else 300)
        size = [max(8, int(edge * rng.uniform(0.7, 1.4))) for _ in range(3)]
        max_it = rng.randint(10, 30 if fp64 else 60)
        exps = rng.choice(["1", "12", "12", "123", "real"])
        if fp64 or exps == "real":
            nt, nb = min(nt, 16), min(nb, 8)
        rel_tol = rng.choice([0.0, 1e-6]) if exps != "real" and not fp64 else 0.0
        deep = not fp64 and exps != "real" and rng.random() < 0.6
        most = (2e8 if fp64 else 5e9 if exps == "real" else 1.5e10 if deep or rel_tol == 0.0
                else 1.2e9)
        while size[0] * size[1] * size[2] * (nt + nb) * max_it > most:
            size = [max(8, int(0.9 * s)) for s in size]
        return {"kind": "field", "x": size[0], "y": size[1], "z": size[2], "nt": nt, "nb": nb,
                "exps": exps, "max_it": max_it,
                "precision": "fp64" if fp64 else "fp32refine",
                "rel_tol": rel_tol, "deep": deep,
                "de": rng.random() < 0.25, "lagrange": nb > 0 and rng.random() < 0.15,
                "rotated": rng.random() < 0.3}
    if kind == "mesh":
        fp64 = rng.random() < 0.35
        res, max_it = _log_int(rng, 24, 56 if fp64 else 256), rng.randint(10, 20 if fp64 else 40)
        if fp64:
            nt, nb = min(nt, 12), min(nb, 6)
        deep = not fp64 and rng.random() < 0.6
        while res ** 3 * (nt + nb) * max_it > (5e7 if fp64 else 6e9 if deep else 1.5e9):
            res = int(0.9 * res)
        return {"kind": "mesh", "res": res, "nt": nt, "nb": nb,
                "exps": "real" if fp64 else rng.choice(["1", "12"]), "max_it": max_it,
                "precision": "fp64" if fp64 else "fp32refine",
                "rel_tol": 0.0 if fp64 else rng.choice([0.0, 1e-6]), "deep": deep}
    if kind == "stored":
        edge = _log_int(rng, 40, 380)
        return {"kind": "stored", "x": int(edge * rng.uniform(0.7, 1.3)),
                "y": int(edge * rng.uniform(0.7, 1.3)), "z": int(edge * rng.uniform(0.7, 1.3))}
    if kind == "objective":
        return {"kind": "objective", "res": _log_int(rng, 20, 100),
                "target": rng.choice([32, 48, 64]), "nt": min(nt, 24), "nb": max(1, min(nb, 12))}
    n = _log_int(rng, 5000, 200_000)
    return {"kind": "energy", "n": n, "nt": _log_int(rng, 8, 64), "nb": max(1, min(nb, 16)),
            "max_it": rng.randint(10, 30), "precision": "fp64" if n < 8000 else "fp32"}


# ------------------------------------------------------------------ inputs

def _np_mul(a, b):
    aw, ax, ay, az = np.moveaxis(a, -1, 0)
    bw, bx, by, bz = np.moveaxis(b, -1, 0)
    return np.stack([aw * bw - ax * bx - ay * by - az * bz, aw * bx + ax * bw + ay * bz - az * by,
                     aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw], -1)


def _np_product(f):
    """The ordered product over axis 1, pairwise."""
    while f.shape[1] > 1:
        k = f.shape[1] // 2
        f = np.concatenate([_np_mul(f[:, 0:2 * k:2], f[:, 1:2 * k:2]), f[:, 2 * k:]], 1)
    return f[:, 0]


def _has_shape(roots, powers, nt, scale, rng, depth):
    """Whether the map bounds a shape: of 64 points in [-1.2, 1.2]^3 some
    escape and some settle, on a limit that draws them in, below the escape
    radius and with a field of at least `depth` (0 is the surface)."""
    q = np.concatenate([rng.uniform(-1.2, 1.2, (64, 3)), np.zeros((64, 1))], 1)
    before = q
    for n in range(24):
        d = q[:, None] - roots[None]
        m, v = np.linalg.norm(d, axis=2), np.linalg.norm(d[..., 1:], axis=2)
        a, t = m ** powers, powers * np.arctan2(v, d[..., 0])
        f = np.concatenate([(a * np.cos(t))[..., None],
                            (a * np.sin(t) / np.maximum(v, 1e-300))[..., None] * d[..., 1:]], -1)
        nq = _np_product(f[:, :nt])
        if nt < len(roots):
            b = _np_product(f[:, nt:])
            nq = _np_mul(nq, b * [1, -1, -1, -1] / (b * b).sum(-1, keepdims=True))
        live = np.linalg.norm(q, axis=1) < 2.0
        before, q = q, np.where(live[:, None], nq * scale, q)
        if n % 2 == 0:
            two_back = before
    inside = np.linalg.norm(q, axis=1) < 2.0
    if not 8 <= inside.sum() <= 56:
        return False
    last = np.stack([before[inside], q[inside]])
    mag = np.linalg.norm(last, axis=2)
    moved = np.linalg.norm(q[inside] - two_back[inside], axis=1)
    return bool((mag < 1.8).all() and (abs(np.log(mag)) > depth).all() and (moved < 1e-6 * mag[1]).all())


def _rootset(rng, nt, nb, exps, depth=0.03):
    """Roots in [-1.2, 1.2]^4 with the conformal scale: exp(-median log|T/B|)
    over cell centres of [-1.5, 1.5]^3, which puts about half of them inside.
    Drawn again until the map bounds a shape, as a user's maps do."""
    a = (np.arange(16) + 0.5) / 16 * 3.0 - 1.5
    p = np.stack(np.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)
    p = np.concatenate([p, np.zeros((len(p), 1))], 1)
    sign = np.where(np.arange(nt + nb) < nt, 1.0, -1.0)
    for _ in range(200):
        roots = rng.uniform(-1.2, 1.2, (nt + nb, 4))
        powers = (rng.uniform(0.5, 2.0, nt + nb) if exps == "real"
                  else rng.choice([float(c) for c in exps], nt + nb))
        logs = np.log(np.linalg.norm(p[:, None, :] - roots[None], axis=2)) @ (sign * powers)
        scale = float(np.exp(-np.median(logs)))
        with np.errstate(all="ignore"):  # points that escaped early may overflow
            if _has_shape(roots, powers, nt, scale, rng, depth):
                break
    return RootSet(top_roots=roots[:nt].copy(), top_powers=powers[:nt].copy(),
                   bottom_roots=roots[nt:].copy(), bottom_powers=powers[nt:].copy(), scale=scale)


def _inputs(c, seed):
    """The host-side inputs of a case: everything but device buffers."""
    rng = np.random.RandomState(seed % (1 << 32))
    if c["kind"] == "field":
        rs = _rootset(rng, c["nt"], c["nb"], c["exps"], 4.2 if c["deep"] else 0.03)
        rot, slab = (1.0, 0.0, 0.0, 0.0), 0.0
        if c["rotated"]:
            v = rng.normal(size=4)
            rot, slab = tuple(float(t) for t in v / np.linalg.norm(v)), 0.05
        if c["x"] >= 2000:  # a slab of a cubic grid, somewhere in its middle half
            z = c["x"]
            z0 = int(rng.randint(z // 4, 3 * z // 4))
        else:
            z, z0 = c["z"], 0
        return rs, Grid((c["x"], c["y"], z), rot=rot, slice=slab), z0, z0 + c["z"]
    if c["kind"] == "mesh":
        depth = 4.2 if c["deep"] else 0.03
        return _rootset(rng, c["nt"], c["nb"], c["exps"], depth), Grid((c["res"],) * 3)
    if c["kind"] == "stored":
        return rng.uniform(-0.5, 0.5, (12, 3)), rng.uniform(0.12, 0.3, 12)
    if c["kind"] == "objective":
        # a fitting problem in the fractal's frame (radius 4): top roots inside
        # the target's spheres, bottom roots around it, the origin root first
        centres, radii = rng.uniform(-0.9, 0.9, (5, 3)), rng.uniform(0.5, 0.9, 5)
        pick = rng.randint(0, 5, c["nt"])
        top = np.zeros((c["nt"], 4))
        top[1:, :3] = (centres[pick] + 0.5 * radii[pick, None]
                       * rng.uniform(-1, 1, (c["nt"], 3)))[1:]
        bot = np.zeros((c["nb"], 4))
        d = rng.normal(size=(c["nb"], 3))
        bot[:, :3] = rng.uniform(1.6, 1.95, (c["nb"], 1)) * d / np.linalg.norm(d, axis=1)[:, None]
        rs = RootSet(top_roots=top, top_powers=rng.uniform(0.4, 2.2, c["nt"]), sigma_top=1.0,
                     bottom_roots=bot, bottom_powers=rng.uniform(0.4, 2.2, c["nb"]),
                     sigma_bottom=1.0)
        return rs, centres, radii
    rs = _rootset(rng, c["nt"], c["nb"], "1")
    xyz = rng.uniform(-1.0, 1.0, (c["n"], 3))
    centres, radii = rng.uniform(-0.45, 0.45, (4, 3)), rng.uniform(0.15, 0.45, 4)
    target = np.min(np.linalg.norm(xyz[:, None] - centres[None], axis=2) - radii[None], axis=1)
    return rs, xyz, target


def _spheres(res, lengths, centres, radii):
    """Signed distance to a union of spheres at the cell centres of a grid
    about the origin (on the GPU, x fastest)."""
    ax = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * (w / n) - 0.5 * w
          for n, w in zip(res, lengths)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    d = torch.full_like(x, 1e30)
    for c, r in zip(centres, radii):
        d = torch.minimum(d, ((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2).sqrt() - r)
    return d


def _objective_grids(c):
    return Grid((c["res"],) * 3, lengths=(4.0,) * 3), Grid((c["target"],) * 3, lengths=(4.0,) * 3)


def _precision(name):
    return {"fp64": lib.QJG_FP64, "fp32": lib.QJG_FP32, "fp32refine": lib.QJG_FP32_REFINE}[name]


def _iter(c, **kw):
    whole = c["exps"] != "real" and c["precision"] == "fp32refine"
    return _ctx().iter_params(c["max_it"], 2.0, precision=_precision(c["precision"]),
                              refine_pow=lib.QJG_REFINE_INT if whole else lib.QJG_REFINE_POW,
                              rel_tol=c["rel_tol"], **kw)


def prepare(case, seed):
    c, s = case, {"case": case}
    inp = _inputs(c, seed)
    if c["kind"] == "field":
        rs, s["grid"], s["z0"], s["z1"] = inp
        s["map"] = _Map(rs)
        s["iter"] = _iter(c, want_de=c["de"], lagrange=c["lagrange"])
        shape = (c["z"], c["y"], c["x"])
        s["field"] = torch.empty(shape, dtype=torch.float64, device="cuda")
        s["de"] = torch.empty(shape, dtype=torch.float32, device="cuda") if c["de"] else None
    elif c["kind"] == "mesh":
        rs, s["grid"] = inp
        s["map"], s["iter"] = _Map(rs), _iter(c)
        s["cap"] = 24 * c["res"] ** 2 + 4096
        _mesh_buffers(s)
    elif c["kind"] == "stored":
        res = (c["x"], c["y"], c["z"])
        s["grid"] = Grid(res, lengths=(2.0, 2.0, 2.0))
        s["field"] = -_spheres(res, (2.0, 2.0, 2.0), *inp)
        s["cap"] = 6 * max(res) ** 2 + 4096
        _mesh_buffers(s)
    elif c["kind"] == "objective":
        rs, centres, radii = inp
        ctx = _ctx()
        s["grid"], s["wgrid"] = _objective_grids(c)
        dist = _spheres(s["wgrid"].res, s["wgrid"].lengths, centres, radii)
        s["weights"] = torch.empty_like(dist)
        ctx.inverted_distance(s["wgrid"].res, dist.data_ptr(), True, s["weights"].data_ptr())
        h = ctx.upload(rs)
        _, _, rs.scale = ctx.conformal_radius(h, s["wgrid"], s["wgrid"], dist.data_ptr())
        ctx.free(h)
        s["map"], s["n_params"] = _Map(rs), 3 + c["nt"] + c["nb"]
        s["field"] = torch.empty((c["res"],) * 3, dtype=torch.float64, device="cuda")
        s["rs"] = rs
    else:
        rs, xyz, target = inp
        s["params"] = torch.from_numpy(lib.params_of(rs)).cuda()
        s["xyz"], s["target"] = torch.from_numpy(xyz).cuda(), torch.from_numpy(target).cuda()
        s["grad"] = torch.empty_like(s["params"])
    return s


def _mesh_buffers(s):
    s["verts"] = torch.zeros((s["cap"], 3), dtype=torch.float32, device="cuda")
    s["tris"] = torch.zeros((2 * s["cap"], 3), dtype=torch.int32, device="cuda")


def run(state):
    s, c, ctx = state, state["case"], _ctx()
    stream = torch.cuda.current_stream().cuda_stream
    if c["kind"] == "field":
        ctx.field(s["map"].handle, s["grid"], s["iter"], s["field"].data_ptr(),
                  d_de=s["de"].data_ptr() if c["de"] else None, z0=s["z0"], z1=s["z1"],
                  stream=stream)
        return [s["field"], s["de"]] if c["de"] else [s["field"]]
    if c["kind"] in ("mesh", "stored"):
        out = dict(d_verts32=s["verts"].data_ptr(), vert_cap=s["cap"], d_tris=s["tris"].data_ptr(),
                   tri_cap=2 * s["cap"], stream=stream)
        if c["kind"] == "mesh":
            _, st = ctx.mesh_stream(s["map"].handle, s["grid"], s["iter"], **out)
        else:
            _, st = ctx.mesh_field(None, s["grid"], None, s["field"].data_ptr(),
                                   lib.QJG_EDGE_LINEAR, **out)
        return [st["n_verts"], st["n_tris"], s["verts"], s["tris"]]
    if c["kind"] == "objective":
        score, grad, _ = ctx.tanh_score_grad(s["map"].handle, s["grid"], 1, s["wgrid"],
                                             s["weights"].data_ptr(), s["n_params"],
                                             d_field=s["field"].data_ptr(), stream=stream)
        return [score, grad, s["field"]]
    e = ctx.energy(s["params"].data_ptr(), c["nt"], c["nb"], c["n"], s["xyz"].data_ptr(),
                   s["target"].data_ptr(), c["max_it"], 2.0, precision=_precision(c["precision"]),
                   d_grad=s["grad"].data_ptr(), stream=stream)
    return [e, s["grad"]]


def work(case):
    """Bytes: inputs read and outputs written once.  Flops: about half of the
    points are inside and run to the cap in a plain escape loop; what no loop
    can leave out is the few applications until an orbit escapes or settles,
    taken as 6 of a map of about 45 operations a root."""
    c = case
    if c["kind"] == "stored":
        n = c["x"] * c["y"] * c["z"]
        return {"bytes": 8 * n + 24 * 6 * max(c["x"], c["y"], c["z"]) ** 2, "flops": n}
    roots = c["nt"] + c["nb"]
    if c["kind"] == "field":
        n = c["x"] * c["y"] * c["z"]
        return {"bytes": n * (12 if c["de"] else 8), "flops": 6 * 45 * roots * n}
    if c["kind"] == "mesh":
        n = c["res"] ** 3
        return {"bytes": 48 * c["res"] ** 2, "flops": 6 * 45 * roots * n}
    if c["kind"] == "objective":
        n = c["res"] ** 3
        return {"bytes": 8 * (n + c["target"] ** 3), "flops": 60 * roots * n}
    return {"bytes": 32 * c["n"], "flops": 6 * 66 * roots * c["n"]}


# ------------------------------------------------------- plain 64-bit values

def _mul(a, b):
    aw, ax, ay, az = a.unbind(-1)
    bw, bx, by, bz = b.unbind(-1)
    return torch.stack([aw * bw - ax * bx - ay * by - az * bz,
                        aw * bx + ax * bw + ay * bz - az * by,
                        aw * by - ax * bz + ay * bw + az * bx,
                        aw * bz + ax * by - ay * bx + az * bw], -1)


def _conj(a):
    return a * torch.tensor([1.0, -1.0, -1.0, -1.0], dtype=a.dtype, device=a.device)


def _pow(d, e):
    """d^e in polar form; e a number."""
    if e in (1.0, 2.0, 3.0):
        return d if e == 1.0 else _mul(d, d) if e == 2.0 else _mul(_mul(d, d), d)
    v = d[..., 1:].norm(dim=-1)
    t = e * torch.atan2(v, d[..., 0])
    a = d.norm(dim=-1) ** e
    return torch.cat([(a * t.cos())[..., None],
                      (a * t.sin() / v.clamp_min(1e-300))[..., None] * d[..., 1:]], -1)


def _escape(q, rs, scale, max_it, lagrange):
    """log|q_N| and the distance estimate of the escape loop from points q."""
    roots = torch.tensor(np.concatenate([rs.top_roots, rs.bottom_roots]), device=q.device)
    exps = [float(e) for e in rs.top_powers] + [float(e) for e in rs.bottom_powers]
    nt, nb = rs.n_top, rs.n_bottom
    n = len(q)
    mag = q.norm(dim=-1)
    dlog = torch.zeros(n, dtype=torch.float64, device=q.device)
    live = torch.nonzero(mag < 2.0)[:, 0]
    for _ in range(max_it):
        if not len(live):
            break
        p = q[live]
        g = torch.zeros_like(p)
        sides = [None, None]
        lag = None
        order = list(range(nt + nb))
        if lagrange:
            order = [i for k in range(max(nt, nb)) for i in ((k,) if k < nt else ()) +
                     ((nt + k,) if k < nb else ())]
        for i in order:
            d = p - roots[i]
            top = i < nt
            g += (exps[i] if top else -exps[i]) * d / (d * d).sum(-1, keepdim=True)
            t = _pow(d, exps[i])
            if lagrange:
                f = t if top else _conj(t) / (t * t).sum(-1, keepdim=True)
                lag = f if lag is None else _mul(lag, f)
            else:
                k = 0 if top else 1
                sides[k] = t if sides[k] is None else _mul(sides[k], t)
        if lagrange:
            p = lag
        elif nb:
            b = sides[1]
            p = _mul(sides[0], _conj(b) / (b * b).sum(-1, keepdim=True))
        else:
            p = sides[0]
        p = p * scale
        m = p.norm(dim=-1)
        dlog[live] += g.norm(dim=-1).log() + m.log()
        q[live], mag[live] = p, m
        live = live[(m < 2.0) & (m >= 10 * 2.0 ** -126)]
    f = mag.log()
    return f, torch.sign(f) * (f.abs().log() + f - dlog).exp()


def _rotation(r):
    w, x, y, z = r
    return torch.tensor([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                         [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                         [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]],
                        dtype=torch.float64, device="cuda")


def _centres(n, length):
    """Cell centres along one axis about 0, rounded as FIELD_3D::cellCenter:
    the sign of a centre next to 0 picks the side of the power's branch cut."""
    dx = length / n
    return (-0.5 * length + torch.arange(n, device="cuda", dtype=torch.float64) * dx) + dx * 0.5


def _exact_field(c, inp):
    n = c["x"] * c["y"] * c["z"]
    cost = 20 if c["exps"] == "real" else 4
    if n * c["max_it"] * (c["nt"] + c["nb"]) * cost > 2e11:
        return None
    rs, g, z0, _ = inp
    axes = [_centres(k, w) for k, w in zip(g.res, g.lengths)]
    rot = _rotation(g.rot)
    field = torch.empty(n, dtype=torch.float64, device="cuda")
    de = torch.empty(n, dtype=torch.float64, device="cuda")
    step = 1 << 21
    for a in range(0, n, step):
        i = torch.arange(a, min(n, a + step), device="cuda")
        p = torch.stack([axes[0][i % c["x"]], axes[1][(i // c["x"]) % c["y"]],
                         axes[2][z0 + i // (c["x"] * c["y"])]], -1) @ rot.T
        q = torch.cat([p, torch.full((len(i), 1), g.slice, dtype=torch.float64, device="cuda")], 1)
        field[a:a + step], de[a:a + step] = _escape(q, rs, rs.scale, c["max_it"], c["lagrange"])
    shape = (c["z"], c["y"], c["x"])
    # the distance estimate is a float32 output: beyond its range it is infinite
    return [field.reshape(shape)] + ([de.float().double().reshape(shape)] if c["de"] else [])


def _trilinear(w, grid, p):
    """Cell-centred lookup; the fractions are single precision, as FIELD_3D's."""
    n = torch.tensor(grid.res, device="cuda")
    length = torch.tensor(grid.lengths, dtype=torch.float64, device="cuda")
    t = (p - (-0.5 * length + 0.5 * length / n)) * (n / length)
    i0 = t.trunc().long()
    i1 = torch.minimum((i0 + 1).clamp_min(0), n - 1)
    i0 = torch.minimum(i0.clamp_min(0), n - 1)
    f1 = (t - i0).float()
    f0 = (1.0 - f1).double()
    f1 = f1.double()
    out = 0.0
    for a, fx in ((i0, f0), (i1, f1)):
        for b, fy in ((i0, f0), (i1, f1)):
            for d, fz in ((i0, f0), (i1, f1)):
                out = out + fx[:, 0] * fy[:, 1] * fz[:, 2] * w[d[:, 2], b[:, 1], a[:, 0]]
    return out


def _exact_objective(c, seed):
    """Score, gradient and field of one map application (the bottom exponents'
    terms by the reference's own formula, T / (-left middle right))."""
    s = prepare(c, seed)  # the weights and the scale are inputs of the call
    rs, grid = s["rs"], s["grid"]
    nt, nb, alpha = c["nt"], c["nb"], 10.0
    k = _centres(c["res"], 4.0)
    z, y, x = torch.meshgrid(k, k, k, indexing="ij")
    p = torch.stack([x, y, z], -1).reshape(-1, 3)
    w = _trilinear(s["weights"], s["wgrid"], p)
    q = torch.cat([p, torch.zeros(len(p), 1, dtype=torch.float64, device="cuda")], 1)
    roots = torch.tensor(np.concatenate([rs.top_roots, rs.bottom_roots]), device="cuda")
    exps = [float(e) for e in rs.top_powers] + [float(e) for e in rs.bottom_powers]
    base = [q - r for r in roots]
    fac = [_pow(d, e) for d, e in zip(base, exps)]

    def qlog(d):
        v = d[:, 1:].norm(dim=-1)
        ang = torch.atan2(v, d[:, 0]) / v.clamp_min(1e-300)
        return torch.cat([d.norm(dim=-1).log()[:, None], ang[:, None] * d[:, 1:]], -1)

    def around(lo, hi):
        one = torch.zeros_like(q)
        one[:, 0] = 1.0
        left, right = [one], [one]
        for i in range(lo, hi):
            left.append(_mul(left[-1], fac[i]))
        for i in range(hi - 1, lo - 1, -1):
            right.append(_mul(fac[i], right[-1]))
        return left, right[::-1]

    tl, tr = around(0, nt)
    bl, br = around(nt, nt + nb)
    T, B = tl[-1], bl[-1]
    Bi = _conj(B) / (B * B).sum(-1, keepdim=True)
    R = _mul(T, Bi)
    # a cell at the origin is not iterated: field 0, no root's terms
    moved = q.norm(dim=-1) >= 1e-8
    F = torch.where(moved, R.norm(dim=-1).log() + math.log(rs.scale), 0.0)
    th = torch.tanh(alpha * F)
    dS = -alpha * w * (1 - th * th)
    grad = torch.zeros(3 + nt + nb, dtype=torch.float64, device="cuda")
    grad[0] = dS.sum()
    RR = 1.0 / (R * R).sum(-1)
    for i in range(nt):
        dT = _mul(_mul(tl[i], _mul(fac[i], qlog(base[i]))), tr[i + 1])
        t = (dS * RR * (R * _mul(dT, Bi)).sum(-1))[moved].sum()
        grad[1 + nb + i] = t
        grad[1 + nb + nt] += rs.top_powers[i] * t
    for j in range(nb):
        lg = qlog(base[nt + j])
        li = _conj(lg) / (lg * lg).sum(-1, keepdim=True)
        dB = _mul(_mul(-bl[j], _mul(fac[nt + j], li)), br[j + 1])
        t = (dS * RR * (R * _mul(T, _conj(dB) / (dB * dB).sum(-1, keepdim=True))).sum(-1))[moved].sum()
        grad[1 + j] = t
        grad[2 + nb + nt] += rs.bottom_powers[j] * t
    return [float((-th * w).sum()), grad.cpu().numpy(), F.reshape(grid.res[::-1])]


def _exact_energy(c, inp):
    if c["n"] * c["max_it"] * (c["nt"] + c["nb"]) > 6e8:
        return None
    rs, xyz, target = inp
    nt, nb = c["nt"], c["nb"]
    nr = nt + nb
    params = torch.from_numpy(lib.params_of(rs)).cuda().requires_grad_()
    sign = torch.where(torch.arange(nr, device="cuda") < nt, 1.0, -1.0).double()
    energy, step = 0.0, 20000
    for a in range(0, c["n"], step):
        p = torch.from_numpy(xyz[a:a + step]).cuda()
        t = torch.from_numpy(target[a:a + step]).cuda()
        roots, exps, scale = params[:4 * nr].reshape(nr, 4), params[4 * nr:5 * nr], params[-1].exp()
        q = torch.cat([p, torch.zeros(len(p), 1, dtype=torch.float64, device="cuda")], 1)
        dlog = torch.zeros(len(p), dtype=torch.float64, device="cuda")
        live = torch.nonzero(q.norm(dim=-1) < 2.0)[:, 0]
        for _ in range(c["max_it"]):
            if not len(live):
                break
            d = q[live][:, None, :] - roots[None]
            g = (sign * exps)[None, :, None] * d / (d * d).sum(-1, keepdim=True)
            v = d[..., 1:].norm(dim=-1)
            ang = exps * torch.atan2(v, d[..., 0])
            amp = (exps * d.norm(dim=-1).log()).exp()
            f = torch.cat([(amp * ang.cos())[..., None],
                           (amp * ang.sin() / v)[..., None] * d[..., 1:]], -1)

            def product(f):
                while f.shape[1] > 1:
                    k = f.shape[1] // 2
                    h = _mul(f[:, 0:2 * k:2], f[:, 1:2 * k:2])
                    f = torch.cat([h, f[:, 2 * k:]], 1)
                return f[:, 0]

            T, B = product(f[:, :nt]), product(f[:, nt:])
            nq = scale * _mul(T, _conj(B) / (B * B).sum(-1, keepdim=True))
            m = nq.norm(dim=-1)
            dlog = dlog.index_add(0, live, g.sum(1).norm(dim=-1).log() + m.log())
            q = q.index_copy(0, live, nq)
            live = live[((m < 2.0) & (m >= 10 * 2.0 ** -126)).detach()]
        m = q.norm(dim=-1)
        ld = m.log().abs().log() + m.log() - dlog
        sat = ld > math.log(20.0)
        val = torch.sign(m.log()) * torch.where(sat, torch.ones_like(ld),
                                                torch.tanh(ld.clamp_max(3.0).exp()))
        e = ((val - t) ** 2).sum()
        e.backward()
        energy += float(e.detach())
    return [energy, params.grad]


def exact(case, seed):
    """What run() returns, in 64 bits by plain torch; meshes have no such
    value (vertex positions come from a bisection to a fixed depth)."""
    if case["kind"] == "field":
        return _exact_field(case, _inputs(case, seed))
    if case["kind"] == "objective":
        return _exact_objective(case, seed)
    if case["kind"] == "energy":
        return _exact_energy(case, _inputs(case, seed))
    return None
