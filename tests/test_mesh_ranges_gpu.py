"""The classification's plane ranges and the emit pass's unit blocks: a mesh
does not depend on the slab depth, whose ranges change with it (one range
below 16 planes, ranges of 8 planes and more above)."""
import numpy as np
import pytest
import torch

from quijibo_gb300 import lib
from quijibo_gb300.rootsets import Grid

pytestmark = pytest.mark.gpu


def mesh(ctx, g, f, slab):
    cap = 6 * g.n_voxels
    v = torch.zeros(3 * cap, dtype=torch.float64, device="cuda")
    t = torch.zeros(3 * cap, dtype=torch.int32, device="cuda")
    _, st = ctx.mesh_field(None, g, None, f.data_ptr(), lib.QJG_EDGE_LINEAR, slab_nz=slab,
                           d_verts64=v.data_ptr(), vert_cap=cap, d_tris=t.data_ptr(), tri_cap=cap)
    torch.cuda.synchronize()
    return v[:3 * st["n_verts"]].cpu().numpy(), t[:3 * st["n_tris"]].cpu().numpy()


# rows of 16-byte aligned pairs (cp.async form) and not; one and several
# segments of 64 voxels; last ranges of one plane
@pytest.mark.parametrize("res", [(20, 9, 70), (21, 9, 66), (130, 6, 33), (67, 5, 18), (64, 4, 17), (2, 2, 2)])
@pytest.mark.parametrize("dense", [True, False])  # random signs; a few flat sheets
def test_mesh_is_the_same_for_every_slab_depth(ctx, oracle, res, dense):
    rng = np.random.RandomState(res[0])
    x, y, z = np.meshgrid(*(np.arange(n) for n in res), indexing="ij")
    f = rng.normal(size=res) if dense else np.sin(0.31 * z + 0.05 * x) * 0.8 + 0.01 * y
    f = torch.from_numpy(np.ascontiguousarray(f.transpose(2, 1, 0))).cuda()
    g = Grid(res)
    v0, t0 = mesh(ctx, g, f, 3)
    assert len(t0) > 0 or not dense
    for slab in (1, 7, 8, 15, 16, 17, 24, 64, 200):
        v, t = mesh(ctx, g, f, slab)
        assert np.array_equal(t, t0) and np.array_equal(v.view(np.uint64), v0.view(np.uint64)), slab


def test_nearly_coincident_vertices_reach_the_exact_length(ctx):
    """Corners a few units above and below 0 put vertices next to grid points:
    edges shorter than 1e-7 beside edges just above it."""
    rng = np.random.RandomState(1)
    res = (24, 24, 24)
    f = rng.choice([-1.0, 1.0], res) * 10.0 ** rng.uniform(-9, 0, res)
    g = Grid(res, lengths=(1.0, 1.0, 1.0))
    t = torch.from_numpy(f).cuda()
    cap = 6 * g.n_voxels
    v = torch.zeros(3 * cap, dtype=torch.float64, device="cuda")
    tr = torch.zeros(3 * cap, dtype=torch.int32, device="cuda")
    _, st = ctx.mesh_field(None, g, None, t.data_ptr(), lib.QJG_EDGE_LINEAR, d_verts64=v.data_ptr(),
                           vert_cap=cap, d_tris=tr.data_ptr(), tri_cap=cap)
    torch.cuda.synchronize()
    assert st["n_degenerate"] > 0
    p = v[:3 * st["n_verts"]].cpu().numpy().reshape(-1, 3)
    k = tr[:3 * st["n_tris"]].cpu().numpy().reshape(-1, 3)
    for a, b in ((0, 1), (0, 2), (1, 2)):
        assert np.linalg.norm(p[k[:, a]] - p[k[:, b]], axis=1).min() >= 1e-7
