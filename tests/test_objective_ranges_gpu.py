"""The objective pass at the edges of its voxel ranges (one warp per range of
32 or 128 voxels) and for each split between dense and sparse steps."""
import numpy as np
import pytest

from quijibo_gb300.rootsets import Grid, cell_centers, conformal_scale, draw_rootset

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# one voxel, one short step, one step and a voxel, ragged, the last grid of
# 32-voxel ranges on 152 SMs (155,648 voxels) and the first of 128-voxel ones
@pytest.mark.parametrize("res", [(1, 1, 1), (7, 4, 1), (33, 1, 1), (19, 13, 11), (64, 64, 38), (61, 57, 45)])
@pytest.mark.parametrize("alpha", [10.0, 0.5])  # mostly saturated (queued voxels); all in the band
@pytest.mark.parametrize("nt,nb", [(12, 6), (3, 1), (1, 2)])
def test_objective_matches_the_oracle(ctx, oracle, res, alpha, nt, nb):
    rng = np.random.RandomState(nt)
    rs = draw_rootset(7, nt, nb, -1.2, 1.2)
    rs.top_powers, rs.bottom_powers = rng.uniform(0.4, 2.2, nt), rng.uniform(0.4, 2.2, nb)
    rs.sigma_top, rs.sigma_bottom = 0.97, 1.03
    g, wg = Grid(res), Grid((9, 8, 7), lengths=(3.1, 3.1, 3.1))
    rs.scale = conformal_scale(rs, Grid((16, 16, 16)))
    c = cell_centers(wg)
    wts = np.cos(c[:, 0] + 2 * c[:, 1])
    sc0, gr0, f0 = oracle.tanh_score_grad(rs, g, wg, wts, 1, alpha=alpha)
    h = ctx.upload(rs)
    w = torch.from_numpy(wts).cuda()
    f = torch.empty(g.n_voxels, dtype=torch.float64, device="cuda")
    sc, gr, _ = ctx.tanh_score_grad(h, g, 1, wg, w.data_ptr(), len(gr0), alpha=alpha, d_field=f.data_ptr())
    ctx.free(h)
    # sums of either sign: their rounding is that of the terms' sizes, at most
    # the weights' sum for the score
    scale = np.abs(wts).max() * g.n_voxels
    assert abs(sc - sc0) <= 1e-12 * scale
    np.testing.assert_allclose(gr, gr0, rtol=1e-9, atol=1e-10 * max(1e-300, np.abs(gr0).max()))
    rel = np.abs(f.cpu().numpy() - f0.ravel()) / np.maximum(np.abs(f0.ravel()), 1e-3)
    assert np.max(rel) <= 1e-11
