"""The fitting energy on orbits that settle: the forward pass ends them early
and fills the adjoint's kept orbit from the last period."""
import numpy as np
import pytest
import torch

from quijibo_gb300 import lib
from test_orbit_period_gpu import settling_map

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", torch.float64)


def _samples(n, seed):
    rng = np.random.RandomState(seed)
    return rng.uniform(-1.2, 1.2, (n, 3)), rng.uniform(-0.3, 0.5, n)


# caps before, at the edges of and past the marks; periods 1, 2 and 6 among the maps
@pytest.mark.parametrize("max_it", [1, 2, 12, 13, 30, 97])
@pytest.mark.parametrize("seed,nt,nb", [(0, 16, 8), (1, 5, 2), (2, 16, 8), (4, 8, 0)])
def test_settled_energy_matches_the_oracle(ctx, oracle, seed, nt, nb, max_it):
    rs = settling_map(seed, nt, nb)
    xyz, t = _samples(700, seed)
    P, X, T = _dev(lib.params_of(rs)), _dev(xyz), _dev(t)
    args = (P.data_ptr(), nt, nb, len(t), X.data_ptr(), T.data_ptr(), max_it, 2.0)
    eo = oracle.sqerr_energy(rs, xyz, t, max_it, 2.0)
    assert abs(ctx.energy(*args, precision=lib.QJG_FP64) - eo) <= 1e-9 * abs(eo)
    assert abs(ctx.energy(*args, precision=lib.QJG_FP32) - eo) <= 1e-4 * abs(eo)


def _settled_sample(ctx, seed, nt, nb, max_it):
    """A map of the seed and one sample whose orbit runs to the cap."""
    rs = settling_map(seed, nt, nb)
    xyz, _ = _samples(3000, seed)
    iters = torch.empty(3000, dtype=torch.int32, device="cuda")
    P, X, T = _dev(lib.params_of(rs)), _dev(xyz), _dev(np.zeros(3000))
    ctx.energy(P.data_ptr(), nt, nb, 3000, X.data_ptr(), T.data_ptr(), max_it, 2.0,
               precision=lib.QJG_FP64, d_iters=iters.data_ptr())
    X = X[iters == max_it][:1].contiguous()
    assert len(X) == 1

    def energy(p, precision=lib.QJG_FP64, grad=None):
        return ctx.energy(p.data_ptr(), nt, nb, 1, X.data_ptr(), T.data_ptr(), max_it, 2.0,
                          precision=precision, d_sat=0.0,
                          d_grad=grad.data_ptr() if grad is not None else 0)
    return P, energy


@pytest.mark.parametrize("seed,nt,nb", [(1, 5, 2), (3, 5, 2)])
def test_gradient_of_settled_samples(ctx, seed, nt, nb):
    """d_sat = 0 gives the settled samples a gradient (E = d^2), so the adjoint
    runs back over the steps that the forward pass left out.  Central
    difference of the FP64 energy along the gradient with h = 1e-7: its
    truncation (h |d log E|)^2 and its rounding 1e-13 / (h |d log E|) stay
    under 1e-4 for |d log E| between 1e-2 and 1e5."""
    P, energy = _settled_sample(ctx, seed, nt, nb, 48)
    g = torch.empty_like(P)
    e = energy(P, lib.QJG_FP64, g)
    assert np.isfinite(e) and bool(torch.isfinite(g).all()) and float(g.norm()) > 0
    u, h = g / g.norm(), 1e-7
    fd = (energy(P + h * u) - energy(P - h * u)) / (2 * h)
    assert abs(float(g.norm()) - fd) <= 1e-4 * abs(fd)


# 48 steps leave the FP32 range here (d^2 = 1e35, its gradient 1e38 and more)
@pytest.mark.parametrize("max_it", [12, 24, 30])
@pytest.mark.parametrize("seed,nt,nb", [(0, 16, 8), (1, 5, 2), (3, 5, 2)])
def test_fp32_gradient_of_settled_samples(ctx, seed, nt, nb, max_it):
    """The FP32 adjoint against the FP64 one on such a sample: FP32 carries
    the direction of 30 contracting steps to 1e-2."""
    P, energy = _settled_sample(ctx, seed, nt, nb, max_it)
    g64, g32 = torch.empty_like(P), torch.empty_like(P)
    e64 = energy(P, lib.QJG_FP64, g64)
    if not e64 < 1e30:
        pytest.skip("d^2 = %.1e is beyond the FP32 adjoint's range" % e64)
    energy(P, lib.QJG_FP32, g32)
    assert float((g32 - g64).norm()) <= 1e-2 * float(g64.norm())
