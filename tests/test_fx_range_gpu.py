"""Maps whose products leave the fixed-point products' range (2^500): the FP64
chain is taken there, with the oracle's overflow.  Finite values: twelve powers
of 2^60, each off by 41 2^-53 through its logarithm, make log|q| uncertain by
6e-14 an application; 1e-11 is allowed."""
import numpy as np
import pytest

from quijibo_gb300 import lib
from quijibo_gb300.rootsets import Grid, RootSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [-60, 30, 60])  # roots about 2^far from the grid's cells
@pytest.mark.parametrize("form,nt,nb", [("pow", 12, 0), ("pow", 12, 12), ("pow", 8, 12), ("int", 12, 0)])
def test_products_beyond_the_range(ctx, oracle, form, nt, nb, far):
    rng = np.random.RandomState(abs(far))
    d = rng.uniform(0.5, 1, (nt + nb, 4)) * rng.choice([-1, 1], (nt + nb, 4)) * 2.0 ** far
    g = Grid((3, 2, 2), lengths=(2.0 ** -58,) * 3 if far < 0 else (3.0, 2.0, 2.0))
    powers = np.ones(nt + nb)
    rs = RootSet(top_roots=d[:nt], top_powers=powers[:nt], bottom_roots=d[nt:], bottom_powers=powers[nt:],
                 scale=2.0 ** (-far * (nt - nb)))
    o = oracle.field(rs, g, 2, 20.0)["field"]
    h = ctx.upload(rs)
    kw = dict(precision=lib.QJG_FP64) if form == "pow" else \
        dict(precision=lib.QJG_FP32_REFINE, refine_pow=lib.QJG_REFINE_INT, rel_tol=1e-30)
    f = ctx.field_host(h, g, ctx.iter_params(2, 20.0, **kw))[0]
    ctx.free(h)
    finite = np.isfinite(o)
    assert np.array_equal(finite, np.isfinite(f)) and np.array_equal(np.isnan(o), np.isnan(f))
    assert (np.abs(f[finite] - o[finite]) <= 1e-11 + 1e-11 * np.abs(o[finite])).all()
