"""Voxels that the double-float re-run cannot bring within rel_tol go to FP64
directly.  The tracked bound is the one the voxels are kept by, so every voxel
lies within rel_tol |f| of FP64 (and 1e-12 for FP64's own rounding), on either
side of the tolerance's rule."""
import numpy as np
import pytest

from quijibo_gb300 import lib
from quijibo_gb300.rootsets import Grid
from test_orbit_period_gpu import settling_map

pytestmark = pytest.mark.gpu


# |f| + 0.2 = ERR_STEP / rel_tol at |f| = 3.8e3 (all hopeless), 3.6, 0.18 and nowhere
@pytest.mark.parametrize("rel_tol", [1e-9, 1e-6, 1e-5, 1e-4])
@pytest.mark.parametrize("seed,nt,nb", [(0, 16, 8), (3, 5, 2), (4, 8, 0)])
@pytest.mark.parametrize("max_it", [2, 3, 20])
def test_kept_voxels_lie_within_the_tolerance(ctx, seed, nt, nb, max_it, rel_tol):
    g = Grid((35, 22, 9))
    h = ctx.upload(settling_map(seed, nt, nb))
    a = ctx.field_host(h, g, ctx.iter_params(max_it, 2.0, precision=lib.QJG_FP32_REFINE,
                                             rel_tol=rel_tol, refine_pow=lib.QJG_REFINE_INT))
    b = ctx.field_host(h, g, ctx.iter_params(max_it, 2.0, precision=lib.QJG_FP32_REFINE,
                                             rel_tol=1e-30, refine_pow=lib.QJG_REFINE_INT))
    ctx.free(h)
    fa, exact = a[0], b[0]
    assert b[2]["refined"] + b[2]["rerun"] >= fa.size  # every voxel left FP32
    assert (np.abs(fa - exact) <= rel_tol * np.abs(exact) + 1e-12).all()
