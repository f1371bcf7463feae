"""Orbits that come back to an iterate bit for bit are finished from their
last period; the one-voxel kernel (field32_kernel) applies the map to every
orbit's end and gives the value each voxel must have."""
import numpy as np
import pytest

from quijibo_gb300 import lib
from quijibo_gb300.rootsets import Grid, RootSet

pytestmark = pytest.mark.gpu


def settling_map(seed, nt, nb):
    """A map whose inside settles (periods 1 to 6 among these seeds)."""
    rng = np.random.RandomState(seed)
    roots = rng.uniform(-1.2, 1.2, (nt + nb, 4))
    powers = rng.choice([1.0, 2.0], nt + nb)
    p = np.concatenate([rng.uniform(-1.5, 1.5, (4000, 3)), np.zeros((4000, 1))], 1)
    sign = np.where(np.arange(nt + nb) < nt, 1.0, -1.0)
    logs = np.log(np.linalg.norm(p[:, None] - roots[None], axis=2)) @ (sign * powers)
    return RootSet(top_roots=roots[:nt], top_powers=powers[:nt], bottom_roots=roots[nt:],
                   bottom_powers=powers[nt:], scale=float(np.exp(-np.median(logs))))


# iteration caps at the edges of the marks (2 apart below 12, 6 above) and past them
@pytest.mark.parametrize("max_it", [1, 2, 3, 12, 13, 19, 40, 97])
@pytest.mark.parametrize("seed,nt,nb", [(0, 16, 8), (1, 5, 2), (2, 16, 8), (3, 5, 2), (4, 8, 0)])
@pytest.mark.parametrize("precision,de", [(lib.QJG_FP32, True), (lib.QJG_FP32, False),
                                          (lib.QJG_FP32_REFINE, True)])
def test_periodic_orbits_equal_the_full_loop(ctx, seed, nt, nb, max_it, precision, de):
    g = Grid((35, 22, 9))
    h = ctx.upload(settling_map(seed, nt, nb))
    it = ctx.iter_params(max_it, 2.0, precision=precision, want_de=de, rel_tol=1e-6,
                         refine_pow=lib.QJG_REFINE_INT)
    out = []
    try:
        for pairs in (True, False):
            lib.set_field32_pairs(pairs)
            out.append(ctx.field_host(h, g, it, de=de))
    finally:
        lib.set_field32_pairs(True)
        ctx.free(h)
    (fa, da, sa), (fb, db, sb) = out
    assert np.array_equal(fa.view(np.uint64), fb.view(np.uint64))
    if de:
        assert np.array_equal(da.view(np.uint32), db.view(np.uint32))
    for k in ("voxel_iters", "refined", "nonfinite", "rerun", "rerun_iters"):
        assert sa[k] == sb[k], k


@pytest.mark.parametrize("max_it", [2, 13, 40])
@pytest.mark.parametrize("seed,nt,nb", [(0, 16, 8), (1, 5, 2), (2, 16, 8), (3, 5, 2)])
def test_fp64_periodic_orbits_equal_the_oracle(ctx, oracle, seed, nt, nb, max_it):
    """With correctly rounded functions the FP64 form has the oracle's bits,
    and its orbit lengths, whether or not its orbits end early; so has its
    field with the distance estimate, whose loop ends early less often."""
    rs, g = settling_map(seed, nt, nb), Grid((13, 10, 6))
    oracle.set_libm(True)
    try:
        o = oracle.field(rs, g, max_it, 2.0, iters=True)
    finally:
        oracle.set_libm(False)
    h = ctx.upload(rs)
    for de in (False, True):
        it = ctx.iter_params(max_it, 2.0, libm=lib.QJG_LIBM_CR, want_de=de)
        f, _, st = ctx.field_host(h, g, it, de=de)
        assert np.array_equal(f.view(np.uint64), o["field"].view(np.uint64))
        assert st["voxel_iters"] == int(o["iters"].sum())
    ctx.free(h)


@pytest.mark.parametrize("refine_pow", [lib.QJG_REFINE_INT, lib.QJG_REFINE_POW])
@pytest.mark.parametrize("seed,nt,nb", [(1, 5, 2), (2, 16, 8)])
def test_refined_field_is_the_same_with_and_without_distances(ctx, seed, nt, nb, refine_pow):
    g = Grid((33, 30, 17))
    h = ctx.upload(settling_map(seed, nt, nb))
    out = [ctx.field_host(h, g, ctx.iter_params(40, 2.0, precision=lib.QJG_FP32_REFINE, rel_tol=1e-6,
                                                refine_pow=refine_pow, want_de=de), de=de)
           for de in (False, True)]
    ctx.free(h)
    assert np.array_equal(out[0][0].view(np.uint64), out[1][0].view(np.uint64))
    assert out[0][2]["refined_iters"] == out[1][2]["refined_iters"] > 0
