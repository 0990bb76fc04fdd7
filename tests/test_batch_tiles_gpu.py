"""A case of a batch stepped by itself after the batch's line tiles have changed: the layout of
the on-chip Poisson sweeps follows the tile, and the words that its blocks exchange start
afresh.  The same bits as a batch that had the tiles from the beginning and as a
context of its own on the per-colour kernels."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import STATE, case_params, make_case, make_gpu

pytestmark = pytest.mark.gpu

# tiles (radial warps, elements, circumferential warps, elements) before and after
TILES = [((1, 1, 1, 1), (4, 1, 4, 1)),      # four warps a line: no two-sweep form
         ((4, 1, 4, 1), (1, 1, 1, 1)),
         ((1, 1, 1, 1), (2, 6, 1, 2)),
         ((2, 1, 2, 1), (1, 12, 4, 4))]      # long chunks: more shared memory than any tile before


def _batch(cases, precision, tiles, **kw):
    b = capi.Batch([case_params(c, precision, refine_sweeps=8, **kw) for c in cases])
    for ctx, c in zip(b.cases, cases):
        ctx.set_grid(c["g"].xg, c["g"].yg)
    b.set_tiles(tiles)
    for ctx, c in zip(b.cases, cases):
        ctx.init(c["du"], c["dv"])
    return b


@pytest.mark.parametrize("precision", [capi.MIXED, capi.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("before,after", TILES)
def test_case_steps_by_itself_after_a_change_of_tiles(before, after, precision):
    cases = [make_case(n_theta=24, n_r=17, skew=0.3, vel_rot=0.2, nswpp=32, resimax=0.0),
             make_case(n_theta=32, n_r=24, seed=2, nswpp=32, resimax=0.0)]
    b, fresh = _batch(cases, precision, before), _batch(cases, precision, after)
    for c in b.cases:
        c.step(2)            # graphs exist, blocks have counted sweeps
    b.set_tiles(after)
    t = dict(tile_r_warps=after[0], tile_r_m=after[1], tile_t_warps=after[2], tile_t_m=after[3])
    for c, f, case in zip(b.cases, fresh.cases, cases):
        c.init(case["du"], case["dv"])
        one = make_gpu(case, precision, refine_sweeps=8, poisson_resident=0, **t)
        for _ in range(3):
            x, y, z = c.step(1), f.step(1), one.step(1)
            for key in ("cd", "cl", "sweeps", "resid"):
                assert x[key] == y[key] == z[key], key
        for nm in STATE:
            assert np.array_equal(c.get(nm), f.get(nm)) and np.array_equal(c.get(nm), one.get(nm)), nm


def test_a_layout_that_the_new_tile_cannot_hold_is_given_up():
    """resident_depth 2 asks for two sweeps per exchange, which four warps a line do not have: the
    change of tiles is accepted and the case steps without it."""
    case = make_case(n_theta=24, n_r=17, nswpp=32, resimax=0.0)
    b = _batch([case], capi.MIXED, (1, 1, 1, 1), resident_depth=2)
    b.cases[0].step(1)
    b.set_tiles((4, 1, 4, 1))
    assert b.cases[0].resident_info()["sweeps_per_exchange"] == 1
    b.cases[0].init(case["du"], case["dv"])
    one = make_gpu(case, capi.MIXED, refine_sweeps=8, poisson_resident=0, tile_r_warps=4, tile_r_m=1, tile_t_warps=4, tile_t_m=1)
    assert b.cases[0].step(2)["cd"] == one.step(2)["cd"]
    assert np.array_equal(b.cases[0].get("P"), one.get("P"))


@pytest.mark.parametrize("before,after", TILES)
def test_transposed_mixed_step_follows_the_tiles(before, after):
    """The scatters around the iteration add in any order: 1e-12 of each array."""
    case = make_case(n_theta=24, n_r=17, skew=0.3, vel_rot=0.2, nswpp=32, resimax=0.0)
    b, fresh = _batch([case], capi.MIXED, before), _batch([case], capi.MIXED, after)
    rng = np.random.default_rng(5)
    lam = {nm: rng.standard_normal(b.cases[0].get("U").shape) for nm in ("U", "V", "P", "NLX", "NLY")}
    b.cases[0].adjoint_vjp(lam)
    b.set_tiles(after)
    b.cases[0].init(case["du"], case["dv"])
    for x in (b, fresh):
        x.cases[0].step(1)
    (x, _, bx), (y, _, by) = b.cases[0].adjoint_vjp(lam), fresh.cases[0].adjoint_vjp(lam)
    for nm in lam:
        assert np.isfinite(x[nm]).all() and np.linalg.norm(x[nm] - y[nm]) <= 1e-12 * np.linalg.norm(y[nm]), nm
    assert np.linalg.norm(bx - by) <= 1e-12 * np.linalg.norm(by)
