"""The transposed systems of the adjoint (coefficients, line factors, drag sensitivities,
split planes) follow the context they were made for: a new grid, another wall geometry and
other line tiles.  Launched scatters add in any order: 1e-12 of each array."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import case_params, make_case, make_gpu

pytestmark = pytest.mark.gpu

NAMES = ("U", "V", "P", "NLX", "NLY")
KW = dict(nswpp=32, resimax=0.0)


def _lam(ctx):
    rng = np.random.default_rng(5)
    return {nm: rng.standard_normal(ctx.get("U").shape) for nm in NAMES}


def _same(ctx, fresh, lam):
    (x, wx, bx), (y, wy, by) = ctx.adjoint_vjp(lam), fresh.adjoint_vjp(lam)
    for nm in NAMES:
        assert np.isfinite(x[nm]).all() and np.linalg.norm(x[nm] - y[nm]) <= 1e-12 * np.linalg.norm(y[nm]), nm
    assert abs(wx - wy) <= 1e-12 * max(1.0, abs(wy)) and np.linalg.norm(bx - by) <= 1e-12 * np.linalg.norm(by)


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
def test_transposed_step_follows_a_new_grid(precision):
    old, new = (make_case(n_theta=24, n_r=17, skew=s, vel_rot=0.2, **KW) for s in (0.0, 0.3))
    kw = dict(precision=precision, refine_sweeps=4)
    ctx, fresh = make_gpu(old, **kw), make_gpu(new, **kw)
    ctx.step(1)
    lam = _lam(ctx)
    ctx.adjoint_vjp(lam)
    ctx.set_grid(new["g"].xg, new["g"].yg)
    ctx.init(new["du"], new["dv"])
    for c in (ctx, fresh):
        c.step(2)
    assert np.array_equal(ctx.get("P"), fresh.get("P"))
    for _ in range(3):   # launched, and from the second on replayed
        _same(ctx, fresh, lam)


def test_drag_gradient_follows_the_wall_geometry():
    """A new grid, and an angle array set by hand: the drag's own sensitivities."""
    old, new = (make_case(n_theta=24, n_r=17, skew=s, vel_rot=0.2, **KW) for s in (0.0, 0.3))
    ctx, fresh = make_gpu(old), make_gpu(new)
    ctx.adjoint_drag_grad(2, 1)
    ctx.set_grid(new["g"].xg, new["g"].yg)
    ctx.init(new["du"], new["dv"])
    for theta in (None, fresh.get("THETA") + 0.1):
        if theta is not None:
            ctx.set("THETA", theta)
            fresh = make_gpu(new)
            fresh.set("THETA", theta)
            ctx.init(new["du"], new["dv"])
        (ja, wa, ba), (jb, wb, bb) = ctx.adjoint_drag_grad(3, 2), fresh.adjoint_drag_grad(3, 2)
        assert ja == jb
        assert abs(wa - wb) <= 1e-11 * max(1.0, abs(wb)) and np.linalg.norm(ba - bb) <= 1e-11 * np.linalg.norm(bb)


# tiles before and after: longer and shorter chunks, more and fewer warps a line
TILES = [((1, 1, 1, 1), (2, 2, 1, 2)), ((1, 1, 1, 1), (4, 1, 4, 1)), ((4, 2, 4, 1), (1, 1, 2, 1))]


def _batch(precision, tiles):
    cases = [make_case(n_theta=24, n_r=17, skew=0.3, vel_rot=0.2, **KW), make_case(n_theta=32, n_r=24, seed=2, **KW)]
    b = capi.Batch([case_params(c, precision, refine_sweeps=4) for c in cases])
    for ctx, c in zip(b.cases, cases):
        ctx.set_grid(c["g"].xg, c["g"].yg)
    b.set_tiles(tiles)
    for ctx, c in zip(b.cases, cases):
        ctx.init(c["du"], c["dv"])
    return b


@pytest.mark.parametrize("before,after", TILES)
def test_transposed_step_of_a_case_follows_the_tiles(before, after):
    b, fresh = _batch(capi.FP64, before), _batch(capi.FP64, after)
    lam = [_lam(c) for c in b.cases]
    for c, v in zip(b.cases, lam):
        c.adjoint_vjp(v)
    b.set_tiles(after)
    for batch in (b, fresh):
        batch.step(1)
    for x, y, v in zip(b.cases, fresh.cases, lam):
        _same(x, y, v)
