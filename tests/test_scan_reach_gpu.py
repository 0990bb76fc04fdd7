"""How far a line solve of the one-launch Poisson iterations carries a value along its line,
against the per-colour kernels: sources of a few cells, whose values fall by many orders of
magnitude along a line, and sources that are not finite, which fill whole lines."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import make_case, make_gpu

pytestmark = pytest.mark.gpu

# theta lines, radial cells, tile, the cell (i, j) whose velocity is set
CASES = [(512, 384, (2, 6), (5, 31)), (512, 384, (2, 6), (377, 500)), (64, 380, (1, 12), (300, 20)),
         (32, 24, (1, 1), (20, 3)), (128, 96, (1, 3), (90, 64))]
CASES64 = CASES + [(512, 100, (4, 1), (3, 77)), (512, 500, (4, 4), (250, 8))]
MIXED = [(capi.MIXED, *c) for c in CASES]
FP64 = [(capi.FP64, *c) for c in CASES64]


def _context(case, precision, tile, resident):
    return make_gpu(case, precision=precision, res_every=2, refine_sweeps=2, poisson_resident=resident,
                    tile_r_warps=tile[0], tile_r_m=tile[1])


def _local(precision, case, tile, at, resident):
    """P after the iteration on a velocity that is zero but for one cell."""
    ctx = _context(case, precision, tile, resident)
    u = np.zeros_like(ctx.get("U"))
    ctx.set("V", u)
    ctx.set("P", u)
    u[at[1], at[0]] = 1.0
    ctx.set("U", u)
    ctx.iter_p()
    p = ctx.get("P")
    ctx.close()
    return p


@pytest.mark.parametrize("precision,n_theta,n_r,tile,at", MIXED + FP64)
def test_a_source_of_a_few_cells(precision, n_theta, n_r, tile, at):
    """Mixed: the same bits.  FP64: the ring leaves out what is below 2^-80 of its source, which in
    32 sweeps is at most 32 units in the last place (2^-53) of the largest value."""
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=32, resimax=0.0)
    a, b = (_local(precision, case, tile, at, r) for r in (1, 0))
    assert np.isfinite(b).all() and np.abs(b).max() > 0.0
    if precision == capi.MIXED:
        assert np.array_equal(a, b)
    else:
        assert np.abs(a - b).max() <= 2.0 ** -48 * np.abs(b).max()


def _finite(precision, case, tile, at, value, resident):
    ctx = _context(case, precision, tile, resident)
    ctx.step(1)
    u = ctx.get("U")
    u[at[1], at[0]] = value
    ctx.set("U", u)
    with pytest.raises(capi.FvmError) as err:
        ctx.iter_p()
    assert err.value.code == capi.FVM_ERR_NAN
    p = ctx.get("P")
    ctx.close()
    return np.isfinite(p)


@pytest.mark.parametrize("value", [np.nan, np.inf], ids=["nan", "inf"])
@pytest.mark.parametrize("precision,n_theta,n_r,tile,at", MIXED + FP64)
def test_a_source_that_is_not_finite(precision, n_theta, n_r, tile, at, value):
    """The same cells of P are not finite."""
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=8, resimax=0.0)
    a, b = (_finite(precision, case, tile, at, value, r) for r in (1, 0))
    assert not a[1:-1, 1:-1].all() and np.array_equal(a, b)
