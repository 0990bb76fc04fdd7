"""The transposed FP64 Poisson iteration in one launch against the per-colour kernels: the same
sweeps of the same system, so a transposed step agrees to rounding (the two sum the
cross term in another order; 64 sweeps keep that below 1e-11 of each array)."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import make_case, make_gpu, rel_l2

pytestmark = pytest.mark.gpu

NAMES = ("U", "V", "P", "NLX", "NLY")
# theta lines, radial cells, tile
CASES = [(4, 5, (0, 0)), (8, 4, (1, 1)), (32, 24, (0, 0)), (64, 33, (1, 2)), (40, 130, (2, 3)), (48, 70, (4, 1)),
         (304, 21, (0, 0)), (308, 40, (0, 0)), (128, 96, (0, 0)), (256, 384, (0, 0))]


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n_theta,n_r,tile", CASES)
def test_transposed_step_equals_per_colour(n_theta, n_r, tile, precision):
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=64, resimax=0.0)
    out = []
    for resident in (1, 0):
        ctx = make_gpu(case, precision=precision, refine_sweeps=8, poisson_resident=resident, tile_r_warps=tile[0],
                       tile_r_m=tile[1])
        ctx.upload(**_state(case))
        lam = {nm: np.random.default_rng(k).standard_normal(ctx.get("U").shape) for k, nm in enumerate(NAMES)}
        a = ctx.adjoint_vjp(lam)
        b = ctx.adjoint_vjp(lam)   # again on the same context: the same start
        for nm in NAMES:
            assert rel_l2(a[0][nm], b[0][nm]) <= 1e-12, nm
        out.append(a)
        ctx.close()
    (x, wx, bx), (y, wy, by) = out
    tol = 1e-11 if precision == capi.FP64 else 1e-6   # mixed: the automatic tiles differ, FP32 rounding
    for nm in NAMES:
        assert np.isfinite(x[nm]).all() and rel_l2(x[nm], y[nm]) <= tol, nm
    assert abs(wx - wy) <= tol * max(abs(wy), 1.0) and rel_l2(bx, by) <= tol


def _state(case):
    """A smooth flow over the whole array (ghost cells included)."""
    g = case["g"]
    th = np.arange(g.nj + 1)[:, None] * (2.0 * np.pi / (g.nj - 1))
    s = np.arange(g.ni + 1)[None, :] / g.ni
    return dict(u=1.0 + 0.3 * s * np.cos(th), v=0.3 * s * np.sin(th), p=0.2 * np.cos(2 * th) * (1 - s))
