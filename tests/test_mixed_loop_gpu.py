"""The mixed Poisson iteration of a step in one launch against the per-colour kernels: skewed
grids (the cross term is there), rings of 3 blocks up, partly filled chunks and tile
columns, uploaded states whose ghost cells disagree with the boundary conditions, and
the pairings and intervals that keep the launch per interval."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import make_case, make_gpu

pytestmark = pytest.mark.gpu

# theta lines, radial cells, tile, sweeps per interval, cap, dd_positional
CASES = [
    (12, 5, (1, 1), 2, 6, 1),
    (16, 33, (0, 0), 8, 40, 1),
    (40, 64, (2, 1), 4, 12, 1),
    (100, 97, (1, 4), 6, 18, 1),
    (128, 96, (0, 0), 16, 64, 1),
    (256, 190, (0, 0), 32, 64, 1),
    (512, 384, (0, 0), 32, 64, 1),
    (512, 510, (0, 0), 2, 4, 1),     # the longest lines: 2 warps x 8 elements, 16 tile columns
    (64, 380, (1, 12), 8, 16, 1),
    (64, 48, (0, 0), 8, 24, 0),      # the cell's own cross term: one launch per interval
    (64, 48, (0, 0), 5, 20, 1),      # an odd interval: one exchange per sweep
]


def _run(case, tile, resident, refine, dd_pos, state):
    ctx = make_gpu(case, precision=capi.MIXED, refine_sweeps=refine, poisson_resident=resident, tile_r_warps=tile[0],
                   tile_r_m=tile[1], dd_positional=dd_pos, poisson_host_loop=0)
    if state is not None:
        ctx.upload(**state)
    rec = [ctx.step(1) for _ in range(2)]
    out = {nm: ctx.get(nm) for nm in ("U", "V", "P")}
    info = ctx.resident_info()
    ctx.close()
    return rec, out, info


@pytest.mark.parametrize("ghosts", [False, True], ids=["init", "uploaded-ghosts"])
@pytest.mark.parametrize("n_theta,n_r,tile,refine,cap,dd_pos", CASES)
def test_loop_equals_per_colour_kernels(n_theta, n_r, tile, refine, cap, dd_pos, ghosts):
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=cap, resimax=0.0)
    g = case["g"]
    state = None
    if ghosts:   # every value of P, ghost cells included, of its own
        rng = np.random.default_rng(7)
        state = dict(p=0.1 * rng.standard_normal((g.nj + 1, g.ni + 1)))
    if (tile[0], tile[1]) == (0, 0):   # the per-colour path picks another automatic tile
        n = n_r
        tile = (1, (n + 31) // 32) if n <= 128 else (2, next(m for m in (1, 2, 3, 4, 6, 8) if 64 * m >= n))
    ra, fa, info = _run(case, tile, 1, refine, dd_pos, state)
    rb, fb, _ = _run(case, tile, 0, refine, dd_pos, state)
    assert info["sweeps_per_exchange"] == 2 and info["lines_per_block"] == 4
    for a, b in zip(ra, rb):
        assert a["sweeps"] == b["sweeps"] and a["resid"] == b["resid"] and a["cd"] == b["cd"]
    for nm in fa:
        assert np.isfinite(fa[nm]).all() and np.array_equal(fa[nm], fb[nm]), nm


def test_loop_and_adjoint_share_the_exchange_words():
    """Steps, a transposed step (launches per interval on the same words) and steps again."""
    case = make_case(n_theta=64, n_r=48, nswpp=48, resimax=0.0)
    a, b = (make_gpu(case, precision=capi.MIXED, refine_sweeps=8, poisson_resident=r) for r in (1, 0))
    for ctx in (a, b):
        ctx.step(2)
    lam = {nm: np.random.default_rng(3).standard_normal(a.get("U").shape) for nm in ("U", "V", "P", "NLX", "NLY")}
    for ctx in (a, b):
        ctx.adjoint_vjp(lam)
        ctx.step(2)
    assert np.array_equal(a.get("P"), b.get("P")) and np.array_equal(a.get("U"), b.get("U"))


# theta lines, radial cells, tile, sweeps per interval, cap, tolerance of the iteration
ADJOINT = [(12, 5, (1, 1), 2, 6, 0.0), (40, 64, (2, 1), 4, 12, 0.0), (100, 97, (1, 4), 6, 18, 0.0),
           (64, 380, (1, 12), 8, 16, 0.0), (512, 510, (2, 8), 2, 4, 0.0), (64, 48, (1, 2), 4, 400, 1e-3)]


@pytest.mark.parametrize("n_theta,n_r,tile,refine,cap,resimax", ADJOINT)
def test_transposed_loop_equals_per_colour_kernels(n_theta, n_r, tile, refine, cap, resimax):
    """The transposed iteration in one launch: the cross term is summed in another order
    (1e-14 of it), which moves an FP32 residual by 2^-24 at most now and then: below 1e-6
    of each array, at the same interval of the iteration."""
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=cap, resimax=resimax)
    names = ("U", "V", "P", "NLX", "NLY")
    out = []
    for resident in (1, 0):
        ctx = make_gpu(case, precision=capi.MIXED, refine_sweeps=refine, poisson_resident=resident, tile_r_warps=tile[0],
                       tile_r_m=tile[1])
        ctx.step(2)
        rng = np.random.default_rng(11)
        out.append(ctx.adjoint_vjp({nm: rng.standard_normal(ctx.get("U").shape) for nm in names}))
        ctx.close()
    (x, wx, bx), (y, wy, by) = out
    for nm in names:
        assert np.isfinite(x[nm]).all() and np.linalg.norm(x[nm] - y[nm]) <= 1e-6 * np.linalg.norm(y[nm]), nm
    assert abs(wx - wy) <= 1e-6 * max(abs(wy), 1.0) and np.linalg.norm(bx - by) <= 1e-6 * np.linalg.norm(by)
