"""Pressure fields whose ghost cells hold values of their own: the first source of the Poisson
iteration reads them as stored, later ones what BCP makes of the current pressure.  The
FP64 ring against the per-colour kernels, and the 3-D mixed residual, which after the first
interval reads the wrapped cells in place of the ghosts."""
import numpy as np
import pytest

from fvm_gb300 import capi, capi3d
from fvm_gb300.grid import o_grid_3d, perturbation_3d
from tests.helpers import make_case, make_gpu, rel_l2

pytestmark = pytest.mark.gpu

# theta lines, radial cells, tile, residual interval
RING = [(4, 5, (1, 1), 2), (8, 4, (1, 1), 4), (32, 24, (1, 1), 2), (64, 130, (2, 3), 6), (48, 70, (4, 1), 2),
        (306, 40, (1, 2), 4), (512, 384, (2, 6), 8)]


@pytest.mark.parametrize("n_theta,n_r,tile,every", RING)
def test_ring_reads_the_stored_ghosts_once(n_theta, n_r, tile, every):
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=3 * every, resimax=0.0)
    out = []
    for resident in (1, 0):
        ctx = make_gpu(case, res_every=every, tile_r_warps=tile[0], tile_r_m=tile[1], poisson_resident=resident)
        ctx.set("P", 0.1 * np.random.default_rng(7).standard_normal(ctx.get("P").shape))
        out.append([(*ctx.iter_p(), ctx.get("P")) for _ in range(2)])
        ctx.close()
    for a, b in zip(*out):
        assert a[:3] == b[:3] and np.isfinite(a[3]).all() and np.array_equal(a[3], b[3])


def _grid():
    """Rings that move along the span and bent span planes: every cross weight is there."""
    g = o_grid_3d(16, 12, 8, lz=np.pi, dr1=0.01, skew=0.3)
    k = np.arange(g.nk + 1).reshape(-1, 1, 1) - 1
    r = np.hypot(g.xg, g.yg)
    s = 2.0 * np.pi * k / (g.nk - 1)
    x, y = g.xg.copy(), g.yg.copy()
    g.xg[1:, 1:, 1:] += (0.02 * r * np.sin(s))[1:, 1:, 1:]
    g.yg[1:, 1:, 1:] += (0.01 * r * np.cos(s))[1:, 1:, 1:]
    g.zg[1:, 1:, 1:] += (0.03 * (x + 0.5 * y) / np.maximum(r, 0.1))[1:, 1:, 1:]
    return g


def _pressure(precision, refine, cap, calls, host_loop):
    g = _grid()
    p = capi3d.default_params(ni=g.ni, nj=g.nj, nk=g.nk, re=1000.0, dt=0.001, resimax=0.0, nswpp=cap, use_les=0, thermal=0,
                              res_every=1, refine_sweeps=refine, precision=precision, poisson_host_loop=host_loop)
    ctx = capi3d.Context3(p)
    ctx.set_grid(g)
    ctx.init(*perturbation_3d(g.ni, g.nj, g.nk, 0.05, 3))
    ctx.set("P", np.random.default_rng(7).standard_normal(ctx.get("P").shape))
    for _ in range(calls):
        ctx.iter_p()
    out = ctx.get("P")
    ctx.close()
    return out


@pytest.mark.parametrize("host_loop", [0, 1], ids=["device-loop", "host-loop"])
def test_3d_residual_reads_the_stored_ghosts_first(host_loop):
    """One interval of one sweep is the FP64 path's first sweep, but for the FP32 correction
    (2^-24 of it, a few operations: 2e-6 of the field)."""
    a, b = (_pressure(q, 1, 1, 1, host_loop) for q in (capi.MIXED, capi.FP64))
    assert np.isfinite(a).all() and rel_l2(a, b) <= 2e-6


@pytest.mark.parametrize("host_loop", [0, 1], ids=["device-loop", "host-loop"])
@pytest.mark.parametrize("refine,intervals", [(1, 2), (2, 3), (4, 2)])
def test_3d_wrapped_cells_are_the_ghosts_of_the_current_pressure(refine, intervals, host_loop):
    """Calls of one interval each, between which BCP sets every ghost, and one call of them all."""
    a = _pressure(capi.MIXED, refine, refine, intervals, host_loop)
    b = _pressure(capi.MIXED, refine, refine * intervals, 1, host_loop)
    assert np.isfinite(a).all() and np.array_equal(a, b)
