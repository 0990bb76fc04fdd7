"""Cross-derivative weights whose direction pairs vanish are left out of the 3-D cross
terms (D3::cwp): grids that need none, one or all three pairs against the CPU
restatement, and a context whose grid changes from one to the other."""
import numpy as np
import pytest

import oracle
from fvm_gb300 import capi, capi3d
from fvm_gb300.grid import o_grid_3d, perturbation_3d
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


def _grid(warp, skew):
    """An extruded grid (warp 0), or one whose rings move along the span and whose span
    planes are bent, so that every product of the metrics is there."""
    g = o_grid_3d(16, 12, 8, lz=np.pi, dr1=0.01, skew=skew)
    k = np.arange(g.nk + 1).reshape(-1, 1, 1) - 1
    r = np.hypot(g.xg, g.yg)
    s = 2.0 * np.pi * k / (g.nk - 1)
    x, y = g.xg.copy(), g.yg.copy()
    g.xg[1:, 1:, 1:] += (warp * 0.02 * r * np.sin(s))[1:, 1:, 1:]
    g.yg[1:, 1:, 1:] += (warp * 0.01 * r * np.cos(s))[1:, 1:, 1:]
    g.zg[1:, 1:, 1:] += (warp * 0.03 * (x + 0.5 * y) / np.maximum(r, 0.1))[1:, 1:, 1:]
    return g


def _pair(g, precision):
    du, dv, dw = perturbation_3d(g.ni, g.nj, g.nk, 0.05, 3)
    kw = dict(re=1000.0, dt=0.001, resimax=0.0, nswpp=24, use_les=True, les_zavg=False, thermal=True, res_every=4,
              ref_a=np.pi)
    o = oracle.Oracle3D(g.ni, g.nj, g.nk, order=oracle.O3_GPU, **kw)
    o.set_grid(g)
    o.init(du, dv, dw)
    p = capi3d.default_params(ni=g.ni, nj=g.nj, nk=g.nk, precision=precision, refine_sweeps=4,
                              **{**kw, "use_les": 1, "les_zavg": 0, "thermal": 1})
    ctx = capi3d.Context3(p)
    ctx.set_grid(g)
    ctx.init(du, dv, dw)
    return o, ctx


@pytest.mark.parametrize("warp,skew", [(0, 0.0), (0, 0.3), (1, 0.3)], ids=["polar", "extruded", "warped"])
def test_steps_match_whatever_pairs_the_grid_needs(warp, skew):
    g = _grid(warp, skew)
    o, ctx = _pair(g, capi.FP64)
    for _ in range(2):
        o.step(1)
        ctx.step(1)
    for nm in ("U", "V", "W", "P", "T"):
        assert rel_l2(ctx.get(nm), o.array(nm)) <= 1e-9, nm


def test_the_pairs_follow_a_new_grid():
    """set_grid with a grid that needs more pairs, on a context that has already run."""
    a, b = _grid(0, 0.0), _grid(1, 0.3)
    du, dv, dw = perturbation_3d(a.ni, a.nj, a.nk, 0.05, 3)
    for precision in (capi.FP64, capi.MIXED):
        _, ctx = _pair(a, precision)
        _, ref = _pair(b, precision)
        ctx.step(1)
        ctx.set_grid(b)
        ctx.init(du, dv, dw)
        x, y = ctx.step(1), ref.step(1)
        assert x["cd"] == y["cd"]
        for nm in ("U", "P", "T"):
            assert np.array_equal(ctx.get(nm), ref.get(nm)), nm
