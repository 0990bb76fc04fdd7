"""J and K line sweeps through shared memory, and the velocity components in shared launches:
lines shorter than a warp, chunks and rows partly filled, one, two and four warps a line,
a last block of lines that is not full.  Against the CPU restatement, and against the same
routines called one component at a time."""
import numpy as np
import pytest

import oracle
from fvm_gb300 import capi, capi3d
from fvm_gb300.grid import o_grid_3d, perturbation_3d
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# theta cells, radial cells, span cells
GRIDS = [(8, 7, 8), (10, 9, 12), (34, 13, 30), (66, 20, 34), (66, 130, 96), (130, 11, 10), (258, 7, 8), (12, 8, 130), (10, 130, 8)]
FIELDS = ("U", "V", "W", "P", "T")


def _case(shape, precision, **kw):
    g = o_grid_3d(*shape, lz=np.pi, dr1=0.02, skew=0.3)
    kw = dict(re=1000.0, dt=0.001, resimax=0.0, nswpp=8, res_every=4, ref_a=np.pi) | kw
    p = capi3d.default_params(ni=g.ni, nj=g.nj, nk=g.nk, precision=precision, refine_sweeps=4, use_les=0, les_zavg=0,
                              thermal=1, **kw)
    ctx = capi3d.Context3(p)
    ctx.set_grid(g)
    d = perturbation_3d(g.ni, g.nj, g.nk, 0.05, 3)
    ctx.init(*d)
    return g, d, kw, ctx


@pytest.mark.parametrize("shape", GRIDS, ids=lambda s: "x".join(map(str, s)))
def test_steps_match_the_restatement(shape):
    g, d, kw, ctx = _case(shape, capi.FP64)
    o = oracle.Oracle3D(g.ni, g.nj, g.nk, order=oracle.O3_GPU, use_les=False, les_zavg=False, thermal=True, **kw)
    o.set_grid(g)
    o.init(*d)
    for _ in range(2):
        o.step(1)
        ctx.step(1)
    for nm in FIELDS:
        assert rel_l2(ctx.get(nm), o.array(nm)) <= 1e-9, nm


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("shape", GRIDS, ids=lambda s: "x".join(map(str, s)))
def test_components_in_one_launch_equal_one_at_a_time(shape, precision):
    a = _case(shape, precision)[3]
    b = _case(shape, precision)[3]
    a.step(1)
    for nm in ("begin_step", "contra_vel", "nl", "dif", "p_source"):
        b.call(nm)
    for comp in (2, 0, 1):
        b.iter_u(comp)
    b.call("remove_grad")
    b.iter_p()
    b.call("correct")
    b.call("iter_t")
    for nm in FIELDS:
        x, y = a.get(nm), b.get(nm)
        assert np.isfinite(x).all() and np.array_equal(x, y), nm
