"""The test filter of the SGS model with its passes fused into other launches: radial cells at
and beside the 30 results of a warp, walks along theta that end early, both walk lengths.
The filtered velocity against the 27-point sum, the model against the CPU restatement."""
import numpy as np
import pytest

import oracle
from fvm_gb300 import capi, capi3d
from fvm_gb300.grid import o_grid_3d, perturbation_3d
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# theta cells, radial cells, span cells; the last one takes the long walks
GRIDS = [(8, 7, 8), (18, 30, 8), (22, 31, 10), (34, 61, 8), (130, 62, 50)]


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("shape", GRIDS, ids=lambda s: "x".join(map(str, s)))
def test_filters_at_the_edges_of_the_tiles(shape, precision):
    g = o_grid_3d(*shape, lz=np.pi, dr1=0.02, skew=0.3)
    kw = dict(re=1000.0, dt=0.001, resimax=0.0, nswpp=4, res_every=4, ref_a=np.pi)
    p = capi3d.default_params(ni=g.ni, nj=g.nj, nk=g.nk, precision=precision, refine_sweeps=4, use_les=1, les_zavg=0,
                              thermal=1, **kw)
    o = oracle.Oracle3D(g.ni, g.nj, g.nk, order=oracle.O3_GPU, use_les=True, les_zavg=False, thermal=True, **kw)
    ctx = capi3d.Context3(p)
    d = perturbation_3d(g.ni, g.nj, g.nk, 0.05, 3)
    for x in (o, ctx):
        x.set_grid(g)
        x.init(*d)
    o.step(1)
    for nm in ("U", "V", "W", "P", "T", "NLX", "NLY", "NLZ", "ADV"):
        ctx.set(nm, o.array(nm))
    c = ctx.sgs()
    for nm in "UVWT":
        o.array(nm + "_N")[...] = o.array(nm)
    o.sgs()
    # a sum of 27 terms: 2^-53 (FP64) or 2^-46 (pairs) per operation
    u, want = o.array("U"), 0.0
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for e in (-1, 0, 1):
                w = (2 - a * a) * (2 - b * b) * (2 - e * e) / 64.0
                want = want + w * u[1 + a:u.shape[0] - 1 + a, 1 + b:u.shape[1] - 1 + b, 1 + e:u.shape[2] - 1 + e]
    assert rel_l2(ctx.get("U_HAT")[1:-1, 1:-1, 1:-1], want) <= (1e-14 if precision == capi.FP64 else 1e-12)
    # the Leonard terms are down to 1e-6 of the products whose rounding they carry
    tol = 1e-8 if precision == capi.FP64 else 1e-6
    assert rel_l2(ctx.get("EDDY_VISCOS"), o.array("EDDY_VISCOS")) <= tol
    assert abs(c["cs2"] - o.coeffs()["cs2"]) <= tol * abs(o.coeffs()["cs2"])
