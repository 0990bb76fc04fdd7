"""A value that is not finite on grids whose cross terms leave direction pairs out: the step ends with
FVM_ERR_NAN, wherever the value stood."""
import numpy as np
import pytest

from fvm_gb300 import capi, capi3d
from fvm_gb300.grid import o_grid_3d, perturbation_3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["U", "P", "W"])
@pytest.mark.parametrize("at", [(4, 5, 20), (1, 1, 1), (7, 12, 23)])
def test_a_step_with_such_a_value_is_refused(name, at, precision):
    g = o_grid_3d(16, 24, 8, lz=np.pi, dr1=0.01, skew=0.0)
    p = capi3d.default_params(ni=g.ni, nj=g.nj, nk=g.nk, re=1000.0, dt=0.001, resimax=0.0, nswpp=4, use_les=1, thermal=1,
                              res_every=2, refine_sweeps=2, precision=precision, ref_a=np.pi)
    ctx = capi3d.Context3(p)
    ctx.set_grid(g)
    ctx.init(*perturbation_3d(g.ni, g.nj, g.nk, 0.05, 3))
    ctx.step(1)
    a = ctx.get(name)
    a[at] = np.nan
    ctx.set(name, a)
    with pytest.raises(capi.FvmError) as err:
        ctx.step(1)
    assert err.value.code == capi.FVM_ERR_NAN
