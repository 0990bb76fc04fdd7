"""A step's launches as graphs from a context's second step on: the same bits and the same
kernel count as the launches, through changes of the controls and of the grid."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import make_case, make_gpu

pytestmark = pytest.mark.gpu

NAMES = ("U", "V", "P", "T", "NLX", "ADV")


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
def test_graph_steps_equal_launched_steps(precision):
    case = make_case(n_theta=24, n_r=17, skew=0.3, vel_rot=0.2, nswpp=16, resimax=0.0)
    kw = dict(precision=precision, refine_sweeps=4)
    a, b = make_gpu(case, **kw), make_gpu(case, **kw)
    recs = []
    for omega in (0.2, 0.2, 0.7):
        a.set_controls(omega)
        for _ in range(3):
            b.set_controls(omega)   # the context has changed: this step launches
            recs.append((a.step(1), b.step(1)))
    for x, y in recs:
        for k in ("time", "cd", "cl", "nu", "resid", "sweeps"):
            assert x[k] == y[k], k
    # a new grid on a context whose graphs exist
    other = make_case(n_theta=24, n_r=17, skew=0.1, vel_rot=0.2, nswpp=16, resimax=0.0)
    a.set_grid(other["g"].xg, other["g"].yg)
    b.set_grid(other["g"].xg, other["g"].yg)
    for _ in range(3):
        b.set_controls(0.7)
        x, y = a.step(1), b.step(1)
        assert x["cd"] == y["cd"] and x["resid"] == y["resid"]
    for nm in NAMES:
        assert np.isfinite(a.get(nm)).all() and np.array_equal(a.get(nm), b.get(nm)), nm


def test_kernels_of_a_graph_are_counted():
    case = make_case(n_theta=24, n_r=17, skew=0.3, vel_rot=0.2, nswpp=16, resimax=0.0)
    ctx = make_gpu(case, precision=capi.FP64)
    counts = []
    for _ in range(4):
        ctx.timing_reset()
        ctx.step(1)
        counts.append(ctx.timing()["kernel_launches"])
    assert len(set(counts)) == 1 and counts[0] > 8, counts


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
def test_transposed_steps_repeat_themselves(precision):
    """Launched and replayed transposed steps, before and after a change of the controls; the
    scatters add in any order: 1e-12 of each array."""
    case = make_case(n_theta=24, n_r=17, skew=0.3, vel_rot=0.2, nswpp=32, resimax=0.0)
    kw = dict(precision=precision, refine_sweeps=4)
    ctx = make_gpu(case, **kw)
    ctx.step(1)
    state = {nm: ctx.get(nm) for nm in ("U", "V", "P", "T", "NLX", "NLY", "ADV")}
    names = ("U", "V", "P", "NLX", "NLY")
    rng = np.random.default_rng(5)
    lam = {nm: rng.standard_normal(state["U"].shape) for nm in names}
    for omega in (0.2, 0.6):
        ctx.set_controls(omega)
        fresh = make_gpu(case, **kw)
        fresh.set_controls(omega)
        for nm, a in state.items():
            fresh.set(nm, a)
        want = fresh.adjoint_vjp(lam)
        for _ in range(6):
            got = ctx.adjoint_vjp(lam)
            for nm in names:
                assert np.linalg.norm(got[0][nm] - want[0][nm]) <= 1e-12 * np.linalg.norm(want[0][nm]), nm
            assert abs(got[1] - want[1]) <= 1e-12 * max(1.0, abs(want[1]))
        for nm, a in state.items():
            assert np.array_equal(ctx.get(nm), a), nm
