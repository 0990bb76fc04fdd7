"""The bounded waits of the one-launch Poisson iterations (FP64 ring, mixed loop, forward and
transposed): with tags that no block publishes each kind of wait runs out, the call
reports FVM_ERR_TIMEOUT, the state stays as it was and the context goes on as one that never
saw it.  Few polls: waits of other kinds may run out as well, in other blocks at other
places."""
import time

import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import make_case, make_gpu

pytestmark = pytest.mark.gpu

NAMES = ("U", "V", "P", "NLX", "NLY")
# theta lines, radial cells: two blocks, one pair of lines a block, two pairs a block with a last
# one of a single pair; mixed: three blocks, 25 and 64
CASES = [(capi.FP64, 4, 5), (capi.FP64, 128, 96), (capi.FP64, 306, 40), (capi.MIXED, 12, 20), (capi.MIXED, 100, 97),
         (capi.MIXED, 256, 190)]


def _advance(ctx):
    """A step's velocity and pressure by its call points (306 lines have a vertical wall face, for
    which the drag formula divides by zero)."""
    ctx.begin_step()
    ctx.contra_vel()
    ctx.iter_u()
    ctx.iter_v()
    ctx.remove_grad()
    resid, sweeps, _ = ctx.iter_p()
    ctx.correct()
    return resid, sweeps


@pytest.mark.parametrize("transposed", [False, True], ids=["forward", "transposed"])
@pytest.mark.parametrize("wait", [1, 2, 3, 4])
@pytest.mark.parametrize("precision,n_theta,n_r", CASES)
def test_each_wait_runs_out_and_the_context_stays_usable(precision, n_theta, n_r, wait, transposed):
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=32, resimax=0.0)
    a, b = (make_gpu(case, precision=precision, res_every=4, refine_sweeps=8) for _ in range(2))
    for c in (a, b):
        _advance(c)
    p = a.get("P")
    rng = np.random.default_rng(3)
    lam = {nm: rng.standard_normal(p.shape) for nm in NAMES}
    for polls in (2048, 16):
        t0 = time.perf_counter()
        rc = a.loop_wait_test(wait, transposed, max_polls=polls)
        assert rc == capi.FVM_ERR_TIMEOUT, capi.STATUS_NAMES.get(rc, rc)
        assert time.perf_counter() - t0 < 10.0 and "bounded wait" in a.last_error()
        assert np.array_equal(a.get("P"), p)
    (x, wx, bx), (y, wy, by) = a.adjoint_vjp(lam), b.adjoint_vjp(lam)
    for nm in NAMES:   # the scatters add in any order
        assert np.linalg.norm(x[nm] - y[nm]) <= 1e-12 * np.linalg.norm(y[nm]), nm
    for _ in range(2):
        assert _advance(a) == _advance(b)
    for nm in ("U", "V", "P"):
        assert np.array_equal(a.get(nm), b.get(nm)), nm


def test_arguments():
    case = make_case(n_theta=16, n_r=12, nswpp=8, resimax=0.0)
    ctx = make_gpu(case)
    assert ctx.loop_wait_test(0) == ctx.loop_wait_test(5) == ctx.loop_wait_test(1, max_polls=0) == capi.FVM_ERR_ARG
    for kw in (dict(poisson_resident=0), dict(dd_positional=0)):
        assert make_gpu(case, **kw).loop_wait_test(1) == capi.FVM_ERR_ARG
    assert make_gpu(case, precision=capi.MIXED, refine_sweeps=5).loop_wait_test(1) == capi.FVM_ERR_ARG
