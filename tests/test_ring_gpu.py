"""The FP64 Poisson iteration in one launch (fvm_ring.cu) against the per-colour kernels
(poisson_resident = 0): the same operations in the same rounding order, so pressure,
scaled residual and sweep count are equal bit for bit."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import make_case, make_gpu

pytestmark = pytest.mark.gpu

# theta lines, radial cells, tile (0, 0: automatic), residual interval, cap, tolerance
CASES = [
    (4, 5, (0, 0), 2, 10, 0.0),          # two blocks of one pair: each is the other's neighbour on both sides
    (8, 4, (1, 1), 2, 2, 0.0),           # one interval
    (32, 24, (0, 0), 2, 20, 1e-4),       # the reference's defaults
    (24, 33, (1, 2), 4, 4000, 1e-9),     # ended by the tolerance; last thread's chunk partly filled
    (64, 130, (2, 3), 6, 60, 0.0),
    (48, 70, (4, 1), 2, 30, 0.0),
    (40, 190, (1, 6), 8, 64, 0.0),
    (304, 21, (0, 0), 4, 24, 0.0),       # 152 blocks of one pair
    (306, 40, (0, 0), 4, 24, 0.0),       # two pairs per block, the last block with one
    (512, 384, (0, 0), 8, 32, 0.0),
    (512, 500, (0, 0), 2, 8, 0.0),       # the longest lines, 4 warps x 4 elements
]


def _iter_p(case, tile, resident, every, passes=2):
    ctx = make_gpu(case, res_every=every, tile_r_warps=tile[0], tile_r_m=tile[1], poisson_resident=resident)
    out = []
    for _ in range(passes):
        ctx.begin_step()
        ctx.contra_vel()
        ctx.iter_u()
        ctx.iter_v()
        ctx.remove_grad()
        resid, sweeps, _ = ctx.iter_p()
        out.append((resid, sweeps, ctx.get("P")))
        ctx.correct()
    ctx.close()
    return out


@pytest.mark.parametrize("n_theta,n_r,tile,every,cap,tol", CASES)
def test_ring_equals_per_colour_kernels(n_theta, n_r, tile, every, cap, tol):
    case = make_case(n_theta=n_theta, n_r=n_r, skew=0.3, vel_rot=0.2, nswpp=cap, resimax=tol)
    for a, b in zip(_iter_p(case, tile, 1, every), _iter_p(case, tile, 0, every)):
        assert a[1] == b[1] and a[0] == b[0]
        assert np.isfinite(a[2]).all() and np.array_equal(a[2], b[2])


def test_per_colour_path_serves_the_cell_local_cross_term():
    """dd_positional = 0 keeps the per-colour kernels whatever poisson_resident says."""
    case = make_case(n_theta=32, n_r=20, skew=0.3, nswpp=12, resimax=0.0)
    a = make_gpu(case, res_every=4, dd_positional=0)
    b = make_gpu(case, res_every=4, dd_positional=0, poisson_resident=0)
    ra, rb = a.step(2), b.step(2)
    assert ra["sweeps"] == rb["sweeps"] and np.array_equal(a.get("P"), b.get("P"))
