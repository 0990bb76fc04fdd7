"""Batches whose mixed Poisson iteration runs one cluster per case (fvm_cluster.cu) against the
same cases one by one on the per-colour kernels: the same bits, for rings of one block
up, blocks without lines, last groups of two lines, every tile width, cases that converge
on their own counts, and batches that keep the per-colour form."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import STATE, case_params, make_case, make_gpu

pytestmark = pytest.mark.gpu

# (theta, r) of the cases, tiles (radial warps, elements, circumferential warps, elements)
BATCHES = [
    ([(4, 5), (8, 6), (12, 20)], (1, 1, 1, 1)),                  # one to three blocks of four lines
    ([(32, 24), (36, 30), (100, 17)], (1, 1, 4, 1)),             # 36: two lines in no block's way; 100: 13 groups
    ([(64, 48), (132, 90), (256, 64)], (2, 2, 4, 2)),            # blocks of 8, 12 and 16 lines
    ([(64, 48), (240, 192), (96, 33)], (2, 3, 4, 2)),            # clusters of 8 and of 16 blocks
    ([(128, 100), (64, 128)], (4, 1, 4, 1)),
    ([(64, 190), (80, 150)], (1, 6, 1, 3)),
    ([(512, 380), (64, 40)], (1, 12, 4, 4)),                     # too large for a block: per-colour kernels
]


def _pair(grids, tiles, refine, **kw):
    cases = [make_case(n_theta=a, n_r=b, seed=k, re=80.0 + 40 * k, skew=0.2 * (k % 2), vel_rot=0.1 * k, **kw)
             for k, (a, b) in enumerate(grids)]
    b = capi.Batch([case_params(c, capi.MIXED, refine_sweeps=refine) for c in cases])
    for ctx, c in zip(b.cases, cases):
        ctx.set_grid(c["g"].xg, c["g"].yg)
    b.set_tiles(tiles)
    for ctx, c in zip(b.cases, cases):
        ctx.init(c["du"], c["dv"])
    t = dict(tile_r_warps=tiles[0], tile_r_m=tiles[1], tile_t_warps=tiles[2], tile_t_m=tiles[3])
    return b, [make_gpu(c, capi.MIXED, refine_sweeps=refine, poisson_resident=0, **t) for c in cases]


def _same(b, singles, steps):
    recs = b.step(steps)
    for k, ctx in enumerate(singles):
        for s in range(steps):
            r = ctx.step(1)
            for key in ("cd", "cl", "nu", "cfl", "sweeps", "resid"):
                assert recs[s][k][key] == r[key], (k, s, key)
        for nm in STATE:
            assert np.array_equal(b.cases[k].get(nm), ctx.get(nm)), (k, nm)
    return recs


@pytest.mark.parametrize("grids,tiles", BATCHES)
@pytest.mark.parametrize("refine", [1, 8])
def test_batch_equals_per_colour_singles(grids, tiles, refine):
    b, singles = _pair(grids, tiles, refine, nswpp=24, resimax=0.0)
    _same(b, singles, 2)


def test_cases_end_on_their_own_counts_and_tiles_may_change():
    b, singles = _pair([(32, 24), (48, 16), (40, 20)], (1, 1, 2, 1), 8, nswpp=40000, resimax=1e-9)
    recs = _same(b, singles, 2)
    assert len({r["sweeps"] for r in recs[-1]}) > 1
    b.set_tiles((2, 1, 2, 1))
    b.step(1)
    assert all(np.isfinite(c.get("P")).all() for c in b.cases)
