"""The timed sweeps of a batch, by which its tiles are chosen, are those that its step runs: one
launch per cluster size where every case has a cluster, two launches a sweep where one has
none."""
import numpy as np
import pytest

from fvm_gb300 import capi
from tests.helpers import STATE, case_params, make_case

pytestmark = pytest.mark.gpu

SWEEPS = 10
# grids, precision, tiles, launches
BATCHES = [([(64, 48), (96, 33)], capi.MIXED, (2, 1, 4, 1), 1),
           ([(64, 48), (240, 192), (96, 33)], capi.MIXED, (2, 3, 4, 2), 2),
           ([(512, 380), (64, 40)], capi.MIXED, (1, 12, 4, 4), 2 * SWEEPS),
           ([(64, 48), (96, 33)], capi.FP64, (2, 1, 4, 1), 2 * SWEEPS)]


def _batch(grids, precision):
    cases = [make_case(n_theta=a, n_r=b, seed=k, nswpp=16, resimax=0.0) for k, (a, b) in enumerate(grids)]
    b = capi.Batch([case_params(c, precision, refine_sweeps=8) for c in cases])
    for ctx, c in zip(b.cases, cases):
        ctx.set_grid(c["g"].xg, c["g"].yg)
        ctx.init(c["du"], c["dv"])
    return b


@pytest.mark.parametrize("grids,precision,tiles,launches", BATCHES)
def test_timed_sweeps_are_those_of_the_step(grids, precision, tiles, launches):
    b = _batch(grids, precision)
    b.set_tiles(tiles)
    b.step(1)
    before = [{nm: c.get(nm) for nm in STATE} for c in b.cases]
    n0 = b.timing()["sweep_span_launches"]
    assert b.time_sweeps(SWEEPS) > 0.0
    assert b.timing()["sweep_span_launches"] - n0 == launches
    for c, was in zip(b.cases, before):
        assert all(np.array_equal(c.get(nm), a) for nm, a in was.items())


def test_the_tuner_times_and_leaves_the_batch_as_it_would_be_with_its_tiles():
    """After the tuner the batch steps as one that was given the tiles it chose."""
    grids = [(64, 48), (240, 192), (96, 33)]
    b, fresh = _batch(grids, capi.MIXED), _batch(grids, capi.MIXED)
    tiles, ms = b.autotune(sweeps=SWEEPS)
    fresh.set_tiles(tiles)
    x, y = b.step(2), fresh.step(2)
    assert ms[0] > 0.0 and [r["cd"] for r in x[-1]] == [r["cd"] for r in y[-1]]
    for c, f in zip(b.cases, fresh.cases):
        assert all(np.array_equal(c.get(nm), f.get(nm)) for nm in STATE)
