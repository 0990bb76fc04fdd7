"""State copies: page-locked buffers (one kernel), pageable ones and mixtures, odd and even
array lengths, unaligned buffers, skipped arrays, one buffer given twice."""
import numpy as np
import pytest
import torch

from fvm_gb300 import capi
from fvm_gb300.grid import o_grid

pytestmark = pytest.mark.gpu

NAMES = ("U", "V", "P", "T", "NLX", "NLY", "ADV")


def _ctx(n_theta, n_r):
    g = o_grid(n_theta, n_r)
    ctx = capi.Context(capi.default_params(ni=g.ni, nj=g.nj))
    ctx.set_grid(g.xg, g.yg)
    ctx.init()
    return ctx, (g.ni + 1) * (g.nj + 1)


def _buffers(n, how, offset):
    """Seven host arrays of n doubles starting `offset` doubles into their allocation."""
    out = []
    for k in range(7):
        a = torch.empty(n + 2, dtype=torch.float64)
        out.append((a.pin_memory() if how == "pinned" or (how == "mixed" and k % 2) else a)[offset:offset + n])
    return out


@pytest.mark.parametrize("how", ["pinned", "pageable", "mixed"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n_theta,n_r", [(4, 4), (64, 41), (256, 200)])
def test_round_trip(n_theta, n_r, how, offset):
    ctx, n = _ctx(n_theta, n_r)
    rng = np.random.default_rng(n)
    src, dst = _buffers(n, how, offset), _buffers(n, how, offset)
    for s, d in zip(src, dst):
        s.copy_(torch.from_numpy(rng.standard_normal(n)))
        d.fill_(-7.0)
    ctx.upload_ptrs([s.data_ptr() for s in src])
    for nm, s in zip(NAMES, src):
        assert np.array_equal(ctx.get(nm).ravel(), s.numpy()), nm
    ctx.download_ptrs([d.data_ptr() if k != 3 else 0 for k, d in enumerate(dst)])
    for k, (s, d) in enumerate(zip(src, dst)):
        assert np.array_equal(d.numpy(), s.numpy() if k != 3 else np.full(n, -7.0)), k


def test_one_target_given_twice_takes_the_last_array():
    ctx, n = _ctx(32, 20)
    src = _buffers(n, "pinned", 0)
    for k, s in enumerate(src):
        s.fill_(float(k))
    ctx.upload_ptrs([s.data_ptr() for s in src])
    d = torch.empty(n, dtype=torch.float64).pin_memory()
    ctx.download_ptrs([d.data_ptr(), d.data_ptr(), 0, 0, 0, 0, 0])
    assert (d == 1.0).all()
