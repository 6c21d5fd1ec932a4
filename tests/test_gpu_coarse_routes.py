"""The coarsest-level solve on its own is the one a V-cycle runs."""
import ctypes

import numpy as np
import pytest

from helpers import make_cfg

pytestmark = pytest.mark.gpu

EDGES = [10, 12, 14, 16, 18, 20, 22, 24, 26, 28, 30, 32]
HS = (1.0, 0.9, 1.1)


def _mg(nc, **kw):
    from warpflow import Multigrid, build_topology
    cfg = make_cfg(2 * nc, levels=2)
    h = 1.0 / (2 * nc)
    return Multigrid(cfg, build_topology(cfg), "cuda:0", *(h * x for x in HS), **kw)


def _no_operator(mg):
    c = mg.case()
    c.mg_cop = c.mg_cop_part = None
    return c


def _coarse_solve(mg, c, rhs):
    from warpflow import _abi
    lev = mg.levels[1]
    lev.rhs.assign(rhs)
    lev.phi.zero_()
    _abi.call("wf_mg_coarse_solve", ctypes.byref(c), lev.phi.ptr, lev.rhs.ptr, mg._stream())
    return lev.phi.numpy()[1:-1, 1:-1, 1:-1]


def _rhs(nc, seed):
    out = np.zeros((nc + 2,) * 3)
    core = np.random.default_rng(seed).standard_normal((nc,) * 3)
    out[1:-1, 1:-1, 1:-1] = core - core.mean()
    return out


@pytest.mark.parametrize("nc", EDGES)
def test_coarse_solve_is_the_vcycles(nc):
    from warpflow import _abi
    mg = _mg(nc)
    mg.n_pre = mg.n_post = 0
    c = _no_operator(mg)
    lev0, lev1 = mg.levels
    lev0.rhs.assign(np.random.default_rng(nc).standard_normal(lev0.shape))
    lev0.phi.zero_()
    _abi.call("wf_mg_vcycle", ctypes.byref(c), lev0.phi.ptr, lev0.rhs.ptr, mg._stream())
    want = lev1.phi.numpy()[1:-1, 1:-1, 1:-1]
    got = _coarse_solve(mg, c, lev1.rhs.numpy())
    assert np.abs(want).max() > 0
    np.testing.assert_array_equal(got, want)
