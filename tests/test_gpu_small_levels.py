"""Small levels (one CTA's shared memory up to 10, 12, 16, and FP32 20 and 24;
a launch per half-sweep above): a relax follows the oracle's sweeps, and
V-cycles whose levels take each of these forms -- with phi known to be zero on
the way down and the rhs read early on the way up -- follow the oracle's."""
import numpy as np
import pytest

from helpers import make_cfg
from oracle import wf_oracle as O

pytestmark = pytest.mark.gpu


def _mg(n, levels, precision="fp64"):
    from warpflow import Multigrid, build_topology
    cfg = make_cfg(n, levels=levels, precision=precision)
    return Multigrid(cfg, build_topology(cfg), "cuda:0", 1.0 / n, 1.0 / n, 1.0 / n)


@pytest.mark.parametrize("sweeps", [1, 6])
@pytest.mark.parametrize("n", [4, 7, 8, 10, 11, 12, 16, 19, 20, 22, 24])
def test_small_relax_follows_the_oracle(n, sweeps):
    mg = _mg(n, 1)
    rng = np.random.default_rng(n)
    omg = O.Multigrid(n, 1, 1.0 / n, 1.0 / n, 1.0 / n)
    lev = omg.levels[0]
    lev.phi[...] = rng.standard_normal(lev.phi.shape)
    lev.rhs[...] = rng.standard_normal(lev.rhs.shape)
    O.mg_refill(lev.phi, n)
    mg.levels[0].phi.assign(lev.phi)
    mg.levels[0].rhs.assign(lev.rhs)
    mg._relax(0, sweeps)
    omg.relax(0, sweeps)
    got = mg.levels[0].phi.numpy()
    # the face rings (edges and corners enter no stencil)
    for s in (np.s_[:, 1:-1, 1:-1], np.s_[1:-1, :, 1:-1], np.s_[1:-1, 1:-1, :]):
        # at most 12 updates in a row of about 8 roundings each
        assert np.abs(got - lev.phi)[s].max() <= 2e-14 * np.abs(lev.phi).max()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-4)])
@pytest.mark.parametrize("n,levels", [(32, 3), (40, 3), (44, 3), (48, 3), (72, 4), (80, 4)])
def test_vcycles_over_small_levels_follow_the_oracle(n, levels, precision, tol):
    mg = _mg(n, levels, precision)
    rng = np.random.default_rng(n)
    omg = O.Multigrid(n, levels, 1.0 / n, 1.0 / n, 1.0 / n)
    lev = omg.levels[0]
    rhs = rng.standard_normal((n,) * 3)
    lev.rhs[1:-1, 1:-1, 1:-1] = rhs - rhs.mean()
    mg.levels[0].rhs.assign(lev.rhs)
    mg.levels[0].phi.zero_()
    for _ in range(2):
        mg._vcycle()
        omg.vcycle()
    got = mg.levels[0].phi.numpy()[1:-1, 1:-1, 1:-1]
    ref = lev.phi[1:-1, 1:-1, 1:-1]
    # fp64: roundings of 300 coarse sweeps; mixed: those of an FP32 V-cycle
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
