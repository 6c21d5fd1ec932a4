"""Prolongation forms (a fine cell per thread, a coarse cell per thread, coarse
cells marching along i with a remainder) and their one-colour variants, and the
first half-sweep made by the kernel that writes a level's rhs: V-cycles of few
sweeps follow the oracle's."""
import numpy as np
import pytest

from helpers import make_cfg
from oracle import wf_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pre,n_post", [(1, 0), (0, 1), (2, 1)])
@pytest.mark.parametrize("n,levels", [(36, 2), (44, 3), (64, 2), (66, 2), (128, 3), (160, 2),
                                      (208, 2)])
def test_vcycle_of_few_sweeps_follows_the_oracle(n, levels, n_pre, n_post):
    from warpflow import Multigrid, build_topology
    cfg = make_cfg(n, levels=levels)
    h = 1.0 / n
    mg = Multigrid(cfg, build_topology(cfg), "cuda:0", h, h, h, coarse="sweeps")
    omg = O.Multigrid(n, levels, h, h, h)
    for m in (mg, omg):
        m.n_pre, m.n_post, m.n_coarse = n_pre, n_post, 2
    rng = np.random.default_rng(n)
    lev = omg.levels[0]
    lev.rhs[1:-1, 1:-1, 1:-1] = rng.standard_normal((n,) * 3)
    lev.phi[...] = rng.standard_normal(lev.phi.shape) / n ** 2
    O.mg_refill(lev.phi, n)
    mg.levels[0].rhs.assign(lev.rhs)
    mg.levels[0].phi.assign(lev.phi)
    for _ in range(2):
        mg._vcycle()
        omg.vcycle()
    got = mg.levels[0].phi.numpy()
    # a few dozen updates of about 8 roundings each
    assert np.abs(got - lev.phi)[1:-1, 1:-1, 1:-1].max() <= 1e-13 * np.abs(lev.phi).max()
