"""The routes a relax can take, where they could part: split copies of the
smallest edges, infinities."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import PKG, ROOT
from helpers import make_cfg
from oracle import wf_oracle as O

pytestmark = pytest.mark.gpu

SOLVE = r"""
import hashlib, sys
sys.path[:0] = [%r, %r, %r]
import numpy as np
from helpers import make_cfg
from warpflow import Multigrid, build_topology
from warpflow.fields import DeviceField
for n, levels in ((4, 2), (12, 3), (12, 2)):     # coarsest 2, 3, 6
    mg = Multigrid(make_cfg(n, levels=levels), build_topology(make_cfg(n)), "cuda:0",
                   1.0 / n, 0.9 / n, 1.1 / n)
    su = DeviceField.zeros((n + 6,) * 3, "cuda:0")
    pp = DeviceField.zeros((n + 6,) * 3, "cuda:0")
    su.assign(np.random.default_rng(n).standard_normal((n + 6,) * 3))
    mg.solve(su, pp, 3)
    print(n, levels, hashlib.sha1(pp.numpy().tobytes()).hexdigest())
""" % (ROOT, PKG, os.path.join(ROOT, "tests"))


def test_split_copies_of_the_smallest_edges():
    """A coarsest level of two cells on the split copy (WF_SPLIT_MIN=2): the
    bits of the default route."""
    out = []
    for extra in ({}, {"WF_SPLIT_MIN": "2"}):
        r = subprocess.run([sys.executable, "-c", SOLVE], capture_output=True, text=True,
                           env=dict(os.environ, **extra), timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        out.append(r.stdout)
    assert out[0] == out[1] and out[0].count("\n") == 3


def _mg(n, levels=1):
    from warpflow import Multigrid, build_topology
    cfg = make_cfg(n, levels=levels)
    return Multigrid(cfg, build_topology(cfg), "cuda:0", 1.0 / n, 1.0 / n, 1.0 / n)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("n", [20, 22, 28, 45, 62, 64, 66, 78])
def test_infinities_stay_infinities(n, sign):
    """An infinite right-hand side: the cells it reaches are the oracle's
    infinities and no NaN, and the other cells the oracle's values (two sweeps
    stay away from the walls, where a zero coefficient meets the infinity)."""
    mg = _mg(n)
    rng = np.random.default_rng(n)
    omg = O.Multigrid(n, 1, 1.0 / n, 1.0 / n, 1.0 / n)
    lev = omg.levels[0]
    lev.rhs[...] = rng.standard_normal(lev.rhs.shape)
    lev.rhs[n // 2, n // 2, n // 2] = sign * np.inf
    mg.levels[0].rhs.assign(lev.rhs)
    mg.levels[0].phi.zero_()
    mg._relax(0, 2)
    with np.errstate(invalid="ignore"):
        omg.relax(0, 2)
    got = mg.levels[0].phi.numpy()[1:-1, 1:-1, 1:-1]
    ref = lev.phi[1:-1, 1:-1, 1:-1]
    fin = np.isfinite(ref)
    assert 1 < (~fin).sum() < 400 and not np.isnan(ref).any()
    np.testing.assert_array_equal(got[~fin], ref[~fin])
    # 4 half-sweeps of a handful of roundings each
    assert np.abs(got[fin] - ref[fin]).max() <= 1e-14 * np.abs(ref[fin]).max()
