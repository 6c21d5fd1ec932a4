"""The routes a relax can take, where they could part: split copies of the
smallest edges."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

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
