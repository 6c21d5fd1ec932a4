"""The half-sweeps on the row-parity-split copy -- with the cells numbered flat
(levels from 64 to below 104 cells, one or two cells per thread), by rows, and
in pairs marching through planes (multiples of 4 from 144) -- give the bits of
the in-place half-sweeps, in both precisions and at the edges of each range;
the in-place ones follow the oracle's sweeps."""
import ctypes

import numpy as np
import pytest

from helpers import make_cfg
from oracle import wf_oracle as O

pytestmark = pytest.mark.gpu


def _mg(n, levels, precision):
    from warpflow import Multigrid, build_topology
    cfg = make_cfg(n, levels=levels, precision=precision)
    return Multigrid(cfg, build_topology(cfg), "cuda:0", 1.0 / n, 1.0 / n, 1.0 / n)


@pytest.mark.parametrize("n", [62, 64, 66, 84, 86, 102, 104, 106, 140, 144, 146, 172, 176,
                               180, 260])
def test_relax_on_split_copy_equals_in_place(n):
    mg = _mg(n, 1, "fp64")
    rng = np.random.default_rng(n)
    phi = rng.standard_normal((n + 2,) * 3)
    rhs = rng.standard_normal((n + 2,) * 3)
    out = []
    for tmp in (mg._tmp64, None):       # without the scratch the level relaxes in place
        mg._tmp64 = tmp
        mg.levels[0].phi.assign(phi)
        mg.levels[0].rhs.assign(rhs)
        mg._relax(0, 3)
        out.append(mg.levels[0].phi.numpy())
    real = np.s_[1:-1, 1:-1, 1:-1]
    np.testing.assert_array_equal(out[0][real], out[1][real])


@pytest.mark.parametrize("n", [28, 33, 45, 64])
def test_relax_in_place_follows_the_oracle(n):
    mg = _mg(n, 1, "fp64")
    mg._tmp64 = None
    rng = np.random.default_rng(n)
    lev = O.Level(n, 1.0 / n, 1.0 / n, 1.0 / n)
    lev.phi[...] = rng.standard_normal(lev.phi.shape)
    lev.rhs[...] = rng.standard_normal(lev.rhs.shape)
    mg.levels[0].phi.assign(lev.phi)
    mg.levels[0].rhs.assign(lev.rhs)
    mg._relax(0, 2)
    for _ in range(2):
        O.rbgs(lev, 0)
        O.rbgs(lev, 1)
        O.mg_refill(lev.phi, n)
    got = mg.levels[0].phi.numpy()
    # a handful of roundings per update, contracted sums: 4 half-sweeps
    assert np.abs(got - lev.phi)[1:-1, 1:-1, 1:-1].max() <= 1e-14 * np.abs(lev.phi).max()


@pytest.mark.parametrize("n,levels", [(64, 3), (80, 3), (96, 3), (128, 4), (144, 4), (184, 4),
                                      (256, 5)])
def test_mixed_solve_on_split_copies_equals_in_place(n, levels):
    from warpflow import _abi
    from warpflow.fields import DeviceField
    mg = _mg(n, levels, "mixed")
    su = DeviceField.zeros((n + 6,) * 3, "cuda:0")
    pp = DeviceField.zeros((n + 6,) * 3, "cuda:0")
    su.assign(np.random.default_rng(n).standard_normal((n + 6,) * 3))
    out = []
    for split in (True, False):
        c = mg.case(su=su, pp=pp)
        for i in range(len(_abi.FIELD_NAMES)):
            c.fld[i] = c.fld[i] or su.ptr
        if not split:
            for l in range(levels):
                c.mg_tmp[l] = None
        _abi.call("wf_mg_solve", ctypes.byref(c), mg._stream())
        out.append(pp.numpy())
    np.testing.assert_array_equal(out[0], out[1])
