"""The coarsest relax from zero of an FP64 level without an operator, summed as
a polynomial of the sweep map, against the sweeps themselves: every edge it
serves, unequal spacings, and sweep counts on both sides of where it applies."""
import numpy as np
import pytest

from helpers import make_cfg

pytestmark = pytest.mark.gpu

HS = (1.0, 0.9, 1.1)


def _coarse(nc, n_coarse):
    from warpflow import Multigrid, build_topology
    h = 1.0 / (2 * nc)
    mg = Multigrid(make_cfg(2 * nc, levels=2), build_topology(make_cfg(2 * nc, levels=2)),
                   "cuda:0", *(h * x for x in HS), coarse="sweeps")
    mg.n_coarse = n_coarse
    rng = np.random.default_rng(nc)
    rhs = np.zeros((nc + 2,) * 3)
    core = rng.standard_normal((nc,) * 3)
    rhs[1:-1, 1:-1, 1:-1] = core - core.mean()
    mg.levels[1].rhs.assign(rhs)
    mg._coarse_solve()
    got = mg.levels[1].phi.numpy()
    one = Multigrid(make_cfg(nc, levels=1), build_topology(make_cfg(nc, levels=1)), "cuda:0",
                    *(2 * h * x for x in HS))
    one.levels[0].rhs.assign(rhs)
    one.levels[0].phi.zero_()
    for part in [12] * (n_coarse // 12) + [n_coarse % 12]:    # few at a time: plain sweeps
        one._relax(0, part)
    return got, one.levels[0].phi.numpy()


# 300 sweeps round at most 300 times: 300 ulp of the solution's size
@pytest.mark.parametrize("nc", [10, 12, 14, 16, 18, 20, 22, 24, 26, 28, 30, 32])
def test_polynomial_equals_the_sweeps(nc):
    got, ref = _coarse(nc, 300)
    assert np.abs(got - ref).max() <= 300 * 2.3e-16 * np.abs(ref).max()


@pytest.mark.parametrize("n_coarse", [63, 64, 150, 600, 1500])
def test_sweep_counts(n_coarse):
    got, ref = _coarse(18, n_coarse)
    assert np.abs(got - ref).max() <= max(n_coarse, 100) * 2.3e-16 * np.abs(ref).max()


@pytest.mark.parametrize("nc", [10, 18, 24])
def test_solve_same_bits_alone_and_in_a_bucket(nc):
    import ctypes
    import torch
    from warpflow import Multigrid, _abi, build_topology
    from warpflow.fields import DeviceField
    n = 4 * nc
    cases, pps, keep = [], [], []
    for q in range(3):
        mg = Multigrid(make_cfg(n), build_topology(make_cfg(n)), "cuda:0", 1.0 / n, 1.0 / n,
                       1.0 / n, coarse="sweeps")
        su = DeviceField.zeros((n + 6,) * 3, "cuda:0")
        pp = DeviceField.zeros((n + 6,) * 3, "cuda:0")
        su.assign(np.random.default_rng(q).standard_normal((n + 6,) * 3))
        c = mg.case(su=su, pp=pp)
        for i in range(len(_abi.FIELD_NAMES)):
            c.fld[i] = c.fld[i] or su.ptr
        cases.append(c)
        pps.append(pp)
        keep.append((mg, su))
    alone = []
    for c, pp in zip(cases, pps):
        _abi.call("wf_mg_solve", ctypes.byref(c), keep[0][0]._stream())
        alone.append(pp.numpy())
    size = ctypes.c_int64()
    _abi.call("wf_mg_bucket_table_bytes", 3, ctypes.byref(size))
    table = torch.zeros(size.value, dtype=torch.uint8, device="cuda:0")
    _abi.call("wf_mg_solve_bucket", (_abi.WfCase * 3)(*cases), 3, table.data_ptr(),
              keep[0][0]._stream())
    for a, pp in zip(alone, pps):
        np.testing.assert_array_equal(a, pp.numpy())
