"""Coarsest edges without an operator or a strategy of their own (10, 14, 18,
22, 26, 30) run many sweeps in a thread-block cluster: the bits are those of
the kernels that run few sweeps of the same level (FP64), and of the one-CTA
relax that a bucket uses (FP32)."""
import ctypes

import numpy as np
import pytest

from helpers import make_cfg

pytestmark = pytest.mark.gpu

EDGES = [6, 10, 14, 18, 22, 26, 30]


def _mg(n, levels, precision):
    from warpflow import Multigrid, build_topology
    cfg = make_cfg(n, levels=levels, precision=precision)
    return Multigrid(cfg, build_topology(cfg), "cuda:0", 1.0 / n, 0.9 / n, 1.1 / n)


@pytest.mark.parametrize("n", EDGES)
def test_many_sweeps_equal_few_at_a_time(n):
    mg = _mg(n, 1, "fp64")
    rng = np.random.default_rng(n)
    phi = rng.standard_normal((n + 2,) * 3)
    mg.levels[0].rhs.assign(rng.standard_normal((n + 2,) * 3))
    out = []
    for parts in ((25,), (12, 12, 1)):
        mg.levels[0].phi.assign(phi)
        for k in parts:
            mg._relax(0, k)
        out.append(mg.levels[0].phi.numpy())
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("n", [4 * e for e in EDGES])
def test_mixed_solve_equals_the_bucket_form(n):
    from warpflow import _abi
    from warpflow.fields import DeviceField
    import torch
    mg = _mg(n, 3, "mixed")
    su = DeviceField.zeros((n + 6,) * 3, "cuda:0")
    pp = DeviceField.zeros((n + 6,) * 3, "cuda:0")
    su.assign(np.random.default_rng(n).standard_normal((n + 6,) * 3))
    c = mg.case(su=su, pp=pp)
    for i in range(len(_abi.FIELD_NAMES)):
        c.fld[i] = c.fld[i] or su.ptr
    _abi.call("wf_mg_solve", ctypes.byref(c), mg._stream())
    a = pp.numpy()
    size = ctypes.c_int64()
    _abi.call("wf_mg_bucket_table_bytes", 1, ctypes.byref(size))
    table = torch.zeros(size.value, dtype=torch.uint8, device="cuda:0")
    _abi.call("wf_mg_solve_bucket", ctypes.byref(c), 1, table.data_ptr(), mg._stream())
    np.testing.assert_array_equal(a, pp.numpy())
