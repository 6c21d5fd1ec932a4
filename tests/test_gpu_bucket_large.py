"""Buckets of levels that relax in pairs and prolong marching through planes: a
case computes the same bits alone and in a bucket, also when the scratch of one
case is aligned to no more than an element (the bucket then keeps to the kernels
that load single elements)."""
import ctypes

import numpy as np
import pytest

from helpers import make_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("odd", [None, 0, 1], ids=["aligned", "first_odd", "second_odd"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [144, 176])
def test_bucket_equals_alone(n, precision, odd):
    import torch
    from warpflow import Multigrid, _abi, build_topology
    from warpflow.fields import DeviceField
    cfg = make_cfg(n, levels=4, precision=precision)
    dt = torch.float32 if precision == "mixed" else torch.float64
    cases, pps, keep = [], [], []
    for q in range(2):
        mg = Multigrid(cfg, build_topology(cfg), "cuda:0", 1.0 / n, 1.0 / n, 1.0 / n)
        mg.n_vcycles = 2
        su = DeviceField.zeros((n + 6,) * 3, "cuda:0")
        pp = DeviceField.zeros((n + 6,) * 3, "cuda:0")
        su.assign(np.random.default_rng(q).standard_normal((n + 6,) * 3))
        c = mg.case(su=su, pp=pp)
        for i in range(len(_abi.FIELD_NAMES)):
            c.fld[i] = c.fld[i] or su.ptr
        if q == odd:
            t = torch.zeros(2 * (n + 2) ** 3 + 1, dtype=dt, device="cuda:0")
            c.mg_tmp[0] = t.data_ptr() + t.element_size()
            keep.append(t)
        cases.append(c)
        pps.append(pp)
        keep.append((mg, su))
    stream = mg._stream()
    alone = []
    for c, pp in zip(cases, pps):
        _abi.call("wf_mg_solve", ctypes.byref(c), stream)
        alone.append(pp.numpy())
    size = ctypes.c_int64()
    _abi.call("wf_mg_bucket_table_bytes", 2, ctypes.byref(size))
    table = torch.zeros(size.value, dtype=torch.uint8, device="cuda:0")
    _abi.call("wf_mg_solve_bucket", (_abi.WfCase * 2)(*cases), 2, table.data_ptr(), stream)
    for a, pp in zip(alone, pps):
        np.testing.assert_array_equal(a, pp.numpy())
