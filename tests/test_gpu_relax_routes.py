"""The routes a relax can take, where they could part: split copies of the
smallest edges, infinities, a ring that was never set, one CTA and launches."""
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


RING_EDGES = [11, 13, 14, 15, 17, 18, 19, 20, 21, 22, 23, 24]


def _nan_ring(a, n):
    out = np.full((n + 2,) * 3, np.nan)
    out[1:-1, 1:-1, 1:-1] = a[1:-1, 1:-1, 1:-1]
    return out


@pytest.mark.parametrize("sweeps", [1, 6, 13])
@pytest.mark.parametrize("n", RING_EDGES)
def test_relax_needs_no_ring(n, sweeps):
    """Up to 24 cells the ring of phi may hold anything: the same cells and the
    same ring come out as with the mirrors in it, from the host and in a graph."""
    import torch
    mg = _mg(n)
    rng = np.random.default_rng(n)
    phi = rng.standard_normal((n + 2,) * 3)
    O.mg_refill(phi, n)
    mg.levels[0].rhs.assign(rng.standard_normal((n + 2,) * 3))
    real = np.s_[1:-1, 1:-1, 1:-1]
    out = []
    for start in (phi, _nan_ring(phi, n)):
        mg.levels[0].phi.assign(start)
        mg._relax(0, sweeps)
        out.append(mg.levels[0].phi.numpy())
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            mg._relax(0, sweeps)
        mg.levels[0].phi.assign(_nan_ring(phi, n))
        g.replay()
        s.synchronize()
        out.append(mg.levels[0].phi.numpy())
    assert np.isfinite(out[0]).all()
    for o in out[1:]:
        np.testing.assert_array_equal(o[real], out[0][real])
        for sl in (np.s_[:, 1:-1, 1:-1], np.s_[1:-1, :, 1:-1], np.s_[1:-1, 1:-1, :]):
            np.testing.assert_array_equal(o[sl], out[0][sl])


@pytest.mark.parametrize("n,levels", [(14, 1), (14, 2), (18, 2), (20, 2), (24, 2), (24, 3),
                                      (13, 1)])
def test_vcycle_needs_no_ring(n, levels):
    mg = _mg(n, levels)
    rng = np.random.default_rng(n)
    phi = rng.standard_normal((n + 2,) * 3)
    O.mg_refill(phi, n)
    mg.levels[0].rhs.assign(rng.standard_normal((n + 2,) * 3))
    out = []
    for start in (phi, _nan_ring(phi, n)):
        mg.levels[0].phi.assign(start)
        mg._vcycle()
        out.append(mg.levels[0].phi.numpy()[1:-1, 1:-1, 1:-1])
    assert np.isfinite(out[0]).all()
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("n", [11, 12, 14, 15, 16, 17, 20, 24])
def test_one_sweep_at_a_time_equals_all(n):
    """One CTA, launches and clusters: 13 sweeps at once, one at a time, and
    recorded in a graph are the same bits off the multiples of four, and the
    same to rounding on them (which multiply by the diagonal's reciprocal)."""
    import torch
    mg = _mg(n)
    rng = np.random.default_rng(n)
    phi = rng.standard_normal((n + 2,) * 3)
    mg.levels[0].rhs.assign(rng.standard_normal((n + 2,) * 3))
    out = []
    for parts in ((13,), (1,) * 13, (6, 7)):
        mg.levels[0].phi.assign(phi)
        for k in parts:
            mg._relax(0, k)
        out.append(mg.levels[0].phi.numpy()[1:-1, 1:-1, 1:-1])
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            mg._relax(0, 13)
        mg.levels[0].phi.assign(phi)
        g.replay()
        s.synchronize()
        out.append(mg.levels[0].phi.numpy()[1:-1, 1:-1, 1:-1])
    for o in out[1:]:
        if n % 4:
            np.testing.assert_array_equal(o, out[0])
        else:   # 26 half-sweeps of two roundings each from the other form
            assert np.abs(o - out[0]).max() <= 26 * 4.4e-16 * np.abs(out[0]).max()


def test_odd_coarsest_level_from_the_host_and_in_a_graph():
    """The 300 sweeps of a 13^3 coarsest level: one launch each when the host
    issues them, 600 in a graph, where a launch costs less; the same fields."""
    import ctypes
    from warpflow import FlowSolver, _abi, build_topology
    counts, fields = [], []
    for mode in ("host", "graph"):
        sol = FlowSolver(make_cfg(52), build_topology(make_cfg(52)), "cuda:0", step_mode=mode)
        for _ in range(2):
            sol.step()
        c = (ctypes.c_int32 * 4)()
        _abi.call("wf_stepper_launch_counts", sol._stepper, c)
        counts.append(c[2])
        fields.append([sol.f[k].numpy() for k in ("u", "v", "w", "p", "pp")])
        sol.close()
    assert counts[0] < 300 and counts[1] - counts[0] == 4 * 599
    for a, b in zip(*fields):
        np.testing.assert_array_equal(a, b)


def test_bucket_keeps_one_cta_for_a_small_coarsest_level():
    """The 14^3 coarsest level of a mixed bucket: one launch for its 300 sweeps,
    and the fields of the cases alone (which sweep in a cluster)."""
    from warpflow import FlowSolver, build_topology
    from warpflow.ensemble import Ensemble, cavity_case
    cfgs = [cavity_case(56, re, 1.0, precision="mixed") for re in (200.0, 900.0)]
    ens = Ensemble(cfgs, nstreams=1, buckets=True)
    assert ens.layout()[1][0][2] < 600          # launches of the multigrid part
    alone = [FlowSolver(c, build_topology(c), "cuda:0") for c in cfgs]
    for _ in range(2):
        assert ens.step() == [s.step() for s in alone]
    for sol, ref in zip(ens.solvers, alone):
        for name in ("u", "v", "w", "p"):
            np.testing.assert_array_equal(sol.f[name].numpy(), ref.f[name].numpy())
    ens.close()


def test_long_coarse_relaxes_leave_the_chip_to_other_cases():
    """Six cases with an 11^3 coarsest level side by side: their long one-CTA
    relaxes run beside one another and beside the other kernels, so a step of
    all takes little longer than a step of one (1.1 times; 1.4 when the kernels
    behind a relax held SMs while it ran)."""
    import torch
    from warpflow.ensemble import Ensemble, cavity_case

    def step_ms(ens):
        for _ in range(3):
            ens.launch()
        best = 1e9
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ens.launch()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    cfgs = [cavity_case(44, 200.0 + 50.0 * q, 1.0, precision="fp64") for q in range(6)]
    one = Ensemble(cfgs[:1], nstreams=1, buckets=False)
    six = Ensemble(cfgs, nstreams=1, buckets=False)
    assert step_ms(six) < 1.25 * step_ms(one)
    one.close()
    six.close()
