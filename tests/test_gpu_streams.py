"""What calls leave behind on a caller's stream that lives on (GPU)."""
import time

import numpy as np
import pytest

import mgcfd
from mgcfd import ops

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _create_seconds():
    """Median set-up time of a small mesh, which allocates some hundred blocks."""
    mesh = mgcfd.HostMesh.generate(17, 3, 5)
    t = []
    for _ in range(9):
        torch.cuda.synchronize()
        a = time.perf_counter()
        s = mgcfd.Solver(mesh, 0.5, 3.0)
        t.append(time.perf_counter() - a)
        s.close()
    return sorted(t)[4]


def _streams(count=32):
    """Live streams, each with a launch in plain order behind it."""
    streams = [torch.cuda.Stream() for _ in range(count)]
    x = torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    for q in streams:
        with torch.cuda.stream(q):
            x.add_(1)
    torch.cuda.synchronize()
    return streams


@pytest.mark.parametrize("form", ["fp64", "dw"])
def test_plans_built_on_live_streams_leave_setup_alone(form):
    """Plans built on 32 streams by programs that make flux calls and residuals
    alone: a later set-up takes what it took before.  (It took 5 times as long
    while the plans' work memory was given back with no plain launch after it;
    twice is the line.)"""
    L = mgcfd.HostMesh.generate(24, 1, 5).levels()[0]
    n = L.nnodes
    var = torch.ones(n, 5, dtype=torch.float64, device="cuda")
    var[:, 4] = 5.0
    old, res, flux = torch.ones_like(var), torch.ones_like(var), torch.zeros_like(var)
    ewt = torch.from_numpy(np.array(L.edge_weights)).cuda()
    streams = _streams()
    maps = [torch.from_numpy(np.array(L.edge_to_nodes)).cuda() for _ in streams]
    before = _create_seconds()
    ops.flux_precision(form)
    try:
        for q, e in zip(streams, maps):
            ops.compute_flux_edge(L.nedges, n, e.data_ptr(), var.data_ptr(), ewt.data_ptr(), 0.1, flux.data_ptr(),
                                  q.cuda_stream)
            ops.residual(n, old.data_ptr(), var.data_ptr(), res.data_ptr(), q.cuda_stream)
        torch.cuda.synchronize()
        after = _create_seconds()
    finally:
        ops.flux_precision("fp64")
        for e in maps:
            ops.plan_release(e.data_ptr())
    assert after < 2 * before, (before, after)


@pytest.mark.parametrize("use_graph", [True, False])
def test_solvers_closed_on_live_streams_leave_setup_alone(use_graph):
    """Solvers closed on 32 streams of the caller's, run from their graph or
    launch by launch: a later set-up takes what it took before (it took 5 times
    as long; twice is the line)."""
    mesh = mgcfd.HostMesh.generate(24, 3, 6)
    streams = _streams()
    before = _create_seconds()
    for q in streams:
        s = mgcfd.Solver(mesh, 0.5, 3.0, precision="mixed", use_graph=use_graph, stream=q.cuda_stream)
        s.run(4)
        assert s.synchronize() == 0
        s.close()
    after = _create_seconds()
    assert after < 2 * before, (before, after)
