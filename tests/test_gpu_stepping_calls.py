"""What a stepping call leaves to its caller: finished uploads, an unaffected
capture, the step state that later launches read, and the kernel it runs.

Comparisons are of the same arithmetic in another order of calls, so they are
exact unless a test says otherwise.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

import ndg_cuda_b200 as ndg
from tests import meshgen

pytestmark = pytest.mark.gpu

FIELDS = ("p", "u", "v")


def _get(mesh):
    return np.concatenate([mesh.get_field(f) for f in FIELDS])


@pytest.mark.parametrize("call", ["run", "stage", "solve"])
def test_a_pinned_buffer_may_be_reused_when_a_stepping_call_returns(call):
    """255 MB of uploads (5 ms) are on the stream when the call is made; what
    the host writes into their buffers after it must not reach the device."""
    zone = meshgen.uniform_zone(64, x_periodic=True, y_periodic=True)
    m = ndg.Mesh2D_t(zone, 8, n_instances=8)
    L, dt = ndg.lib(), ndg.Solver2D_t.get_delta_t(m)
    n = m.field_size * m.n_instances
    rng = np.random.default_rng(0)
    values = [torch.from_numpy(rng.standard_normal(n)) for _ in FIELDS]
    pinned = [torch.empty(n, dtype=torch.float64, pin_memory=True) for _ in FIELDS]
    results = []
    for overwrite in (False, False, True):  # the first pass also captures the graphs
        for b, v in zip(pinned, values):
            b.copy_(v)
        for _ in range(4):
            for i, b in enumerate(pinned):
                assert L.ndg_set_field(m.handle, -1, i, b.data_ptr()) == 0
        if call == "run":
            ndg.Solver2D_t.run(m, 1)
        elif call == "stage":
            ndg.Solver2D_t.stage(m, 0, 0.0, dt)
        else:  # the wrapper's solve sets the CFL number first, which waits
            t, steps = C.c_double(0.0), C.c_int64()
            assert L.ndg_solve(m.handle, 0.5 * dt, C.byref(t), C.byref(steps)) == 0
        if overwrite:
            for b in pinned:
                b.fill_(7.0)
        results.append(_get(m))
    m.close()
    assert np.array_equal(results[1], results[0])
    assert np.array_equal(results[2], results[0])


def test_a_stepping_call_on_a_capturing_stream_is_refused():
    """And leaves the capture usable."""
    zone = meshgen.uniform_zone(16, x_periodic=True, y_periodic=True)
    stream = torch.cuda.Stream()
    m = ndg.Mesh2D_t(zone, 4, stream=stream.cuda_stream)
    m.initial_conditions()
    ndg.Solver2D_t.run(m, 9)
    m.synchronize()
    before = _get(m)
    x = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        x += 1
        for call in (lambda: ndg.Solver2D_t.run(m, 9), lambda: ndg.Solver2D_t.run(m, 0), lambda: ndg.Solver2D_t.stage(m, 1, 0.0, 1e-3)):
            with pytest.raises(ndg.NdgError, match="captured"):
                call()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, torch.ones_like(x))
    assert np.array_equal(_get(m), before)
    m.close()


@pytest.mark.parametrize("N", [3, 6])
@pytest.mark.parametrize("steps", [0, 1, 2, 9])
def test_timed_stages_run_at_the_state_the_last_call_left(N, steps):
    """ndg_time_stage's launches are stages at the time and step the last
    stepping call left (the inflow boundary takes its values from them), in a
    row, after autotuning and after the mesh became a mixed-order one."""
    zone = meshgen.uniform_zone(12, order="rowmajor", boundary=meshgen.INFLOW, x_min=0.0, x_max=1.0, y_min=0.0, y_max=1.0)
    K = 144

    def after(mesh):
        mesh.initial_conditions()
        return ndg.Solver2D_t.run(mesh, steps, 0.1)

    a, b = (ndg.Mesh2D_t(zone, N, maximum_N=N + 2) for _ in range(2))
    dt = ndg.Solver2D_t.get_delta_t(a)

    def compare(t, m, n):
        a.time_stage(m, n)
        for _ in range(n):
            ndg.Solver2D_t.stage(b, m, t, dt)
        assert np.array_equal(_get(a), _get(b)), (m, n)

    t = after(a)
    assert after(b) == t
    for m, n in ((1, 3), (2, 4), (0, 1)):
        compare(t, m, n)
    ndg.Solver2D_t.stage(a, 1, t + 0.3, dt)
    ndg.Solver2D_t.stage(b, 1, t + 0.3, dt)
    compare(t + 0.3, 1, 2)
    a.autotune(3)
    a.set_tile(0)
    compare(t + 0.3, 1, 3)
    t = after(a)
    after(b)
    for mesh in (a, b):
        mesh.adapt((np.arange(K) % 3 == 0).astype(np.int32), np.full(K, 2.0))
    compare(t, 1, 2)
    for mesh in (a, b):
        mesh.close()
