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


def _launched(mesh, steps=1):
    """Names of the stage kernels a run launches, as CUPTI records them."""
    from torch.profiler import ProfilerActivity, profile
    ndg.Solver2D_t.run(mesh, steps)
    mesh.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        ndg.Solver2D_t.run(mesh, steps)
        mesh.synchronize()
    names = [e.name for e in prof.events() if "stage_kernel" in e.name]
    return {n.replace("void ", "").replace("ndg::dev::", "").split("(")[0] for n in names}


def _is(name, launched):
    """stage_kernel() leaves out the line kernel's argument type."""
    return len(launched) == 1 and (launched == {name} or next(iter(launched)).startswith(name[:-1] + ", "))


@pytest.mark.parametrize("precision", [ndg.FP64, ndg.FP32])
@pytest.mark.parametrize("N,res", [(3, 8), (6, 40), (6, 8), (8, 40), (10, 40)])
def test_tiles_are_those_of_the_kernel_that_runs(N, res, precision):
    """With keep_derivative the three-threads-a-line kernel runs, so its tiles
    are the candidates and take effect; without, the line kernel's where it
    runs. Switching keeps a tile that both kernels have, and the fields do not
    depend on any of it beyond rounding (4 steps; the bounds of
    tests/test_gpu_line_stage.py)."""
    tol = 1e-13 if precision == ndg.FP64 else 2e-6
    mesh = ndg.Mesh2D_t(meshgen.uniform_zone(res, boundary=meshgen.WALL, jitter=0.1, seed=2, order="rowmajor"), N, precision=precision)
    rng = np.random.default_rng(N)
    start = [rng.standard_normal(mesh.field_size) for _ in FIELDS]

    def fields():
        for f, v in zip(FIELDS, start):
            mesh.set_field(f, v)
        ndg.Solver2D_t.run(mesh, 4)
        return _get(mesh)

    reference = fields()
    line = N <= 4 or res >= 40
    assert mesh.stage_kernel().startswith("line_stage_kernel" if line else "stage_kernel")
    seen = {}
    for keep in (1, 0, 1):
        assert ndg.lib().ndg_ctx_keep_derivative(mesh.handle, keep) == 0
        candidates, default = mesh.tile_candidates()
        mesh.set_tile(0)
        names = {mesh.stage_kernel()}
        for tile in candidates:
            mesh.set_tile(tile)
            name = mesh.stage_kernel()
            names.add(name)
            assert name.startswith("line_") == (line and not keep and tile < ndg.TENSOR_TILE), (keep, tile, name)
            assert _is(name, _launched(mesh)), (keep, tile, name)
            got = fields()
            assert np.linalg.norm(got - reference) <= tol * np.linalg.norm(reference), (keep, tile)
        assert len(names) >= len(candidates)  # every tile is a kernel of its own; the default may be one of them
        assert default > 0
        seen[keep] = candidates
    assert set(seen[1]) <= set(seen[0])
    # 4 elements: a tile of both kernels; 16 at order 10: only the line kernel's
    mesh.set_tile(4)
    assert ndg.lib().ndg_ctx_keep_derivative(mesh.handle, 0) == 0
    assert ", 4" in mesh.stage_kernel()
    extra = sorted(set(seen[0]) - set(seen[1]))
    if extra:
        mesh.set_tile(extra[-1])
        assert ndg.lib().ndg_ctx_keep_derivative(mesh.handle, 1) == 0
        assert ", 0, false>" in mesh.stage_kernel()
    got = fields()
    assert np.linalg.norm(got - reference) <= tol * np.linalg.norm(reference)
    tile, ms = mesh.autotune(3)
    assert ms > 0 and (tile == 0 or tile in mesh.tile_candidates()[0])
    mesh.close()


@pytest.mark.parametrize("kind", ["uniform", "uniform fp32", "mixed", "mixed fp32", "adjoint"])
def test_a_mesh_of_lower_order_loaded_meanwhile_changes_nothing(kind):
    """Kernels take their order's coefficients from tables that every context
    shares; another context's mesh of lower orders must not take them away,
    from launches, captures of a later run, estimates or the adjoint."""
    zone = meshgen.uniform_zone(8, boundary=meshgen.WALL)
    precision = ndg.FP32 if "fp32" in kind else ndg.FP64

    def low():
        m = ndg.Mesh2D_t(zone, 2)
        m.initial_conditions()
        ndg.Solver2D_t.run(m, 1)
        m.synchronize()
        m.close()

    results = []
    for between in (lambda: None, low):
        m = ndg.Mesh2D_t(zone, 5, maximum_N=9, precision=precision, tolerance_min=1e-12)
        m.initial_conditions()
        if kind == "adjoint":
            adj = ndg.Adjoint2D_t(m, [[0.3, 0.2]])
            p0 = m.get_field("p")
            dt = adj.delta_t(0.5)
            out = []
            for _ in range(2):
                between()
                out += [adj.forward(p0, dt, 3, targets=np.zeros((4, 1)))[1].ravel(), adj.backward()["c"]]
            adj.close()
        else:
            if "mixed" in kind:
                between()
                m.adapt((np.arange(64) % 2).astype(np.int32), np.full(64, 2.0))
            t = ndg.Solver2D_t.run(m, 8)
            between()
            t = ndg.Solver2D_t.run(m, 1, t)  # a run that captures anew
            between()
            ndg.Solver2D_t.stage(m, 1, t, 1e-3)
            between()
            m.estimate_error()
            out = [m.get_field(f) for f in ("p", "u", "v", "k_p")] + [m.error()[k] for k in ("p_error", "p_sigma")]
        m.close()
        results.append(np.concatenate(out))
    assert np.isfinite(results[0]).all() and np.linalg.norm(results[0]) > 0
    assert np.array_equal(results[0], results[1])


@pytest.mark.parametrize("precision", [ndg.FP64, ndg.FP32])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_a_mixed_mesh_with_smaller_tiles_loaded_meanwhile_changes_nothing(mode, precision):
    """Split meshes need larger mixed-order tiles than p-adapted ones of the
    same orders; the kernels' shared-memory limit is one for all contexts."""
    zone = meshgen.uniform_zone(8, boundary=meshgen.WALL)

    def mixed(split):
        m = ndg.Mesh2D_t(zone, 8, maximum_N=12, max_split_level=2 if split else 0, precision=precision)
        m.set_mixed_launch(mode)
        m.initial_conditions()
        for _ in range(2):
            K = m.n_elements_
            m.adapt((np.arange(K) % 3 == 0).astype(np.int32), np.where(np.arange(K) % 2 == 0, 0.5, 2.0) if split else np.full(K, 2.0))
        return m

    results = []
    for between in (False, True):
        m = mixed(True)
        t = ndg.Solver2D_t.run(m, 1)
        if between:
            other = mixed(False)
            ndg.Solver2D_t.run(other, 1)
            other.synchronize()
            other.close()
        t = ndg.Solver2D_t.run(m, 2, t)  # captures the graph of the other parity
        ndg.Solver2D_t.stage(m, 1, t, 1e-4)
        results.append(_get(m))
        m.close()
    assert np.isfinite(results[0]).all() and np.array_equal(results[0], results[1])


_TABLES_FIRST = """
import sys
import numpy as np
import ndg_cuda_b200 as ndg
from tests import meshgen

if sys.argv[1] == "tables":
    class Context(ndg._Context):
        def __init__(self, *args):
            super().__init__(*args)
            assert ndg.lib().ndg_tables_build(self.h, 9, 2) == 0
    ndg._Context = Context
m = ndg.Mesh2D_t(meshgen.uniform_zone(8, boundary=meshgen.WALL), 4, maximum_N=8)
m.initial_conditions()
m.adapt((np.arange(64) % 2).astype(np.int32), np.full(64, 2.0))
ndg.Solver2D_t.run(m, 3)
np.save(sys.argv[2], np.concatenate([m.get_field(f) for f in "puv"]))
"""


def test_tables_built_before_the_mesh_serve_mixed_orders(tmp_path):
    """ndg_tables_build, then a mesh in the same context, which uses those
    tables and becomes a mixed-order one; in processes that load nothing else."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = []
    for how in ("mesh", "tables"):
        path = str(tmp_path / f"{how}.npy")
        subprocess.run([sys.executable, "-c", _TABLES_FIRST, how, path], check=True, cwd=root, capture_output=True, text=True, timeout=300)
        out.append(np.load(path))
    assert np.isfinite(out[0]).all() and np.linalg.norm(out[0]) > 0
    assert np.array_equal(out[0], out[1])
