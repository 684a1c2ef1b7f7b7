"""The uniform stage kernel with one thread per element line, against the
three-threads-a-line kernel (which keep_derivative selects) and the oracle.

Every order it runs in either form, every boundary kind, one and several
instances, element counts above the size rule (1,536 times the instances) that
are multiples of the tile, odd and ragged; each arm's kernel is checked by
name, and the dispatch on both sides of the rules. Runs of nine steps take an
eight-step graph and a single step. Both kernels evaluate the same operator in
FP64 (or the FP32 form's FP32 part), so the difference after a few steps is
rounding: with n + 1 = N + 2 term sums and a dozen operations per stage, 1e-13
relative L2 leaves a factor of ten over FP64's 2^-53 times the terms and
stages; the FP32 form is held to its own 1e-6 of FP64 on either side, 2e-6
between them.
"""
from __future__ import annotations

import numpy as np
import pytest

import ndg_cuda_b200 as ndg
from oracle.pyoracle import OracleSolver
from tests import meshgen

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


LINE_ORDERS = {ndg.FP64: range(1, 15), ndg.FP32: (1, 2, 3, 4, 5, 6, 8, 10)}
EVERY_SIZE = 4  # orders up to here run it on meshes of any size


def _run(zone, N, precision, keep, fields, n_inst, steps, tiles=(0,)):
    m = ndg.Mesh2D_t(zone, N, precision=precision, n_instances=n_inst, keep_derivative=keep)
    assert m.stage_kernel().startswith("stage_kernel" if keep else "line_stage_kernel")
    out = []
    for tile in tiles:
        m.set_tile(tile)
        for f, v in zip(("p", "u", "v"), fields):
            m.set_field(f, v)
        ndg.Solver2D_t.run(m, steps)
        out.append(np.concatenate([m.get_field(f) for f in ("p", "u", "v", "k_p", "k_u", "k_v")]))
    m.close()
    return out


CASES = [("periodic", 40, 1, 0.1), ("wall", 41, 1, 0.1), ("outflow", 21, 4, 0.0), ("inflow", 41, 1, 0.1)]


@pytest.mark.parametrize("precision,N", [(p, N) for p, orders in LINE_ORDERS.items() for N in orders])
@pytest.mark.parametrize("kind,res,n_inst,jitter", CASES)
def test_line_kernel_against_three_threads_a_line(N, precision, kind, res, n_inst, jitter):
    kw = {"periodic": dict(x_periodic=True, y_periodic=True), "wall": dict(x_periodic=True, boundary=meshgen.WALL),
          "outflow": dict(boundary=meshgen.OUTFLOW), "inflow": dict(boundary=meshgen.INFLOW, x_min=0.0, x_max=1.0, y_min=0.0, y_max=1.0)}[kind]
    zone = meshgen.uniform_zone(res, order="rowmajor", jitter=jitter, seed=res, **kw)
    rng = np.random.default_rng(N)
    K = res * res
    fields = [rng.standard_normal(n_inst * K * (N + 1) ** 2) for _ in range(3)]
    # the scheme is unstable at N = 2 and CFL 0.5, which magnifies FP32 rounding
    steps = 2 if precision == ndg.FP32 and N == 2 else 9
    line, = _run(zone, N, precision, False, fields, n_inst, steps)
    three, = _run(zone, N, precision, True, fields, n_inst, steps)
    assert rel_l2(line, three) < (1e-13 if precision == ndg.FP64 else 2e-6)


@pytest.mark.parametrize("precision", [ndg.FP64, ndg.FP32])
def test_where_the_line_kernel_runs(precision):
    """The rules on orders, sizes and forms, on both sides of each line."""
    def kernel(res, N, n_inst=1, **kw):
        m = ndg.Mesh2D_t(meshgen.uniform_zone(res, order="rowmajor", boundary=meshgen.WALL), N, n_instances=n_inst, **{"precision": precision, **kw})
        name = m.stage_kernel()
        m.close()
        return name.startswith("line_stage_kernel")

    for N in range(1, 17):
        assert kernel(40, N) == (N in LINE_ORDERS[precision]), N
        assert not kernel(40, N, keep_derivative=True)
    for N in (5, 6, 8):
        assert not kernel(39, N) and not kernel(16, N, 5) and kernel(16, N, 6)
    for N in range(1, EVERY_SIZE + 1):
        assert kernel(2, N)
    assert not kernel(40, 4, precision=ndg.FP64_STRICT)


@pytest.mark.parametrize("precision", [ndg.FP64, ndg.FP32])
@pytest.mark.parametrize("N", [4, 8])
def test_kernels_switched_between_runs(N, precision):
    """The two kernels lay the same trace buffers out differently: runs that
    switch between them, by keep_derivative or by a tensor-core tile, go on as
    one run does."""
    zone = meshgen.uniform_zone(40, order="rowmajor", boundary=meshgen.INFLOW, x_min=0.0, x_max=1.0, y_min=0.0, y_max=1.0, jitter=0.1, seed=6)
    rng = np.random.default_rng(N)
    fields = [rng.standard_normal(1600 * (N + 1) ** 2) for _ in range(3)]
    want, = _run(zone, N, precision, False, fields, 1, 21)
    m = ndg.Mesh2D_t(zone, N, precision=precision)
    for f, v in zip(("p", "u", "v"), fields):
        m.set_field(f, v)
    tensor = max(m.tile_candidates()[0])
    switches = [lambda: ndg.lib().ndg_ctx_keep_derivative(m.handle, 1), lambda: ndg.lib().ndg_ctx_keep_derivative(m.handle, 0)]
    if tensor >= ndg.TENSOR_TILE:
        switches += [lambda: m.set_tile(tensor), lambda: m.set_tile(0)]
    t, names = ndg.Solver2D_t.run(m, 1), [m.stage_kernel()]
    for switch, steps in zip(switches * 2, (3, 1, 9, 2, 1, 2, 1, 1)):
        switch()
        names.append(m.stage_kernel())
        t = ndg.Solver2D_t.run(m, steps, t)
    if tensor < ndg.TENSOR_TILE:
        t = ndg.Solver2D_t.run(m, 5, t)
    got = np.concatenate([m.get_field(f) for f in ("p", "u", "v", "k_p", "k_u", "k_v")])
    m.close()
    assert all(n.startswith("line_") == (i % 2 == 0) for i, n in enumerate(names)), names
    assert rel_l2(got, want) < (1e-12 if precision == ndg.FP64 and tensor >= ndg.TENSOR_TILE else 1e-13 if precision == ndg.FP64 else 2e-6)


@pytest.mark.parametrize("precision,N", [(ndg.FP64, 7), (ndg.FP64, 8), (ndg.FP64, 11), (ndg.FP32, 5), (ndg.FP32, 8)])
def test_line_tiles_agree_and_runs_split_anywhere(N, precision):
    """Tiles give the same bits, and so does a run stopped and resumed after
    its traces were rebuilt from q."""
    zone = meshgen.uniform_zone(40, order="rowmajor", x_periodic=True, boundary=meshgen.WALL, jitter=0.1, seed=3)
    m = ndg.Mesh2D_t(zone, N, precision=precision)
    tiles = [0] + [t for t in m.tile_candidates()[0] if t < ndg.TENSOR_TILE]
    rng = np.random.default_rng(0)
    fields = [rng.standard_normal(m.field_size) for _ in range(3)]
    m.close()
    runs = _run(zone, N, precision, False, fields, 1, 4, tiles)
    for t, r in zip(tiles[1:], runs[1:]):
        assert np.array_equal(r, runs[0]), t
    m = ndg.Mesh2D_t(zone, N, precision=precision)
    for f, v in zip(("p", "u", "v"), fields):
        m.set_field(f, v)
    ndg.Solver2D_t.run(m, 2)
    m.set_field("u", m.get_field("u"))
    ndg.Solver2D_t.run(m, 2)
    got = np.concatenate([m.get_field(f) for f in ("p", "u", "v", "k_p", "k_u", "k_v")])
    m.close()
    assert np.array_equal(got, runs[0])


@pytest.mark.parametrize("N", [5, 8])
def test_line_kernel_against_the_oracle(N):
    zone = meshgen.uniform_zone(40, order="rowmajor", boundary=meshgen.WALL, jitter=0.1, seed=5)
    o = OracleSolver(zone, N)
    o.initial_conditions()
    m = ndg.Mesh2D_t(zone, N)
    for f in ("p", "u", "v"):
        m.set_field(f, o.field(f))
    o.run(4)
    ndg.Solver2D_t.run(m, 4)
    for f in ("p", "u", "v"):
        assert rel_l2(m.get_field(f), o.field(f)) < 1e-12, f
    m.close()


@pytest.mark.parametrize("precision,N", [(ndg.FP64, N) for N in range(4, 13)] + [(ndg.FP32, N) for N in (4, 5, 6, 8, 10)])
@pytest.mark.parametrize("boundary", ["wall", "periodic", "outflow"])
def test_variable_speed_line_stage(N, precision, boundary):
    """The variable-speed stage in the line kernel: the operator and the
    gradient (kept stage inputs, samples, recomputation) against the oracle's
    CPU adjoint, to the tolerances of the adjoint's own tests."""
    from tests import adjoint_setup as A
    kw = {"wall": dict(boundary=meshgen.WALL), "outflow": dict(boundary=meshgen.OUTFLOW), "periodic": dict(x_periodic=True, y_periodic=True)}[boundary]
    zone = meshgen.uniform_zone(41, order="rowmajor", jitter=0.1, seed=2, **kw)
    rng = np.random.default_rng(N)
    c = 1.0 + 0.2 * rng.random(41 * 41)
    xy = A.circle_receivers(5, 0.6)
    mesh = ndg.Mesh2D_t(zone, N)
    adj = ndg.Adjoint2D_t(mesh, xy, speed=c, precision=precision)
    o, el, w = A.oracle_problem(zone, N, c, xy)
    x, y = rng.standard_normal(3 * mesh.field_size), rng.standard_normal(3 * mesh.field_size)
    Lx, LTy, dc = adj.operator(x, y)
    LTy_o, dc_o = o.operator_transpose(x, y)
    for got, want in ((Lx, o.operator(x)), (LTy, LTy_o), (dc, dc_o)):
        assert rel_l2(got, want) < (1e-12 if precision == ndg.FP64 else 1e-6)
    p0 = A.gaussian_pulse(zone, N, sigma=0.3)
    dt, steps = adj.delta_t(0.5), 5
    target = 0.1 * rng.standard_normal((steps + 1, el.size))
    J, samples = adj.forward(p0, dt, steps, targets=target, checkpoint_interval=2)
    g = adj.backward()
    ref = o.adjoint_solve(p0, dt, steps, el, w, targets=target)
    assert rel_l2(samples, ref["samples"]) < (1e-12 if precision == ndg.FP64 else 1e-6)
    for k in ("p0", "u0", "v0", "c"):
        assert rel_l2(g[k], ref[k]) < (1e-10 if precision == ndg.FP64 else 1e-4), k
    adj.close()
    mesh.close()


@pytest.mark.parametrize("N", [8, 10])
def test_fp32_speed_derivative_keeps_its_accuracy(N):
    """The line kernel's FP32 speed derivative against the three-threads-a-line
    kernel's, which runs below the size rule: on meshes of 40^2 and 38^2
    elements of the same shapes and data the RMS difference from the FP64 form
    is a sample of 1,600 and 1,444 elements, so the two agree within about 2%
    (1 / sqrt(2 K) each) where both sum alike. 1.15 leaves room for the order
    of the sums; one FP32 accumulator over the three fields shows 1.27 (N = 8)
    and 1.31 (N = 10), one per field 1.04 and 1.07. The state has a mean, so
    the sums grow along the lines."""
    def rms(res):
        zone = meshgen.uniform_zone(res, order="rowmajor", x_periodic=True, y_periodic=True, jitter=0.1, seed=3)
        mesh = ndg.Mesh2D_t(zone, N)
        err, size = 0.0, 0.0
        for seed in range(2):
            rng = np.random.default_rng(seed)
            x, y = 3.0 + rng.standard_normal(3 * mesh.field_size), rng.standard_normal(3 * mesh.field_size)
            c = 1.0 + 0.2 * rng.random(res * res)
            dc = []
            for precision in (ndg.FP64, ndg.FP32):
                adj = ndg.Adjoint2D_t(mesh, speed=c, precision=precision)
                dc.append(adj.operator(x, y)[2])
                adj.close()
            err, size = err + np.mean((dc[1] - dc[0]) ** 2), size + np.mean(dc[0] ** 2)
        mesh.close()
        return np.sqrt(err / size)

    assert rms(40) < 1.15 * rms(38)


def _seam_zone(kind):
    """Periodic squares whose seam sides are not exactly antiparallel: turned
    by 0.3 rad (translates, normals equal to the rounding of the coordinates),
    and bent into a ring's sector (the y seam's normals 0.5 rad apart)."""
    zone = meshgen.uniform_zone(41, order="rowmajor", x_periodic=kind == "turned", y_periodic=True, boundary=meshgen.WALL, jitter=0.1, seed=4)
    x, y = zone["x"].copy(), zone["y"].copy()
    if kind == "turned":
        zone["x"], zone["y"] = np.cos(0.3) * x - np.sin(0.3) * y, np.sin(0.3) * x + np.cos(0.3) * y
    else:
        zone["x"], zone["y"] = (3 + x) * np.cos(0.25 * y), (3 + x) * np.sin(0.25 * y)
    return zone


@pytest.mark.parametrize("precision", [ndg.FP64, ndg.FP32])
@pytest.mark.parametrize("N", [3, 6, 8])
@pytest.mark.parametrize("kind", ["turned", "sector"])
def test_seams_whose_normals_are_not_opposite(N, kind, precision):
    """The line kernel runs there too, and gives what the three-threads-a-line
    kernel and the oracle give, forward, operator and transpose."""
    zone = _seam_zone(kind)
    o = OracleSolver(zone, N)
    o.initial_conditions()
    rng = np.random.default_rng(N)
    m = ndg.Mesh2D_t(zone, N, precision=precision)
    fields = [rng.standard_normal(m.field_size) for _ in range(3)]
    assert m.stage_kernel().startswith("line_stage_kernel")
    m.close()
    line, = _run(zone, N, precision, False, fields, 1, 9)
    three, = _run(zone, N, precision, True, fields, 1, 9)
    assert rel_l2(line, three) < (1e-13 if precision == ndg.FP64 else 2e-6)
    for f, v in zip(("p", "u", "v"), fields):
        o.set_field(f, v)
    o.run(9)
    want = np.concatenate([o.field(f) for f in ("p", "u", "v")])
    assert rel_l2(line[:want.size], want) < (1e-12 if precision == ndg.FP64 else 2e-6)
    mesh = ndg.Mesh2D_t(zone, N)
    c = 1.0 + 0.2 * rng.random(mesh.n_elements_)
    adj = ndg.Adjoint2D_t(mesh, speed=c, precision=precision)
    o.set_speed(c)
    x, y = rng.standard_normal(3 * mesh.field_size), rng.standard_normal(3 * mesh.field_size)
    Lx, LTy, dc = adj.operator(x, y)
    LTy_o, dc_o = o.operator_transpose(x, y)
    for got, ref in ((Lx, o.operator(x)), (LTy, LTy_o), (dc, dc_o)):
        assert rel_l2(got, ref) < (1e-12 if precision == ndg.FP64 else 1e-6)
    adj.close()
    mesh.close()


def test_degenerate_elements_run_the_other_kernel():
    """An element whose Jacobian vanishes at its nodes gives infinities in the
    three-threads-a-line kernel, as an IEEE division does; the line kernel's
    reciprocal has no special cases, so such a mesh does not run it. The same
    mesh before its element collapses does, and so does one with a corner of an
    element collapsed, whose nodes are regular."""
    zone = meshgen.uniform_zone(41, order="rowmajor", boundary=meshgen.WALL)
    quad = zone["sections"][0][4].reshape(-1, 4)[20 * 41 + 20] - 1

    def kernel(points):
        z = dict(zone, x=zone["x"].copy(), y=zone["y"].copy())
        for node, (px, py) in points.items():
            z["x"][quad[node]], z["y"][quad[node]] = px, py
        out = []
        for keep in (False, True):
            m = ndg.Mesh2D_t(z, 6, keep_derivative=keep)
            rng = np.random.default_rng(1)
            for f in ("p", "u", "v"):
                m.set_field(f, rng.standard_normal(m.field_size))
            ndg.Solver2D_t.stage(m, 0, 0.0, 1e-3)
            out.append(np.concatenate([m.get_field(f) for f in ("p", "u", "v", "k_p", "k_u", "k_v")]))
            name = m.stage_kernel() if not keep else name
            m.close()
        return name, out[0], out[1]

    name, line, three = kernel({})
    assert name.startswith("line_stage_kernel") and rel_l2(line, three) < 1e-13
    x, y = zone["x"][quad], zone["y"][quad]
    name, line, three = kernel({2: (0.5 * (x[1] + x[3]), 0.5 * (y[1] + y[3]))})  # a triangle
    assert name.startswith("line_stage_kernel") and rel_l2(line, three) < 1e-13
    flat = {i: (0.25 * i, 0.0) for i in range(4)}  # four corners on a line
    name, line, three = kernel(flat)
    assert name.startswith("stage_kernel") and np.isinf(three).any()
    assert np.array_equal(line, three, equal_nan=True)


def test_line_reciprocal(tmp_path):
    """line_rcp against the correctly rounded reciprocal, 6e7 arguments of both
    signs: Jacobians of ordinary meshes (2^-60 to 2^60) and the whole range that
    the kernels take (2^-1000 to 2^1000). Its error before the last rounding is
    below 2^-79, so it may miss the correct rounding by one unit where 1 / x lies
    that close to a boundary between two results: one random argument in 2^26,
    and (2 - 2^-52) 2^k, whose reciprocal lies 2^-106 off one."""
    import ctypes
    import os
    import subprocess

    import torch
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = str(tmp_path / "liblinercp.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(root, "include"), "-I", os.path.join(root, "ndg_cuda_b200", "csrc"),
                    os.path.join(root, "tests", "cpp", "line_rcp.cu"), "-o", out], check=True, capture_output=True, text=True)
    compare = ctypes.CDLL(out).compare_reciprocals
    compare.argtypes = [ctypes.c_ulonglong, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    torch.cuda.synchronize()
    for low, high, near in ((-60, 60, 0), (-1000, 1000, 0), (-60, 60, 1), (-1000, 1000, 1)):
        counts = torch.zeros(4, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        total = 592 * 256 * 400
        assert compare(12345, low, high, near, 400, counts.data_ptr()) == 0
        same, one, two, more = counts.tolist()
        assert same + one == total and one <= (total / 15 if near else 20), (low, high, near, counts.tolist())
