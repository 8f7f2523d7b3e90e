"""Whole steps with red-black SOR whose pairs a launch are chosen by the grid
(fl_params.rb_pairs 0): as a graph and eagerly, to a budget and to a tolerance,
with no sweeps, one, a ragged row and the vortex street's own 60 or 100. The
depth changes no result, so every step equals that of four pairs a launch; the
solve with residual tests equals the float32 oracle's."""
import ctypes

import numpy as np
import pytest

from flowlab_gb300 import autotune, configs, native
from flowlab_gb300.native import f32, ptr
from tests.test_gpu_smoother import problem, same

pytestmark = pytest.mark.gpu


def run(nx, ny, prm, graph):
    g, f, _ = configs.karman(nx, ny)
    eng = native.Engine(g.nx, g.ny, g.h, params=prm)
    try:
        eng.call("fl_upload_fields", native.FL_F32, ptr(f32(f.u)), ptr(f32(f.v)), ptr(f32(f.p)), ptr(f.label),
                 ptr(f32(f.dye)))
        if not graph:
            eng.profile(True)  # profiled steps run eagerly
        iters = ctypes.c_int(-1)
        eng.call("fl_step_auto", 3, ctypes.byref(iters))
        u, v, p = (np.empty(n, np.float32) for n in (eng.ufaces, eng.vfaces, eng.cells))
        eng.call("fl_read_velocity", native.FL_F32, ptr(u), ptr(v))
        eng.call("fl_read_pressure", native.FL_F32, ptr(p))
    finally:
        eng.close()
    return iters.value, u, v, p


@pytest.mark.parametrize("nx,ny", [(128, 128), (201, 97)])
@pytest.mark.parametrize("iters", [0, 1, 13, 60])
@pytest.mark.parametrize("tol,graph", [(0.0, True), (0.0, False), (1e-3, False)])
def test_chosen_depth_steps_as_four_pairs(nx, ny, iters, tol, graph):
    base = autotune.with_params(configs.karman_params(), pressure_iters=iters, tol=tol)
    want = run(nx, ny, autotune.with_params(base, rb_pairs=4), graph)
    got = run(nx, ny, autotune.with_params(base, rb_pairs=0), graph)
    assert got[0] == want[0] <= iters
    for name, a, b in zip(("u", "v", "p"), want[1:], got[1:]):
        assert np.isfinite(a).all() and np.array_equal(a, b), "%s: %d values differ" % (name, (a != b).sum())


@pytest.mark.parametrize("nx,ny", [(40, 32), (128, 128), (517, 389), (640, 480)])
@pytest.mark.parametrize("tol", [1e-30, 0.3])
def test_residual_tests_between_launches(o32, nx, ny, tol):
    label, div, p0 = problem(nx, ny)
    eng = native.Engine(nx, ny)
    try:
        p, used = p0.copy(), ctypes.c_int()
        eng.call("fl_rb_solve", ptr(p), ptr(div), ptr(label), 0.02, 43, 1.7, tol, ctypes.byref(used))
    finally:
        eng.close()
    exp, n = o32.rb_solve(nx, ny, p0, div, label, 0.02, 43, 1.7, tol)
    assert used.value == n
    same(exp, p, "%dx%d" % (nx, ny))
