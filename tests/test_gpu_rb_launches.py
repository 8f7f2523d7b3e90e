"""Red-black SOR with the pairs a launch and the region shape chosen by the
grid (csrc/fl_multigrid.cu, rb_launch_pairs and rb_shape): on both sides of
each line of the choice, with row lengths that do not divide the iterations,
against the float32 oracle. The same operations in the same order, so
identical results."""
import pytest

from flowlab_gb300 import native
from flowlab_gb300.native import ptr
from tests.test_gpu_smoother import problem, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3, 2), (40, 8), (41, 9), (129, 127), (200, 192), (245, 250), (255, 258), (384, 300),
                                   (517, 389), (640, 480), (801, 603), (1030, 700)])
@pytest.mark.parametrize("iters,omega", [(5, 1.9), (12, 1.0), (23, 1.7)])
def test_chosen_launches(o32, nx, ny, iters, omega):
    label, div, p0 = problem(nx, ny)
    eng = native.Engine(nx, ny)
    try:
        p, used = p0.copy(), native.ctypes.c_int()
        eng.call("fl_rb_solve", ptr(p), ptr(div), ptr(label), 0.02, iters, omega, 0.0, native.ctypes.byref(used))
    finally:
        eng.close()
    same(o32.rb_solve(nx, ny, p0, div, label, 0.02, iters, omega, 0.0)[0], p, "%dx%d, %d" % (nx, ny, iters))
