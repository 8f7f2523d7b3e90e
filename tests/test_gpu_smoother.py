"""The register-blocked smoother (csrc/fl_multigrid.cu, smooth_tile) at the
sizes where its regions, warps and column pairs end, on both of its region
shapes, against the float32 oracle: the same operations in the same order, so
identical results. Every cell starts nonzero, solid and open ones too (which
keep their value)."""
import numpy as np
import pytest

from flowlab_gb300 import native
from flowlab_gb300.native import f32, ptr
from tests import fixtures as fx

pytestmark = pytest.mark.gpu


def problem(nx, ny):
    label = fx.scaled_block_labels(nx, ny)
    if nx > 8 and ny > 8:  # single solid cells: link counts 3, 2 and 1 next to the walls
        lab = label.reshape(ny, nx)
        lab[1, 2] = lab[ny - 2, 1] = lab[ny - 1, nx // 2] = lab[3, 0] = fx.SOLID
    vals = fx.js_lcg_uniform(2 * nx * ny, 4242)
    return label, f32(vals[:nx * ny]), f32(0.1 * vals[nx * ny:])


def same(exp, got, what):
    bad = np.asarray(exp, np.float32) != got
    assert not bad.any(), "%s: %d of %d values differ, first at %d" % (what, bad.sum(), bad.size, np.nonzero(bad)[0][0])


@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 50), (48, 16), (49, 17), (56, 33), (60, 64), (97, 31), (130, 66),
                                   (700, 690), (701, 689)])
@pytest.mark.parametrize("pairs,omega", [(1, 1.0), (2, 1.9), (3, 1.0), (4, 1.9)])
def test_sor_regions(o32, nx, ny, pairs, omega):
    label, div, p0 = problem(nx, ny)
    eng = native.Engine(nx, ny, params=native.default_params(rb_pairs=pairs))
    try:
        p, used = p0.copy(), native.ctypes.c_int()
        eng.call("fl_rb_solve", ptr(p), ptr(div), ptr(label), 0.02, 9, omega, 0.0, native.ctypes.byref(used))
    finally:
        eng.close()
    same(o32.rb_solve(nx, ny, p0, div, label, 0.02, 9, omega, 0.0)[0], p, "%dx%d, %d pairs" % (nx, ny, pairs))


@pytest.mark.parametrize("nx,ny", [(40, 9), (52, 36), (53, 37), (105, 129), (700, 690), (701, 689)])
@pytest.mark.parametrize("pre,post", [(0, 1), (1, 0), (2, 3), (3, 2), (4, 4)])
def test_multigrid_regions(o32, nx, ny, pre, post):
    label, div, p0 = problem(nx, ny)
    prm = native.default_params(mg_pre=pre, mg_post=post, mg_coarsest=4, mg_tail_side=8)
    eng = native.Engine(nx, ny, params=prm)
    try:
        p, used, rr = p0.copy(), native.ctypes.c_int(), native.ctypes.c_double()
        eng.call("fl_mg_solve", ptr(p), ptr(div), ptr(label), 0.02, 2, 1e-30, native.ctypes.byref(used),
                 native.ctypes.byref(rr))
    finally:
        eng.close()
    exp, _, rr32 = o32.mg_solve(nx, ny, p0, div, label, 0.02, 2, 1e-30, pre, post, 8, 4)
    same(exp, p, "%dx%d, V(%d,%d)" % (nx, ny, pre, post))
    # a sum of float squares in another order of float64 additions
    assert abs(rr.value - rr32) <= 1e-9 * rr32


@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 5), (8, 8), (9, 16), (17, 32), (32, 31), (33, 2), (64, 3), (3, 64),
                                   (63, 40), (64, 64), (100, 77)])
@pytest.mark.parametrize("side,coarsest,sweeps,pre,post", [(0, 8, 16, 3, 3), (64, 4, 8, 2, 2), (64, 1, 3, 0, 1),
                                                           (16, 2, 0, 1, 0), (64, 64, 5, 1, 1)])
def test_tail_frames(o32, nx, ny, side, coarsest, sweeps, pre, post):
    """The single-CTA tail: levels that fill their frame or not, in both
    directions, first level finest or not, one level or several, no sweeps."""
    label, div, p0 = problem(nx, ny)
    prm = native.default_params(mg_pre=pre, mg_post=post, mg_coarse_sweeps=sweeps, mg_coarsest=coarsest,
                                mg_tail_side=side)
    eng = native.Engine(nx, ny, params=prm)
    try:
        p, used, rr = p0.copy(), native.ctypes.c_int(), native.ctypes.c_double()
        eng.call("fl_mg_solve", ptr(p), ptr(div), ptr(label), 0.02, 2, 1e-30, native.ctypes.byref(used),
                 native.ctypes.byref(rr))
    finally:
        eng.close()
    exp, _, rr32 = o32.mg_solve(nx, ny, p0, div, label, 0.02, 2, 1e-30, pre, post, sweeps, coarsest)
    same(exp, p, "%dx%d" % (nx, ny))
    assert used.value == 2 and abs(rr.value - rr32) <= 1e-9 * rr32


@pytest.mark.parametrize("mixed", [1, 2])
@pytest.mark.parametrize("nx,ny", [(3, 2), (29, 8), (30, 9), (61, 33), (130, 66), (517, 389), (724, 500), (1100, 1060)])
def test_defect_pass_rows(o32, nx, ny, mixed):
    """The defect-correction passes where their blocks' columns and rows end
    and at sizes that take each number of rows a warp: the refined pressure
    of two cycles, bit for bit."""
    label, div, _ = problem(nx, ny)
    prm = native.default_params(mg_pre=1, mg_post=1, mg_coarse_sweeps=4, mg_coarsest=4, mixed=mixed)
    eng = native.Engine(nx, ny, params=prm)
    try:
        p, used, rr = np.zeros(nx * ny), native.ctypes.c_int(), native.ctypes.c_double()
        eng.call("fl_mg_solve_mixed", ptr(p), ptr(div), ptr(label), 0.02, 2, 1e-30, native.ctypes.byref(used),
                 native.ctypes.byref(rr))
    finally:
        eng.close()
    solve = o32.mg_solve_mixed if mixed == 1 else o32.mg_solve_df
    exp, used32, rr32 = solve(nx, ny, np.zeros(nx * ny), div, label, 0.02, 2, 1e-30, 1, 1, 4, 4)
    assert used.value == used32
    assert np.array_equal(np.asarray(exp, np.float64), p)
    # sums of the same squares in another order, float64 or double-float
    assert abs(rr.value - rr32) <= 1e-9 * rr32
