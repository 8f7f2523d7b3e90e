"""The plans that only large grids and batches enter (csrc/fl_multigrid.cu):
the defect passes' widest row counts, and a work-list batch whose phases take
the 64 x 64 regions, both region shapes, eight rows a warp or a tail from 64^2.
The regions and blocks are counted here for a device of 152 SMs by the rules of
launch_smooth and defect_rows, so that each case is in the plan it names."""
import numpy as np
import pytest

from flowlab_gb300 import autotune, batch, configs, native
from flowlab_gb300.native import ptr
from tests.test_gpu_batch import assert_same
from tests.test_gpu_smoother import problem

pytestmark = pytest.mark.gpu

SMS = 152


def blocks(nx, ny, df, rows):
    return -(-nx // (60 if df else 30)) * -(-ny // (4 * rows))


def rows(sizes, df):
    """Rows a warp of the defect pass over these grids together."""
    total = lambda r: sum(blocks(nx, ny, df, r) for nx, ny in sizes)
    if not df:
        return 2 if total(2) <= 2 * SMS else 4 if total(4) <= 26 * SMS else 8
    return next((r for r in (2, 4, 6) if total(r) <= 6 * SMS), 8)


@pytest.mark.parametrize("mixed,nx,ny,want", [(2, 724, 724, 4), (2, 723, 725, 4), (2, 1200, 1204, 8), (2, 1203, 1201, 8),
                                              (1, 1400, 1408, 8), (1, 1403, 1397, 8)])
def test_defect_pass_widest_rows(o32, mixed, nx, ny, want):
    assert rows([(nx, ny)], mixed == 2) == want
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


def engines(sides, mixed, tails):
    tol = 1e-4 if mixed == 0 else 1e-6
    base = configs.random_scene_params(tol=tol, max_cycles=12, mixed=mixed)
    return [batch.make_engines([n], seed=31 + k, params=autotune.with_params(base, mg_tail_side=t))[0]
            for k, (n, t) in enumerate(zip(sides, tails))]


@pytest.mark.parametrize("mixed", [0, 1, 2])
@pytest.mark.parametrize("tails", [(0, 0, 0, 0, 0), (64, 0, 64, 64, 32)])
def test_large_batch_equals_engines_stepped_alone(mixed, tails):
    sides = [1024, 1024, 256, 64, 32]
    # the two largest levels in 64 x 64 regions, those below in the small ones
    regions = lambda n: (-(-n // (64 - 2 * 6))) ** 2  # V(3,3) from zero: a halo of 6
    assert 2 * regions(512) >= 176 > 3 * regions(256)
    if mixed:
        assert rows([(n, n) for n in sides], mixed == 2) == 8
    alone, together = engines(sides, mixed, tails), engines(sides, mixed, tails)
    try:
        for e in alone:
            e.call("fl_step_auto", 2, None)
        b = native.Batch(together)
        try:
            assert b.worklist
            b.step(2)
        finally:
            b.close()
        assert_same(alone, together, "mixed %d" % mixed)
    finally:
        batch.close_all(alone + together)
