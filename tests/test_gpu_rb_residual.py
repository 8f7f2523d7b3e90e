"""The red-black solver's stopping test (csrc/fl_multigrid.cu,
k_rms_remaining): the reported relative residual against the same sums in
numpy, where rows, columns and blocks end and for scales of both of its
divisions. Every term is rounded alike, so the tolerance is that of summing
n squares in another order (n * 2^-53), twice, and a quotient and two roots."""
import ctypes

import numpy as np
import pytest

from flowlab_gb300 import native
from flowlab_gb300.native import f32, ptr
from tests import fixtures as fx

FLUID = 0

pytestmark = pytest.mark.gpu


def remaining(nx, ny, p, div, label, scale):
    p2, lab = p.reshape(ny, nx), label.reshape(ny, nx)
    total = np.zeros((ny, nx), np.float32)
    count = np.zeros((ny, nx), np.int64)
    for dj, di in ((0, 1), (1, 0), (0, -1), (-1, 0)):
        src = (slice(max(dj, 0), ny + min(dj, 0)), slice(max(di, 0), nx + min(di, 0)))
        dst = (slice(max(-dj, 0), ny + min(-dj, 0)), slice(max(-di, 0), nx + min(-di, 0)))
        open_ = lab[src] != fx.SOLID
        count[dst] += open_
        total[dst] += np.where(open_, p2[src], np.float32(0))
    with np.errstate(divide="ignore", invalid="ignore"):
        r = div.reshape(ny, nx).astype(np.float64) + (
            count * p2.astype(np.float64) - total.astype(np.float64)) / np.float64(np.float32(scale))
    use = (lab == FLUID) & (count > 0)
    return np.sqrt(np.sum(r[use] ** 2) / max(1, use.sum()))


@pytest.mark.parametrize("nx,ny", [(2, 2), (7, 5), (33, 9), (31, 700), (640, 480), (1001, 75)])
@pytest.mark.parametrize("scale", [0.02, 3e-39, 1e30, 0.0])
def test_reported_residual(nx, ny, scale):
    label = fx.scaled_block_labels(nx, ny)
    vals = fx.js_lcg_uniform(2 * nx * ny, 77)
    div, p = f32(vals[:nx * ny]), f32(0.1 * vals[nx * ny:])
    p0 = p.copy()
    eng = native.Engine(nx, ny)
    try:
        used = ctypes.c_int()
        eng.call("fl_rb_solve", ptr(p), ptr(div), ptr(label), scale, 12, 1.0, 1e-300, ctypes.byref(used))
        st = eng.stats()
    finally:
        eng.close()
    assert used.value == 12 and not np.array_equal(p, p0)
    fluid = label == FLUID
    rms = np.sqrt(np.sum(div[fluid].astype(np.float64) ** 2) / fluid.sum())
    tol = nx * ny * 2.0 ** -53 * 2 + 1e-14
    assert abs(st["div_rms"] - rms) <= tol * rms
    want = remaining(nx, ny, p, div, label, scale) / rms
    got = st["rel_residual"]
    if np.isfinite(want):
        assert abs(got - want) <= tol * want
    else:
        assert np.isnan(got) == np.isnan(want) and (np.isnan(got) or got == want)
