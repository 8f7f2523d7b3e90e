"""Advection on cell sizes that are and are not powers of two (multiplied and
divided positions), at sizes where blocks end, with positions far outside the
grid, on walls and beside solids: identical to the float32 oracle; and NaN and
infinite velocities, which reach the same values as there."""
import ctypes

import numpy as np
import pytest

from flowlab_gb300 import native
from flowlab_gb300.native import f32, ptr
from tests import fixtures as fx

pytestmark = pytest.mark.gpu


def run(o32, nx, ny, h, scale, mac, u, v, label, dye, dt):
    eng = native.Engine(nx, ny, h, scale)
    nd = nx * ny * scale * scale
    try:
        uo, vo = np.empty_like(u), np.empty_like(v)
        eng.call("fl_advect_velocity", int(mac), ptr(u), ptr(v), ptr(uo), ptr(vo), ptr(label), np.float32(dt))
        qi = [dye[c * nd:(c + 1) * nd].copy() for c in range(3)]
        qo = [np.empty(nd, np.float32) for _ in range(3)]
        planes = lambda ps: (ctypes.c_void_p * 3)(*[a.ctypes.data for a in ps])  # noqa: E731
        eng.call("fl_advect_dye", int(mac), ptr(u), ptr(v), planes(qi), planes(qo), ptr(label), np.float32(dt))
    finally:
        eng.close()
    hf, dtf, dh = float(np.float32(h)), float(np.float32(dt)), float(np.float32(h / scale))
    eu, ev = o32.advect_velocity(nx, ny, hf, mac, u, v, label, dtf)
    eq = o32.advect_dye(nx, ny, hf, nx * scale, ny * scale, dh, mac, u, v, dye, label, dtf)
    return (("u", eu, uo), ("v", ev, vo), ("dye", eq, np.concatenate(qo)))


@pytest.mark.parametrize("mac", [False, True])
@pytest.mark.parametrize("nx,ny,h,scale", [(2, 2, 0.5, 1), (3, 7, 0.1, 2), (31, 9, 1 / 9, 1), (32, 8, 1 / 8, 2),
                                           (33, 65, 1 / 65, 1), (130, 64, 1 / 64, 1), (257, 129, 0.037, 3)])
def test_samplers_identical(o32, nx, ny, h, scale, mac):
    rng = np.random.default_rng(nx * 1000 + ny)
    label = fx.scaled_block_labels(nx, ny)
    u, v = f32(rng.uniform(-1, 1, (nx + 1) * ny)), f32(rng.uniform(-1, 1, nx * (ny + 1)))
    u[::17] = 0.0
    v[::13] *= 200.0  # far outside the grid
    dye = f32(rng.uniform(0, 1, 3 * nx * ny * scale * scale))
    for name, exp, got in run(o32, nx, ny, h, scale, mac, u, v, label, dye, 2.0 * h):
        assert np.array_equal(np.asarray(exp, np.float32), got), name


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("h", [1 / 16, 1 / 17])
def test_samplers_nonfinite(o32, h, bad):
    nx, ny = 24, 16
    rng = np.random.default_rng(5)
    label = fx.scaled_block_labels(nx, ny)
    u, v = f32(rng.uniform(-1, 1, (nx + 1) * ny)), f32(rng.uniform(-1, 1, nx * (ny + 1)))
    u[5 * (nx + 1) + 3] = v[9 * nx + 7] = bad
    dye = f32(rng.uniform(0, 1, 3 * nx * ny))
    for name, exp, got in run(o32, nx, ny, h, 1, True, u, v, label, dye, h):
        assert np.array_equal(np.asarray(exp, np.float32), got, equal_nan=True), name
