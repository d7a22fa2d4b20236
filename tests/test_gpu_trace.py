"""The tiled WENO6 backtrace of both forms against the oracle's vertex by vertex one: grids of one
tile and of many, remainders along every axis, small and large tiles.  Bounds of
tests/test_gpu_parity.py (1e-13) and tests/test_gpu_fp32.py (1e-6 of a cell)."""
import numpy as np
import pytest

import scenes
from oracle import Oracle

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu

O = Oracle()


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 7, 16), (4, 3, 33), (9, 16, 31), (47, 41, 65), (64, 63, 40)])
@pytest.mark.parametrize("comp", [-1, 0, 1, 2])
def test_trace_tiles(shape, comp):
    n = max(shape)
    h = 1.0 / n
    nx, ny, nz = shape
    u, v, w = scenes.fourier_velocity(n, seed=8)
    u = u.reshape(n + 1, n, n)[:nx + 1, :ny, :nz].ravel()
    v = v.reshape(n, n + 1, n)[:nx, :ny + 1, :nz].ravel()
    w = w.reshape(n, n, n + 1)[:nx, :ny, :nz + 1].ravel()
    dt = 1.3 * h
    ref = O.backtrace_vertices(shape, h, u, v, w, dt, comp, 0)
    for precision, bound in ((fia.FIA_FP64, 1e-13), (fia.FIA_FP32C, 1e-6 * h)):
        g = fia.Grid3D(nx, ny, nz, h, precision=precision)
        for name, a in (("u", u), ("v", v), ("w", w)):
            g.set(name, a)
        got = g.debug_backtrace(comp, dt, 0)
        g.close()
        assert np.abs(got - ref).max() <= bound
