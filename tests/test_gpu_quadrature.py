"""The per-piece quadrature of both forms at the edges of its stencils and point groups: grids
smaller than the six-node stencil along each axis (every z-record clamped), Gauss rules around
the group of three points, and WENO6 psi points off the node rows (use_integral 0).

Fields and tolerance of tests/test_gpu_fp32.py: 2e-6 relative L2 of a single FP32 flux pass outside
at most four cells whose pieces fall on the other side of a y-face in FP32, 5e-4 with them.
"""
import numpy as np
import pytest

import scenes
from oracle import Oracle

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu

O = Oracle()


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 7, 2), (9, 2, 5), (12, 9, 33)])
@pytest.mark.parametrize("comp", [-1, 0, 1, 2])
@pytest.mark.parametrize("k,integral", [(1, 1), (5, 1), (15, 1), (3, 0)])
def test_fp32_weno_pass_small_grids(shape, comp, k, integral):
    n = max(shape)
    h = 1.0 / n
    nx, ny, nz = shape
    u, v, w = scenes.fourier_velocity(n, seed=3)
    u = u.reshape(n + 1, n, n)[:nx + 1, :ny, :nz].ravel()
    v = v.reshape(n, n + 1, n)[:nx, :ny + 1, :nz].ravel()
    w = w.reshape(n, n, n + 1)[:nx, :ny, :nz + 1].ravel()
    f = (u, v, w)[comp] if comp >= 0 else scenes.gaussian_blobs(n, seed=4).reshape(n, n, n)[:nx, :ny, :nz].ravel()
    dt = 1.7 * h
    ref, _, _, _ = O.flux_pass(shape, h, u, v, w, comp, f, dt, 0, 1, integral, 0, (0.5, 0.5), k)
    g = fia.Grid3D(*shape, h, precision=fia.FIA_FP32C)
    for name, a in (("u", u), ("v", v), ("w", w)):
        g.set(name, a)
    got, st = g.debug_flux_pass(comp, f, dt, 0, 1, integral, 0, (0.5, 0.5), k)
    g.close()
    assert st == 0
    d = np.abs(got - ref)
    keep = np.argsort(d)[:-4]
    assert np.linalg.norm(d[keep]) < 2e-6 * np.linalg.norm(ref)
    assert np.linalg.norm(d) < 5e-4 * np.linalg.norm(ref)


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 7, 2), (9, 2, 5), (12, 9, 33)])
@pytest.mark.parametrize("comp", [-1, 0, 1, 2])
@pytest.mark.parametrize("k,integral,zero", [(1, 1, 0), (5, 1, 0), (15, 1, 0), (3, 0, 0), (3, 0, 1)])
def test_fp64_weno_pass_small_grids(shape, comp, k, integral, zero):
    """the plain form at its parity bound, 1e-10"""
    n = max(shape)
    h = 1.0 / n
    nx, ny, nz = shape
    u, v, w = scenes.fourier_velocity(n, seed=3)
    u = u.reshape(n + 1, n, n)[:nx + 1, :ny, :nz].ravel()
    v = v.reshape(n, n + 1, n)[:nx, :ny + 1, :nz].ravel()
    w = w.reshape(n, n, n + 1)[:nx, :ny, :nz + 1].ravel()
    f = (u, v, w)[comp] if comp >= 0 else scenes.gaussian_blobs(n, seed=4).reshape(n, n, n)[:nx, :ny, :nz].ravel()
    dt = 1.7 * h
    ref, _, _, _ = O.flux_pass(shape, h, u, v, w, comp, f, dt, 0, 1, integral, zero, (0.5, 0.5), k)
    g = fia.Grid3D(*shape, h)
    for name, a in (("u", u), ("v", v), ("w", w)):
        g.set(name, a)
    got, st = g.debug_flux_pass(comp, f, dt, 0, 1, integral, zero, (0.5, 0.5), k)
    g.close()
    assert st == 0
    assert np.linalg.norm(got - ref) < 1e-10 * np.linalg.norm(ref)


def test_fp32_weno_weights_keep_their_range():
    """a density of 1e9 (squared indicators of 1e38 and more): as close to the oracle as at 1"""
    n, scale = 12, 1e9
    u, v, w = scenes.fourier_velocity(n, seed=5)
    rho = scenes.gaussian_blobs(n, seed=6) * scale
    g = fia.Grid3D(n, n, n, 1.0 / n, precision=fia.FIA_FP32C)
    for name, a in (("density", rho), ("u", u), ("v", v), ("w", w)):
        g.set(name, a)
    g.move_substances_3D(2.0 / n, fia.advect_params())
    assert g.last_status() == 0
    got = g.get("density")
    g.close()
    ref, _ = O.move_substances_3D((n, n, n), 1.0 / n, u, v, w, rho, 2.0 / n)
    assert np.linalg.norm(got - ref) < 2e-6 * np.linalg.norm(ref)
