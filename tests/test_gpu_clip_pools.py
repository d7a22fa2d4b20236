"""The face clipper with its shared-memory pools (k_clip32, k_clip32_deferred) against the
local-memory clipper on every face: the same pieces in the same order, so the same bits, for
families of unequal size in one launch and for faces that outgrow the first pool, the second, or
both."""
import numpy as np
import pytest

import scenes

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2), (2, 9, 3), (7, 2, 33), (19, 12, 5), (24, 24, 24)])
@pytest.mark.parametrize("cfl", [0.0, 3.0, 9.0])
def test_clip_pools_match_local_clipper(shape, cfl):
    n = max(shape)
    nx, ny, nz = shape
    u, v, w = scenes.fourier_velocity(n, seed=6)
    u = u.reshape(n + 1, n, n)[:nx + 1, :ny, :nz].ravel()
    v = v.reshape(n, n + 1, n)[:nx, :ny + 1, :nz].ravel()
    w = w.reshape(n, n, n + 1)[:nx, :ny, :nz + 1].ravel()
    rho = scenes.gaussian_blobs(n, seed=4).reshape(n, n, n)[:nx, :ny, :nz].ravel()
    out = []
    for fast in (1, 0):
        g = fia.Grid3D(nx, ny, nz, 1.0 / n, precision=fia.FIA_FP32C)
        for name, a in (("u", u), ("v", v), ("w", w), ("density", rho)):
            g.set(name, a)
        before = g.debug_clip_fast(fast)
        g.move_substances_3D(cfl / n, fia.advect_params())
        g.advect_velocity_xyz_flux_advection_3D(cfl / n, fia.advect_params())
        listed = g.debug_clip_fast() - before
        out.append(([g.get(c) for c in ("density", "u", "v", "w")], listed, list(g.pass_counters())[:3]))
        g.close()
    (f1, n1, c1), (f0, n0, c0) = out
    for a, b in zip(f1, f0):
        assert np.array_equal(a, b)
    assert c1 == c0
    assert n0 == c0[0] and n1 <= n0
