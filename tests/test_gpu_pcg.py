"""The one-kernel Jacobi-PCG where its shape changes: one block and several, chunks that end inside a
z-line, rows of any length (one, two or four cells a thread step), solids and the pinned cell
they move, fewer and more iterations than a launch makes.

The pressure's residual is formed here in 64 bits from the operator's definition.  Tolerance: the
requested one, 1e-10, twice over for the recursive residual's drift in FP64; the FP32 form's
report is itself a 64-bit residual of its pressure.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import fia  # noqa: E402
import unet_oracle as U  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spheres", [0, 2])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 7), (16, 16, 16), (17, 16, 20), (9, 40, 33), (64, 37, 30),
                                   (70, 64, 68)])
def test_pcg_solves_its_operator(shape, spheres):
    if spheres and min(shape) < 9:
        pytest.skip("no room for a sphere")
    nx, ny, nz = shape
    h = 1.0 / max(shape)
    rng = np.random.default_rng(11)
    vel = [rng.normal(size=(nx + 1, ny, nz)), rng.normal(size=(nx, ny + 1, nz)), rng.normal(size=(nx, ny, nz + 1))]
    for d, f in enumerate(vel):
        f[(slice(None),) * d + (0,)] = 0.0
        f[(slice(None),) * d + (-1,)] = 0.0
    for precision, tol in ((fia.FIA_FP64, 1e-10), (fia.FIA_FP32C, 1e-6)):
        g = fia.Grid3D(nx, ny, nz, h, precision=precision)
        for name, f in zip("uvw", vel):
            g.set(name, f.ravel())
        if spheres:
            # one of them over the last cell, which then is not the pinned one
            g.set_solid_spheres([[nx * h, ny * h, nz * h], [0.4 * nx * h, 0.5 * ny * h, 0.4 * nz * h]], [2.5 * h, 3.2 * h])
        mask = g.solid_mask()
        pin = int(np.nonzero(mask == 0)[0][-1])
        u, v, w = (g.get(c).reshape(f.shape) for c, f in zip("uvw", vel))
        b = h * (np.diff(u, axis=0) + np.diff(v, axis=1) + np.diff(w, axis=2))
        b.reshape(-1)[mask.astype(bool)] = 0.0
        b.reshape(-1)[pin] = 0.0
        rep = g.calc_pressure_3D(fia.solver_params(tol=tol, max_iter=20000))
        p = g.get("pressure").reshape(shape)
        g.close()
        assert rep.status == 0
        assert rep.rel_residual <= tol
        if precision == fia.FIA_FP64:
            r = U.apply_B(p, shape, pin, mask if spheres else None) + b      # B p = -b
            assert np.linalg.norm(r) <= 2 * tol * np.linalg.norm(b)


def test_pcg_stops_at_the_iteration_cap():
    g = fia.Grid3D(48, 40, 44, 1.0 / 48)
    rng = np.random.default_rng(5)
    for name in "uvw":
        g.set(name, rng.normal(size=g.sizes()[name]))
    for cap in (1, 17, 300):
        rep = g.calc_pressure_3D(fia.solver_params(tol=1e-14, max_iter=cap))
        assert rep.iterations == cap
        assert rep.status == fia.FIA_STATUS_SOLVER_CAP
    g.close()
