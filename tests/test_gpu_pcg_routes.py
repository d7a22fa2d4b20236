"""Jacobi-PCG on every route that the size of the grid decides, one grid each: the one-kernel solver with
four, three and two vectors in shared memory, its cells' places kept or formed at each visit, rows of whole
groups and of single cells; and the two kernels of the grids above.  The residual is formed here in 64
bits from the operator's definition (FP64 form; tolerance twice the requested one for the recursive
residual's drift), or is the report's own 64-bit residual of its pressure (FP32 form)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import fia  # noqa: E402
import unet_oracle as U  # noqa: E402

pytestmark = pytest.mark.gpu

# with 152 SMs, of which it takes 148
FP32 = [(132, 130, 132), (140, 140, 140), (160, 158, 156), (176, 160, 168),      # three vectors, + places, two, none
        (89, 87, 85), (141, 139, 141), (151, 149, 151)]                          # four, three, none; single cells
FP64 = [(106, 104, 106), (116, 112, 114), (132, 130, 134),                       # three, two, none
        (101, 99, 101), (107, 107, 105), (115, 113, 115), (131, 133, 133)]       # four, three, two, none; single cells


@pytest.mark.parametrize("precision,shape", [("fp32", s) for s in FP32] + [("fp64", s) for s in FP64])
@pytest.mark.parametrize("spheres", [0, 2])
def test_routes(precision, shape, spheres):
    nx, ny, nz = shape
    h = 1.0 / max(shape)
    rng = np.random.default_rng(3)
    vel = [rng.normal(size=(nx + 1, ny, nz)), rng.normal(size=(nx, ny + 1, nz)), rng.normal(size=(nx, ny, nz + 1))]
    for d, f in enumerate(vel):
        f[(slice(None),) * d + (0,)] = 0.0
        f[(slice(None),) * d + (-1,)] = 0.0
    fp64 = precision == "fp64"
    tol = 1e-8 if fp64 else 1e-6
    g = fia.Grid3D(nx, ny, nz, h, precision=fia.FIA_FP64 if fp64 else fia.FIA_FP32C)
    for name, f in zip("uvw", vel):
        g.set(name, f.ravel())
    if spheres:
        g.set_solid_spheres([[nx * h, ny * h, nz * h], [0.4 * nx * h, 0.5 * ny * h, 0.4 * nz * h]], [2.5 * h, 9.2 * h])
    rep = g.calc_pressure_3D(fia.solver_params(tol=tol, max_iter=20000))
    assert rep.status == 0
    assert rep.rel_residual <= tol
    if fp64:
        mask = g.solid_mask()
        pin = int(np.nonzero(mask == 0)[0][-1])
        u, v, w = (g.get(c).reshape(f.shape) for c, f in zip("uvw", vel))
        b = h * (np.diff(u, axis=0) + np.diff(v, axis=1) + np.diff(w, axis=2))
        b.reshape(-1)[mask.astype(bool)] = 0.0
        b.reshape(-1)[pin] = 0.0
        r = U.apply_B(g.get("pressure").reshape(shape), shape, pin, mask if spheres else None) + b
        assert np.linalg.norm(r) <= 2 * tol * np.linalg.norm(b)
    g.close()


@pytest.mark.parametrize("precision", [fia.FIA_FP32C, fia.FIA_FP64])
def test_a_wait_that_ran_out_is_an_error(precision):
    g = fia.Grid3D(32, 30, 28, 1.0 / 32, precision=precision)
    rng = np.random.default_rng(5)
    for name in "uvw":
        g.set(name, rng.normal(size=g.sizes()[name]))
    sp = fia.solver_params(tol=1e-6)
    g.debug_pcg_stuck(1)
    with pytest.raises(fia.FiaError):
        g.calc_pressure_3D(sp)
    g.debug_pcg_stuck(0)
    rep = g.calc_pressure_3D(sp)
    g.close()
    assert rep.status == 0 and rep.rel_residual <= 1e-6
