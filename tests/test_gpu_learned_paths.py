"""The learned preconditioner's kernels at the sizes where their dispatch changes: convolutions of
four x-planes a CTA with ragged tiles and one-CTA-per-SM layers against the mma.sync kernel (bound of
tests/test_gpu_learned.py), and flexible CG with z-lines of whole and broken groups of four cells,
with and without solids, judged by the FP64 residual formed apart from the solver."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu

WEIGHTS = os.path.join(ROOT, "flux-interpolated-advection_gb300", "weights", "unet_precond.f32")


@pytest.mark.parametrize("fine", [(260, 184, 180), (146, 250, 258)])
def test_plane_by_plane_convolutions_match_mma_path(fine):
    g = fia.Grid3D(*fine, 1.0 / fine[0], precision=fia.FIA_FP32C)
    g.learned_init(5)
    x0 = np.random.default_rng(4).normal(size=tuple(g.learned_level_dims(0))).astype(np.float32)
    assert g.debug_learned_tc(1) == 0
    y_tc = g.debug_unet_forward(x0)
    st = g.debug_learned_tc(0)
    y_ref = g.debug_unet_forward(x0)
    g.close()
    assert st == 0
    assert np.all(np.isfinite(y_tc))
    assert np.linalg.norm(y_tc - y_ref) < 1e-2 * np.linalg.norm(y_ref)


@pytest.mark.parametrize("shape", [(24, 20, 32), (20, 24, 30), (33, 18, 21)])
@pytest.mark.parametrize("solid", [False, True])
def test_fcg_direction_counts_and_groups(shape, solid):
    nx, ny, nz = shape
    h = 1.0 / nx
    g = fia.Grid3D(nx, ny, nz, h, precision=fia.FIA_FP32C)
    g.learned_set_weights(np.fromfile(WEIGHTS, dtype="<f4"))
    if solid:
        g.set_solid_spheres([[0.5, 0.4 * ny * h, 0.5 * nz * h]], [0.17])
    rng = np.random.default_rng(11)
    u = rng.normal(size=(nx + 1, ny, nz)); v = rng.normal(size=(nx, ny + 1, nz)); w = rng.normal(size=(nx, ny, nz + 1))
    u[[0, nx]] = 0.0
    v[:, [0, ny]] = 0.0
    w[:, :, [0, nz]] = 0.0
    for name, a in (("u", u), ("v", v), ("w", w)):
        g.set(name, a.ravel())
    rep = g.calc_pressure_gradient_term_3D(fia.solver_params(tol=1e-6, max_iter=5000, method=fia.FIA_SOLVER_FCG_LEARNED,
                                                             fallback_iter=400))
    g.close()
    assert rep.rel_residual <= 1e-6
    assert rep.fcg_iterations > 8     # every count of kept directions, the full ring last
