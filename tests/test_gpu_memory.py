"""What a session allocates after its creation, when there is no memory for it (the allocation made to
fail on the host): the z-records are given back and the call succeeds, with the outputs of a session that
had none; where that does not help, the call fails and succeeds later."""
import os

import numpy as np
import pytest

import scenes

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu

N = 16
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WEIGHTS = os.path.join(ROOT, "flux-interpolated-advection_gb300", "weights", "unet_precond.f32")


def small_store(g):
    g.debug_set_piece_capacity(64)


def weights(g):
    g.learned_set_weights(np.fromfile(WEIGHTS, dtype="<f4"))


def pair(g):
    rng = np.random.default_rng(2)
    return g.learned_add_pair(*(rng.normal(size=(2, N ** 3)).astype(np.float32)))


def learned(g):
    return g.calc_pressure_gradient_term_3D(fia.solver_params(tol=1e-4, method=fia.FIA_SOLVER_FCG_LEARNED, fallback_iter=50))


# what comes before, the call, and the forms it exists in
CALLS = {
    "pieces": (small_store, lambda g: g.move_substances_3D(2.0 / N, fia.advect_params()), (0, 1)),
    "maccormack": (None, lambda g: g.move_substances_3D(2.0 / N, fia.advect_params(use_MacCormack_scheme=True)), (0, 1)),
    "volumes": (None, lambda g: g.move_substances_3D(2.0 / N, fia.advect_params(enable_cell_volume_correction=True)), (0, 1)),
    "solids": (None, lambda g: g.set_solid_spheres([[0.5, 0.5, 0.5]], [0.2]), (0, 1)),
    "refinement": (None, lambda g: g.calc_pressure_gradient_term_3D(fia.solver_params(tol=1e-5)), (1,)),
    "network": (None, weights, (1,)),
    "pair": (weights, pair, (1,)),
    "directions": (weights, learned, (1,)),
}


def session(fp32, before):
    g = fia.Grid3D(N, N, N, 1.0 / N, precision=fia.FIA_FP32C if fp32 else fia.FIA_FP64)
    for name, a in zip(("u", "v", "w", "density"), (*scenes.fourier_velocity(N, seed=6), scenes.gaussian_blobs(N, seed=4))):
        g.set(name, a)
    if before:
        before(g)
    return g


def fields(g):
    return [g.get(c) for c in ("density", "u", "v", "w")]


@pytest.mark.parametrize("name,fp32", [(n, f) for n, c in CALLS.items() for f in c[2]])
def test_records_give_way(name, fp32):
    before, call, _ = CALLS[name]
    g = session(fp32, before)
    g.debug_records(0)
    call(g)
    want = fields(g)
    g.close()

    g = session(fp32, before)
    assert g.debug_records() == 1
    g.debug_fail_allocations(1)
    call(g)
    assert g.debug_fail_allocations() == 0 and g.debug_records() == 0
    got = fields(g)
    g.close()
    # the records may have served part of the call: the bound between both routes
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) <= (2e-6 if fp32 else 1e-10) * np.linalg.norm(b)


@pytest.mark.parametrize("name,fp32", [(n, f) for n, c in CALLS.items() for f in c[2]])
def test_no_memory_at_all(name, fp32):
    before, call, _ = CALLS[name]
    g = session(fp32, before)
    start = fields(g)
    g.debug_fail_allocations(1000)
    with pytest.raises(fia.FiaError):
        call(g)
    g.debug_fail_allocations(0)
    for a, b in zip(fields(g), start):
        assert np.array_equal(a, b)
    call(g)
    got = fields(g)
    g.close()
    g = session(fp32, before)
    g.debug_records(0)
    call(g)
    want = fields(g)
    g.close()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
