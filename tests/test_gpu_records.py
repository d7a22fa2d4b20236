"""WENO6 quadrature in a session without z-records (no memory for them): the same stencils, formed from
the samples.  Velocity passes of the FP32 form are the same bits either way; the others hold the
bounds of tests/test_gpu_quadrature.py against the oracle."""
import numpy as np
import pytest

import scenes
from oracle import Oracle

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu

O = Oracle()


def scene(shape, comp):
    n = max(shape)
    nx, ny, nz = shape
    u, v, w = scenes.fourier_velocity(n, seed=3)
    u = u.reshape(n + 1, n, n)[:nx + 1, :ny, :nz].ravel()
    v = v.reshape(n, n + 1, n)[:nx, :ny + 1, :nz].ravel()
    w = w.reshape(n, n, n + 1)[:nx, :ny, :nz + 1].ravel()
    f = (u, v, w)[comp] if comp >= 0 else scenes.gaussian_blobs(n, seed=4).reshape(n, n, n)[:nx, :ny, :nz].ravel()
    return u, v, w, f


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 7, 2), (12, 9, 33)])
@pytest.mark.parametrize("comp", [-1, 0, 1, 2])
@pytest.mark.parametrize("k,integral,zero", [(1, 1, 0), (5, 1, 0), (3, 0, 0), (3, 0, 1)])
def test_pass_without_records(shape, comp, k, integral, zero):
    u, v, w, f = scene(shape, comp)
    h = 1.0 / max(shape)
    dt = 1.7 * h
    ref, _, _, _ = O.flux_pass(shape, h, u, v, w, comp, f, dt, 0, 1, integral, zero, (0.5, 0.5), k)
    for precision in (fia.FIA_FP64, fia.FIA_FP32C):
        g = fia.Grid3D(*shape, h, precision=precision)
        for name, a in (("u", u), ("v", v), ("w", w)):
            g.set(name, a)
        assert g.debug_records() == 1
        kept, _ = g.debug_flux_pass(comp, f, dt, 0, 1, integral, zero, (0.5, 0.5), k)
        assert g.debug_records(0) == 0
        got, st = g.debug_flux_pass(comp, f, dt, 0, 1, integral, zero, (0.5, 0.5), k)
        assert g.debug_records(1) == 1
        again, _ = g.debug_flux_pass(comp, f, dt, 0, 1, integral, zero, (0.5, 0.5), k)
        g.close()
        assert st == 0
        assert np.array_equal(again, kept)
        d = np.abs(got - ref)
        if precision == fia.FIA_FP64:
            assert np.linalg.norm(d) < 1e-10 * np.linalg.norm(ref)
        else:
            assert np.linalg.norm(d[np.argsort(d)[:-4]]) < 2e-6 * np.linalg.norm(ref)
            assert np.linalg.norm(d) < 5e-4 * np.linalg.norm(ref)
            if comp >= 0:
                assert np.array_equal(got, kept)


@pytest.mark.parametrize("precision", [fia.FIA_FP64, fia.FIA_FP32C])
def test_maccormack_step_without_records(precision):
    n = 20
    u, v, w, f = scene((n, n, n), -1)
    out = []
    for records in (1, 0):
        g = fia.Grid3D(n, n, n, 1.0 / n, precision=precision)
        for name, a in (("u", u), ("v", v), ("w", w), ("density", f)):
            g.set(name, a)
        g.debug_records(records)
        assert g.move_substances_3D(2.0 / n, fia.advect_params(use_MacCormack_scheme=True)) == 0
        out.append((g.get("density"), list(g.pass_counters())[:4]))
        g.close()
    bound = 1e-10 if precision == fia.FIA_FP64 else 2e-6
    assert np.linalg.norm(out[1][0] - out[0][0]) < bound * np.linalg.norm(out[0][0])
    assert out[0][1] == out[1][1]
