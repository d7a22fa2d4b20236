"""Faces that outgrow the clipper's shared-memory pools, on the routes their number decides: a short
list finished by one kernel, a long one whose rest goes to the local-memory clipper's kernel, and
one whose rest the list array has no room for a second time.  Against the local-memory clipper on
every face: the same pieces in the same order, so the same bits."""
import numpy as np
import pytest

import scenes

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu

SHORT = 152 * 4 * 2     # a face a warp of k_clip32_deferred


def step(n, vel, cfl, fast):
    g = fia.Grid3D(n, n, n, 1.0 / n, precision=fia.FIA_FP32C)
    for name, a in zip(("u", "v", "w", "density"), (*vel, scenes.gaussian_blobs(n, seed=4))):
        g.set(name, a.ravel())
    before = g.debug_clip_fast(fast)
    st = g.move_substances_3D(cfl / n, fia.advect_params(enable_eliminate_zero_velocity_false_diffusion=False))
    out = g.get("density"), g.debug_clip_fast() - before, list(g.pass_counters())[:3], st
    g.close()
    return out


@pytest.mark.parametrize("n,cfl,long", [(12, 3.0, False), (24, 16.0, True), (64, 8.0, True)])
def test_listed_faces(n, cfl, long):
    vel = scenes.fourier_velocity(n, seed=6)
    a, listed, ca, sa = step(n, vel, cfl, 1)
    b, faces, cb, sb = step(n, vel, cfl, 0)
    assert (listed > SHORT) == long and listed > 0 and faces == ca[0]
    assert sa == sb == 0
    assert ca == cb
    assert np.array_equal(a, b)


def test_no_room_for_the_rest_of_the_list():
    """vertices displaced by four cells to and fro along x: every second y- and z-face spans nine cells in
    x, the others seven, but for the four layers at either wall, and both pools end before the seventh
    iso-line (4 + 2 vertices a line, 15 and 16 at most).  So more faces are left over than the list array
    has room for behind the list."""
    n = 48
    u = np.zeros((n + 1, n, n))
    u[:] = np.where(np.arange(n + 1) % 2, 1.0, -1.0)[:, None, None]
    vel = (u, np.zeros((n, n + 1, n)), np.zeros((n, n, n + 1)))
    a, listed, ca, sa = step(n, vel, 4.0, 1)
    b, faces, cb, sb = step(n, vel, 4.0, 0)
    assert listed + 2 * (n - 8) * n * (n + 1) > 3 * (n + 2) ** 3 and faces == ca[0]
    assert sa == sb == 0
    assert ca == cb
    assert np.array_equal(a, b)
