"""A projection beside a long kernel of another stream that holds one SM: the one-kernel solver does not
wait for it, at a size whose blocks take all the SMs it asks for."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [fia.FIA_FP32C, fia.FIA_FP64])
def test_projection_does_not_wait_for_a_resident_kernel(precision):
    n = 112
    g = fia.Grid3D(n, n, n, 1.0 / n, precision=precision)
    rng = np.random.default_rng(1)
    for c in "uvw":
        g.set(c, rng.normal(size=g.sizes()[c]))
    sp = fia.solver_params(tol=1e-4)
    want = g.calc_pressure_3D(sp)
    g.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(2 * 10 ** 9)      # one thread, about a second
    got = g.calc_pressure_3D(sp)
    running = not side.query()
    side.synchronize()
    g.close()
    assert running
    assert got.status == 0 and got.iterations == want.iterations
