"""psi (the running y-integral) in both forms at the edges of its runs of four cells and batches of
sixteen rows, for Gauss rules of one to fifteen points.  Bounds of tests/test_gpu_parity.py and
tests/test_gpu_fp32.py: 1e-12 of the largest value in the plain form, 2e-7 in the chosen form."""
import numpy as np
import pytest

import scenes
from oracle import Oracle

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu

O = Oracle()


@pytest.mark.parametrize("ny", [2, 3, 4, 5, 15, 16, 17, 33])
@pytest.mark.parametrize("comp", [-1, 0, 1, 2])
@pytest.mark.parametrize("mode,k", [(0, 1), (1, 1), (1, 3), (1, 15), (2, 1)])
def test_psi_rows(ny, comp, mode, k):
    n, shape = 35, (3, ny, 5)
    h = 1.0 / n
    M = [shape[d] + (d == comp) for d in range(3)]
    f = np.ascontiguousarray(scenes.gaussian_blobs(n, seed=4).reshape(n, n, n)[14:14 + M[0], :M[1], 15:15 + M[2]]).ravel()
    off = [0.0 if d == comp else 0.5 for d in range(3)]
    for precision, bound in ((fia.FIA_FP64, 1e-12), (fia.FIA_FP32C, 2e-7)):
        g = fia.Grid3D(*shape, h, precision=precision)
        a = f if precision == fia.FIA_FP64 else f.astype(np.float32).astype(np.float64)
        ref = O.psi(a, M, off, h, mode, k)
        got = g.debug_psi(comp, a, mode, k)
        g.close()
        assert np.abs(got - ref).max() <= bound * max(np.abs(ref).max(), 1.0 if bound < 1e-9 else 0.0)
