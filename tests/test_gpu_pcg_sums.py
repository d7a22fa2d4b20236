"""The sums of the one-kernel Jacobi-PCG, FP64 from the warps' float pairs on.

A right-hand side of isolated cells 6 * 2^k inside the grid makes the first iteration exact: z = 2^k
there, B z = 6 * 2^k there and -2^k at the six neighbours, alpha = 1, and the residual is 2^k at the
neighbours.  With one cell k = 0 and others k = -13 and k = -24 the sums of squares are multiples of
2^-48 below 2^3, and of 9 * 2^-46 below 2^6: exact in FP64, and exact in a float pair within every warp (no small cell is near the
large one's lines), but not in a float pair across warps or blocks.  So the reported residual is the
rounded quotient's root to the last bit.
"""
import math

import numpy as np
import pytest

fia = pytest.importorskip("fia")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
def test_residual_sum_is_exact(seed):
    n = 32
    rng = np.random.default_rng(seed)
    exponent = rng.choice([-13, -24], size=(10, 10, 10))
    exponent[:3, 3:6] = -99
    exponent[1, 4, 4] = 0
    used = exponent > -99
    rhs = np.zeros((n, n, n))
    rhs[1:29:3, 1:29:3, 1:29:3] = np.where(used, 6.0 * 2.0 ** np.maximum(exponent, -30), 0.0)
    units = sum(4 ** int(24 + e) for e in exponent[used])     # the sum of 4^k in units of 4^-24
    bb, rr = 36 * units * 2.0 ** -48, 6 * units * 2.0 ** -48
    assert 9 * units < 2 ** 53
    g = fia.Grid3D(n, n, n, 1.0, precision=fia.FIA_FP32C)
    x, rep = g.debug_solve_rhs(rhs.astype(np.float32), fia.solver_params(tol=1e-9, max_iter=1))
    g.close()
    assert rep.iterations == 1
    assert np.array_equal(x.reshape(rhs.shape), rhs / 6.0)
    assert rep.rel_residual == math.sqrt(rr / bb)
