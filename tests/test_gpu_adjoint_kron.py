"""Adjoint of the Kronecker-core operators on every route of its quadratic
form: Hadamard transforms of the full space (one, two and three tile passes,
both signs of betaJ), of the half space (flip-symmetric vectors), and pruned
along the prefix tree (odd and even widths, 3D), against central differences.

Bar: 2e-6 of max(|grad|, 1), as the other finite-difference checks (eigenvalues
to 1e-13, step 1e-5).
"""
import numpy as np
import pytest

import latttmat_gb300 as lt

pytestmark = pytest.mark.gpu
STEP = 1e-5


def _solve(pt, bj, k, h):
    model, dim, ax, ec, _, _, _, size = pt
    op = lt.TMatOp(model, dim, ax, bj, k, h, size, 0.0, ec)
    vals, vecs, _, _ = op.eigs(1, ncv=12, tol=1e-13, vectors=True)
    return op, vals[0], vecs[0]


@pytest.mark.parametrize("pt", [
    ("A", 2, 1, 0, 0.4, 0.3, 0.1, 8), ("A", 2, 1, 0, -0.4, 0.3, 0.1, 11), ("A", 2, 1, 0, 0.4, 0.3, 0.1, 19),
    ("A", 2, 5, 2, 0.4, 0.3, 0.05, 9), ("A", 2, 5, 2, 0.4, 0.6, 0.05, 13), ("A", 2, 5, 0, 0.4, 0.3, 0.0, 13),
    ("A", 2, 5, 2, -0.3, 0.3, 0.05, 15), ("A", 2, 5, 0, 0.4, 0.3, 0.0, 16), ("A", 2, 5, 2, 0.3, 0.6, 0.05, 18),
    ("A", 2, 13, 2, 0.4, 0.6, 0.05, 13), ("A", 3, 1, 0, 0.25, 0.4, 0.05, (3, 5)), ("A", 3, 1, 0, 0.25, 0.4, 0.0, (3, 5)),
])
def test_grad_routes(pt):
    bj, k, h = pt[4:7]
    op, lam, v = _solve(pt, bj, k, h)
    g = op.grad(v, lam * op.getnormfactor())
    again = op.grad(v, lam * op.getnormfactor())  # tables built by the first call are kept
    np.testing.assert_array_equal(g, again)
    for t, dp in ((0, (STEP, 0.0, 0.0)), (1, (0.0, STEP, 0.0)), (3, (0.0, 0.0, STEP))):
        if t == 3 and h == 0.0:
            continue  # the flip-reduced sector is only defined at h = 0
        up = _solve(pt, bj + dp[0], k + dp[1], h + dp[2])[1]
        dn = _solve(pt, bj - dp[0], k - dp[1], h - dp[2])[1]
        fd = (np.log(up) - np.log(dn)) / (2 * STEP)
        assert abs(g[t] - fd) < 2e-6 * max(1.0, abs(fd)), (t, g[t], fd)
