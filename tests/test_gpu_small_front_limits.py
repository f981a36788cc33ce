"""Fronts factored whole and solved by one warp at the borders of their rows per lane, up to
the largest that small_front_max allows, below the cut of the solves (six trees of two
fronts) and above it."""
import numpy as np
import pytest

from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import ScalarCSC

pytestmark = pytest.mark.gpu

FRONTS = [64, 65, 96, 97, 160, 161, 169, 170, 192, 193, 241]


@pytest.mark.parametrize("cut", [0, 6])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("front", FRONTS)
def test_front_rows_match_dense(front, single, cut):
    limit = 241 if single else 170
    if front > limit:
        pytest.skip("above the largest front of the type")
    trees, w = 6, 35
    rng = np.random.default_rng(front)
    A = rng.uniform(-1.0, 1.0, size=(front, front)) / front   # eigenvalues of A + A^T within 2 of 0
    A = A + A.T + 4.0 * np.eye(front)
    cols = [np.arange(j + 1) for j in range(front)]
    one = np.concatenate([A[c, j] for j, c in enumerate(cols)])
    Ap = np.concatenate([[0], np.cumsum(np.tile([c.size for c in cols], trees))]).astype(np.int64)
    Ai = np.concatenate([np.concatenate(cols) + t * front for t in range(trees)]).astype(np.int64)
    H = ScalarCSC(trees * front, Ap, Ai, np.tile(one, trees))
    f = B200Factorizer(single, orderingMethod=OrderingMethod.Native, relax=False, small_front_max=limit,
                       solve_subtrees=cut)
    f.factorizeSymbolic(H, supernode_sizes=[w, front - w] * trees)
    f.factorizeNumeric(H)
    # condition about 3: n eps of the factor's type, times a constant of the triangular solves
    tol = front * (1.2e-7 if single else 2.3e-16) * 8
    for nrhs in (1, 3, 5, 8):
        B = rng.normal(size=(H.n, nrhs))
        want = np.concatenate([np.linalg.solve(A, b) for b in np.split(B, trees)])
        assert np.abs(f.solveMultiRHS(B) - want).max() <= tol * np.abs(want).max(), nrhs
