"""An infinite diagonal entry (a penalty beyond the factor's range) in a front factored in
shared memory: its variable solves to zero, the others to the system without it."""
import numpy as np
import pytest

from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import ScalarCSC

pytestmark = pytest.mark.gpu


def upper(A):
    n = A.shape[0]
    cols = [np.arange(j + 1) for j in range(n)]
    Ap = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int64)
    return ScalarCSC(n, Ap, np.concatenate(cols).astype(np.int64), np.concatenate([A[c, j] for j, c in enumerate(cols)]))


@pytest.mark.parametrize("n,at", [(1, 0), (12, 0), (12, 6), (12, 11), (97, 42)])
@pytest.mark.parametrize("single", [False, True])
def test_infinite_diagonal_solves_to_zero(n, at, single):
    rng = np.random.default_rng(n + at)
    A = rng.normal(size=(n, n)) / n
    A = A + A.T + 4.0 * np.eye(n)
    A[at, at] = 1e39 if single else np.inf                # 1e39: infinite in the FP32 factor
    cols = [np.arange(j + 1) for j in range(n)]
    Ap = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int64)
    H = ScalarCSC(n, Ap, np.concatenate(cols).astype(np.int64), np.concatenate([A[c, j] for j, c in enumerate(cols)]))
    f = B200Factorizer(single, refine=False, orderingMethod=OrderingMethod.Native)
    f.factorizeSymbolic(H)
    f.factorizeNumeric(H)
    b = rng.normal(size=(n, 2))
    x = f.solveMultiRHS(b)
    others = np.delete(np.arange(n), at)
    want = np.zeros((n, 2))
    want[others] = np.linalg.solve(A[np.ix_(others, others)], b[others])
    # condition about 3: n eps of the factor's type
    tol = n * (1.2e-7 if single else 2.3e-16) * 8
    assert np.all(x[at] == 0.0)
    assert np.abs(x - want).max() <= tol * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("w", [5, 6, 7, 8, 65, 70])
@pytest.mark.parametrize("single", [False, True])
def test_infinite_diagonal_in_the_last_columns_of_a_front_with_structure(w, single):
    # two dense fronts: the structure rows of the first start at w, its boxes at a multiple of 4
    n, at = w + 30, w - 1
    rng = np.random.default_rng(n)
    A = rng.uniform(-1.0, 1.0, size=(n, n)) / n           # eigenvalues of A + A^T within 2 of 0
    A = A + A.T + 4.0 * np.eye(n)
    A[at, at] = 1e39 if single else np.inf
    H = upper(A)
    f = B200Factorizer(single, refine=False, orderingMethod=OrderingMethod.Native, relax=False)
    f.factorizeSymbolic(H, supernode_sizes=[w, 30])
    f.factorizeNumeric(H)
    for nrhs in (1, 2, 3, 8):
        b = rng.normal(size=(n, nrhs))
        x = f.solveMultiRHS(b)
        others = np.delete(np.arange(n), at)
        want = np.zeros((n, nrhs))
        want[others] = np.linalg.solve(A[np.ix_(others, others)], b[others])
        tol = n * (1.2e-7 if single else 2.3e-16) * 8
        assert np.all(x[at] == 0.0)
        assert np.abs(x - want).max() <= tol * max(1.0, np.abs(want).max())
