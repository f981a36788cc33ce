"""An infinite diagonal entry (a penalty beyond the factor's range) in a front factored in
shared memory: its variable solves to zero, the others to the system without it."""
import numpy as np
import pytest

from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import ScalarCSC

pytestmark = pytest.mark.gpu


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
