"""The one-launch forward and backward solves above the cut: widths around the 64-row parts,
the 256-row superblocks and the 4-row alignment of the structure rows, one or several
children, every vector count of a pass and one more."""
import numpy as np
import pytest

from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import ScalarCSC

pytestmark = pytest.mark.gpu

# supernode widths and, for each, whether it starts a new chain below the last one
SHAPES = {
    "chain": ([1, 63, 64, 65, 130], None),
    "superblocks": ([255, 256, 257, 513], None),
    "two_children": ([66, 301, 194], 2),
    "five_children": ([5, 70, 3, 128, 259, 67], 5),
}


def matrix(widths, leaves):
    """Diagonally dominant: dense (a chain), or `leaves` dense blocks coupled to the last."""
    n = sum(widths)
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n)) / n
    if leaves:
        start = np.concatenate([[0], np.cumsum(widths)])
        for i in range(leaves):
            for j in range(leaves):
                if i != j:
                    A[start[i]:start[i + 1], start[j]:start[j + 1]] = 0.0
    A = A + A.T + 4.0 * np.eye(n)
    U = np.triu(A)
    cols = [np.nonzero(U[:, j])[0] for j in range(n)]
    Ap = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int64)
    Ai = np.concatenate(cols).astype(np.int64)
    return A, ScalarCSC(n, Ap, Ai, np.concatenate([U[c, j] for j, c in enumerate(cols)]))


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_one_launch_solves_match_dense(shape, single):
    widths, leaves = SHAPES[shape]
    A, H = matrix(widths, leaves)
    f = B200Factorizer(single, refine=single, orderingMethod=OrderingMethod.Native, relax=False)
    f.factorizeSymbolic(H, supernode_sizes=widths)
    f.factorizeNumeric(H)
    rng = np.random.default_rng(1)
    for nrhs in (1, 2, 3, 4, 5, 8, 9):
        B = rng.normal(size=(H.n, nrhs))
        X = f.solveMultiRHS(B)
        want = np.linalg.solve(A, B)
        # condition about 3: FP64 to n eps, the refined FP32 factor to its residual target
        tol = 3e-10 if single else 1e-12
        assert np.abs(X - want).max() <= tol * np.abs(want).max(), nrhs
