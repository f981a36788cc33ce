"""Superblock inverses of a forest: diagonal blocks without stored inverses, few of them
(substitution per 16 columns) and many (inverted first), beside fronts with stored ones."""
import numpy as np
import pytest

from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import ScalarCSC

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 100, 257]


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("single", [False, True])
def test_block_diagonal_solves_match_dense(single, many):
    # one dense block per size, the sizes up to 64 a hundred times each when there are many
    sizes = np.concatenate([np.repeat([s for s in SIZES if s <= 64], 100 if many else 1), [s for s in SIZES if s > 64]])
    rng = np.random.default_rng(int(sizes.size))
    blocks, Ap, Ai, Ax = [], [0], [], []
    for n in sizes:
        A = rng.uniform(-1.0, 1.0, size=(n, n)) / n       # eigenvalues of A + A^T within 2 of 0
        A = A + A.T + 4.0 * np.eye(n)
        start = len(Ap) - 1
        for j in range(n):
            Ai.append(start + np.arange(j + 1))
            Ax.append(A[:j + 1, j])
            Ap.append(Ap[-1] + j + 1)
        blocks.append(A)
    H = ScalarCSC(len(Ap) - 1, np.array(Ap, dtype=np.int64), np.concatenate(Ai).astype(np.int64), np.concatenate(Ax))
    f = B200Factorizer(single, orderingMethod=OrderingMethod.Native)
    f.factorizeSymbolic(H)
    f.factorizeNumeric(H)
    B = rng.normal(size=(H.n, 2))
    X = f.solveMultiRHS(B)
    want = np.concatenate([np.linalg.solve(A, b) for A, b in zip(blocks, np.split(B, np.cumsum(sizes)[:-1]))])
    # condition about 3: n eps of the factor's type, times a constant of the triangular solves
    tol = 257 * (1.2e-7 if single else 2.3e-16) * 8
    assert np.abs(X - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("single", [False, True])
def test_many_superblocks_match_dense(single, many):
    # on both sides of the superblock count from which FP32 inverses take 32 columns a CTA
    sizes = np.repeat([65, 70, 129, 161, 200, 257], 90 if many else 20)
    rng = np.random.default_rng(int(sizes.size))
    blocks, Ap, Ai, Ax = [], [np.zeros(1, dtype=np.int64)], [], []
    start = 0
    for n in sizes:
        A = rng.uniform(-1.0, 1.0, size=(n, n)) / n       # eigenvalues of A + A^T within 2 of 0
        A = A + A.T + 4.0 * np.eye(n)
        j, i = np.tril_indices(n)                         # the upper triangle by columns
        Ai.append(start + i)
        Ax.append(A[i, j])
        Ap.append(Ap[-1][-1] + np.cumsum(np.arange(1, n + 1)))
        blocks.append(A)
        start += n
    H = ScalarCSC(start, np.concatenate(Ap).astype(np.int64), np.concatenate(Ai).astype(np.int64), np.concatenate(Ax))
    f = B200Factorizer(single, orderingMethod=OrderingMethod.Native)
    f.factorizeSymbolic(H)
    f.factorizeNumeric(H)
    B = rng.normal(size=(start, 2))
    X = f.solveMultiRHS(B)
    want = np.concatenate([np.linalg.solve(A, b) for A, b in zip(blocks, np.split(B, np.cumsum(sizes)[:-1]))])
    # condition about 3: n eps of the factor's type, times a constant of the triangular solves
    tol = 257 * (1.2e-7 if single else 2.3e-16) * 8
    assert np.abs(X - want).max() <= tol * np.abs(want).max()
