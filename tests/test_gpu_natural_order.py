"""Elimination orders that are no postorder of their forest: trees whose variables take turns in
the order (natural and user orders), with enough trees for a cut of the solves by default
and with few and one asked for."""
import numpy as np
import pytest

from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import BlockCSCHessian

pytestmark = pytest.mark.gpu


def interleaved(trees, rows, bs, shuffle):
    """`trees` binary trees of `rows` nodes (node i's parent is i // 2 from the last on), node by node
    across the trees; shuffled: parents after their children, else anything."""
    rng = np.random.default_rng(trees + rows)
    place = np.arange(trees * rows).reshape(rows, trees).T.copy()      # [tree][node, children first]
    if shuffle:
        depth = np.floor(np.log2(rows - np.arange(rows))).astype(int)
        order = np.lexsort((rng.random(trees * rows), -np.tile(depth, trees)))
        place = np.empty(trees * rows, dtype=np.int64)
        place[order] = np.arange(trees * rows)
        place = place.reshape(trees, rows)
    n = trees * rows
    pairs = {(j, j) for j in range(n)}
    for t in range(trees):
        for i in range(rows - 1):                         # node rows - k has the parent rows - k // 2
            a, b = place[t, i], place[t, rows - (rows - i) // 2]
            pairs.add((min(a, b), max(a, b)))
    pairs = sorted(pairs, key=lambda p: (p[1], p[0]))
    Ap = np.concatenate([[0], np.cumsum(np.bincount([j for _, j in pairs], minlength=n))]).astype(np.int64)
    A = np.zeros((n * bs, n * bs))
    Ax = []
    for i, j in pairs:
        B = rng.uniform(-1.0, 1.0, size=(bs, bs))
        if i == j:
            B = B + B.T + 12.0 * bs * np.eye(bs)
        A[i * bs:(i + 1) * bs, j * bs:(j + 1) * bs] = B
        A[j * bs:(j + 1) * bs, i * bs:(i + 1) * bs] = B.T
        Ax.append(B.T.reshape(-1))
    return A, BlockCSCHessian(n, Ap, np.array([i for i, _ in pairs], dtype=np.int64), bs, np.concatenate(Ax))


@pytest.mark.parametrize("order", ["natural", "user"])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("relax", [False, True])
@pytest.mark.parametrize("trees,rows,bs,cut,shuffle", [(160, 7, 1, 0, False), (160, 7, 1, 0, True), (5, 31, 3, 2, False),
                                                        (5, 31, 3, 4, True), (3, 100, 2, 2, True)])
def test_interleaved_trees_match_dense(trees, rows, bs, cut, shuffle, relax, single, order):
    A, H = interleaved(trees, rows, bs, shuffle)
    f = B200Factorizer(single, orderingMethod=OrderingMethod.Native if order == "natural" else OrderingMethod.User,
                       relax=relax, solve_subtrees=cut)
    f.factorizeSymbolic(H, **({} if order == "natural" else {"user_perm": np.arange(H.numBlocks)}))
    f.factorizeNumeric(H)
    # diagonally dominant, condition below 3: n eps of the factor's type
    tol = rows * bs * (1.2e-7 if single else 2.3e-16) * 8
    for nrhs in (1, 6):
        B = np.random.default_rng(1).normal(size=(A.shape[0], nrhs))
        want = np.linalg.solve(A, B)
        assert np.abs(f.solveMultiRHS(B) - want).max() <= tol * np.abs(want).max()
