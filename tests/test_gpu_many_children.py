"""Fronts with many children (a wide separator over many small parts): at the number of
children from which on a front has lists of them, lists of more and fewer than 32 entries,
children of more and fewer than 32 rows, hubs factored whole and by blocks, with and without
a front above them, above and below the cut of the solves."""
import numpy as np
import pytest

from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import BlockCSCHessian

pytestmark = pytest.mark.gpu


def hub_matrix(leaves, wl, hub, per, top, bs, seed):
    """`leaves` dense parts of wl nodes, each coupled to `per` of the hub's nodes; the hub dense and
    coupled to `top` nodes above it. Diagonally dominant: dense A and its block Hessian."""
    rng = np.random.default_rng(seed)
    nb = leaves * wl + hub + top
    P = np.zeros((nb, nb), dtype=bool)
    h0 = leaves * wl
    for i in range(leaves):
        part = slice(i * wl, (i + 1) * wl)
        P[part, part] = True
        P[part, h0 + rng.choice(hub, size=per, replace=False)] = True
    P[h0:, h0:] = True
    P = np.triu(P)
    A = np.kron(P, np.ones((bs, bs))) * rng.uniform(-1.0, 1.0, size=(nb * bs, nb * bs))
    A = np.triu(A, 1)
    A = A + A.T
    A[np.arange(nb * bs), np.arange(nb * bs)] = np.abs(A).sum(axis=1) + 1.0
    Ap, Ai, Ax = [0], [], []
    for j in range(nb):
        rows = np.nonzero(P[:, j])[0]
        Ai.append(rows)
        Ap.append(Ap[-1] + rows.size)
        for i in rows:                                    # a block column-major
            Ax.append(A[i * bs:(i + 1) * bs, j * bs:(j + 1) * bs].T.reshape(-1))
    return A, BlockCSCHessian(nb, np.array(Ap, dtype=np.int64), np.concatenate(Ai).astype(np.int64), bs, np.concatenate(Ax))


CASES = {
    # leaves, nodes of a leaf, hub, hub nodes of a leaf, top, block size
    "sixteen": (16, 2, 20, 5, 0, 1),
    "seventeen": (17, 2, 20, 5, 0, 1),
    "structure": (17, 3, 21, 5, 9, 1),
    "long_lists": (90, 1, 7, 5, 6, 1),
    "long_rows": (20, 2, 90, 70, 10, 1),
    "large_hub": (40, 2, 270, 45, 30, 1),
    "blocks": (40, 1, 17, 4, 3, 3),
    "large_blocks": (24, 2, 90, 13, 12, 3),
}


@pytest.mark.parametrize("cut", [0, 8])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("case", sorted(CASES))
def test_many_children_match_dense(case, single, cut):
    leaves, wl, hub, per, top, bs = CASES[case]
    A, H = hub_matrix(leaves, wl, hub, per, top, bs, seed=len(case))
    f = B200Factorizer(single, orderingMethod=OrderingMethod.Native, relax=False, solve_subtrees=cut)
    f.factorizeSymbolic(H, supernode_sizes=[wl] * leaves + [hub] + ([top] if top else []))
    f.factorizeNumeric(H)
    rng = np.random.default_rng(7)
    # diagonally dominant: each row's error within a few eps of its sums
    tol = A.shape[0] * (1.2e-7 if single else 2.3e-16) * 8
    for nrhs in (1, 3, 9):
        B = rng.normal(size=(A.shape[0], nrhs))
        want = np.linalg.solve(A, B)
        assert np.abs(f.solveMultiRHS(B) - want).max() <= tol * np.abs(want).max(), nrhs


def test_memory_of_a_wide_separator_over_many_leaves():
    # a map per child of as many entries as the hub has rows would be 160 MB
    torch = pytest.importorskip("torch")
    leaves, hub, per = 40000, 1000, 3
    rng = np.random.default_rng(0)
    touch = (rng.integers(0, hub // per, size=(leaves, 1)) + hub // per * np.arange(per)).astype(np.int64)
    by_hub = np.argsort(touch.reshape(-1), kind="stable") // per
    count = np.bincount(touch.reshape(-1), minlength=hub)
    start = np.concatenate([[0], np.cumsum(count)])
    Ai = [np.arange(leaves)] + [np.concatenate([by_hub[start[j]:start[j + 1]], leaves + np.arange(j + 1)])
                                for j in range(hub)]
    Ap = np.concatenate([np.arange(leaves + 1), leaves + np.cumsum(count + np.arange(1, hub + 1))])
    H = BlockCSCHessian(leaves + hub, Ap.astype(np.int64), np.concatenate(Ai).astype(np.int64), 1)
    f = B200Factorizer(orderingMethod=OrderingMethod.Native, relax=False)
    f.factorizeSymbolic(BlockCSCHessian(1, [0, 1], [0], 1))            # the context and what every handle has
    free = torch.cuda.mem_get_info()[0]
    f.factorizeSymbolic(H, supernode_sizes=[1] * leaves + [hub])
    grown = free - torch.cuda.mem_get_info()[0]
    reported = f.stats()["device_bytes"]
    assert grown < 120e6
    assert reported > grown - 32e6
