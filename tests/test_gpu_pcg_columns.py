"""The PCG's convergence, settled on the device: columns that end at different iterations, a
zero one among them, and caps inside and at the ends of the batches of iterations that
are launched ahead."""
import numpy as np
import pytest
import scipy.linalg

from meshfemsparse_b200 import B200Factorizer, SystemAssembler, fem
from meshfemsparse_b200.learned import pcg_solve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    nodes, tets = fem.tet_cube(3, jitter=0.1, seed=4)
    H = SystemAssembler(nodes.shape[0]).blockSparsityPattern(tets)
    f = B200Factorizer()
    pins = fem.bottom_pins(nodes)
    f.factorizeSymbolic(H, pins)
    f.setElements(tets)
    H.Ax = f.assemble(fem.linear_elastic_hessians(nodes, tets, np.ones(tets.shape[0]), 0.3))
    free = np.delete(np.arange(3 * nodes.shape[0]), pins)
    A = H.toScalar().to_dense()[np.ix_(free, free)]
    return f, A, free, 3 * nodes.shape[0]


def columns(A):
    """Right-hand sides that Jacobi PCG solves in 1 and 3 iterations, a zero and a general one."""
    D = np.diag(np.diag(A))
    _, V = scipy.linalg.eigh(A, D)
    n = A.shape[0]
    k = [0, n // 2, n - 1]
    return np.stack([D @ V[:, k[1]], (D @ V[:, k]).sum(axis=1), np.zeros(n),
                     np.random.default_rng(0).normal(size=n)], axis=1)


def iterations(A, b, tol):
    """Jacobi PCG in FP64: the iterations of one column."""
    if not b.any():
        return 0
    d = np.diag(A)
    x, r = np.zeros_like(b), b.copy()
    z = r / d
    p, rz = z.copy(), r @ z
    for it in range(1, 10000):
        q = A @ p
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        if np.linalg.norm(r) <= tol * np.linalg.norm(b):
            return it
        z = r / d
        rz, old = r @ z, rz
        p = z + rz / old * p
    raise AssertionError("no convergence")


@pytest.mark.parametrize("which", [[0], [2], [0, 2], [1, 0], [0, 1, 2, 3], [3]])
def test_columns_end_at_their_own_iterations(system, which):
    f, A, free, n = system
    tol = 1e-8
    b = columns(A)[:, which]
    B = np.zeros((n, len(which)))
    B[free] = b
    X, it, fallback = pcg_solve(f, B, None, maxit=2000, tol=tol)
    want = max(iterations(A, b[:, c], tol) for c in range(b.shape[1]))
    # the sums' order differs: a column next to its tolerance may take an iteration more or less in 30
    assert not fallback and abs(it - want) <= 1 + want // 30
    res = np.linalg.norm(A @ X[free] - b, axis=0)
    # the recurrence's residual and the true one differ by rounding
    assert np.all(res <= 1.01 * tol * np.linalg.norm(b, axis=0) + 1e-300)


@pytest.mark.parametrize("maxit", [1, 3, 4, 5, 13])
def test_caps(system, maxit):
    f, A, free, n = system
    B = np.zeros((n, 4))
    b = columns(A)
    B[free] = b
    X, it, fallback = pcg_solve(f, B, None, maxit=maxit, tol=1e-8)
    assert fallback and it == maxit                       # (the general column is not done)
    assert np.abs(A @ X[free] - b).max() <= 1e-10 * np.abs(b).max()
    X, it, fallback = pcg_solve(f, B[:, :3], None, maxit=maxit, tol=1e-8)
    assert fallback == (maxit < 3) and it == min(maxit, 3)
