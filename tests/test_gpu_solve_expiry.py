"""A dependency wait of the solves above the cut that runs into its limit: the call reports
MFS_TIMEOUT, and the handle solves again once the counts are right."""
import ctypes

import numpy as np
import pytest

from meshfemsparse_b200 import _lib
from meshfemsparse_b200.factorizer import B200Factorizer, OrderingMethod
from meshfemsparse_b200.hessian import ScalarCSC

pytestmark = pytest.mark.gpu

WIDTHS = [66, 301, 130]                                   # two fronts below one of three 64-row parts


def matrix():
    n = sum(WIDTHS)
    rng = np.random.default_rng(7)
    A = rng.normal(size=(n, n)) / n
    A[:WIDTHS[0], WIDTHS[0]:WIDTHS[0] + WIDTHS[1]] = 0.0
    A = np.triu(A) + np.triu(A, 1).T + 4.0 * np.eye(n)
    cols = [np.nonzero(A[:j + 1, j])[0] for j in range(n)]
    Ap = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int64)
    return A, ScalarCSC(n, Ap, np.concatenate(cols).astype(np.int64),
                        np.concatenate([A[c, j] for j, c in enumerate(cols)]))


def add_to_counts(f, forward, delta):
    _lib.check(_lib.load().mfs_debug_solve_counts(f._h, int(forward), delta), f._h)


@pytest.mark.parametrize("nrhs", [1, 9])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("forward", [True, False])
def test_expired_wait_is_reported_and_leaves_the_handle_usable(forward, single, nrhs):
    A, H = matrix()
    f = B200Factorizer(single, refine=single, orderingMethod=OrderingMethod.Native, relax=False)
    f.factorizeSymbolic(H, supernode_sizes=WIDTHS)
    f.factorizeNumeric(H)
    B = np.random.default_rng(1).normal(size=(H.n, nrhs))
    add_to_counts(f, forward, 1)
    with pytest.raises(_lib.MFSError) as e:
        f.solveMultiRHS(B)
    assert e.value.status == _lib.MFS_TIMEOUT
    add_to_counts(f, forward, -1)
    X = f.solveMultiRHS(B)
    want = np.linalg.solve(A, B)
    # condition about 3: FP64 to n eps, the refined FP32 factor to its residual target
    assert np.abs(X - want).max() <= (3e-10 if single else 1e-12) * np.abs(want).max()


def test_counts_hook_refuses_a_handle_without_an_analysis():
    f = B200Factorizer()
    assert _lib.load().mfs_debug_solve_counts(f._h, 1, 1) == _lib.MFS_INVALID_ARG
    assert _lib.load().mfs_debug_solve_counts(ctypes.c_void_p(), 1, 1) == _lib.MFS_INVALID_ARG
