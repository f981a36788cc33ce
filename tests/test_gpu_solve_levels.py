"""The solves by levels above the cut (solve_chain = 1): widths around the 64-row blocks, several
children, more right-hand sides than a pass, and the switch between the two forms on a
handle that has a factor."""
import numpy as np
import pytest

from meshfemsparse_b200 import B200Factorizer, SystemAssembler, fem
from meshfemsparse_b200.factorizer import OrderingMethod
from test_gpu_solve_dataflow import SHAPES, matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_solves_by_levels_match_dense(shape, single):
    widths, leaves = SHAPES[shape]
    A, H = matrix(widths, leaves)
    f = B200Factorizer(single, refine=single, orderingMethod=OrderingMethod.Native, relax=False, solve_chain=1)
    f.factorizeSymbolic(H, supernode_sizes=widths)
    f.factorizeNumeric(H)
    rng = np.random.default_rng(1)
    for nrhs in (1, 9, 17):
        B = rng.normal(size=(H.n, nrhs))
        want = np.linalg.solve(A, B)
        # condition about 3: FP64 to n eps, the refined FP32 factor to its residual target
        tol = 3e-10 if single else 1e-12
        assert np.abs(f.solveMultiRHS(B) - want).max() <= tol * np.abs(want).max(), nrhs


@pytest.mark.parametrize("first", [0, 1])
def test_both_forms_solve_the_same_cube(first):
    nodes, tets = fem.tet_cube(9, jitter=0.1, seed=2)
    H = SystemAssembler(nodes.shape[0]).blockSparsityPattern(tets)
    pins = fem.bottom_pins(nodes)
    b = np.random.default_rng(3).normal(size=(3 * nodes.shape[0], 3))
    b[pins] = 0.0
    X = []
    for chain in (first, 1 - first):
        f = B200Factorizer(solve_chain=chain, solve_subtrees=16)
        f.factorizeSymbolic(H, pins)
        f.setElements(tets)
        f.assemble(fem.linear_elastic_hessians(nodes, tets, np.ones(tets.shape[0]), 0.3), return_values=False)
        f.factorizeAssembled()
        X.append(f.solveMultiRHS(b))
        # backward stable solves with one factor: residuals of n eps
        r = np.abs(f.apply(X[-1]) - b)
        r[pins] = 0.0
        assert r.max() <= 1e-10 * np.abs(b).max()
    assert np.abs(X[0] - X[1]).max() <= 1e-10 * np.abs(X[0]).max()
