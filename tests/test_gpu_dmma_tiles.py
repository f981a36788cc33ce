"""FP64 GEMM on both sides of the tile count from which whole tiles are used, with odd operand
offsets, against a host FP64 product."""
import numpy as np
import pytest

from test_gpu_gemm_kernels import expected, lens, run_case, task

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lower", [0, 1])
@pytest.mark.parametrize("m,n", [(1535, 768), (1537, 830)])   # 12 x 12 tiles, 12 x 13 with the odd offset, 13 x 13
@pytest.mark.parametrize("da,db", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_many_tiles(m, n, da, db, lower):
    k = 37
    if lower:
        db = da
    t = [task(2 + da, 4 + db, 1, m + 4 - m % 2, m + 6 - m % 2, m + 3, m, n, k, lower=lower)]
    a_len, b_len, c_len = lens(t)
    A, B, C0, C = run_case(t, a_len, b_len, c_len, np.float64, 0, seed=m + n)
    ref, scale, written = expected(t, A, B, C0)
    prod = (ref - C0)[written]
    # k products and a subtraction: a few eps
    assert np.linalg.norm((C - ref)[written]) <= 1e-13 * np.linalg.norm(prod)
    assert np.array_equal(C[~written], C0[~written])
