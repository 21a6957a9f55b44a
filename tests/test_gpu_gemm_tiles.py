"""The batched GEMM at the edges of its tiles (32 x 8, 16 x 16), of a fragment (8 x 8,
4 of k), of the single buffer (k = 96) and of a chunk of the ring (k = 48), with both
operands plain and adjoint.  Tolerance as in test_gpu_gemm: 1e-13 of |A| |B|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 8), (33, 7), (32, 9), (17, 16), (15, 17), (64, 33)])
@pytest.mark.parametrize("k", [1, 3, 4, 47, 95, 96, 97, 145])
def test_tile_edges(m, n, k):
    import aifmm_ls_b200 as A
    K = A.LSKernel(depth=2)
    rng = np.random.default_rng(1000 * m + 10 * n + k)
    cn = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    for opA in (0, 1):
        for opB in (0, 1):
            a, b = (cn(k, m) if opA else cn(m, k)), (cn(n, k) if opB else cn(k, n))
            oa, ob = (a.conj().T if opA else a), (b.conj().T if opB else b)
            c = K.zgemm(a, b, opA=opA, opB=opB)
            assert np.all(np.abs(c - oa @ ob) <= 1e-13 * (np.abs(oa) @ np.abs(ob))), (opA, opB)


def test_rows_and_columns_outside_do_not_leak():
    """A NaN in one row of A or one column of B stays in that row or column of C."""
    import aifmm_ls_b200 as A
    K = A.LSKernel(depth=2)
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((19, 6)) + 0j, rng.standard_normal((6, 11)) + 0j
    a[4, 2] = np.nan
    b[1, 9] = np.nan
    c = K.zgemm(a, b)
    bad = np.zeros((19, 11), bool)
    bad[4] = bad[:, 9] = True
    assert np.array_equal(np.isnan(c), bad)
