"""Which rows of dense_matvec need no series: those whose far entries are all zero by the
bound that the entries themselves use, whatever the size of the caller's tables.  Sampled
rows of the product against the rows of getMatrix times x.

Tolerance: test_gpu_dense_product's 1e-12 of sum |a_ij| |x_j|, and 1e-16 of sum |x_j|
for the far entries that are below 1e-16, zero in the matrix and part of the sum in the product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("factor", [1.0, 1e26, 1e-20])
@pytest.mark.parametrize("n_cheb,depth,q_kind", [(4, 3, "gaussian160"), (6, 2, "gaussian160"), (3, 4, "disk")])
def test_rows_outside_the_contrast(factor, n_cheb, depth, q_kind):
    import aifmm_ls_b200 as A
    K = A.LSKernel(n_cheb=n_cheb, kappa=8.0, degree=2, depth=depth, q_kind=q_kind)
    K.tables_compute()
    M, near = K.tables_get()
    K.tables_set(factor * M, factor * near)
    rng = np.random.default_rng(2)
    x = rng.standard_normal((2, K.N)) + 1j * rng.standard_normal((2, K.N))
    y = K.dense_matvec(x)
    r2 = np.sum(K.gridPoints ** 2, axis=1)
    rows = np.argsort(r2)[np.linspace(0, K.N - 1, min(K.N, 150)).astype(int)].astype(np.int32)  # the middle to the corners
    R = K.getMatrix(rows, np.arange(K.N, dtype=np.int32))
    want, scale = x @ R.T, np.abs(x) @ np.abs(R).T
    bound = 1e-12 * scale + 1e-16 * np.abs(x).sum(axis=1)[:, None]
    assert np.all(np.abs(y[:, rows] - want) <= bound)
    outside = (np.abs(R) > 0).sum(axis=1) == 1  # the identity alone
    assert outside.any() and (factor < 1 or not outside.all())
