"""The dense products by leaf moments (dense_matvec, total_field) against the
entries themselves: sampled rows from getMatrix times x.

Tolerance: an entry agrees with the oracle's to 1e-12 relative
(test_gpu_parity.py); a row of the product may differ from the sum of its entries
by that much of sum |a_ij| |x_j|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cheb,depth,nrhs,kappa,q_kind", [
    (2, 2, 1, 0.5, "gauss_aw"),     # 64 points: less than one block of rows, small arguments of the Bessel functions
    (3, 3, 2, 12.0, "disk"),        # rows not a multiple of the block; rows outside the contrast
    (5, 3, 3, 60.0, "gauss_aw"),
    (6, 3, 4, 250.0, "gauss_aw"),   # arguments above the series length: the recurrence starts higher
    (4, 4, 5, 7.0, "gaussian160"),  # rows whose contrast underflows
    (8, 2, 6, 30.0, "disk"),
    (4, 3, 7, 20.0, "gauss_aw"),
    (2, 7, 8, 40.0, "gauss_aw"),    # 16,384 leaves and 8 columns: the moments take several chunks
])
def test_rows_of_the_product(n_cheb, depth, nrhs, kappa, q_kind):
    import aifmm_ls_b200 as A
    K = A.LSKernel(n_cheb=n_cheb, kappa=kappa, degree=min(2, n_cheb - 1), depth=depth, q_kind=q_kind)
    K.tables_compute()
    rng = np.random.default_rng(11)
    x = rng.standard_normal((nrhs, K.N)) + 1j * rng.standard_normal((nrhs, K.N))
    y = K.dense_matvec(x)
    rows = np.unique(np.r_[0, K.N // 2, K.N - 1, rng.integers(0, K.N, 29)]).astype(np.int32)
    R = K.getMatrix(rows, np.arange(K.N, dtype=np.int32))
    want, scale = x @ R.T, np.abs(x) @ np.abs(R).T
    assert np.all(np.abs(y[:, rows] - want) <= 1e-12 * scale)
    # total_field: u - u_inc = G x with kappa^2 q G = A - I, on the rows with a contrast
    th = rng.uniform(0, 2 * np.pi, nrhs)
    u = K.total_field(th, x)
    xy = K.gridPoints[rows]
    inc = np.exp(1j * kappa * (np.outer(np.cos(th), xy[:, 0]) + np.outer(np.sin(th), xy[:, 1])))
    b = K.rhs_plane_wave(th)[:, rows]          # -kappa^2 q u_inc
    kq = -(b / inc).real
    on = np.abs(kq[0]) > 1e-3
    off = R.copy()
    off[np.arange(len(rows)), rows] -= 1.0
    # 1 + a is rounded at the diagonal: that rounding is divided by kappa^2 q
    bound = 1e-12 * (np.abs(x) @ np.abs(off).T) / np.abs(kq) + 4e-16 * np.abs(x[:, rows]) / np.abs(kq) + 1e-13
    assert np.all(np.abs((u[:, rows] - inc) - (x @ off.T) / kq)[:, on] <= bound[:, on])
