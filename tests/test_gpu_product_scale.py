"""dense_matvec and total_field of vectors of any size: a power of two in front of the vector
comes out in front of the product.  Every operation on the vector is linear and a power
of two is exact, so only the order of the final sums (atomics) may differ: 1e-13 of
sum |a_ij| |x_j|, estimated by the product with |x|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cheb,depth,kappa", [(2, 2, 0.05), (4, 3, 20.0), (6, 3, 400.0)])
@pytest.mark.parametrize("e", [-1040, -900, -600, -300, 300, 600, 900, 1000])
def test_powers_of_two(n_cheb, depth, kappa, e):
    import aifmm_ls_b200 as A
    K = A.LSKernel(n_cheb=n_cheb, kappa=kappa, degree=2, depth=depth, q_kind="gauss_aw")
    K.tables_compute()
    rng = np.random.default_rng(4)
    x = rng.standard_normal((3, K.N)) + 1j * rng.standard_normal((3, K.N))
    if e < -1000:
        x = np.round(x * 1024)  # whole numbers: their products with 2^e are exact, subnormal ones too
    y = K.dense_matvec(x)

    def times(v, p):  # exact where the result is normal
        return np.ldexp(v.real, p) + 1j * np.ldexp(v.imag, p)

    got = times(K.dense_matvec(times(x, e)), -e)
    scale = np.abs(x).sum(axis=1).max()
    # sums of subnormals: half a unit an addition, of the near entries and of the leaves' far sums,
    # which kappa^2 q <= 1.5 kappa^2 multiplies
    units = 18 * K.rank + (2 * 4 ** depth + 4) * max(1.0, 1.5 * kappa ** 2)
    tiny = np.ldexp(units, -1074 - e) if e < -1000 else 0.0
    assert np.all(np.abs(got - y) <= 1e-13 * scale + tiny)


def test_columns_and_leaves_of_different_size():
    import aifmm_ls_b200 as A
    K = A.LSKernel(n_cheb=4, kappa=20.0, degree=2, depth=3, q_kind="gauss_aw")
    K.tables_compute()
    rng = np.random.default_rng(6)
    x = rng.standard_normal((4, K.N)) + 1j * rng.standard_normal((4, K.N))
    size = np.array([1.0, 2.0 ** 700, 2.0 ** -700, 0.0])[:, None]
    y, z = K.dense_matvec(x), K.dense_matvec(x * size)
    assert np.all(np.abs(z[:3] / size[:3] - y[:3]) <= 1e-13 * np.abs(x).sum(axis=1).max()) and not z[3].any()
    # one leaf far larger than the others: its own part of the product decides
    big = np.zeros_like(x[:1])
    big[:, 5 * 16:6 * 16] = x[:1, 5 * 16:6 * 16]
    w = K.dense_matvec(x[:1] + big * 2.0 ** 800)
    assert np.all(np.abs(w / 2.0 ** 800 - K.dense_matvec(big)) <= 1e-13 * np.abs(big).sum())


@pytest.mark.parametrize("e", [-700, 700])
def test_field_of_scaled_densities(e):
    import aifmm_ls_b200 as A
    K = A.LSKernel(n_cheb=4, kappa=20.0, degree=2, depth=3, q_kind="gauss_aw")
    K.tables_compute()
    rng = np.random.default_rng(8)
    x = rng.standard_normal((1, K.N)) + 1j * rng.standard_normal((1, K.N))
    th = [0.4]
    inc = K.total_field(th, np.zeros_like(x))
    s = K.total_field(th, x) - inc
    if e > 0:  # the incident field is lost in the sum
        assert np.all(np.abs(K.total_field(th, x * 2.0 ** e) / 2.0 ** e - s) <= 1e-13 * np.abs(x).sum())
    else:      # the scattered one is
        assert np.array_equal(K.total_field(th, x * 2.0 ** e), inc)
