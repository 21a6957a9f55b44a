"""The register and the shared-memory QR give the same bits for the same block: factors,
coefficients, permutation, pivot count and rank.  Blocks at the edges of the register
classes (20, 36, 64, 96 and 144 rows), rows that do not fill a lane's four, more columns
than rows and fewer; random, with tied norms, of deficient rank, the identity."""
import numpy as np
import pytest

from test_gpu_qr_nan import REG, SMEM, factor

pytestmark = pytest.mark.gpu


def _block(kind, m, n, dtype):
    rng = np.random.default_rng(m * 1000 + n)
    a = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    if kind == "tied":      # equal columns, and columns of equal norm
        a[:, n // 2:] = a[:, :n - n // 2]
        a[:, n // 3] = 1j * a[:, 0]
    elif kind == "rank":    # three columns span all, with noise at the threshold
        k = min(3, n)
        a = a[:, :k] @ (rng.standard_normal((k, n)) + 0j) + 1e-15 * a
    elif kind == "eye":
        a = np.eye(m, n) + 0j
    elif kind == "graded":  # norms over many decades: recomputed norms
        a *= 10.0 ** -np.linspace(0, 12, n)
    return a.astype(dtype)


@pytest.mark.parametrize("m,n", [(1, 1), (4, 9), (19, 57), (20, 128), (21, 36), (36, 57), (33, 90), (37, 64), (64, 96),
                                 (63, 20), (65, 80), (96, 96), (94, 31), (97, 60), (141, 64), (144, 33)])
@pytest.mark.parametrize("kind", ["random", "tied", "rank", "eye", "graded"])
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_same_bits(m, n, kind, dtype):
    a = _block(kind, m, n, dtype)
    for r, s in zip(factor(REG, a), factor(SMEM, a)):
        assert np.array_equal(r, s)
