"""The 6-digit round trip of the leaf tables on the device against printf's "%.6g" and
strtod on the host, bit for bit, over the values that the tables take: entries, the
rounding noise of symmetry zeros (down to 1e-25), exact zeros.  Rounding the unrounded
tables on the host must give the rounded ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cheb,degree,kappa,depth", [(6, 6, 10.0, 5), (8, 6, 80.0, 4), (4, 3, 0.5, 8), (2, 1, 40.0, 2),
                                                       (9, 10, 30.0, 3), (6, 6, 1e-3, 9)])
def test_rounded_tables_are_the_text_round_trip(n_cheb, degree, kappa, depth):
    import aifmm_ls_b200 as A
    K = A.LSKernel(n_cheb=n_cheb, degree=degree, kappa=kappa, depth=depth)
    K.tables_compute(round6=False)
    v = np.concatenate([t.ravel() for t in K.tables_get()]).view(np.float64)
    K.tables_compute(round6=True)
    r = np.concatenate([t.ravel() for t in K.tables_get()]).view(np.float64)
    want = np.array([float("%.6g" % x) for x in v])
    small = np.abs(v[v != 0])
    print("%d values, %.1e .. %.1e, %d zeros" % (v.size, small.min(), small.max(), int((v == 0).sum())))
    assert np.array_equal(r, want, equal_nan=True)  # degree 10 on 9 nodes: a singular fit, NaN tables
