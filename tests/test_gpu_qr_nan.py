"""Pivoted QR of blocks whose norms are not numbers.  Where the largest norm is a NaN no
columns change places (it orders above every number, and nothing compares equal to it),
so the permutation is the identity, the columns before the first NaN hold the QR
without pivoting, and every index stays inside the block.  The register kernel, the
shared-memory kernel and the global-memory kernel, called by their launchers; then a
whole solve with near tables that are NaN."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REG = "_Z26aifmm_launch_qr_factor_regPK5QRJobS1_iiiiP11CUstream_st"
SMEM = "_Z27aifmm_launch_qr_factor_smemPK5QRJobimiP11CUstream_st"
GLOBAL = "_Z22aifmm_launch_qr_factorPK5QRJobiiiiP11CUstream_st"


class QRJob(ctypes.Structure):
    _fields_ = [("a", ctypes.c_void_p), ("lda", ctypes.c_int), ("m", ctypes.c_int), ("n", ctypes.c_int),
                ("tau", ctypes.c_void_p), ("perm", ctypes.c_void_p), ("norms", ctypes.c_void_p),
                ("thr", ctypes.c_double), ("info", ctypes.c_void_p), ("maxpiv", ctypes.c_void_p)]


def factor(kernel, a):
    """The factors of a (m x n, complex128 or complex64): qr, tau, perm, (pivots, rank)."""
    import torch
    import aifmm_ls_b200 as A
    lib = A.load()
    m, n = a.shape
    es = a.dtype.itemsize
    dt = torch.complex128 if es == 16 else torch.complex64
    d = torch.from_numpy(np.ascontiguousarray(a.T)).to("cuda")
    tau = torch.zeros(min(m, n), dtype=dt, device="cuda")
    perm = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    info = torch.zeros(4, dtype=torch.int32, device="cuda")
    norms = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    job = QRJob(d.data_ptr(), m, m, n, tau.data_ptr(), perm.data_ptr(), norms.data_ptr(), 0.0, info.data_ptr(), None)
    dj = torch.frombuffer(bytearray(bytes(job)), dtype=torch.uint8).to("cuda")
    torch.cuda.synchronize()
    p = ctypes.c_void_p(dj.data_ptr())
    if kernel == REG:
        cls = getattr(lib, "_Z14aifmm_qr_classii")(m, n)
        assert cls >= 0
        e = getattr(lib, REG)(p, None, 1, cls, n, es, None)
    elif kernel == SMEM:
        size = getattr(lib, "_Z19aifmm_qr_smem_bytesiii")
        size.restype = ctypes.c_size_t
        e = getattr(lib, SMEM)(p, 1, ctypes.c_size_t(size(m, n, es)), es, None)
    else:
        e = getattr(lib, GLOBAL)(p, 1, m, n, es, None)
    assert e == 0
    torch.cuda.synchronize()
    return d.cpu().numpy().T, tau.cpu().numpy(), perm.cpu().numpy(), info.cpu().numpy()[:2]


@pytest.mark.parametrize("kernel,m,n", [(REG, 36, 57), (SMEM, 100, 100), (SMEM, 7, 3), (SMEM, 61, 130), (GLOBAL, 130, 121)])
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("where", ["all", "first", "middle", "last"])
def test_no_swap_where_a_norm_is_not_a_number(kernel, m, n, dtype, where):
    rng = np.random.default_rng(3)
    a = (rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))).astype(dtype)
    j = {"all": 0, "first": 0, "middle": n // 2, "last": n - 1}[where]
    if where == "all":
        a[:] = complex(np.nan, np.nan)
    else:
        a[m // 2, j] = complex(np.nan, 1.0)
    qr, tau, perm, info = factor(kernel, a)
    assert np.array_equal(perm, np.arange(n))
    assert info[0] == min(m, n)
    k = min(j, m, n)
    if k:  # columns before the NaN: |R_kk| of the QR without pivoting, to 100 units of rounding
        r = np.abs(np.diag(np.linalg.qr(a[:, :k].astype(np.complex128), mode="r")))
        got = np.abs(np.diag(qr[:k, :k]))
        assert np.all(np.abs(got - r) <= 100 * np.finfo(dtype).eps * np.linalg.norm(a[:, :k]))


@pytest.mark.parametrize("n_cheb", [6, 10, 11])
def test_solve_with_tables_that_are_not_numbers(n_cheb):
    import aifmm_ls_b200 as A
    K = A.LSKernel(n_cheb=n_cheb, kappa=10.0, degree=3, depth=2, tol_pow=6, q_kind="gauss_aw")
    K.tables_compute()
    M, near = K.tables_get()
    K.tables_set(M, np.full_like(near, complex(np.nan, np.nan)))
    T = A.FMM2DTree(K)
    T.createTree()
    T.assemble()
    b = K.rhs_plane_wave([0.3])
    try:
        assert np.isnan(T.solve(b)).any()
    except RuntimeError:
        pass  # a status is as good
    K.tables_set(M, near)  # the handle works on
    T.createTree()
    T.assemble()
    assert np.isfinite(T.solve(b)).all()
