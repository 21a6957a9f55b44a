"""A handle after a call that failed for want of device memory, in the middle of the
elimination, of an assembly or of a recorded solve: nothing of the failed call is left
running, queued or recorded.  Entries, products and a new factorisation on the same
handle give the bits of a handle that never failed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KW = dict(n_cheb=6, kappa=40.0, degree=6, depth=5, tol_pow=8, q_kind="gauss_aw")


def _handle():
    import aifmm_ls_b200 as A
    K = A.LSKernel(**KW)
    K.tables_compute()
    T = A.FMM2DTree(K)
    T.createTree()
    return K, T


class _Full:
    """The device's memory taken but for `leave` bytes."""
    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        self.held = []
        for chunk in (1 << 30, 2 << 20):
            n = (torch.cuda.mem_get_info()[0] - self.leave) // chunk * chunk
            if n > 0:
                self.held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))

    def __exit__(self, *a):
        import torch
        self.held = None
        torch.cuda.empty_cache()


def _pool(T):
    return int(T.stats()["pool_bytes"])


@pytest.fixture(scope="module")
def reference():
    K, T = _handle()
    T.assemble()
    before = _pool(T)
    b = K.rhs_plane_wave([0.3, 1.0, 2.0])
    T.factorize()
    grown = _pool(T) - before
    x = T.solve_factored(b)
    assert np.array_equal(T.solve_factored(b, graph=True), x)  # and its kernels are loaded
    rng = np.random.default_rng(1)
    I, J = rng.integers(0, K.N, 5000), rng.integers(0, K.N, 5000)
    v = rng.standard_normal((2, K.N)) + 0j
    return dict(b=b, x=x, grown=grown, I=I, J=J, e=K.entries(I, J), v=v, y=K.dense_matvec(v))


def _check(K, T, r, x=True):
    assert np.array_equal(K.entries(r["I"], r["J"]), r["e"])
    y = K.dense_matvec(r["v"])  # summed by atomics, in no fixed order
    assert np.linalg.norm(y - r["y"]) <= 1e-14 * np.linalg.norm(r["y"])
    if x:
        T.createTree()
        T.assemble()
        T.factorize()
        assert np.array_equal(T.solve_factored(r["b"]), r["x"])


@pytest.mark.parametrize("part", [0.25, 0.5, 0.75])
def test_after_a_failed_factorisation(reference, part):
    import aifmm_ls_b200 as A
    K, T = _handle()
    T.assemble()
    with _Full(int(part * reference["grown"])):
        with pytest.raises(A.AifmmError, match="cudaMalloc"):
            T.factorize()
    _check(K, T, reference)


@pytest.mark.parametrize("part", [0.2, 0.5, 0.85])
def test_a_kept_assembly_survives_a_failed_factorisation(reference, part):
    import aifmm_ls_b200 as A
    K, T = _handle()
    T.assemble()
    before = _pool(T)
    T.factorize(keep_assembly=True)
    grown = _pool(T) - before
    K, T = _handle()
    T.assemble()
    with _Full(int(part * grown)):  # in the copy of the assembly, or in the elimination
        with pytest.raises(A.AifmmError, match="cudaMalloc"):
            T.factorize(keep_assembly=True)
    T.factorize(keep_assembly=True)
    assert np.array_equal(T.solve_factored(reference["b"]), reference["x"])


def test_after_a_failed_assembly(reference):
    import aifmm_ls_b200 as A
    K, T = _handle()
    with _Full(100 << 20):
        with pytest.raises(A.AifmmError, match="cudaMalloc"):
            T.assemble()
    with pytest.raises(A.AifmmError):
        T.factorize()
    _check(K, T, reference)


def test_after_a_failed_recording(reference):
    import aifmm_ls_b200 as A
    K, T = _handle()
    T.assemble()
    T.factorize()
    b = np.tile(reference["b"], (80, 1))  # 142 MB of right-hand sides: blocks of their own
    with _Full(200 << 20):
        with pytest.raises(A.AifmmError, match="cudaMalloc"):
            T.solve_factored(b, graph=True)
    for graph in (False, True):
        assert np.array_equal(T.solve_factored(reference["b"], graph=graph), reference["x"])
    _check(K, T, reference, x=False)
