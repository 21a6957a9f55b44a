"""Blocks of 121 and 144 rows, whose pivoted QR runs on the matrix in global memory, whole
and with columns and rows that do not fill the last warp: solutions against the CPU oracle
with the same tables, under the bound of test_gpu_block_sizes: max(1e-8, 5 x what the
oracle's own solution moves by when every entry is perturbed by 1e-16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cheb,depth,kappa,tol_pow", [(11, 2, 15.0, 7), (12, 2, 6.0, 5)])
def test_solution_with_blocks_in_global_memory(oracle_mod, n_cheb, depth, kappa, tol_pow):
    import aifmm_ls_b200 as A
    kw = dict(n_cheb=n_cheb, kappa=kappa, degree=4, depth=depth, tol_pow=tol_pow, q_kind="gauss_aw")
    p = oracle_mod.params(**kw)
    M, near, _ = oracle_mod.tables(p)
    K = A.LSKernel(**kw)
    K.tables_set(M, near)
    T = A.FMM2DTree(K)
    T.createTree()
    T.assemble()
    P = oracle_mod.Problem(p, M, near)
    b = P.rhs_plane_wave([0.3, 2.0])
    xo, _ = P.solve(b)
    x = T.solve(b)
    spread = 0.0
    for eps in (1e-16, -1e-16, 3e-16):
        Q = oracle_mod.Problem(p, M, near)
        Q.set_perturbation(eps)
        x1, _ = Q.solve(b)
        spread = max(spread, np.linalg.norm(x1 - xo) / np.linalg.norm(xo))
    rel = np.linalg.norm(x - xo) / np.linalg.norm(xo)
    print("n_cheb %d: |x - x_oracle| %.2e, oracle spread %.2e" % (n_cheb, rel, spread))
    assert rel <= max(1e-8, 5.0 * spread)
