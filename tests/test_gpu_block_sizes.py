"""The solver over block sizes: 4 to 100 rows at the leaves and the mosaics of the
level above, so that every kernel of the pivoted QR and of the recompression (rows
up to 20, 36, 64, 96, 144 in registers, then shared and global memory) is taken,
with rows that do not fill a lane's last group of four.  Against the CPU oracle
with the same tables, under the bound of test_gpu_parity.test_solution_matches_oracle:
max(1e-8, 5 x what the oracle's own solution moves by when every entry is perturbed
by 1e-16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cheb,depth,kappa,tol_pow", [
    (2, 3, 5.0, 6), (3, 3, 8.0, 8), (4, 4, 10.0, 8), (5, 3, 20.0, 10), (7, 3, 20.0, 9), (8, 3, 30.0, 9),
    (9, 2, 20.0, 8), (10, 2, 30.0, 8)])
def test_solution_over_block_sizes(oracle_mod, n_cheb, depth, kappa, tol_pow):
    import aifmm_ls_b200 as A
    kw = dict(n_cheb=n_cheb, kappa=kappa, degree=min(n_cheb, 4), depth=depth, tol_pow=tol_pow, q_kind="gauss_aw")
    p = oracle_mod.params(**kw)
    M, near, _ = oracle_mod.tables(p)
    K = A.LSKernel(**kw)
    K.tables_set(M, near)
    T = A.FMM2DTree(K)
    T.createTree()
    T.assemble()
    P = oracle_mod.Problem(p, M, near)
    b = P.rhs_plane_wave([0.0, 1.1, 4.0])
    xo, _ = P.solve(b)
    x = T.solve(b)
    spread = 0.0
    for eps in (1e-16, -1e-16, 3e-16):
        Q = oracle_mod.Problem(p, M, near)
        Q.set_perturbation(eps)
        x1, _ = Q.solve(b)
        spread = max(spread, np.linalg.norm(x1 - xo) / np.linalg.norm(xo))
    rel = np.linalg.norm(x - xo) / np.linalg.norm(xo)
    print("n_cheb %d depth %d: |x - x_oracle| %.2e, oracle spread %.2e" % (n_cheb, depth, rel, spread))
    assert rel <= max(1e-8, 5.0 * spread)
