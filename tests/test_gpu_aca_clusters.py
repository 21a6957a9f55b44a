"""Skeletons and ranks against the CPU oracle, index for index, where the clusters of the
ACA kernel are at their edges: two CTAs a job (depth 5) with four nodes a box, more
positions than the magnitudes a thread keeps, more terms than the coefficients held in
shared memory, rows outside the contrast's support.  And entries whose bound decides
that they are zero: those rows of the matrix against the oracle's, around 1e-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(oracle_mod, table_cache, **kw):
    import aifmm_ls_b200 as A
    p, tabs = table_cache(**kw)
    names = {v: k for k, v in oracle_mod.Q_KINDS.items()}
    K = A.LSKernel(n_cheb=p.n_cheb, kappa=p.kappa, degree=p.degree, L=p.L, depth=p.depth, tol_pow=p.tol_pow,
                   q_kind=names[p.q_kind], q_amp=p.q_amp, q_width=p.q_width, q_radius=p.q_radius)
    K.tables_set(tabs[0], tabs[1])
    return K, oracle_mod.Problem(p, *tabs[:2]), p


@pytest.mark.parametrize("n_cheb,degree,depth,kappa,tol_pow,q_kind,least", [
    (2, 2, 5, 10.0, 6, "gauss_aw", 1), (9, 6, 4, 5.0, 4, "gauss_aw", 1), (8, 6, 2, 120.0, 9, "gauss_aw", 33),
    (3, 3, 4, 20.0, 8, "gaussian160", 1), (7, 5, 3, 30.0, 9, "disk", 1)])
def test_skeletons_at_the_edges_of_a_cluster(oracle_mod, table_cache, n_cheb, degree, depth, kappa, tol_pow, q_kind, least):
    import aifmm_ls_b200 as A
    K, P, p = _pair(oracle_mod, table_cache, n_cheb=n_cheb, degree=degree, depth=depth, kappa=kappa, tol_pow=tol_pow,
                    q_kind=q_kind)
    T = A.FMM2DTree(K)
    T.createTree()
    T.assemble()
    P.solve(P.rhs_plane_wave([0.0]))
    top = 0
    for lev in range(2, depth + 1):
        for a, b in zip(T.level_ranks(lev), P.level_ranks(lev)):
            assert np.array_equal(a, b), lev
            top = max(top, int(np.max(a)))
        for box in range(0, 4 ** lev, max(1, 4 ** lev // 23)):
            for which in range(4):
                assert np.array_equal(T.box_skeleton(lev, box, which), P.box_skeleton(lev, box, which)), (lev, box, which)
    assert top >= least


@pytest.mark.parametrize("n_cheb,degree,depth,kappa,q_kind", [
    (6, 6, 4, 10.0, "gaussian160"), (4, 3, 6, 1.0, "gaussian160"), (8, 6, 3, 80.0, "gaussian160"), (6, 6, 3, 20.0, "disk")])
def test_bounded_entries_are_zero_where_they_were(oracle_mod, table_cache, n_cheb, degree, depth, kappa, q_kind):
    K, P, p = _pair(oracle_mod, table_cache, n_cheb=n_cheb, degree=degree, depth=depth, kappa=kappa, q_kind=q_kind)
    rng = np.random.default_rng(5)
    r2 = np.sum(np.asarray(K.gridPoints).reshape(K.N, -1)[:, :2] ** 2, axis=1)
    q = 1.5 * np.exp(-160 * r2)
    band = np.nonzero((q > 1e-20) & (q < 1e-9))[0] if q_kind == "gaussian160" else np.arange(K.N)
    I = rng.choice(band, 6000)
    J = rng.integers(0, K.N, 6000)
    g, o = K.entries(I, J), P.entries(I, J)
    edge = 1e-16 * (1 + 1e-9)
    either = ((g == 0) & (np.abs(o) <= edge)) | ((o == 0) & (np.abs(g) <= edge))
    print("%d zero of %d" % (int((g == 0).sum()), g.size))
    assert ((np.abs(g - o) <= 1e-12 * np.abs(o)) | either).all()
    assert (g == 0).any() and (g != 0).any()
