"""Products with long rows in one launch, finer tiles, and the one-pass step of
a diagonal Q (engine.cu, rowblock.cuh)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_long", [0, 1, 255, 256, 257])
def test_long_rows_beside_tiles(engine_lib, n_long):
    """Rows of more than 1024 entries among short and empty ones: up to 256 of
    them are finished by the last chunk CTA, more by a kernel of their own.
    Tolerance: 64-bit sums of len entries, 2 len eps sum |a_ij x_j|."""
    import scipy.sparse as sp

    rng = np.random.default_rng(n_long)
    ncol = 3000
    lens = np.concatenate([np.full(n_long, 1025) + rng.integers(0, 1100, n_long), rng.integers(0, 40, 700)])
    rng.shuffle(lens)
    indptr = np.concatenate([[0], np.cumsum(lens)])
    indices = np.concatenate([np.sort(rng.choice(ncol, l, replace=False)) for l in lens]).astype(np.int64)
    data = rng.standard_normal(len(indices))
    x = rng.standard_normal(ncol)
    M = sp.csr_matrix((data, indices, indptr), shape=(len(lens), ncol))
    scale = abs(M) @ abs(x)
    for _ in range(2):  # a second launch finds the chunk counter as the first did
        y, _ = engine_lib.spmv(indptr, indices, data, ncol, x, reps=2)
        assert np.all(np.abs(y - M @ x) <= 2 * np.finfo(float).eps * np.maximum(lens, 1) * scale)


@pytest.mark.parametrize("n", [1, 31, 1000, 40001])
def test_diagonal_step_equals_general_step(engine_lib, n):
    """A Q of its diagonal alone against the same Q with stored zeros beside
    it, which takes the two products: the same iterates, bit for bit (zeros
    add nothing to a row's sum, and no reduction enters the first steps)."""
    from hprqp import instances

    inst = instances.plain_qp(5, n=max(n, 2), m=max(1, n // 3), a_density=min(0.3, 6.0 / n), m_rows=1, m_density=0.1,
                              n_eq=0)
    n = inst.n
    d = np.random.default_rng(n).uniform(0.1, 2.0, n)
    plain = instances.CSR(n, n, np.arange(n + 1), np.arange(n), d)
    rows = np.repeat(np.arange(n), 2)
    cols = np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)
    vals = np.stack([d, np.zeros(n)], 1)
    o = np.argsort(cols, axis=1)
    padded = instances.CSR(n, n, 2 * np.arange(n + 1), np.take_along_axis(cols, o, 1).ravel(),
                           np.take_along_axis(vals, o, 1).ravel())
    assert len(rows) == padded.nnz
    old = engine_lib.set_single_cta_max_work(0)  # the device-wide engine
    try:
        got = []
        for Q in (plain, padded):
            inst.Q = Q
            r = engine_lib.optimize(engine_lib.build_from_instance(inst),
                                    engine_lib.Parameters(verbose=False, stoptol=1e-30, max_iter=57), as_numpy=True)
            got.append(r)
        for f in ("x", "y", "z", "w"):
            np.testing.assert_array_equal(getattr(got[0], f), getattr(got[1], f), err_msg=f)
    finally:
        engine_lib.set_single_cta_max_work(old)


@pytest.mark.parametrize("n", [1025, 2100])
def test_scaling_of_long_rows(engine_lib, n):
    """Ruiz x10 and Pock-Chambolle with rows longer than a chunk, against the
    same passes in numpy.  Each of the 11 passes rounds a value three times,
    the last one's sums have chains of at most n / 32 + 5 additions: 35 + 2 *
    71 eps, taken as 200."""
    import scipy.sparse as sp
    from hprqp import instances

    rng = np.random.default_rng(n)
    inst = instances.plain_qp(3, n=n, m=40, a_density=0.01, m_rows=30, m_density=0.02, n_eq=10)
    A = inst.A.to_scipy().tolil()
    A[0, :] = rng.standard_normal(n)
    A[7, : n - 1] = 10.0 * rng.standard_normal(n - 1)
    A = A.tocsr()
    A.sort_indices()
    inst.A = instances.CSR(40, n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data)
    model = engine_lib.build_from_instance(inst)
    got = engine_lib.setup_info(model, dump=True)
    arrays = engine_lib.model_arrays(model)
    Q, A = (sp.csr_matrix((arrays[k + "_data"], arrays[k + "_indices"], arrays[k + "_indptr"]), shape=(r, n)).toarray()
            for k, r in (("q", n), ("a", arrays["m"])))
    rows = np.repeat(np.arange(arrays["m"]), np.diff(arrays["a_indptr"]))
    rn, cn = np.ones(A.shape[0]), np.ones(n)
    for p in range(11):
        if p < 10:
            rf, cf = abs(A).max(1), np.maximum(abs(A).max(0), abs(Q).max(0))
        else:
            rf, cf = abs(A).sum(1), abs(A).sum(0) + abs(Q).sum(0)
        rf, cf = np.sqrt(np.where(rf > 0, rf, 1.0)), np.sqrt(np.where(cf > 0, cf, 1.0))
        A, Q = A / rf[:, None] / cf, Q / cf[:, None] / cf
        rn, cn = rn * rf, cn * cf
    np.testing.assert_allclose(got["row_norm"], rn, rtol=200 * np.finfo(float).eps)
    np.testing.assert_allclose(got["col_norm"], cn, rtol=200 * np.finfo(float).eps)
    np.testing.assert_allclose(got["a_val"], A[rows, arrays["a_indices"]], rtol=200 * np.finfo(float).eps)


@pytest.mark.parametrize("long_q", [False, True])
@pytest.mark.parametrize("long_a", [0, 2, 257])
def test_two_products_in_one_launch(engine_lib, long_q, long_a):
    """MINRES, whose Q v and A v share a launch, with and without rows longer
    than a chunk (257 long rows of A keep the products apart): the solution
    satisfies the active-set KKT system assembled on the host to 1e-8 (the
    bound of test_single_adjoint_large_kkt_residual), and a second backward
    gives the same bits (tolerance 0)."""
    import scipy.sparse as sp
    from hprqp import instances

    n, m = 1100, 300
    rng = np.random.default_rng(7 * long_a + long_q)
    inst = instances.plain_qp(11, n=n, m=m, a_density=0.02, m_rows=30, m_density=0.01, n_eq=20)

    def csr(M):
        M = M.tocsr()
        M.sort_indices()
        return instances.CSR(*M.shape, M.indptr.astype(np.int64), M.indices.astype(np.int64), M.data)

    if long_a:
        A = inst.A.to_scipy().tolil()
        long_rows = rng.choice(m, long_a, replace=False)
        A[long_rows, :] = rng.standard_normal((long_a, n)) / n
        inst.A, inst.AL[long_rows], inst.AU[long_rows] = csr(A), -1.0, 1.0
    if long_q:  # two dense rows and columns, and a diagonal that dominates
        arrow = np.zeros((n, n))
        arrow[[3, 500], :] = rng.uniform(-1, 1, (2, n)) / n
        Q = inst.Q.to_scipy() + sp.csr_matrix(arrow + arrow.T)
        inst.Q = csr(Q + sp.diags(np.asarray(abs(Q).sum(1)).ravel()))
    model = engine_lib.build_from_instance(inst)
    r, state = engine_lib.solve_for_backward(model, engine_lib.Parameters(verbose=False, stoptol=1e-8, max_iter=20000))
    assert r.status_code == engine_lib.STATUS_OPTIMAL
    try:
        gx = rng.standard_normal(n)
        g, again = state.backward(gx, tol=1e-12), state.backward(gx, tol=1e-12)
    finally:
        state.close()
    a = engine_lib.model_arrays(model)
    Q, A = (sp.csr_matrix((a[k + "_data"], a[k + "_indices"], a[k + "_indptr"]), shape=(rows, n))
            for k, rows in (("q", n), ("a", a["m"])))
    F, R = np.nonzero(r.z == 0.0)[0], np.nonzero(r.y != 0.0)[0]
    AF = A[R][:, F]
    res = np.concatenate([Q[F][:, F] @ g["lam"][F] + AF.T @ g["mu"][R] - gx[F], AF @ g["lam"][F]])
    assert np.linalg.norm(res) <= 1e-8 * np.linalg.norm(gx[F])
    for k in ("dc", "lam", "mu", "dQ_values", "dA_values"):
        np.testing.assert_array_equal(again[k], g[k], err_msg=k)
