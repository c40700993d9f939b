"""Restarts of the host-driven engine where rows of A share a column of more
than 1024 entries: the restart kernel's product is A' y, whose long rows are
summed by the first CTAs of its grid (engine.cu, rowblock.cuh)."""
from __future__ import annotations

import functools

import numpy as np
import pytest

import pyoracle
from hprqp import instances

pytestmark = pytest.mark.gpu

# (n, m, full columns of A): one chunk CTA, several, more long rows of A' than
# the last chunk CTA finishes (k_long_epi)
SHAPES = [(2000, 3000, 1), (1300, 1025, 9), (700, 2100, 257)]


@pytest.fixture
def device_wide(engine_lib):
    old = engine_lib.set_single_cta_max_work(0)
    yield engine_lib
    engine_lib.set_single_cta_max_work(old)


@functools.lru_cache(maxsize=None)
def _qp(n, m, cols, kind):
    rng = np.random.default_rng(n + cols)
    inst = instances.plain_qp(31 + cols, n=n, m=m, a_density=0.01, m_rows=n // 5, m_density=0.005, n_eq=n // 10)
    A = inst.A.to_scipy().tolil()
    at = rng.choice(n, cols, replace=False)
    A[:, at] = rng.standard_normal((m, cols)) / np.sqrt(cols)
    inst.A = instances._csr_from_scipy(A)
    inst.AL, inst.AU = instances._feasible_rows(rng, inst.A, n, n // 10)
    if kind == "free":  # the step without bounds (noC)
        free = rng.random(n) < 0.95
        inst.l[free], inst.u[free] = -np.inf, np.inf
    return inst


@functools.lru_cache(maxsize=None)
def _oracle(n, m, cols, kind, stoptol, max_iter):
    return pyoracle.OracleModel(_qp(n, m, cols, kind)).solve(mode=pyoracle.MODE_GPU_REF, stoptol=stoptol,
                                                             max_iter=max_iter)


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(1.0, float(np.max(np.abs(b)))))


@pytest.mark.parametrize("kind", ["boxed", "free"])
@pytest.mark.parametrize("n,m,cols", SHAPES)
def test_iterates_past_a_restart(device_wide, n, m, cols, kind):
    """150 steps, the first restart after 100: iterates within 1e-6 of the
    oracle's.  A restart chooses sigma by comparing values near a minimum,
    which finds it to sqrt(eps) = 1.5e-8 only: one unit in the last place of c
    moves the oracle's own iterates by up to 3e-8."""
    o = _oracle(n, m, cols, kind, 1e-30, 150)
    r = device_wide.optimize(device_wide.build_from_instance(_qp(n, m, cols, kind)),
                             device_wide.Parameters(verbose=False, stoptol=1e-30, max_iter=150), as_numpy=True)
    assert r.iter == o["iter"] == 150
    for f in ("x", "y", "z", "w"):
        assert _rel(getattr(r, f), np.asarray(o[f])) <= 1e-6, f


@pytest.mark.parametrize("kind", ["boxed", "free"])
@pytest.mark.parametrize("n,m,cols", SHAPES)
def test_converges_like_the_oracle(device_wide, n, m, cols, kind):
    o = _oracle(n, m, cols, kind, 1e-6, 20000)
    r = device_wide.optimize(device_wide.build_from_instance(_qp(n, m, cols, kind)),
                             device_wide.Parameters(verbose=False, stoptol=1e-6, max_iter=20000), as_numpy=True)
    assert r.status_code == o["status"] == device_wide.STATUS_OPTIMAL
    assert abs(r.objective - o["primal_obj"]) <= 1e-6 * max(1.0, abs(o["primal_obj"]))
    assert abs(r.iter - o["iter"]) <= max(20, o["iter"] // 10)


def test_backward_after_restarts(device_wide):
    """solve_for_backward takes this engine whatever the size: as many
    iterations as the oracle, and an adjoint."""
    n, m, cols = SHAPES[0]
    o = _oracle(n, m, cols, "boxed", 1e-6, 20000)
    r, state = device_wide.solve_for_backward(device_wide.build_from_instance(_qp(n, m, cols, "boxed")),
                                              device_wide.Parameters(verbose=False, stoptol=1e-6, max_iter=20000))
    try:
        assert r.status_code == device_wide.STATUS_OPTIMAL
        assert abs(r.iter - o["iter"]) <= max(20, o["iter"] // 10)
        assert np.all(np.isfinite(state.backward(np.ones(n), tol=1e-10)["dc"]))
    finally:
        state.close()


def test_cone_model(device_wide):
    """A cone of two variables, |v| <= t, and a full column of A: the QP with
    the rows t - v >= 0 and t + v >= 0 in its place has the same optimum
    (objectives within 1e-6, both solved to 1e-8)."""
    n, m, _ = SHAPES[0]
    inst = _qp(n, m, 1, "boxed")
    Q = np.zeros((n + 2, n + 2))
    Q[:n, :n] = inst.Q.to_scipy().toarray()
    A = np.zeros((m + 1, n + 2))
    A[:m, :n] = inst.A.to_scipy().toarray()
    A[m, :3], A[m, n + 1] = 1.0, -1.0  # v = x_0 + x_1 + x_2 - 5
    c = np.concatenate([inst.c, [2.0, 0.0]])
    l, u = (np.concatenate([b, s * np.full(2, np.inf)]) for b, s in ((inst.l, -1), (inst.u, 1)))
    AL, AU = np.append(inst.AL, 5.0), np.append(inst.AU, 5.0)
    import scipy.sparse as sp

    model = device_wide.build_from_qabc_soc(sp.csr_matrix(Q), c, sp.csr_matrix(A), AL, AU, l, u,
                                            var_cone_offsets=[n, n + 2])
    r = device_wide.optimize(model, device_wide.Parameters(verbose=False, stoptol=1e-8, max_iter=50000), as_numpy=True)
    rows = np.zeros((2, n + 2))
    rows[:, n], rows[:, n + 1] = 1.0, [-1.0, 1.0]
    flat = instances.QPInstance(instances._csr_from_scipy(sp.csr_matrix(Q)),
                                instances._csr_from_scipy(sp.csr_matrix(np.vstack([A, rows]))), c,
                                np.append(AL, [0.0, 0.0]), np.append(AU, [np.inf, np.inf]), l, u)
    o = pyoracle.OracleModel(flat).solve(mode=pyoracle.MODE_GPU_REF, stoptol=1e-8, max_iter=50000)
    assert r.status_code == o["status"] == device_wide.STATUS_OPTIMAL
    assert abs(r.objective - o["primal_obj"]) <= 1e-6 * max(1.0, abs(o["primal_obj"]))
