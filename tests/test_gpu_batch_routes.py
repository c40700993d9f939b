"""What a call answers does not depend on the kernel that an instance of a
batch runs on (k_batch_solve, or k_cluster_solve with one or several CTAs),
nor on the instances beside it."""
from __future__ import annotations

import numpy as np
import pytest

from hprqp import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(60, 1), (641, 1), (60, 200), (60, 300), (700, 300)],
                         ids=["cluster", "cluster_1024", "one_cta_512", "one_cta_640", "k_batch_solve"])
def test_warm_start_without_a_step(engine_lib, n, count):
    """A solve that ends before its first step returns the starting point: x, y
    and w are scaled and unscaled once, two roundings."""
    from hprqp.batch import Batch, pack

    inst = instances.plain_qp(5, n=n, m=n // 2, a_density=0.02, m_rows=20, m_density=0.02, n_eq=n // 8)
    rng = np.random.default_rng(n + count)
    b = Batch(pack([inst] * count))
    x, w, y = rng.uniform(-1, 1, b.n), rng.uniform(-1, 1, b.n), rng.standard_normal(b.m)
    y[np.tile(np.diff(inst.A.indptr) == 0, count)] = 0.0  # rows that the builder takes out
    b.set_warm_start(x, y, w)
    b.solve(stoptol=1e-30, max_iter=0)
    r = b.results()
    b.close()
    assert np.all(r.iter == 0)
    for got, want in ((r.x, x), (r.w, w), (r.y, y)):
        np.testing.assert_allclose(got, want, rtol=4 * np.finfo(float).eps, atol=0)


def test_movable_instances_do_not_wait_for_others(engine_lib):
    """Seven small QPs beside one that no cluster takes (n > 8190) and that
    runs into the time limit: the small ones, 60,000 steps of a few
    microseconds, end by their iteration limit long before it."""
    from hprqp.batch import Batch, pack

    small = [instances.plain_qp(60 + i, n=n, m=n // 2, a_density=0.1, m_rows=10, m_density=0.05, n_eq=5)
             for i, n in enumerate([40] * 6 + [500])]
    large = instances.plain_qp(70, n=8200, m=2000, a_density=0.002, m_rows=1640, m_density=0.002, n_eq=500)
    b = Batch(pack(small + [large]))
    b.solve(stoptol=1e-30, max_iter=60000, time_limit=2.0)
    r = b.results(vectors=False)
    b.close()
    assert r.status[-1] == 5 and 0 < r.iter[-1] < 60000, (r.status[-1], r.iter[-1])
    np.testing.assert_array_equal(r.status[:-1], 4)
    np.testing.assert_array_equal(r.iter[:-1], 60000)


def _mixed(kind):
    """Shapes that a large batch leaves to k_batch_solve: 640-thread ones whose
    matrices are dense enough, 1024-thread ones, and small ones that the
    one-CTA form of k_cluster_solve takes."""
    out = []
    diag = kind == "diagonal"
    for i, (n, m, da, dm) in enumerate([(600, 300, 0.07 if diag else 0.03, 0.01),
                                        (320, 310, 0.13 if diag else 0.07, 0.03),
                                        (640, 640, 0.03 if diag else 0.012, 0.01), (97, 33, 0.1, 0.1),
                                        (700, 300, 0.02, 0.01), (1250, 400, 0.01, 0.005)]):
        inst = instances.plain_qp(300 + i, n=n, m=m, a_density=da, m_rows=n // 3, m_density=dm, n_eq=m // 3)
        if kind == "free":
            free = np.random.default_rng(i).random(n) < 0.95
            inst.l[free], inst.u[free] = -np.inf, np.inf
        if diag:
            inst.Q = instances.CSR(n, n, np.arange(n + 1), np.arange(n), np.random.default_rng(i).uniform(0.1, 2.0, n))
        out.append(inst)
    return out


@pytest.mark.parametrize("count", [200, 312])
@pytest.mark.parametrize("kind", ["boxed", "free", "diagonal"])
def test_every_copy_gets_the_same_bits(engine_lib, kind, count):
    """Copies of six QPs, 353 steps with restarts: most end on the kernel that
    they started on, the last quarter of the running ones are handed over to
    clusters, and none of it shows.  With more than two instances per SM each
    also equals the solve of it alone, on a cluster from the start."""
    from hprqp.batch import Batch, pack

    insts = _mixed(kind)
    kw = dict(stoptol=1e-30, max_iter=353)
    b = Batch(pack([insts[i % 6] for i in range(count)]))
    b.solve(**kw)
    r = b.results()
    parts = {f: b.split(getattr(r, f), "y" if f == "y" else "x") for f in ("x", "y", "z", "w")}
    scalars = ("objective", "residual", "gap", "sigma", "iter", "status")
    b.close()
    for i, inst in enumerate(insts):
        want = {f: parts[f][i] for f in parts} | {f: getattr(r, f)[i] for f in scalars}
        if count > 296:
            alone = Batch(pack([inst]))
            alone.solve(**kw)
            s = alone.results()
            alone.close()
            want = {f: getattr(s, f) for f in parts} | {f: getattr(s, f)[0] for f in scalars}
        for k in range(i, count, 6):
            for f in parts:
                np.testing.assert_array_equal(parts[f][k], want[f], err_msg=f"{f} of copy {k}")
            for f in scalars:
                assert getattr(r, f)[k] == want[f], (f, k)
