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
