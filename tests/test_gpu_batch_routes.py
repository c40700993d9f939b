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
