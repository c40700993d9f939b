"""Blocks, streams and pinned words shared between solves (pool.cpp): solves
in several threads and of several sizes give what each gives alone."""
from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_concurrent_solves_share_the_pool(engine_lib):
    from hprqp import instances
    from hprqp.batch import solve_batch

    insts = [instances.plain_qp(40 + i, n=80 + 160 * i, m=30 + 60 * i, a_density=0.03, m_rows=20, m_density=0.02,
                                n_eq=10) for i in range(8)]

    def single(i):
        r = engine_lib.optimize(engine_lib.build_from_instance(insts[i]),
                                engine_lib.Parameters(verbose=False, stoptol=1e-6, max_iter=500), as_numpy=True)
        return r.x, r.y

    def batch(i):
        r = solve_batch(insts[: 2 + i], stoptol=1e-6, max_iter=500)
        return r.x, r.y

    jobs = [(f, i) for i in range(8) for f in (single, batch)]
    old = engine_lib.set_single_cta_max_work(20000)  # the small ones on clusters, the larger ones device-wide
    try:
        alone = [f(i) for f, i in jobs]
        with ThreadPoolExecutor(4) as ex:
            for _ in range(3):
                for (a, b) in zip(alone, ex.map(lambda j: j[0](j[1]), jobs)):
                    np.testing.assert_array_equal(a[0], b[0])
                    np.testing.assert_array_equal(a[1], b[1])
    finally:
        engine_lib.set_single_cta_max_work(old)
