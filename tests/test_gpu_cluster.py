"""Thread-block clusters (k_cluster_solve): an instance gets the same answer,
bit for bit, whether a cluster solves it alone, one CTA of a large batch
solves it, or it is handed from one CTA to a cluster on the way.

The reference is the one-CTA kernel itself: in a batch of more than two
instances per SM every instance starts on one CTA of the shape it would have
alone, so the same arithmetic in the same order must give the same bits
(tolerance 0).  Its parity with the oracle is test_gpu_batch's subject."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free_vars(inst, seed):
    free = np.random.default_rng(seed).random(inst.n) < 0.95  # the step without bounds (noC)
    inst.l[free], inst.u[free] = -np.inf, np.inf
    return inst


# (n, m): rows that do not divide among the CTAs, the edge between the 640-
# and 1024-thread shapes, fewer rows of A than CTAs, more rows than variables,
# matrices that fill or exceed the CTAs' shared memory
SIZES = [(33, 16), (60, 1), (121, 60), (320, 3), (640, 257), (641, 300), (900, 899), (1000, 500), (257, 400),
         (1531, 1013), (2047, 700)]


def _instances(kind):
    from hprqp import instances

    out = []
    for i, (n, m) in enumerate(SIZES):
        inst = instances.plain_qp(77 + i, n=n, m=m, a_density=min(0.3, 12.0 / n), m_rows=max(1, n // 5),
                                  m_density=min(0.5, 6.0 / n), n_eq=m // 2)
        out.append(_free_vars(inst, i) if kind == "free" else inst)
    return out


@pytest.mark.parametrize("max_iter", [1, 230])
@pytest.mark.parametrize("kind", ["boxed", "free"])
def test_cluster_equals_one_cta(engine_lib, kind, max_iter):
    from hprqp.batch import Batch, pack

    insts = _instances(kind)
    kw = dict(stoptol=1e-30, max_iter=max_iter)  # no instance ends early: none is handed over
    many = Batch(pack(insts * 28))  # 308 instances: one CTA each
    many.solve(**kw)
    ref = many.results()
    few = Batch(pack(insts))  # all at once, SMs spread over them
    few.solve(**kw)
    got = few.results()
    for f in ("status", "iter", "objective", "residual", "gap", "sigma"):
        np.testing.assert_array_equal(getattr(got, f), getattr(ref, f)[:len(insts)], err_msg=f)
    for f, size in (("x", few.n), ("w", few.n), ("z", few.n), ("y", few.m)):
        np.testing.assert_array_equal(getattr(got, f), getattr(ref, f)[:size], err_msg=f)
    for k, inst in enumerate(insts):
        alone = Batch(pack([inst]))
        alone.solve(**kw)
        r = alone.results()
        for f, kind_ in (("x", "x"), ("w", "x"), ("z", "x"), ("y", "y")):
            np.testing.assert_array_equal(getattr(r, f), few.split(getattr(got, f), kind_)[k], err_msg=f"{f} {SIZES[k]}")


@pytest.mark.parametrize("count", [16, 200, 310])
def test_handed_over_instances(engine_lib, count):
    """Batches whose instances end at different times: the last ones move to
    clusters.  Every instance equals the solve of it alone."""
    from hprqp import instances
    from hprqp.batch import Batch, pack

    insts = [instances.plain_qp(900 + i, n=60 + (i * 53) % 700, m=20 + (i * 17) % 90, a_density=0.03, m_rows=40,
                                m_density=0.02, n_eq=10) for i in range(count)]
    kw = dict(stoptol=1e-7, max_iter=6000)
    b = Batch(pack(insts))
    b.solve(**kw)
    r = b.results()
    b.solve(**kw)
    again = b.results()
    for f in ("x", "y", "z", "w", "iter", "status", "objective"):
        np.testing.assert_array_equal(getattr(again, f), getattr(r, f), err_msg=f)
    if 148 < count <= 296:
        return  # the 512-thread shape: a single solve sums in another order
    xs = b.split(r.x, "x")
    for k in np.argsort(-r.iter)[:8]:  # the ones that ran longest
        alone = Batch(pack([insts[k]]))
        alone.solve(**kw)
        s = alone.results()
        assert s.iter[0] == r.iter[k] and s.status[0] == r.status[k]
        np.testing.assert_array_equal(s.x, xs[k])


@pytest.mark.parametrize("max_iter", [1, 230])
@pytest.mark.parametrize("kind", ["boxed", "free"])
@pytest.mark.parametrize("count", [200, 308])
def test_diagonal_q_equals_one_cta(engine_lib, count, kind, max_iter):
    """Instances whose Q is diagonal: on the one-CTA kernel (the batch of 308
    holds shapes that k_cluster_solve takes and shapes that it does not) and
    on clusters the same bits, so a hand-over does not show."""
    from hprqp import instances
    from hprqp.batch import Batch, pack

    insts = []
    for i, inst in enumerate(_instances(kind)):
        n = inst.n
        d = np.random.default_rng(i).uniform(0.1, 2.0, n)
        inst.Q = instances.CSR(n, n, np.arange(n + 1), np.arange(n), d)
        insts.append(inst)
    kw = dict(stoptol=1e-30, max_iter=max_iter)
    many = Batch(pack((insts * 28)[:count]))
    many.solve(**kw)
    ref = many.results()
    many.solve(**kw)
    again = many.results()
    few = Batch(pack(insts))
    few.solve(**kw)
    got = few.results()
    for f, size in (("x", few.n), ("w", few.n), ("z", few.n), ("y", few.m)):
        np.testing.assert_array_equal(getattr(again, f), getattr(ref, f), err_msg=f)
        if count > 296:  # (up to 296 instances the sums are taken in another order)
            np.testing.assert_array_equal(getattr(got, f), getattr(ref, f)[:size], err_msg=f)
