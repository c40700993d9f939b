"""hprqp_b200_release_memory: what closed handles leave goes back to the
device, and solves go on as before."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_memory_comes_back(engine_lib):
    import torch
    from hprqp import instances
    from hprqp.batch import Batch, pack

    insts = [instances.plain_qp(9, n=600, m=300)] * 300
    kw = dict(stoptol=1e-6, max_iter=300)

    def solve():
        b = Batch(pack(insts))
        b.solve(**kw)
        r = b.results()
        b.close()
        return r.x, r.y

    first = solve()  # loads the kernels too
    engine_lib.release_memory()
    free = torch.cuda.mem_get_info(0)[0]
    again = solve()
    kept = free - torch.cuda.mem_get_info(0)[0]
    engine_lib.release_memory()
    assert kept > 16 << 20  # the workspaces alone, 32 vectors of 608 and 12 of 320 for 148 CTAs, are 27 MB
    assert abs(free - torch.cuda.mem_get_info(0)[0]) <= 4 << 20
    for a, b in zip(first, again):
        np.testing.assert_array_equal(a, b)
    open_handle = Batch(pack(insts[:4]))
    engine_lib.release_memory()
    open_handle.solve(**kw)
    np.testing.assert_array_equal(open_handle.results().status, 4)
    open_handle.close()
    with pytest.raises(RuntimeError):
        engine_lib.release_memory(999)
