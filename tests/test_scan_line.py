"""Which scan a batch takes (scan_mma_pays in csrc/erq_capi.cu): by pairs and by
the size of the clusters, from other numbers on in a plan, and the same results
on both sides of each line."""
import os

import numpy as np
import pytest

from test_refine_windows import _index

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _scans(fn):
    """fn()'s result and the scan kernels it launched (1: lookups, 2: products)."""
    from erq_b200 import _lib

    _lib.profile_enable(True)
    _lib.profile_reset()
    try:
        out = fn()
        torch.cuda.synchronize()
        return _lib.profile_read()["scan"][0], out
    finally:
        _lib.profile_enable(False)


@pytest.mark.parametrize("sizes,search,plan", [
    # nprobe, queries -> kernels
    ([20] * 300, {(2, 1024): 1, (2, 3071): 1, (2, 3073): 2}, {(4, 1000): 1, (1, 1023): 1, (1, 1024): 2, (6, 1000): 2}),
    ([250] * 40, {(2, 600): 1, (4, 500): 1, (4, 550): 2}, {(2, 550): 1, (2, 600): 2}),
    ([2100] + [90] * 30, {(1, 511): 1, (1, 700): 2}, {(1, 700): 2}),
])
def test_both_sides_of_the_lines(tmp_path, oracle_mod, sizes, search, plan):
    from erq_b200 import Plan

    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, 1536, sizes, 4, len(sizes))
    nq = max(n for _, n in [*search, *plan])
    pick = torch.randint(0, len(sizes), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, 1536, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    ref = {p: o.search(q, 10, p, nthreads=8) for p in {p for p, _ in [*search, *plan]}}
    o.close()

    def check(nprobe, n, got):
        assert (got[0] == ref[nprobe][0][:n]).all(), (nprobe, n)
        assert (got[1].view(np.uint32) == ref[nprobe][1][:n].view(np.uint32)).all(), (nprobe, n)

    for (nprobe, n), kernels in search.items():
        seen, got = _scans(lambda: idx.search_batch(q[:n], 10, nprobe))
        assert seen == kernels, (nprobe, n)
        check(nprobe, n, got)
    for (nprobe, n), kernels in plan.items():
        p = Plan(idx, n, 10, nprobe)
        p.set_graphs(False)
        seen, got = _scans(lambda: p.search(q[:n]))
        assert seen == kernels, (nprobe, n)
        check(nprobe, n, got)
        p.free()
    idx.free()
