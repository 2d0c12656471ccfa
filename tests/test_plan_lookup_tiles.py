"""Every tile of a plan's lookup scan (csrc/scan_batch.cuh) on uneven clusters, in
a batch below the line from which plans scan on the tensor cores, against the C
oracle, ids and distance bits equal."""
import os

import pytest

from test_plan import SHAPES
from test_refine_windows import _index, _same
from test_scan_line import _scans

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dim,nq,nprobe", [(128, 1300, 6), (1024, 250, 4)])
def test_every_tile(tmp_path, oracle_mod, dim, nq, nprobe):
    from erq_b200 import Plan

    path = os.path.join(tmp_path, "i.index")
    sizes = [int(4000 / (i + 1) ** 1.3) for i in range(60)] + [0, 1]
    idx, g, cent = _index(path, dim, sizes, 7, dim)
    pick = (62 * torch.rand(nq, generator=g) ** 2).long()
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    ref = o.search(q, 100, nprobe, nthreads=8)
    o.close()
    plan = Plan(idx, nq, 100, nprobe)
    plan.set_graphs(False)
    for qb, w in SHAPES:
        for cb in (1, 3, 16, 64):
            plan.set_tuning(nq, qb, cb, w)
            n, got = _scans(lambda: plan.search(q))
            assert n == 1
            _same(got[:2], ref)
    plan.free()
    idx.free()
