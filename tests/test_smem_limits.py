"""Shared-memory limits are properties of a kernel, not of an index: a search of
a small index between the making of a plan on a large one and the first search
of a batch size (which launches and captures) changes nothing."""
import os

import numpy as np
import pytest

from test_refine_windows import _index

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _same(got, ref):
    assert (got[0] == ref[0]).all()
    assert (got[1].view(np.uint32) == ref[1].view(np.uint32)).all()


@pytest.mark.parametrize("dim", [1024, 1536, 2048])
def test_a_small_index_lowers_no_limit(tmp_path, dim):
    from erq_b200 import Plan

    big, g, cent = _index(os.path.join(tmp_path, "big.index"), dim, [1 + (5 * i) % 40 for i in range(300)], 4, dim)
    # of the same and of a smaller class of dimensions of the plans' tile kernels
    smalls = [_index(os.path.join(tmp_path, f"s{d}.index"), d, [40] * 20, 4, d)[0] for d in (64, dim - 192)]
    pick = torch.randint(0, 300, (500,), generator=g)
    q = big.rotate((cent[pick] + 0.7 * torch.randn(500, dim, generator=g)).numpy())
    ref = big.search_batch(q, 10, 4)
    plan = Plan(big, 500, 10, 4)

    def others():
        for s in smalls:
            qs = np.random.default_rng(1).standard_normal((5, s.D)).astype(np.float32)
            p = Plan(s, 5, 10, 4)
            _same(p.search(qs)[:2], s.search_batch(qs, 10, 4))
            p.free()

    for n in (1, 50, 200, 500):  # lookups, products; probes by blocks and by warps
        others()
        _same(plan.search(q[:n])[:2], (ref[0][:n], ref[1][:n]))
    plan.set_graphs(False)
    for qb, w in ((1, 4), (1, 8), (2, 8), (4, 8)):
        plan.set_tuning(50, qb, 8, w)
        others()
        _same(plan.search(q[:50])[:2], (ref[0][:50], ref[1][:50]))
    plan.free()
    for i in (big, *smalls):
        i.free()
