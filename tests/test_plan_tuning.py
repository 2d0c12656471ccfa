"""What a plan's tuning selects: a refinement form asked for by its warps is the
one that runs, and what the autotuner did not time is not fixed for other batch
sizes.  Results are the same in every case."""
import os

import numpy as np
import pytest

from test_refine_windows import _index

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _same(got, ref):
    assert (got[0] == ref[0]).all()
    assert (got[1].view(np.uint32) == ref[1].view(np.uint32)).all()


def test_refine_warps_selects_the_form(tmp_path):
    """40 clusters of 6 vectors and a pool that never fills: a window holds as
    many clusters as unit queries are staged, 8 with 4 warps, 12 with 8, 16 with
    16, so each form shows in the number of windows."""
    from erq_b200 import Plan, _lib

    idx, g, cent = _index(os.path.join(tmp_path, "i.index"), 64, [6] * 40, 5, 2)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    q = idx.rotate(torch.randn(3 * sms + 1, 64, generator=g).numpy())
    plan = Plan(idx, len(q), 250, 40)
    plan.set_graphs(False)
    ref = plan.search(q)
    for n in (1, sms, sms + 1, 3 * sms, 3 * sms + 1):
        by_size = 3 if n <= sms else (4 if n <= 3 * sms else 5)
        for rw, windows in ((4, 5), (32, 3), (0, by_size)):
            plan.set_tuning(n, 1, 16, 4, rw)
            assert plan.tuning(n)["refine_warps"] == rw
            _lib.refine_stats(enable=True)
            got = plan.search(q[:n])
            assert _lib.refine_stats()["windows"] == windows * n, (n, rw)
            _same(got[:2], (ref[0][:n], ref[1][:n]))
    plan.free()
    idx.free()


def test_autotune_fixes_what_it_timed(tmp_path):
    from erq_b200 import Plan

    idx, g, cent = _index(os.path.join(tmp_path, "i.index"), 128, [90] * 60, 4, 3)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    q = idx.rotate((cent[torch.randint(0, 60, (2000,), generator=g)] +
                    0.7 * torch.randn(2000, 128, generator=g)).numpy())
    ref = idx.search_batch(q, 10, 8)

    def tile(t):
        return t["queries_per_item"], t["blocks_per_item"], t["warps"]

    # 16,000 pairs: on the tensor cores, no tile is timed
    plan = Plan(idx, 2000, 10, 8)
    default = {n: tile(plan.tuning(n)) for n in (1, 60, sms, 2000)}
    t, _ = plan.autotune(q, reps=2)
    assert plan.tuning(2000) == t and t["refine_warps"] in (4, 32)
    for n in (1, 60, sms):
        assert tile(plan.tuning(n)) == default[n]
        _same(plan.search(q[:n])[:2], (ref[0][:n], ref[1][:n]))
    if t["refine_warps"] == 4:  # the default of this size: others keep theirs
        assert plan.tuning(sms)["refine_warps"] == 32
        assert plan.tuning(sms + 1)["refine_warps"] == 0
    plan.free()
    # 400 pairs: by lookups, the tile goes with the tuning
    plan = Plan(idx, 50, 10, 8)
    t, _ = plan.autotune(q[:50], reps=2)
    assert plan.tuning(50) == t
    assert tile(plan.tuning(1)) == tile(t)
    _same(plan.search(q[:50])[:2], (ref[0][:50], ref[1][:50]))
    plan.free()
    idx.free()
