"""Searches and plans on a device that is nearly full.

The quantized rows of the tensor-core scan are the one buffer that a search can
do without (it scans by lookups then), so they never take the room of another:
what fits without them is not refused, and every result is the same."""
import os

import numpy as np
import pytest

from test_refine_windows import _index

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _same(got, ref):
    assert (got[0] == ref[0]).all()
    assert (got[1].view(np.uint32) == ref[1].view(np.uint32)).all()


class _limit:
    def __init__(self, n):
        self.n = n

    def __enter__(self):
        from erq_b200 import _lib

        _lib.check(_lib.load_library().erq_debug_set_memory_limit(self.n))

    def __exit__(self, *a):
        from erq_b200 import _lib

        _lib.check(_lib.load_library().erq_debug_set_memory_limit(0))


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


@pytest.fixture(scope="module")
def case(tmp_path_factory):
    from erq_b200 import learned

    path = os.path.join(tmp_path_factory.mktemp("mem"), "i.index")
    sizes = [1 + (7 * i) % 70 for i in range(300)]
    idx, g, cent = _index(path, 1024, sizes, 4, 7)
    nq = 1100
    pick = torch.randint(0, 300, (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, 1024, generator=g)).numpy())
    labels = np.random.default_rng(1).integers(0, 8, nq).astype(np.uint8)
    model = learned.ProbeModel.train(learned.probe_features(idx, q), labels, epochs=1, batch=256)
    yield idx, q, model
    model.free()
    idx.free()


@pytest.mark.parametrize("with_model", [False, True])
def test_a_plan_does_without_the_rows(case, with_model):
    from erq_b200 import Plan, _lib

    idx, q, model = case

    def make():
        p = Plan(idx, len(q), 10, 5, model=model if with_model else None)
        p.set_graphs(False)
        return p

    p = make()
    full = p.device_bytes()
    n, ref = _scans(lambda: p.search(q))
    assert n == 2
    p.free()
    with _limit(full - 1):  # all but the rows
        p = make()
    least = p.device_bytes()
    assert least < full
    n, got = _scans(lambda: p.search(q))
    assert n == 1
    _same(got[:2], ref[:2])
    p.free()
    with _limit(least):
        make().free()
    with _limit(least - 1), pytest.raises(_lib.ErqError, match="OUT_OF_MEMORY"):
        make()


@pytest.mark.parametrize("with_model", [False, True])
def test_a_search_does_without_the_rows(case, with_model):
    from erq_b200 import _lib, learned

    idx, q, model = case

    def search():
        if with_model:
            return learned.search_learned(idx, model, q, 10, 5)[:2]
        return idx.search_batch(q, 10, 5)

    _, ref = _scans(search)
    seen = []
    for mib in np.concatenate([np.linspace(4, 64, 121), np.geomspace(65, 1024, 12)]):
        with _limit(int(mib * (1 << 20))):
            try:
                n, got = _scans(search)
            except _lib.ErqError as e:
                assert "OUT_OF_MEMORY" in str(e)
                seen.append(0)
                continue
        _same(got, ref)
        seen.append(n)
    # refused, then by lookups, then by products: in this order
    assert seen == sorted(seen) and set(seen) == {0, 1, 2}, seen


def test_a_large_call_keeps_to_the_budget_with_the_rows(tmp_path):
    """25,000 queries whose workspace takes 2.9 of the 3 GiB without the rows (0.9
    GB): two batches of products within the budget and the eighth that rows may add,
    not one beyond it."""
    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, 1024, [57 * 32] * 20, 4, 9)
    nq, k, nprobe = 25_000, 10, 16
    pick = torch.randint(0, 20, (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, 1024, generator=g)).cuda())
    with _limit((3 << 30) + (448 << 20)):
        n, (ids, d) = _scans(lambda: idx.search_batch(q, k, nprobe))
    assert n == 4
    for at in (0, 12_000, 19_000, nq - 30):  # by lookups
        n, few = _scans(lambda: idx.search_batch(q[at:at + 30].contiguous(), k, nprobe))
        assert n == 1
        assert (few[0] == ids[at:at + 30]).all() and (few[1] == d[at:at + 30]).all()
    idx.free()
