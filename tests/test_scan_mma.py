"""The tensor-core scan (csrc/scan_mma.cuh) at the edges of its tiles.

Sums are exact integers, so ids and distances must equal the C oracle's bit
for bit: clusters around a block (32 vectors), a tile (4 blocks) and a work
item (32 blocks), empty ones too; query groups around 8 rows and around the
32 queries of an item; padded dimensions whose 96-dim chunks do and do not
fill the 128-dim blocks of the query operand; per-query depths.  Batches below
the dispatch's line take the lookup scan, which the launch counts show."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

EDGES = [0, 1, 31, 32, 33, 127, 128, 129, 160, 1023, 1024, 1025, 1060, 2100]


def _index(path, dim, sizes, bits, seed):
    from erq_b200 import IVF, build_index, indexfile

    g = torch.Generator().manual_seed(seed)
    K = len(sizes)
    cent = torch.randn(K, dim, generator=g)
    ids = torch.repeat_interleave(torch.arange(K), torch.tensor(sizes))
    ids = ids[torch.randperm(ids.numel(), generator=g)]
    base = cent[ids] + 0.7 * torch.randn(ids.numel(), dim, generator=g)
    arr = build_index.build_index_torch(base.cuda(), cent.cuda(), ids.cuda(), bits, seed=seed)
    indexfile.write_index(path, arr)
    return IVF(path), g, cent


def _scan_launches(fn):
    from erq_b200 import _lib

    _lib.profile_enable(True)
    _lib.profile_reset()
    try:
        out = fn()
        torch.cuda.synchronize()
        return _lib.profile_read()["scan"][0], out
    finally:
        _lib.profile_enable(False)


def _same(got, ref):
    assert (got[0] == ref[0]).all()
    assert (got[1].view(np.uint32) == ref[1].view(np.uint32)).all()


@pytest.mark.parametrize("dim,bits,nq", [(64, 4, 1171), (100, 8, 601), (768, 9, 98), (960, 3, 79),
                                         (1536, 8, 49), (1500, 5, 65), (2048, 7, 37)])
def test_every_cluster_and_group_size(tmp_path, oracle_mod, dim, bits, nq):
    """All clusters probed by every query: groups of ceil(nq / 32) even parts."""
    from erq_b200 import Plan

    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, dim, EDGES, bits, 100 + dim)
    pick = torch.randint(0, len(EDGES), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    q[3] = q[2]  # equal queries
    o = oracle_mod.Oracle(path)
    q[0] = o.centroids()[5]  # a query on a centroid: the unit query is constant
    ref = o.search(q, 20, len(EDGES), nthreads=8)
    o.close()
    n, got = _scan_launches(lambda: idx.search_batch(q, 20, len(EDGES)))
    assert n == 2  # quantization and products
    _same(got, ref)
    plan = Plan(idx, nq, 20, len(EDGES))
    for _ in range(2):
        _same(plan.search(q)[:2], ref)
    # below the line: lookups, the same results
    few = q[:3]
    n, got = _scan_launches(lambda: idx.search_batch(few, 20, len(EDGES)))
    assert n == 1
    _same(got, (ref[0][:3], ref[1][:3]))
    plan.free()
    idx.free()


def test_small_groups_and_learned_depths(tmp_path, oracle_mod):
    """Many small clusters with a few queries each, and per-query depths."""
    from erq_b200 import Plan, learned

    path = os.path.join(tmp_path, "i.index")
    sizes = [1 + (7 * i) % 70 for i in range(300)]
    idx, g, cent = _index(path, 1024, sizes, 8, 7)
    nq, nprobe = 1100, 5
    pick = torch.randint(0, 300, (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, 1024, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    n, got = _scan_launches(lambda: idx.search_batch(q, 10, nprobe))
    assert n == 2
    _same(got, o.search(q, 10, nprobe, nthreads=8))
    feats = learned.probe_features(idx, q)
    labels = np.random.default_rng(1).integers(0, 8, nq).astype(np.uint8)
    model = learned.ProbeModel.train(feats, labels, epochs=2, batch=256)
    ids, d, used = learned.search_learned(idx, model, q, 10, nprobe, confidence=0.6)
    assert len(np.unique(used)) > 1
    for depth in np.unique(used):
        at = used == depth
        _same((ids[at], d[at]), o.search(q[at], 10, int(depth), nthreads=8))
    plan = Plan(idx, nq, 10, nprobe, model=model)
    plan.set_learned(0.6)
    pid, pd, pu = plan.search(q, with_nprobe=True)
    assert (pu == used).all()
    _same((pid, pd), (ids, d))
    o.close()
    plan.free()
    idx.free()
