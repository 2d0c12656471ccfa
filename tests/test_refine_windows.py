"""The refinement's windows and pools (csrc/refine.cuh) at their edges, against
the C oracle, ids and distance bits equal: pools of every kind (registers up to
128 entries, shared memory above, never filled), both launch forms (at most one
query per SM, more), windows cut by full lists, by the number of staged
clusters and by the pool's filling, more probes and blocks than one pass of the
window search holds, rows of 8-, 4- and 2-bit codes that do and do not fill
whole 16-byte words, equal distances, and unit queries outside the range of the
scaled codes."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _index(path, dim, sizes, bits, seed, sigma=0.7, P=None, dup=0, zero_dims=0):
    from erq_b200 import IVF, build_index, indexfile

    g = torch.Generator().manual_seed(seed)
    K = len(sizes)
    cent = torch.randn(K, dim, generator=g)
    if zero_dims:
        cent[:, :zero_dims] = 0
    ids = torch.repeat_interleave(torch.arange(K), torch.tensor(sizes))
    base = cent[ids] + sigma * torch.randn(ids.numel(), dim, generator=g)
    if dup:  # runs of equal vectors: equal distances in pools and at their end
        base = base[torch.arange(ids.numel()) // dup * dup]
        ids = ids[torch.arange(ids.numel()) // dup * dup]
    arr = build_index.build_index_torch(base.cuda(), cent.cuda(), ids.cuda(), bits, P=P, seed=seed)
    indexfile.write_index(path, arr)
    return IVF(path), g, cent


def _same(got, ref):
    assert (got[0] == ref[0]).all()
    assert (got[1].view(np.uint32) == ref[1].view(np.uint32)).all()


@pytest.mark.parametrize("dim,bits", [(64, 3), (192, 4), (320, 5), (128, 7), (960, 8), (256, 9), (1536, 4)])
def test_pools_forms_and_rows(tmp_path, oracle_mod, dim, bits):
    path = os.path.join(tmp_path, "i.index")
    sizes = [1 + (37 * i) % 61 for i in range(90)] + [700, 1500, 0, 33]
    idx, g, cent = _index(path, dim, sizes, bits, dim + bits)
    nq = 160  # more than one query per SM
    pick = torch.randint(0, len(sizes), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k, nprobe in ((1, 3), (10, 94), (100, 40), (128, 94), (129, 94), (300, 60), (1024, 94)):
        ref = o.search(q, k, nprobe, nthreads=8)
        _same(idx.search_batch(q, k, nprobe), ref)
        _same(idx.search_batch(q[:9], k, nprobe), (ref[0][:9], ref[1][:9]))
    o.close()
    idx.free()


def test_many_probes_and_blocks(tmp_path, oracle_mod):
    """Over 256 probes and over 1,024 blocks per query; pools that stay short."""
    path = os.path.join(tmp_path, "i.index")
    sizes = [(13 * i) % 97 for i in range(700)]
    idx, g, cent = _index(path, 64, sizes, 5, 3, sigma=2.0)
    q = idx.rotate((2.0 * torch.randn(155, 64, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k, nprobe in ((100, 700), (7, 300), (600, 2)):
        ref = o.search(q, k, nprobe, nthreads=8)
        _same(idx.search_batch(q, k, nprobe), ref)
        _same(idx.search_batch(q[:5], k, nprobe), (ref[0][:5], ref[1][:5]))
    o.close()
    idx.free()


def test_equal_distances(tmp_path, oracle_mod):
    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, 128, [400, 96, 300, 64, 900, 31], 8, 5, dup=9)
    pick = torch.randint(0, 6, (150,), generator=g)
    q = idx.rotate((cent[pick] + 0.5 * torch.randn(150, 128, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k in (1, 20, 100, 128, 200):
        ref = o.search(q, k, 6, nthreads=8)
        _same(idx.search_batch(q, k, 6), ref)
        _same(idx.search_batch(q[:6], k, 6), (ref[0][:6], ref[1][:6]))
    o.close()
    idx.free()


@pytest.mark.parametrize("tiny", [1e-35, 1e-30, 1e-43])
def test_unit_queries_outside_the_scaled_range(tmp_path, oracle_mod, tiny):
    """An identity rotation and dims where the centroids are zero: queries with
    tiny values there have unit components below 2^-96 (1e-30: just above)."""
    path = os.path.join(tmp_path, "i.index")
    P = np.eye(128, dtype=np.float32)
    idx, g, cent = _index(path, 128, [300, 200, 500, 50], 8, 11, P=P, zero_dims=70)
    q = torch.zeros(152, 128)
    q[:, 70:] = cent[torch.randint(0, 4, (152,), generator=g)][:, 70:] + 0.5 * torch.randn(152, 58, generator=g)
    q[::2, :70] = tiny * torch.randn(76, 70, generator=g)  # every other query leaves the range
    q = q.numpy()
    o = oracle_mod.Oracle(path)
    ref = o.search(q, 50, 4, nthreads=8)
    _same(idx.search_batch(q, 50, 4), ref)
    _same(idx.search_batch(q[:8], 50, 4), (ref[0][:8], ref[1][:8]))
    o.close()
    idx.free()
