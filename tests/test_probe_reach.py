"""The probe's fallback (probe_exact_kernel in csrc/probe.cuh) where its list of
centroids in reach is longer than one round of it holds, where the bound on the
reach is not a number, and where K is just above a round, against the C oracle."""
import os

import numpy as np
import pytest

from test_refine_windows import _same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("K,dim,nprobe", [(1025, 64, 7), (3000, 128, 40), (2049, 64, 300), (5003, 192, 20)])
def test_most_centroids_in_reach(tmp_path, oracle_mod, K, dim, nprobe):
    """Centroids closer together than the estimates are exact: a cut that is not
    proven has most of them in reach."""
    from erq_b200 import IVF, _lib, build_index, indexfile

    path = os.path.join(tmp_path, "i.index")
    g = torch.Generator().manual_seed(K)
    point = torch.randn(1, dim, generator=g)
    cent = point + 3e-5 * torch.randn(K, dim, generator=g)
    cent[K // 2:K // 2 + 5] = cent[3]  # ties
    ids = torch.arange(K).repeat(3)
    base = cent[ids] + 0.5 * torch.randn(ids.numel(), dim, generator=g)
    arr = build_index.build_index_torch(base.cuda(), cent.cuda(), ids.cuda(), 4, seed=1)
    indexfile.write_index(path, arr)
    idx = IVF(path)
    nq = 40
    q = idx.rotate((point + torch.randn(nq, dim, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    ref = o.search(q, 10, nprobe, nthreads=8)
    o.close()
    _lib.probe_fallbacks(0, reset=True)
    _same(idx.search_batch(q, 10, nprobe), ref)
    assert _lib.probe_fallbacks(0, reset=True) > nq // 2
    # queries without a bound leave the others of their batch as they are
    bad = q.copy()
    bad[5, 3] = np.nan
    bad[6, 0] = np.inf
    bad[7] = 3e19  # a norm past the floats
    ids, d = idx.search_batch(bad, 10, nprobe)
    keep = [i for i in range(nq) if i not in (5, 6, 7)]
    _same((ids[keep], d[keep]), (ref[0][keep], ref[1][keep]))
    idx.free()
