"""The 4-warp refinement with windows across clusters (csrc/refine.cuh), which
batches above three queries per SM take, at the edges of its windows and pools,
against the C oracle, ids and distance bits equal: codes of every storage size,
pools on both sides of the register limit and of the largest k, over 128 and 256
probes, equal distances, and unit queries outside the range of the scaled codes."""
import os

import numpy as np
import pytest

from test_refine_windows import _index, _same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _batch():
    return 3 * torch.cuda.get_device_properties(0).multi_processor_count + 1


@pytest.mark.parametrize("dim,bits", [(64, 3), (128, 7), (256, 9), (1536, 8)])
def test_pools_and_rows(tmp_path, oracle_mod, dim, bits):
    path = os.path.join(tmp_path, "i.index")
    sizes = [1 + (37 * i) % 61 for i in range(150)] + [33, 0]
    idx, g, cent = _index(path, dim, sizes, bits, 3 * dim + bits)
    nq = _batch()
    pick = torch.randint(0, len(sizes), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k, nprobe in ((1, 9), (32, 5), (33, 152), (128, 40), (256, 60), (257, 60), (1024, 130)):
        _same(idx.search_batch(q, k, nprobe), o.search(q, k, nprobe, nthreads=8))
    o.close()
    idx.free()


def test_many_probes(tmp_path, oracle_mod):
    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, 64, [(13 * i) % 97 for i in range(500)], 9, 3, sigma=2.0)
    q = idx.rotate((2.0 * torch.randn(_batch(), 64, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k, nprobe in ((100, 500), (7, 300), (300, 129)):
        _same(idx.search_batch(q, k, nprobe), o.search(q, k, nprobe, nthreads=8))
    o.close()
    idx.free()


def test_equal_distances(tmp_path, oracle_mod):
    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, 128, [150, 96, 100, 64, 90, 31, 40], 8, 5, dup=9)
    pick = torch.randint(0, 7, (_batch(),), generator=g)
    q = idx.rotate((cent[pick] + 0.5 * torch.randn(len(pick), 128, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k in (1, 20, 100, 200, 256, 300):
        _same(idx.search_batch(q, k, 7), o.search(q, k, 7, nthreads=8))
    o.close()
    idx.free()


@pytest.mark.parametrize("tiny", [1e-35, 1e-43])
def test_unit_queries_outside_the_scaled_range(tmp_path, oracle_mod, tiny):
    """More clusters than unit queries are staged at once, some with the plain
    codes: an identity rotation and dims where every second query is tiny."""
    path = os.path.join(tmp_path, "i.index")
    P = np.eye(128, dtype=np.float32)
    idx, g, cent = _index(path, 128, [40, 70, 25, 90, 33, 60, 64, 10, 80, 55, 31, 20], 8, 11, P=P, zero_dims=70)
    nq = _batch()
    q = torch.zeros(nq, 128)
    q[:, 70:] = cent[torch.randint(0, 12, (nq,), generator=g)][:, 70:] + 0.5 * torch.randn(nq, 58, generator=g)
    q[::2, :70] = tiny * torch.randn((nq + 1) // 2, 70, generator=g)
    q = q.numpy()
    o = oracle_mod.Oracle(path)
    _same(idx.search_batch(q, 50, 12), o.search(q, 50, 12, nthreads=8))
    o.close()
    idx.free()
