"""The coarse probe by blocks and by warps (csrc/erq_capi.cu, probe_block_pays)
on both sides of each line - nprobe x D, six and eight queries per SM, more
clusters than are staged - against the C oracle's search, ids and distance bits
equal."""
import os

import pytest

from test_refine_windows import _index, _same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dim,clusters", [(64, 300), (256, 131), (768, 1031), (64, 4099)])
def test_forms_by_work_and_batch(tmp_path, oracle_mod, dim, clusters):
    path = os.path.join(tmp_path, "i.index")
    sizes = [1 + (7 * i) % 5 for i in range(clusters)]
    idx, g, cent = _index(path, dim, sizes, 4, dim + clusters)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nq = 8 * sms + 1
    pick = torch.randint(0, clusters, (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    near = -(-3072 // dim)
    far = min(63, -(-12288 // dim))
    for nprobe in sorted({1, min(near, 63) - 1, min(near, 63), far - 1, far}):
        ref = o.search(q, 5, nprobe, nthreads=8)
        for n in (1, 6 * sms, 6 * sms + 1, 8 * sms, nq):
            _same(idx.search_batch(q[:n], 5, nprobe), (ref[0][:n], ref[1][:n]))
    o.close()
    idx.free()
