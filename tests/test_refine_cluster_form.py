"""The refinement with windows per cluster (csrc/refine_cluster.cuh) on both sides
of the lines that choose it (refine_by_cluster in csrc/erq_capi.cu): pools of 256
and 257, up to and above a wave of queries, 4 probes and 5, codes of 8 bits and
smaller, clusters around 6 and 32 blocks, k up to a cluster's size, one wave and
more - against the C oracle, ids and distance bits equal."""
import os

import pytest

from test_refine_windows import _index, _same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHORT = [1 + (37 * i) % 150 for i in range(60)] + [0, 33]
LONG = [1800, 1100, 64, 0, 1031]


@pytest.mark.parametrize("dim,bits,sizes", [(64, 9, SHORT), (192, 7, [170 + i % 40 for i in range(24)]),
                                            (1024, 8, SHORT), (128, 4, SHORT), (100, 5, LONG), (1088, 9, SHORT)])
def test_windows_per_cluster(tmp_path, oracle_mod, dim, bits, sizes):
    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, dim, sizes, bits, 5 * dim + bits, dup=3)  # equal distances too
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nq = 8 * sms + 1
    pick = torch.randint(0, len(sizes), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k, nprobe in ((1, 1), (4, 2), (5, 4), (20, 4), (20, 5), (129, 1), (300, 1), (256, 4), (257, 4), (1024, 5)):
        ref = o.search(q, k, nprobe, nthreads=8)
        for n in (3, 3 * sms + 1, 6 * sms, 6 * sms + 1, 8 * sms, nq):
            _same(idx.search_batch(q[:n], k, nprobe), (ref[0][:n], ref[1][:n]))
    o.close()
    idx.free()


def test_one_cluster_of_most_blocks(tmp_path, oracle_mod):
    """Over Zipf clusters the wide form for large pools goes by the size of the
    last cluster probed, and large batches of small k by their queries."""
    path = os.path.join(tmp_path, "i.index")
    idx, g, cent = _index(path, 64, [6000, 900, 700, 40, 3], 7, 12)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nq = 24 * sms + 1
    q = idx.rotate((cent[torch.randint(0, 5, (nq,), generator=g)] + 0.7 * torch.randn(nq, 64, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k, nprobe, n in ((257, 1, 9), (257, 2, 9), (257, 3, 9), (300, 4, sms), (10, 1, nq), (64, 5, nq), (65, 2, nq)):
        _same(idx.search_batch(q[:n], k, nprobe), o.search(q[:n], k, nprobe, nthreads=8))
    o.close()
    idx.free()
