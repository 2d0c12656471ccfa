"""The refinement's pools (csrc/refine.cuh) with distances that are not finite,
which only an index with damaged factors has."""
import os

import numpy as np
import pytest

from test_refine_windows import _index

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _damaged(tmp_path, path, at, value):
    """The index at `path` with the factors of the vectors `at` replaced."""
    from erq_b200 import IVF, indexfile

    a = indexfile.read_index(path)
    a.xipnorm = np.array(a.xipnorm)
    a.xipnorm[at] = value
    out = os.path.join(tmp_path, "damaged.index")
    indexfile.write_index(out, a)
    return IVF(out), out, np.array(a.ids)[at]


def _batches():
    """One per launch form: up to a query per SM, up to three, more."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 9, sms + 1, 3 * sms + 1


@pytest.mark.parametrize("k", [20, 64, 200, 300])
def test_not_a_number_counts_as_infinite(tmp_path, k):
    """Every result is one of the index's ids, none twice, in ascending distance,
    at the distance it has in the sound index; the damaged vectors come only
    where the sound ones run out, at infinity."""
    path = os.path.join(tmp_path, "i.index")
    n = 330
    idx, g, cent = _index(path, 128, [n], 8, 3)
    bad, _, bad_ids = _damaged(tmp_path, path, np.arange(3, n, 5), np.nan)
    for nq in _batches():
        q = idx.rotate((cent[0] + 0.7 * torch.randn(nq, 128, generator=g)).numpy())
        all_ids, all_d = idx.search_batch(q, n, 1)
        ids, d = bad.search_batch(q, k, 1)
        for i in range(nq):
            sound = dict(zip(all_ids[i].tolist(), all_d[i].tolist()))
            assert len(set(ids[i].tolist())) == k, (nq, i)
            assert (np.diff(d[i]) >= 0).all() or np.isinf(d[i][-1])
            for v, x in zip(ids[i].tolist(), d[i].tolist()):
                assert x == (np.inf if v in bad_ids else sound[v]), (nq, i, v)
            assert np.isinf(d[i]).sum() == max(0, k - (n - len(bad_ids))), (nq, i)
    bad.free()
    idx.free()


@pytest.mark.parametrize("k", [55, 70, 80, 90])
def test_infinite_distances_keep_their_order(tmp_path, oracle_mod, k):
    """Infinite distances are ordered like any others - equal ones newest first,
    in the block that fills a pool too - as the C oracle does, bit for bit."""
    path = os.path.join(tmp_path, "i.index")
    sizes = [45, 20, 31]
    idx, g, cent = _index(path, 128, sizes, 8, 4)
    n = sum(sizes)
    # about half of the distances infinite, half of them -infinity
    bad, out, _ = _damaged(tmp_path, path, np.flatnonzero(np.arange(n) % 9), np.float32(-3e38))
    o = oracle_mod.Oracle(out)
    nq = _batches()[-1]
    pick = torch.randint(0, len(sizes), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 2.0 * torch.randn(nq, 128, generator=g)).numpy())
    ref = o.search(q, k, len(sizes), nthreads=8)
    assert np.isinf(ref[1]).any()
    for m in _batches():
        ids, d = bad.search_batch(q[:m], k, len(sizes))
        assert (ids == ref[0][:m]).all(), m
        assert (d.view(np.uint32) == ref[1][:m].view(np.uint32)).all(), m
    o.close()
    bad.free()
    idx.free()
