"""Every pipeline wait of the tensor-core scan is bounded.  With a limit of one
poll the roles give up, at different points: the search must report
ERQ_ERR_TIMEOUT (its blocks wait for their copies and products, free their tensor
memory and exit), and with the default limit the next one is right again."""
import os

import numpy as np
import pytest

from test_scan_mma import EDGES, _index

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dim,bits,nq", [(64, 4, 1171), (1536, 8, 60)])
def test_wait_limit_reports_timeout_and_recovers(tmp_path, dim, bits, nq):
    from erq_b200 import _lib

    lib = _lib.load_library()
    idx, g, cent = _index(os.path.join(tmp_path, "i.index"), dim, EDGES, bits, dim)
    pick = torch.randint(0, len(EDGES), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    ref = idx.search_batch(q, 20, len(EDGES))
    timeouts = {}
    for polls in (1, 2, 3):  # a poll itself waits a while: more of them may suffice
        _lib.check(lib.erq_debug_set_scan_wait_limit(polls))
        timeouts[polls] = False
        try:
            got = idx.search_batch(q, 20, len(EDGES))
        except _lib.ErqError as e:
            assert "TIMEOUT" in str(e)
            timeouts[polls] = True
        finally:
            _lib.check(lib.erq_debug_set_scan_wait_limit(0))
        if timeouts[polls]:
            got = idx.search_batch(q, 20, len(EDGES))
        assert (got[0] == ref[0]).all()
        assert (got[1].view(np.uint32) == ref[1].view(np.uint32)).all()
    assert timeouts[1], timeouts
    idx.free()
