"""The refinement's three forms by batch size (csrc/refine.cuh: up to a query per
SM, up to three, more) on both sides of each line, against the C oracle, ids and
distance bits equal; pools in registers, in shared memory and never filled,
more probes than a form keeps."""
import os

import pytest

from test_refine_windows import _index, _same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dim,bits", [(64, 3), (320, 5), (960, 8), (1536, 4)])
def test_forms_by_batch_size(tmp_path, oracle_mod, dim, bits):
    path = os.path.join(tmp_path, "i.index")
    sizes = [1 + (37 * i) % 61 for i in range(150)] + [700, 1500, 0, 33]
    idx, g, cent = _index(path, dim, sizes, bits, 7 * dim + bits)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nq = 3 * sms + 1
    pick = torch.randint(0, len(sizes), (nq,), generator=g)
    q = idx.rotate((cent[pick] + 0.7 * torch.randn(nq, dim, generator=g)).numpy())
    o = oracle_mod.Oracle(path)
    for k, nprobe in ((1, 3), (10, 154), (100, 40), (128, 20), (300, 60)):
        ref = o.search(q, k, nprobe, nthreads=8)
        for n in (sms, sms + 1, 3 * sms, nq):
            _same(idx.search_batch(q[:n], k, nprobe), (ref[0][:n], ref[1][:n]))
    o.close()
    idx.free()
