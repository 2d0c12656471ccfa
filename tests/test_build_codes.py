"""The EX-bit codes of the GPU index builder against a float64 restatement of
fast_quantize (inc/index/Quantizer.hpp:138-219) with a priority queue: every
code byte and xipnorm equal, on vectors whose critical factors tie, vanish,
span many octaves (sums that round) or are absent (a zero residual)."""
import heapq
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _fast_quantize(o, EX):
    o = [float(v) for v in o]
    cap = (1 << EX) - 1
    mx = max(o)
    if mx == 0.0:  # no factor is finite: codes 0, ipnorm 1
        return [0] * len(o), np.float32(1.0)
    t_start, t_end = (cap // 3) / mx, (cap + 10) / mx
    num, den = 0.0, len(o) * 0.25
    cur, heap = [], []
    for i, v in enumerate(o):
        c = int(t_start * v + 1e-5)
        cur.append(c)
        den += c * c + c
        num += (c + 0.5) * v
        heap.append(((c + 1) / v if v else math.inf, i))
    heapq.heapify(heap)
    best, t = 0.0, 0.0
    while heap:
        ct, i = heap[0]
        cur[i] += 1
        den += 2 * cur[i]
        num += o[i]
        ip = num / math.sqrt(den)
        if ip > best:
            best, t = ip, ct
        tn = (cur[i] + 1) / o[i] if o[i] and cur[i] < cap else math.inf
        if tn < t_end:
            heapq.heapreplace(heap, (tn, i))
        else:
            heapq.heappop(heap)
    code = [min(int(t * v + 1e-5), cap) for v in o]
    num2 = 0.0
    for c, v in zip(code, o):
        num2 += (c + 0.5) * v
    return code, np.float32(1.0 / num2)


@pytest.mark.parametrize("dim,bits", [(64, 3), (64, 9), (100, 5), (200, 4), (200, 8), (768, 7), (768, 9),
                                      (1024, 8), (1088, 9), (2048, 5)])
def test_codes_equal_the_sweep(tmp_path, dim, bits):
    from erq_b200 import indexfile
    from erq_b200.build_index import build_index_gpu, pack_ex_codes

    EX, D = bits - 1, (dim + 63) // 64 * 64
    rng = np.random.default_rng(dim + bits)
    x = [rng.standard_normal(dim) for _ in range(6)]
    x.append(rng.integers(-3, 4, dim))                                   # ties
    x.append(np.where(rng.random(dim) < 0.5, 1.0, -1.0))                 # one value
    x.append(np.where(np.arange(dim) == dim // 2, 2.0, 0.0))             # one dim
    x.append(np.where(rng.random(dim) < 0.9, 0.0, rng.standard_normal(dim)))
    x.append(rng.standard_normal(dim) * 10.0 ** rng.uniform(-12, 0, dim))  # rounding sums
    x.append(rng.standard_normal(dim) * 10.0 ** rng.uniform(-36, 0, dim))  # denormals
    x.append(rng.standard_normal(dim) * np.where(np.arange(dim) % 7, 1.0, 1e-6))
    x.append(np.zeros(dim))                                              # no factor
    x = np.stack(x).astype(np.float32)
    n = len(x)
    path = str(tmp_path / "codes.index")
    build_index_gpu(x, np.zeros((1, dim), np.float32), np.zeros(n, np.uint32), bits, path,
                    P=np.eye(D, dtype=np.float32))
    got = indexfile.read_index(path)
    long_code = np.asarray(got.long_code).reshape(n, -1)
    onorm = np.asarray(got.short).reshape(-1)[4 * D:4 * D + 4 * n].copy().view(np.float32)
    for r in range(n):
        xp = np.zeros(D, np.float32)
        xp[:dim] = x[r]
        sq = 0.0
        for v in xp.astype(np.float64):
            sq += v * v
        xn = xp / np.float32(math.sqrt(sq)) if sq > 0 else xp
        code, ipn = _fast_quantize(np.abs(xn), EX)
        code = np.array(code, np.uint8)
        code = np.where(xp > 0, code, ~code & ((1 << EX) - 1)).astype(np.uint8)
        want = pack_ex_codes(torch.from_numpy(code[None]), EX).numpy()[0]
        assert (long_code[r] == want).all(), r
        assert np.float32(got.xipnorm.reshape(-1)[r]) == ipn * np.float32(2) * onorm[r], r
