"""The work that programs built on this package have it do, as timed cases.

Each case goes through a public entry point (``IVF``, ``Plan``, ``clustering``,
``build_index``, ``learned``) the way a user's program calls it, over the sizes
of the repository's own workloads (bench.py, tests/): 128-d, 768-d and 1536-d
data, 4- to 9-bit indexes, one query to 10,000 queries per call, even and
Zipf-sized clusters, host and device buffers, search, clustering, index
construction and training of the probe model.

An index is what a program loads once and keeps: it depends on the case alone
(its sizes), is built once per process and is shared by the states of the
cases that search it.  Queries, training data and the data that is clustered
or indexed are drawn from the seed.
"""
from __future__ import annotations

import collections
import math
import os
import sys
import tempfile

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "extended-rabitq_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from erq_b200 import IVF, Plan, build_index, clustering, datasets, indexfile, learned  # noqa: E402

# The indexes of the listed search cases (sizes of the repository's workloads;
# the Zipf ones with fewer vectors, so that a process builds them in seconds).
_GAUSS128 = dict(gen="gauss", n=100_000, dim=128, clusters=1024, comps=256, bits=4, zipf=False)
_SPHERE1536 = dict(gen="sphere", n=1_000_000, dim=1536, clusters=4096, comps=4096, bits=8, zipf=False)
_ZIPF1536 = dict(gen="sphere", n=400_000, dim=1536, clusters=2048, comps=2048, bits=7, zipf=True)
_ZIPF768 = dict(gen="gauss", n=600_000, dim=768, clusters=4096, comps=4096, bits=9, zipf=True)


def listed():
    return [
        # an interactive program: one query per call, device buffers; latency and launches
        dict(name="one_query_128", path="search", raw=True, nq=1, k=100, nprobe=32, **_GAUSS128),
        # a program that batches a thousand small queries per call
        dict(name="batch_128", path="search", raw=True, nq=1000, k=100, nprobe=32, **_GAUSS128),
        # the headline workload at its fixed depth: a tuned plan, 10,000 queries per step
        dict(name="plan_1536", path="plan", raw=True, nq=10_000, k=100, nprobe=2, tune=True,
             **_SPHERE1536),
        # the headline workload with the learned probe depth
        dict(name="learned_1536", path="learned", raw=True, nq=10_000, k=100, nprobe=2, tune=True,
             **_SPHERE1536),
        # a high-recall search of already rotated queries without a plan, deep probes
        dict(name="deep_1536", path="search", raw=False, nq=2000, k=100, nprobe=64, **_SPHERE1536),
        # an offline job over very uneven clusters, a batch of no round size
        dict(name="zipf_1536", path="plan", raw=True, nq=2047, k=100, nprobe=96, tune=False,
             **_ZIPF1536),
        # a serving loop: 64 requests at a time, pinned host buffers in and out
        dict(name="serve_64", path="host", raw=True, nq=64, k=10, nprobe=128, **_ZIPF1536),
        # 9-bit codes, small top-k, uneven clusters, an odd batch
        dict(name="zipf_768", path="plan", raw=True, nq=1023, k=10, nprobe=64, tune=False,
             **_ZIPF768),
        # the rotation alone, for a program that searches the same queries at several depths
        dict(name="rotate_1536", path="rotate", nq=10_000, **_SPHERE1536),
        # the clustering that precedes an index
        dict(name="kmeans_128", path="kmeans", gen="gauss", n=200_000, dim=128, comps=256,
             clusters=1024, iters=10, zipf=False),
        # the index construction itself (clusters and rotation given, file out)
        dict(name="build_768", path="build", gen="sphere", n=20_000, dim=768, comps=64, clusters=64,
             bits=8, zipf=False),
        # training of the probe model on labelled features
        dict(name="train_probe", path="train", n=16_384, epochs=2, batch=1024),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: the same paths, sizes over the whole range of the listed ones."""
    path = rng.choice(("search", "search", "search", "plan", "plan", "learned", "host", "rotate",
                       "kmeans", "build", "train"))
    if path == "train":
        return dict(path="train", n=_log_int(rng, 1000, 16_384), epochs=rng.choice((1, 2)),
                    batch=rng.choice((256, 500, 1024)))
    gen = rng.choice(("gauss", "sphere"))
    dim = _log_int(rng, 64, 1536)
    if rng.random() < 0.6:
        dim = max(64, dim // 64 * 64)
    if path == "kmeans":
        n = _log_int(rng, 5000, min(200_000, 60_000_000 // dim))
        k = _log_int(rng, 16, min(1024, n // 40))
        return dict(path="kmeans", gen=gen, n=n, dim=dim, comps=max(16, k // 4), clusters=k,
                    iters=rng.choice((3, 5, 10)), zipf=rng.random() < 0.3)
    bits = rng.choice((3, 4, 5, 7, 8, 9))
    if path == "build":
        dim = min(dim, 768)
        n = _log_int(rng, 500, min(20_000, 15_000_000 // dim))
        k = _log_int(rng, 8, max(8, n // 100))
        return dict(path="build", gen=gen, n=n, dim=dim, comps=k, clusters=k, bits=min(bits, 8), zipf=False)
    n = _log_int(rng, 20_000, min(400_000, 150_000_000 // dim))
    k_c = _log_int(rng, 150, min(4096, n // 40))
    zipf = rng.random() < 0.4
    idx = dict(gen=gen, n=n, dim=dim, clusters=k_c, comps=max(32, k_c // rng.choice((1, 2, 4))),
               bits=bits, zipf=zipf)
    if path == "rotate":
        return dict(path="rotate", nq=_log_int(rng, 1, 10_000), **idx)
    nprobe = _log_int(rng, 1, 128)
    # scanned codes bounded by those of the listed cases
    most = int(4e11 / (nprobe * (n / k_c) * (8 if zipf else 2) * dim))
    nq = _log_int(rng, 1, max(2, min(10_000, most)))
    if path == "host":
        nq = min(nq, 256)
    c = dict(path=path, raw=rng.random() < 0.6, nq=nq, k=rng.choice((1, 10, 37, 100, 100, 200)),
             nprobe=nprobe, **idx)
    if path in ("plan", "learned"):
        c["tune"] = False
    return c


# ------------------------------------------------------------------ inputs
def _centres(case, g, dev):
    c = torch.randn(case["comps"], case["dim"], generator=g, device=dev)
    return c / c.norm(dim=1, keepdim=True) if case["gen"] == "sphere" else c


def _components(case, n, g):
    """The mixture component of n points: even or Zipf(1.1) weights."""
    m = case["comps"]
    if case["zipf"]:
        w = torch.arange(1, m + 1, device="cuda", dtype=torch.float64) ** -1.1
        return torch.multinomial(w, n, replacement=True, generator=g)
    return torch.randint(0, m, (n,), generator=g, device="cuda")


def _points(case, centres, n, g, comp=None):
    """n points of the case's mixture: unit-norm with tangent noise 0.05, or
    Gaussian with sigma 0.3."""
    dev = centres.device
    if comp is None:
        comp = _components(case, n, g)
    out = torch.empty(n, centres.shape[1], device=dev)
    for s in range(0, n, 1 << 17):
        c = centres[comp[s:s + (1 << 17)]]
        z = torch.randn(c.shape, generator=g, device=dev)
        if case["gen"] == "sphere":
            z -= (z * c).sum(1, keepdim=True) * c
            p = c + 0.05 * z
            out[s:s + (1 << 17)] = p / p.norm(dim=1, keepdim=True)
        else:
            out[s:s + (1 << 17)] = c + 0.3 * z
    return out


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


_INDEX_SEED = 20241
_INDEX_KEYS = ("gen", "n", "dim", "clusters", "comps", "bits", "zipf")


def _arrays(case):
    """The case's index in file form, and its mixture's centres."""
    g = _gen(_INDEX_SEED)
    centres = _centres(case, g, "cuda")
    base = _points(case, centres, case["n"], g)
    cent, ids = datasets.kmeans_torch(base, case["clusters"], iters=8, seed=_INDEX_SEED + 1)
    a = build_index.build_index_torch(base, cent, ids, case["bits"], seed=_INDEX_SEED + 2)
    return a, centres


class _Loaded:
    """A loaded index, its mixture's centres and, once asked for, its probe model."""

    def __init__(self, case):
        a, self.centres = _arrays(case)
        with tempfile.TemporaryDirectory(prefix="erq_cases_", dir=_tmp()) as d:
            path = os.path.join(d, "ivf.index")
            indexfile.write_index(path, a)
            self.ivf = IVF(path)
        self.case = {k: case[k] for k in _INDEX_KEYS}
        self.models = {}

    def queries(self, nq, seed):
        return _points(self.case, self.centres, nq, _gen(seed))

    def model(self, k, nprobe):
        """The probe model for this depth, trained on the index's own queries."""
        if (k, nprobe) not in self.models:
            bins = learned.scaled_bins(nprobe, self.ivf.K)
            q = self.queries(8192, _INDEX_SEED + 3)
            rot = self.ivf.rotate(q).cpu().numpy()
            labels = learned.make_labels(self.ivf, rot, k, bins)
            feats = learned.probe_features(self.ivf, rot)
            self.models[k, nprobe] = learned.ProbeModel.train(feats, labels, bins, epochs=6,
                                                              batch=512, seed=_INDEX_SEED + 4)
        return self.models[k, nprobe]


def _tmp():
    """Where index files go: memory where there is a memory file system."""
    return "/dev/shm" if os.access("/dev/shm", os.W_OK) else None


_loaded = collections.OrderedDict()
_MOST_LOADED = 4


def _index(case):
    key = tuple(case[k] for k in _INDEX_KEYS)
    if key not in _loaded:
        while len(_loaded) >= _MOST_LOADED:
            _loaded.popitem(last=False)
        _loaded[key] = _Loaded(case)
    _loaded.move_to_end(key)
    return _loaded[key]


def _train_data(case, seed):
    """Standard features of the probe model (256 sketch dims, then the log of
    the nearest centroid's distance and 63 growing ratios) and labels that
    follow the ratios."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    f = np.empty((n, learned.N_FEATURES), np.float32)
    f[:, :256] = rng.standard_normal((n, 256), np.float32)
    f[:, 256] = np.log(0.3 + 0.5 * rng.random(n))
    f[:, 257:] = np.cumsum(rng.exponential(0.03, (n, 63)), axis=1)
    score = f[:, 264] + 0.1 * f[:, 0] + 0.05 * rng.standard_normal(n)
    cuts = np.quantile(score, np.linspace(0, 1, learned.N_BINS + 1)[1:-1])
    return f, (learned.N_BINS - 1 - np.searchsorted(cuts, score)).astype(np.uint8)


def prepare(case, seed):
    path = case["path"]
    if path == "train":
        f, y = _train_data(case, seed)
        return dict(path=path, features=f, labels=y, epochs=case["epochs"], batch=case["batch"])
    if path in ("kmeans", "build"):
        g = _gen(seed)
        centres = _centres(case, g, "cuda")
        if path == "kmeans":
            return dict(path=path, base=_points(case, centres, case["n"], g),
                        clusters=case["clusters"], iters=case["iters"])
        # the clusters are the mixture's components, of the same uneven sizes for
        # every seed (the file's length depends on them), about their means
        ids = _components(case, case["n"], _gen(_INDEX_SEED))
        base = _points(case, centres, case["n"], g, ids)
        K = case["clusters"]
        cent = torch.zeros(K, case["dim"], dtype=torch.float64, device="cuda").index_add_(0, ids, base.double())
        cent = (cent / torch.bincount(ids, minlength=K).clamp_min(1)[:, None]).float()
        s = dict(path=path, base=base)
        d = tempfile.TemporaryDirectory(prefix="erq_build_", dir=_tmp())
        s.update(centroids=cent, ids=ids.to(torch.int32), bits=case["bits"], dir=d,
                 file=os.path.join(d.name, "built.index"),
                 rotation=build_index.random_rotation((case["dim"] + 63) // 64 * 64, seed % 1000).cuda())
        return s
    loaded = _index(case)
    ivf = loaded.ivf
    q = loaded.queries(case["nq"], seed)
    if path == "rotate":
        return dict(path=path, ivf=ivf, q=q, out=torch.empty(case["nq"], ivf.D, device="cuda"))
    if not case["raw"]:
        q = ivf.rotate(q)
    nq, k = case["nq"], case["k"]
    s = dict(path=path, ivf=ivf, q=q, k=k, nprobe=case["nprobe"], raw=case["raw"],
             ids=torch.empty(nq, k, dtype=torch.int32, device="cuda"),
             dists=torch.empty(nq, k, device="cuda"))
    if path == "search":
        return s
    if path == "learned":
        model = loaded.model(k, case["nprobe"])
        s["plan"] = Plan(ivf, nq, k, case["nprobe"], model=model, raw=case["raw"])
        s["plan"].set_learned(0.005, 0.25)
        s["used"] = torch.empty(nq, dtype=torch.int32, device="cuda")
    else:
        s["plan"] = Plan(ivf, nq, k, case["nprobe"], raw=case["raw"])
    if case.get("tune"):
        s["plan"].autotune(q.cpu().numpy(), reps=2)
    if path == "host":
        for name in ("q", "ids", "dists"):
            s[name] = s[name].cpu().pin_memory()
    return s


# --------------------------------------------------------------------- run
def run(state):
    path = state["path"]
    if path == "train":
        m = learned.ProbeModel.train(state["features"], state["labels"], epochs=state["epochs"],
                                     batch=state["batch"], lr=1e-3, seed=7)
        params, mean, std, _ = m.params()
        m.free()
        return dict(params=params, mean=mean, std=std, loss=m.final_loss)
    if path == "kmeans":
        cent, assign = clustering.kmeans(state["base"], state["clusters"], iters=state["iters"], seed=5)
        return dict(centroids=cent, assign=assign.view(np.int32))
    if path == "build":
        build_index.build_index_gpu(state["base"], state["centroids"], state["ids"], state["bits"],
                                    state["file"], P=state["rotation"])
        return dict(file=np.memmap(state["file"], np.uint8, "r"))
    if path == "rotate":
        return dict(rotated=state["ivf"].rotate(state["q"], out=state["out"]))
    ids, dists = state["ids"], state["dists"]
    if path == "search":
        fn = state["ivf"].search_raw if state["raw"] else state["ivf"].search_batch
        fn(state["q"], state["k"], state["nprobe"], ids=ids, dists=dists)
        return dict(ids=ids, dists=dists)
    if path == "learned":
        state["plan"].search_buffers(state["q"], ids, dists, state["used"])
        return dict(ids=ids, dists=dists, used=state["used"])
    state["plan"].search_buffers(state["q"], ids, dists)
    return dict(ids=ids, dists=dists)


# -------------------------------------------------------------------- work
def work(case):
    path = case["path"]
    if path == "train":
        rows = case["n"] * case["epochs"]
        layers = 320 * 256 + 256 * 256 + 256 * 8
        return dict(bytes=4.0 * 320 * rows, flops=6.0 * rows * layers)
    n, dim, K = case["n"], case["dim"], case["clusters"]
    D = (dim + 63) // 64 * 64
    if path == "kmeans":  # one assignment per iteration and a last one, and the means
        return dict(bytes=4.0 * n * dim * case["iters"],
                    flops=(case["iters"] + 1) * 2.0 * n * dim * K + case["iters"] * 1.0 * n * dim)
    ex = case["bits"] - 1
    if path == "build":  # the rotation, and one step per critical factor of the sweep
        steps = D * 2 ** ex / 4
        return dict(bytes=n * (4.0 * dim + D * (ex + 1) / 8 + 8) + 4.0 * D * D,
                    flops=2.0 * n * D * D + 6.0 * n * steps)
    nq = case["nq"]
    if path == "rotate":
        return dict(bytes=4.0 * (nq * (dim + D) + D * D), flops=2.0 * nq * D * D)
    pairs, k = nq * case["nprobe"], case["k"]
    per = n / K  # vectors of a probed cluster
    seen = min(1.0, pairs / K)  # share of the clusters that are read
    refined = min(3.0 * k * nq, pairs * per)  # candidates that need their exact distance
    flops = 2.0 * nq * K * D + 2.0 * pairs * per * D + 2.0 * refined * D
    if case["raw"]:
        flops += 2.0 * nq * D * D
    byts = (4.0 * nq * (dim if case["raw"] else D) + 8.0 * nq * k + seen * n * (D / 8 + 4) +
            min(refined, n) * (D * ex / 8 + 8) + 4.0 * K * D)
    return dict(bytes=byts, flops=flops)


# ------------------------------------------------------- results in 64 bits
_PERM = (0, 8, 1, 9, 2, 10, 3, 11, 4, 12, 5, 13, 6, 14, 7, 15)


def _sign_bits(codes, D):
    """1-bit codes of FastScan blocks [nb, 4D] uint8 -> [nb * 32, D] (0 or 1)."""
    nb = codes.shape[0]
    c = codes.view(nb, D // 4, 16)
    inv = torch.argsort(torch.tensor(_PERM, device=codes.device))
    nib = torch.cat([(c & 15)[:, :, inv], (c >> 4)[:, :, inv]], 2)  # [nb, D/4, vector]
    nib = nib.permute(0, 2, 1)
    return torch.stack([(nib >> s) & 1 for s in (3, 2, 1, 0)], 3).reshape(nb * 32, D)


def _ex_codes(rows, D, ex):
    """EX-bit codes of file rows [n, D * ex / 8] uint8 -> [n, D] uint8."""
    n = rows.shape[0]
    if ex == 8:
        return rows
    if ex == 4:
        g = rows.view(n, D // 32, 16)
        return torch.stack([g & 15, g >> 4], 2).reshape(n, D)
    g = rows.view(n, D // 64, 8 * ex)
    if ex in (2, 3):
        v = torch.stack([(g[:, :, :16] >> (2 * s)) & 3 for s in range(4)], 2).reshape(n, -1, 64)
        bit, top = 2, g[:, :, 16:]
    else:
        c1, c2, c3 = g[:, :, :16], g[:, :, 16:32], g[:, :, 32:48]
        v = torch.stack([c1 & 63, c2 & 63, ((c1 >> 2) & 48) | (c3 & 15), ((c2 >> 2) & 48) | (c3 >> 4)],
                        2).reshape(n, -1, 64)
        bit, top = 6, g[:, :, 48:]
    if ex in (3, 7):  # bit j of byte m is the top bit of dim 8j + m
        v = v | torch.stack([((top >> j) & 1) << bit for j in range(8)], 2).reshape(n, -1, 64)
    return v.reshape(n, D)


def _estimates(a, q, nprobe, k):
    """The k smallest distance estimates of each rotated query (float64) over
    the vectors of its nprobe nearest clusters."""
    dev, D, nq = q.device, a.D, q.shape[0]
    cent = torch.from_numpy(np.array(a.centroids)).to(dev).double()
    best = torch.full((nq, nprobe, k), math.inf, dtype=torch.float64, device=dev)
    d2 = (q * q).sum(1, keepdim=True) + (cent * cent).sum(1)[None, :] - 2.0 * q @ cent.T
    probe = d2.topk(nprobe, dim=1, largest=False).indices
    del d2
    order = torch.argsort(probe.reshape(-1), stable=True)
    ends = torch.bincount(probe.reshape(-1), minlength=a.K).cumsum(0).tolist()
    fb, fv, sizes = a.first_block(), a.first_vec(), a.sizes.astype(np.int64)
    short = torch.from_numpy(np.array(a.short)).to(dev)
    rows = torch.from_numpy(np.array(a.long_code)).to(dev)
    xip = torch.from_numpy(np.array(a.xipnorm)).to(dev).double()
    scale = float(1 << a.EX)
    for c in range(a.K):
        pairs = order[(ends[c - 1] if c else 0):ends[c]]
        n = int(sizes[c])
        if not len(pairs) or not n:
            continue
        blk = short[int(fb[c]):int(fb[c]) + (n + 31) // 32]
        bits = _sign_bits(blk[:, :4 * D].contiguous(), D)[:n].double()
        on = blk[:, 4 * D:].contiguous().view(torch.float32).reshape(-1)[:n].double()
        code = _ex_codes(rows[int(fv[c]):int(fv[c]) + n], D, a.EX).double()
        for s in range(0, len(pairs), 4096):
            p = pairs[s:s + 4096]
            r = q[p // nprobe] - cent[c]
            y = r.norm(dim=1, keepdim=True)
            u = r / y
            delta = u.abs().amax(1, keepdim=True) / 8191.0
            coarse = (torch.round(u / delta) @ bits.T) * delta
            ip = scale * coarse + u @ code.T - (scale - 0.5) * u.sum(1, keepdim=True)
            est = on[None, :] ** 2 + y * y - xip[int(fv[c]):int(fv[c]) + n][None, :] * y * ip
            m = min(k, n)
            best[p // nprobe, p % nprobe, :m] = est.topk(m, dim=1, largest=False).values
    return best.view(nq, -1).topk(k, dim=1, largest=False).values


def exact(case, seed):
    path = case["path"]
    if path == "rotate":
        loaded = _index(case)
        D = loaded.ivf.D
        q = torch.zeros(case["nq"], D, dtype=torch.float64, device="cuda")
        q[:, :case["dim"]] = loaded.queries(case["nq"], seed).double()
        return dict(rotated=q @ build_index.random_rotation(D, _INDEX_SEED + 2).cuda().double())
    if path not in ("search", "plan", "host"):
        return None  # a trajectory of rounded steps, file bytes, or a depth chosen per query
    a, centres = _arrays(case)
    q = torch.zeros(case["nq"], a.D, dtype=torch.float64, device="cuda")
    q[:, :case["dim"]] = _points(case, centres, case["nq"], _gen(seed)).double()
    q = q @ torch.from_numpy(np.array(a.P)).cuda().double()
    return dict(ids=None, dists=_estimates(a, q, case["nprobe"], case["k"]))
