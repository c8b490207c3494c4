"""The work a user has this library do, as cases that can be timed.

A case is a dict of plain values; `path` says which entry point it calls:

  search     IVF.search: `nq` queries of one call, uniform (`nprobe`, `topk`) or
             uneven (each query's own nprobe and k), device or host buffers
  search_tc  IVF.search_tc: the batched tensor-core form
  estimate   IVF.estimate over every vector of the index (all clusters probed)
  construct  IVF.construct of a new index, read back whole through IVF.estimate
             over all of its clusters
  encode     caq_encode: residual vectors to codes and factors

An index is described by n, dim, clusters, bits, seg and data.  The data are
drawn in the coordinates PCA leaves (axes by descending variance):

  zipf       unit-norm vectors, cluster sizes by Zipf(1.1), centres with
             spectrum i^-0.8, offsets with spectrum i^-1.6 (scale 0.2)
  mixture    Gaussian mixture, centres N(0, 1), offsets N(0, 0.5^2)
  aniso      unit-norm vectors with spectrum i^-0.8 and no cluster structure,
             one k-means step from sampled centroids

A program that searches keeps one index and gets ever new queries, so an index
is built once per description and kept while cases of that description follow
one another; the queries come from the seed.  construct and encode take
everything from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from saq_gb300 import ivf as saq

FLT_MAX = float(np.finfo(np.float32).max)
CHUNK = 1 << 18

# 100,000 x 960 mixture and 1,000,000 x 1024 without clusters: the plain
# single-query configurations; 10,000,000 x 1024 with Zipf clusters: the batched
# one; 1,000,000 x 1536 at 6 and 8 bits: the precision one.
MIX100K = dict(n=100_000, dim=960, clusters=1024, bits=4.0, seg=True, data="mixture")
ANISO1M = dict(n=1_000_000, dim=1024, clusters=4096, bits=4.0, seg=True, data="aniso")
ZIPF10M = dict(n=10_000_000, dim=1024, clusters=16384, bits=4.0, seg=True, data="zipf")
WIDE1M = dict(n=1_000_000, dim=1536, clusters=4096, bits=6.0, seg=False, data="aniso")


def listed():
    return [
        # one query per call from host memory: the drop-in for a program that
        # calls the reference's search; the smallest call
        dict(name="single query, host", path="search", **MIX100K, nq=1, nprobe=32, topk=10, uneven=False, host=True),
        # the estimator over a whole index: an accuracy run's step
        dict(name="estimate, 100k", path="estimate", **MIX100K),
        # one query per call, the query already on the GPU
        dict(name="single query, device", path="search", **ANISO1M, nq=1, nprobe=64, topk=10, uneven=False, host=False),
        # what a small service gathers in a moment: an odd number of queries, k 100
        dict(name="37 queries, k 100", path="search", **ANISO1M, nq=37, nprobe=128, topk=100, uneven=False,
             host=False),
        # the smaller of the precision configuration's batches, exact form
        dict(name="256 queries, 1536-d", path="search", **WIDE1M, nq=256, nprobe=32, topk=10, uneven=False, host=False),
        # the larger one in the tensor-core form, codes of 6 bits
        dict(name="tensor-core, 2048 queries", path="search_tc", **WIDE1M, nq=2048, nprobe=32, topk=10, shortlist=40),
        # the headline: a batch of 4,096 over ten million vectors
        dict(name="batch 4096, 10M", path="search", **ZIPF10M, nq=4096, nprobe=16, topk=10, uneven=False, host=False),
        # a serving loop's batch: nprobe 16-256 and k 10 or 100 mixed; the largest call
        dict(name="uneven batch, 10M", path="search", **ZIPF10M, nq=4096, nprobe=256, topk=100, uneven=True,
             host=False),
        # the headline batch in the tensor-core form
        dict(name="tensor-core, 10M", path="search_tc", **ZIPF10M, nq=4096, nprobe=16, topk=10, shortlist=40),
        # index builds: segmented with the variance at hand, and one segment
        # with the variance left to the library (an odd number of vectors)
        dict(name="build 100k x 960", path="construct", **MIX100K, variance=True),
        dict(name="build 250k x 1024, no seg", path="construct", n=250_007, dim=1024, clusters=1024, bits=4.0,
             seg=False, data="zipf", variance=False),
        # the encoder alone, from and to host memory
        dict(name="encode 8191 x 960, host", path="encode", n=8191, dim=960, bits=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_index(rng, n_max, dim_max=1536):
    n = _log_int(rng, 50_000, n_max)
    clusters = min(16384, max(64, int(n / rng.uniform(80, 640))))
    data = rng.choice(["zipf", "mixture", "aniso"] if n <= 1_000_000 else ["zipf"])
    return dict(n=n, dim=64 * rng.randint(2, dim_max // 64), clusters=clusters,
                bits=rng.choice([1.5, 2.0, 3.0, 4.0, 5.0, 6.0, 8.0]), seg=rng.random() < 0.6, data=data)


def draw(rng):
    """One more case: indexes from 50,000 vectors to the 10 million of the
    batched configuration (1,024 dimensions there), calls of 1 to 4,096 queries."""
    path = rng.choice(["search"] * 5 + ["search_tc", "estimate", "construct", "construct", "encode"])
    if path == "encode":
        return dict(path=path, n=_log_int(rng, 500, 16_000), dim=64 * rng.randint(1, 16), bits=rng.randint(1, 9))
    if path == "construct":
        c = dict(path=path, **_draw_index(rng, 250_000, 1024))
        c["variance"] = c["seg"]
        return c
    if path == "estimate":
        return dict(path=path, **_draw_index(rng, 400_000, 1024))
    c = dict(path=path, **_draw_index(rng, 10_000_000 if rng.random() < 0.3 else 1_000_000))
    if c["n"] > 2_000_000:
        c.update(dim=1024, bits=4.0)
    nq = _log_int(rng, 1, 4096)
    nprobe = min(c["clusters"], _log_int(rng, 4, 256))
    topk = rng.choice([1, 10, 10, 33, 100])
    if path == "search_tc":
        return dict(c, seg=False, nq=max(16, nq), nprobe=min(64, nprobe), topk=topk, shortlist=4 * topk)
    host = rng.random() < 0.3
    uneven = nq >= 8 and rng.random() < 0.3
    return dict(c, nq=nq, nprobe=min(nprobe, max(4, 500_000 // nq)), topk=topk, uneven=uneven, host=host)


# ---------------------------------------------------------------- data
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _spectrum(dim, alpha):
    return torch.arange(1, dim + 1, device="cuda", dtype=torch.float64).pow(-alpha / 2).float()


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


class _Source:
    """Draws base vectors with their cluster ids, then queries, of a description."""

    def __init__(self, case, seed):
        torch.backends.cuda.matmul.allow_tf32 = False
        self.case, self.g = case, _generator(seed)
        k, d, self.kind = case["clusters"], case["dim"], case["data"]
        self.centroids = None
        if self.kind == "zipf":
            self.scale = _spectrum(d, 1.6)
            self.scale = self.scale * (0.2 * _spectrum(d, 0.8).norm() / self.scale.norm())
            self.centroids = _unit(torch.randn(k, d, generator=self.g, device="cuda") * _spectrum(d, 0.8))
        elif self.kind == "mixture":
            self.scale = torch.full((d,), 0.5, device="cuda")
            self.centroids = torch.randn(k, d, generator=self.g, device="cuda")
        else:
            self.scale = _spectrum(d, 0.8)

    def _rows(self, labels, m, g):
        d = self.case["dim"]
        out = torch.empty(m, d, device="cuda")
        for a in range(0, m, CHUNK):
            b = min(m, a + CHUNK)
            v = torch.randn(b - a, d, generator=g, device="cuda").mul_(self.scale)
            if labels is not None:
                v += self.centroids[labels[a:b]]
            out[a:b] = v if self.kind == "mixture" else _unit(v)
        return out

    def _nearest(self, x):
        cn = (self.centroids * self.centroids).sum(1)
        near = torch.empty(x.shape[0], dtype=torch.int64, device="cuda")
        for a in range(0, x.shape[0], CHUNK):
            near[a:a + CHUNK] = torch.argmin(cn[None, :] - 2.0 * (x[a:a + CHUNK] @ self.centroids.T), dim=1)
        return near

    def base(self):
        n, k = self.case["n"], self.case["clusters"]
        if self.kind == "aniso":
            x = self._rows(None, n, self.g)
            self.centroids = x[torch.randperm(n, generator=self.g, device="cuda")[:k]].clone()
            near = self._nearest(x)
            sums = torch.zeros(k, x.shape[1], dtype=torch.float64, device="cuda")
            for a in range(0, n, CHUNK):
                sums.index_add_(0, near[a:a + CHUNK], x[a:a + CHUNK].double())
            count = torch.bincount(near, minlength=k)
            # sums that the order of atomics cannot change any more
            self.centroids = (sums / count[:, None].clamp(min=1)).float().mul(4096).round().div(4096)
            return x, self._nearest(x)
        if self.kind == "zipf":
            w = torch.arange(1, k + 1, dtype=torch.float64).pow(-1.1)
            sizes = (w / w.sum() * n).floor().long()
            sizes[: n - int(sizes.sum())] += 1
            labels = torch.repeat_interleave(torch.arange(k, device="cuda"), sizes.cuda())
            labels = labels[torch.randperm(n, generator=self.g, device="cuda")]
        else:
            labels = torch.randint(0, k, (n,), generator=self.g, device="cuda")
        return self._rows(labels, n, self.g), labels

    def queries(self, nq, seed):
        """Queries of the base's distribution, the clusters of a clustered base taken evenly."""
        g = _generator(1_000_003 + seed)
        labels = None
        if self.kind != "aniso":
            labels = torch.randint(0, self.case["clusters"], (nq,), generator=g, device="cuda")
        return self._rows(labels, nq, g)


def _variance(x):
    s = torch.zeros(x.shape[1], dtype=torch.float64, device="cuda")
    s2 = torch.zeros_like(s)
    for a in range(0, x.shape[0], CHUNK):
        b = x[a:a + CHUNK].double()
        s += b.sum(0)
        s2 += (b * b).sum(0)
    mean = s / x.shape[0]
    return (s2 / x.shape[0] - mean * mean).float().cpu().numpy()


def _rotations(plan, seed):
    """A random orthogonal matrix per segment, concatenated, as a program hands them over."""
    g, mats = _generator(seed), []
    for dim, _ in plan:
        q, r = torch.linalg.qr(torch.randn(dim, dim, generator=g, device="cuda", dtype=torch.float64))
        mats.append((q * torch.sign(torch.diagonal(r))).float().reshape(-1))
    return torch.cat(mats).cpu().numpy()


def _config(case):
    return saq.QuantizeConfig(avg_bits=float(case["bits"]), enable_segmentation=bool(case["seg"]))


def _build_inputs(case, seed):
    src = _Source(case, seed)
    x, labels = src.base()
    variance = _variance(x)
    plan = saq.plan_gpu(variance, float(case["bits"]), bool(case["seg"]))
    return src, dict(x=x, cent=src.centroids.cpu().numpy(), cids=labels.to(torch.int32).cpu().numpy().view(np.uint32),
                     variance=variance, rotations=_rotations(plan, seed + 1))


def _build(case, b, variance=True):
    index = saq.IVF(case["n"], case["dim"], case["clusters"], _config(case))
    if variance:
        index.set_variance(b["variance"])
    index.construct(b["x"], b["cent"], b["cids"], rotations=b["rotations"])
    return index


_kept = {}  # the index of the latest description: {description: (index, source)}


def _index(case):
    key = tuple(case[k] for k in ("n", "dim", "clusters", "bits", "seg", "data"))
    if key not in _kept:
        _kept.clear()
        torch.cuda.empty_cache()
        src, b = _build_inputs(case, 7)
        index = _build(case, b)
        del b
        torch.cuda.empty_cache()
        _kept[key] = (index, src)
    return _kept[key]


def _shapes(case, seed):
    """Per-query nprobe in [16, nprobe] and k in {10, topk} of an uneven batch."""
    r = np.random.default_rng(seed)
    nps = r.integers(min(16, case["nprobe"]), case["nprobe"] + 1, case["nq"])
    ks = np.where(r.random(case["nq"]) < 0.5, min(10, case["topk"]), case["topk"])
    nps[0], ks[0] = case["nprobe"], case["topk"]
    return nps.astype(np.int32), ks.astype(np.int32)


# ---------------------------------------------------------------- the cases
def prepare(case, seed):
    state = dict(case=case)
    path = case["path"]
    if path == "encode":
        g = _generator(seed)
        # rotated residuals of a cluster: near-Gaussian, and the centroid they are taken from
        state["resid"] = (0.2 * torch.randn(case["n"], case["dim"], generator=g, device="cuda")).cpu().numpy()
        state["centroid"] = torch.randn(case["dim"], generator=g, device="cuda").cpu().numpy()
    elif path == "construct":
        src, state["inputs"] = _build_inputs(case, seed)
        state["query"] = src.queries(1, seed)[0].cpu().numpy()
    else:
        state["index"], src = _index(case)
        nq = case.get("nq", 1)
        q = src.queries(nq, seed)
        if path == "estimate":
            q = q[0].cpu().numpy()
        elif case.get("host"):
            q = (q[0] if nq == 1 else q).cpu().numpy()
        state["query"] = q
        state["nprobe"], state["topk"] = case.get("nprobe"), case.get("topk")
        if case.get("uneven"):
            state["nprobe"], state["topk"] = _shapes(case, seed)
    return state


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "search":
        return state["index"].search(state["query"], state["topk"], state["nprobe"], return_dists=True)
    if path == "search_tc":
        return state["index"].search_tc(state["query"], state["topk"], state["nprobe"], shortlist=case["shortlist"],
                                        return_dists=True, return_approx=True)
    if path == "estimate":
        return state["index"].estimate(state["query"], case["clusters"])
    if path == "construct":
        index = _build(case, state["inputs"], case["variance"])
        return index.estimate(state["query"], case["clusters"])
    return saq.caq_encode(state["resid"], case["bits"], state["centroid"])


def work(case):
    """Bytes: queries in, the centroids and the codes and norms of the probed
    vectors once, results out.  Operations: ranking and rotation products, and a
    lookup and an add per four dimensions of a scanned vector (two per dimension
    for every form that computes whole inner products)."""
    d, path = case["dim"], case["path"]
    if path == "encode":
        return dict(bytes=case["n"] * (8 * d + 16), flops=10 * case["n"] * d)
    n, k = case["n"], case["clusters"]
    code = d * float(case["bits"]) / 8
    rotation = 2 * d * d if not case["seg"] else d * d // 2
    if path == "construct":
        return dict(bytes=n * (4 * d + code + 20) + 4 * k * d, flops=n * (rotation + 10 * d))
    nq, nprobe = case.get("nq", 1), case.get("nprobe", k)
    if case.get("uneven"):
        nprobe = (16 + nprobe) / 2
    scanned = nq * nprobe * n / k
    distinct = min(n, scanned)
    per_vec = d / 8 + 8 if path == "search" else code + 8
    out = 16 * distinct if path == "estimate" else 8 * nq * case["topk"]
    per_scan = d / 2 if path == "search" else 2 * d
    return dict(bytes=4 * nq * d + 4 * k * d + distinct * per_vec + out,
                flops=nq * (2 * k * d + rotation) + scanned * per_scan)


# ---------------------------------------------------------------- 64 bits
def _nearest64(x, q, k):
    """Squared distances to the k nearest rows of x, ascending (FP32 shortlist, FP64 distances)."""
    short = min(x.shape[0], k + 64)
    best_d, best_i = None, None
    for a in range(0, x.shape[0], CHUNK):
        xb = x[a:a + CHUNK]
        v, i = torch.topk((xb * xb).sum(1)[None, :] - 2.0 * (q @ xb.T), min(short, xb.shape[0]), dim=1, largest=False)
        i += a
        if best_d is not None:
            v, i = torch.cat([best_d, v], 1), torch.cat([best_i, i], 1)
        o = torch.topk(v, min(short, v.shape[1]), dim=1, largest=False).indices
        best_d, best_i = torch.gather(v, 1, o), torch.gather(i, 1, o)
    out = torch.empty(q.shape[0], k, dtype=torch.float64, device="cuda")
    for a in range(0, q.shape[0], 256):
        diff = x[best_i[a:a + 256]].double() - q[a:a + 256, None, :].double()
        out[a:a + 256] = (diff * diff).sum(-1).sort(dim=1).values[:, :k]
    return out


def _all64(x, labels, cent, q):
    """Squared distances to every vector, nearest cluster first, ids ascending within a cluster."""
    q = q.double()
    rank = torch.argsort(torch.argsort(((cent.double() - q) ** 2).sum(1)))
    rows = torch.argsort(rank[labels], stable=True)
    return torch.cat([((x[rows[a:a + CHUNK]].double() - q) ** 2).sum(1) for a in range(0, rows.numel(), CHUNK)])


def exact(case, seed):
    """What the estimated distances stand for: the true squared distances, to the
    nearest vectors (search) or to each listed vector (estimate, construct).  Ids
    and codes are the quantizer's own and have no such value."""
    path = case["path"]
    if path == "encode":
        return None
    src = _Source(case, seed if path == "construct" else 7)
    x, labels = src.base()
    q = src.queries(case.get("nq", 1), seed)
    if path in ("estimate", "construct"):
        return None, _all64(x, labels, src.centroids, q[0]), None, None
    if path == "search" and not case["seg"] and case["data"] == "zipf":
        return None  # one segment prunes by its 1-bit estimate: among tight clusters the true nearest may be passed over
    d = _nearest64(x, q, case["topk"])
    if case.get("uneven"):
        ks = torch.from_numpy(_shapes(case, seed)[1]).cuda()
        d[torch.arange(case["topk"], device="cuda")[None, :] >= ks[:, None]] = FLT_MAX
    if path == "search_tc":
        return None, d, d
    return None, (d[0] if case["host"] and case["nq"] == 1 else d)
