"""Which candidates the tensor-core form's shortlist keeps: with one cluster probed and a
shortlist of 1,024 (the radix selection) every approximate distance that can matter is
known, and a shorter shortlist has to hold exactly the smallest of them, equal ones in
scan order, and to return them by exact distance, the later-scanned of equal ones first."""
import numpy as np
import pytest

SIZES = (900, 6000, 4097)  # within 1,024; two selection chunks; one vector into the second


def _index(dup):
    from saq_gb300 import ivf
    rng = np.random.default_rng(5)
    D, K = 128, len(SIZES)
    cids = np.repeat(np.arange(K), SIZES).astype(np.uint32)
    rng.shuffle(cids)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.5 * rng.standard_normal((len(cids), D))).astype(np.float32)
    if dup:  # many vectors alike, so that equal keys pass what the selection collects
        like = rng.random(len(x)) < 0.5
        x[like] = cent[cids[like]] + 0.05
    ix = ivf.IVF(len(x), D, K, ivf.QuantizeConfig(avg_bits=4.0, enable_segmentation=False))
    ix.construct(x, cent, cids, seed=2)
    q = (cent[rng.integers(0, K, 70)] + 0.5 * rng.standard_normal((70, D))).astype(np.float32)
    return ix, q


@pytest.mark.gpu
@pytest.mark.parametrize("dup", [False, True])
def test_shortlist_holds_the_smallest(dup):
    ix, q = _index(dup)
    ids, d, apx = ix.search_tc(q, 1024, 1, shortlist=1024, return_dists=True, return_approx=True)
    for L in (1, 7, 8, 9, 40, 128, 200, 255, 256, 257, 512):
        got, gd = ix.search_tc(q, L, 1, shortlist=L, return_dists=True)
        for a, b, i, e, v in zip(got, gd, ids, d, apx):
            some = e < np.finfo(np.float32).max  # fewer than 1,024 vectors: the rest is padding
            i, e, v = i[some], e[some], v[some]
            keep = np.lexsort((i, v))[:L]  # ids ascend in a cluster's scan order
            order = keep[np.lexsort((-i[keep].astype(np.int64), e[keep]))]
            assert np.array_equal(a, i[order]), L
            assert np.array_equal(b.view(np.uint32), e[order].view(np.uint32)), L


@pytest.mark.gpu
def test_longest_collected_shortlist_is_not_slower_than_the_radix_one():
    """At 256 entries, the longest that the selection collects under a bound, the bound has
    to keep what is collected well below its limit: over it the collection is lost work and
    the radix selection follows (1.6 times the time of 264 entries then, less than it now)."""
    import torch
    from saq_gb300 import ivf
    rng = np.random.default_rng(1)
    n, D, K, nq = 50000, 64, 8, 512
    cids = rng.integers(0, K, n).astype(np.uint32)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + rng.standard_normal((n, D))).astype(np.float32)
    ix = ivf.IVF(n, D, K, ivf.QuantizeConfig(avg_bits=2.0, enable_segmentation=False))
    ix.construct(x, cent, cids, seed=2)
    q = torch.from_numpy((cent[rng.integers(0, K, nq)] + rng.standard_normal((nq, D))).astype(np.float32)).cuda()
    ms = {L: min(ix.search_tc(q, 10, K, shortlist=L, stats=True)[-1]["ms_select"] for _ in range(8)) for L in (256, 264)}
    assert ms[256] < 1.2 * ms[264], ms
