"""The tensor-core form's shortlist and re-rank at their edges: shortlists on both sides
of the few-of-many selection and of its work items, equal approximate distances (the
radix path), one and several segments, an uncoded width and wide ones.  With a
shortlist that holds every candidate the answer is the exact distance's top-k, so a
long shortlist checks a short one's distances bit for bit."""
import numpy as np
import pytest


def _index(D, bits, seg, eqseg, dup):
    from saq_gb300 import ivf
    rng = np.random.default_rng(int(bits) + D)
    K, n = 6, 6 * 900
    cent = rng.standard_normal((K, D)).astype(np.float32)
    cids = rng.integers(0, K, n).astype(np.uint32)
    x = (cent[cids] + 0.5 * rng.standard_normal((n, D))).astype(np.float32)
    if dup:  # many vectors alike: equal distances beyond what the selection collects
        x[: n // 2] = cent[cids[: n // 2]] + 0.25
    ix = ivf.IVF(n, D, K, ivf.QuantizeConfig(avg_bits=bits, enable_segmentation=seg, seg_eqseg=eqseg))
    ix.construct(x, cent, cids, seed=2)
    q = (cent[rng.integers(0, K, 70)] + 0.5 * rng.standard_normal((70, D))).astype(np.float32)
    return ix, q


@pytest.mark.gpu
@pytest.mark.parametrize("dup", [False, True])
@pytest.mark.parametrize("D,bits,seg,eqseg", [(128, 4.0, False, 0), (192, 4.0, True, 3), (128, 1.0, False, 0),
                                              (64, 8.0, False, 0), (256, 10.0, True, 2)])
def test_shortlists_agree(D, bits, seg, eqseg, dup):
    ix, q = _index(D, bits, seg, eqseg, dup)
    full_ids, full_d = ix.search_tc(q, 512, 4, shortlist=1024, return_dists=True)
    dist = [dict(zip(i.tolist(), d.view(np.uint32).tolist())) for i, d in zip(full_ids, full_d)]
    known = matched = 0
    for L in (1, 7, 8, 9, 31, 40, 255, 256, 257, 1000):
        k = min(L, 10)
        ids, d = ix.search_tc(q, k, 4, shortlist=L, return_dists=True)
        assert np.all(np.diff(d, axis=1) >= 0)
        for a, b, m in zip(ids, d.view(np.uint32), dist):
            assert len(set(a.tolist())) == k
            for i, v in zip(a.tolist(), b.tolist()):
                known += 1
                if i in m:
                    matched += 1
                    assert m[i] == v, L
    assert matched > 0.9 * known or dup
