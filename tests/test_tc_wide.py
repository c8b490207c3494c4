"""The tensor-core form on wide vectors, whose residuals leave the re-rank room for three
warps instead of four: its distances are the exact search's."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("D,segs", [(14080, 4), (14144, 4), (14336, 4), (16384, 1)])
def test_rerank_of_wide_vectors(D, segs):
    from saq_gb300 import ivf
    rng = np.random.default_rng(D)
    n, K = 300, 3
    cids = rng.integers(0, K, n).astype(np.uint32)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.6 * rng.standard_normal((n, D))).astype(np.float32)
    q = (cent[rng.integers(0, K, 5)] + 0.6 * rng.standard_normal((5, D))).astype(np.float32)
    ix = ivf.IVF(n, D, K, ivf.QuantizeConfig(avg_bits=4.0, seg_eqseg=segs, random_rotation=False))
    ix.construct(x, cent, cids)
    ids, d = ix.search_tc(q, n, K, shortlist=n, return_dists=True)  # every vector is re-ranked
    near, near_d = ix.search(q, 10, K, return_dists=True)
    for a, b, c, e in zip(ids, d, near, near_d):
        full = dict(zip(a.tolist(), b.view(np.uint32).tolist()))
        assert len(full) == n and np.all(np.diff(b) >= 0)
        assert [full[i] for i in c.tolist()] == e.view(np.uint32).tolist()
