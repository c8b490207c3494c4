"""Query rotation and prune bounds at the edges of their kernels (saq_gb300/csrc
rotate.cuh, k_qprep_few, k_qprep_tiled): one query to over a tile of them, one chain
(64 dimensions) and block chains, queries that are not 16-byte aligned, and rows of an
index build on both sides of a tile.  Everything downstream is bit-exact, so ids and
distances equal to the oracle's show it."""
import numpy as np
import pytest

import oracle as O
from saq_gb300 import data
from test_configs import _same_index


def _index(tmp_path, n, D, k, bits, seg, n_query):
    from saq_gb300 import ivf
    x, q = data.anisotropic(n, D, 0.8, seed=D + k, n_query=n_query)
    rng = np.random.default_rng(3)
    cent = x[rng.choice(n, k, replace=False)].copy()
    cids = data.assign_nearest(x, cent)
    var = x.var(axis=0).astype(np.float32)
    plan = ivf.plan(var, bits, seg)
    rots = np.concatenate([data.random_orthogonal(d, rng).astype(np.float32).reshape(-1) for d, _ in plan])
    ix = ivf.IVF(n, D, k, ivf.QuantizeConfig(avg_bits=bits, enable_segmentation=seg))
    ix.set_variance(var)
    ix.construct(x, cent, cids, rotations=rots)
    path = str(tmp_path / "i.index")
    ix.save(path)
    ref = str(tmp_path / "o.index")
    O.build_index(ref, x, cent, cids, bits, seg, 0, rots, variance=var)
    _same_index(path, ref)  # centroids are vectors here: their error factor is a NaN of the host's sign
    return ix, O.OracleIndex(ref), q


@pytest.mark.gpu
@pytest.mark.parametrize("n,D,k,seg", [(129, 64, 5, False), (300, 128, 131, False), (2001, 640, 20, False),
                                       (2001, 1024, 20, True)])
def test_rotated_queries_equal_oracle(tmp_path, n, D, k, seg):
    import torch
    ix, ref, q = _index(tmp_path, n, D, k, 4.0, seg, 1030)
    oi, od = ref.search(q, 5, 4, with_dists=True)
    buf = torch.empty(q.size + 4, device="cuda")
    for nq in (1, 7, 8, 9, 16, 129, 1030):
        for shift in (0, 1):
            t = buf[shift:shift + nq * D].view(nq, D)
            t.copy_(torch.from_numpy(q[:nq]))
            ids, d = ix.search(t, 5, 4, return_dists=True)
            assert np.array_equal(ids.cpu().numpy().view(np.uint32), oi[:nq]), (nq, shift)
            assert np.array_equal(d.cpu().numpy().view(np.uint32), od[:nq].view(np.uint32)), (nq, shift)
