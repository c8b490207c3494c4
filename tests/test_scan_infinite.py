"""Estimated distances that overflow to minus infinity (an index whose vectors carry huge
rescale factors) take their places in the pool as in the reference: ids and distances
against the oracle, in every scan form and pool size."""
import numpy as np
import pytest

import oracle as O
from saq_gb300 import index_format as F


@pytest.mark.gpu
@pytest.mark.parametrize("D,segs", [(128, 1), (192, 3)])
def test_minus_infinity(D, segs, tmp_path, monkeypatch):
    from saq_gb300 import ivf
    rng = np.random.default_rng(D)
    n, K = 2400, 4
    cids = rng.integers(0, K, n).astype(np.uint32)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.7 * rng.standard_normal((n, D))).astype(np.float32)
    q = (cent[rng.integers(0, K, 30)] + 0.7 * rng.standard_normal((30, D))).astype(np.float32)
    path = str(tmp_path / "i.index")
    O.build_index(path, x, cent, cids, 4.0, segs > 1, segs if segs > 1 else 0, None)
    f = F.load(path)
    for c in f.clusters:
        at = rng.choice(c.num_vec, 3, replace=False)
        c.long_factors[at, rng.integers(0, segs, 3), 0] = 3e38
    F.save(f, path)
    ref, ix = O.OracleIndex(path), ivf.IVF.load(path)
    for k in (2, 10, 40, 100, 200):
        oi, od = ref.search(q, k, K, with_dists=True)
        assert np.isneginf(od).any() and np.isfinite(od[np.isneginf(od).any(1)]).any()
        for mode in ("", "split", "seq", "ws", "warp"):
            if mode:
                monkeypatch.setenv("SAQG_SCAN_MODE", mode)
            else:
                monkeypatch.delenv("SAQG_SCAN_MODE", raising=False)
            for nq in (1, 30):
                ids, d = ix.search(q[:nq], k, K, return_dists=True)
                assert np.array_equal(ids, oi[:nq]), (k, mode, nq)
                assert np.array_equal(d.view(np.uint32), od[:nq].view(np.uint32)), (k, mode, nq)
