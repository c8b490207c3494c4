"""Plans of many segments and large k, whose tiles, pools and records fill most of a
CTA's shared memory: one query (split pass), a batch below the deferral line (CTA scan)
and one above it (both), against the oracle, ids and distances bit for bit."""
import numpy as np
import pytest

import oracle as O

SIZES = (6000, 3100, 2000, 950)  # 190, 97, 63 and 30 blocks: nprobe 1 stays below the line of 256 blocks, 4 passes it


@pytest.mark.gpu
@pytest.mark.parametrize("D,segs,k", [(960, 15, 1000), (1024, 16, 10), (1024, 16, 4096), (768, 12, 4096)])
def test_many_segments_and_large_k(D, segs, k, tmp_path):
    from saq_gb300 import ivf
    rng = np.random.default_rng(D + k)
    K = len(SIZES)
    cids = np.repeat(np.arange(K), SIZES).astype(np.uint32)
    rng.shuffle(cids)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.6 * rng.standard_normal((len(cids), D))).astype(np.float32)
    q = (cent[rng.integers(0, K, 20)] + 0.6 * rng.standard_normal((20, D))).astype(np.float32)
    ix = ivf.IVF(len(cids), D, K, ivf.QuantizeConfig(avg_bits=3.0, seg_eqseg=segs))
    ix.construct(x, cent, cids, seed=3)
    assert len(ix.info()["plan"]) == segs
    path = str(tmp_path / "w.index")
    ix.save(path)
    ref = O.OracleIndex(path)
    for nprobe in (1, 4):
        oi, od = ref.search(q, k, nprobe, threads=8, with_dists=True)
        for nq in (1, 20):
            ids, d = ix.search(q[:nq], k, nprobe, return_dists=True)
            assert np.array_equal(ids, oi[:nq]), (nprobe, nq)
            assert np.array_equal(d.view(np.uint32), od[:nq].view(np.uint32)), (nprobe, nq)


@pytest.mark.gpu
@pytest.mark.parametrize("D,segs,k", [(11200, 16, 100), (14080, 7, 512)])
def test_largest_scan(D, segs, k, tmp_path):
    """Shapes whose scan state fills the shared memory that a scan may take."""
    from saq_gb300 import ivf
    rng = np.random.default_rng(D)
    n, K = 700, 3
    cids = rng.integers(0, K, n).astype(np.uint32)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.6 * rng.standard_normal((n, D))).astype(np.float32)
    q = (cent[rng.integers(0, K, 20)] + 0.6 * rng.standard_normal((20, D))).astype(np.float32)
    ix = ivf.IVF(n, D, K, ivf.QuantizeConfig(avg_bits=2.0, seg_eqseg=segs, random_rotation=False))
    ix.construct(x, cent, cids)
    path = str(tmp_path / "l.index")
    ix.save(path)
    oi, od = O.OracleIndex(path).search(q, k, K, threads=8, with_dists=True)
    ids, d = ix.search(q, k, K, return_dists=True)
    assert np.array_equal(ids, oi) and np.array_equal(d.view(np.uint32), od.view(np.uint32))
