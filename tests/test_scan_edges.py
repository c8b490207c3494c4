"""The exact scan against the oracle, ids and distances bit for bit, where its tiles,
filters and pools have their edges: every ex-code width (half-warp and one-thread
products), one to seven segments (the stage-0 filter, sums held in registers up to
four), clusters around a block, a group of four blocks, a pass of 128 blocks and more,
k around the rows of the register pool, tied distances, and each scan form."""
import numpy as np
import pytest

import oracle as O

SIZES = (0, 1, 31, 32, 33, 127, 129, 511, 4200, 64, 300)  # 4,200 vectors: 132 blocks


def _clustered(D, seed, grid=False):
    rng = np.random.default_rng(seed)
    K = len(SIZES)
    cids = np.repeat(np.arange(K), SIZES)
    rng.shuffle(cids)
    scale = (np.arange(1, D + 1) ** -0.5).astype(np.float32)
    if grid:
        cent = np.zeros((K, D), np.float32)
        cent[:, 0] = np.arange(K) - 5
        x = cent[cids] + rng.integers(-2, 3, (len(cids), D)).astype(np.float32)
        q = x[rng.choice(len(x), 40)] + rng.integers(-1, 2, (40, D)).astype(np.float32)
    else:
        cent = (rng.standard_normal((K, D)) * scale).astype(np.float32)
        x = (cent[cids] + 0.7 * rng.standard_normal((len(cids), D)) * scale).astype(np.float32)
        q = (cent[rng.integers(0, K, 40)] + 0.7 * rng.standard_normal((40, D)) * scale).astype(np.float32)
    return x, cent, cids.astype(np.uint32), q.astype(np.float32)


def _check(tmp_path, monkeypatch, D, bits, seg, eqseg, ks, grid=False, modes=("", "split", "seq", "ws")):
    from saq_gb300 import ivf
    x, cent, cids, q = _clustered(D, int(bits * 10) + eqseg, grid)
    path = str(tmp_path / "e.index")
    O.build_index(path, x, cent, cids, bits, seg, eqseg, None)
    ref, ix = O.OracleIndex(path), ivf.IVF.load(path)
    for k in ks:
        oi, od = ref.search(q, k, 9, with_dists=True)
        for mode in modes:
            if mode:
                monkeypatch.setenv("SAQG_SCAN_MODE", mode)
            else:
                monkeypatch.delenv("SAQG_SCAN_MODE", raising=False)
            for nq in (2, 40):
                ids, d = ix.search(q[:nq], k, 9, return_dists=True)
                assert np.array_equal(ids, oi[:nq]), (k, mode, nq)
                assert np.array_equal(d.view(np.uint32), od[:nq].view(np.uint32)), (k, mode, nq)
        monkeypatch.setenv("SAQG_DEFER_BLOCKS", "40")  # part of the batch on the split pass
        monkeypatch.delenv("SAQG_SCAN_MODE", raising=False)
        ids, d = ix.search(q, k, 9, return_dists=True)
        assert np.array_equal(ids, oi) and np.array_equal(d.view(np.uint32), od.view(np.uint32)), (k, "deferred")
        monkeypatch.delenv("SAQG_DEFER_BLOCKS")


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 13])
def test_one_segment_every_width(bits, tmp_path, monkeypatch):
    _check(tmp_path, monkeypatch, 192, float(bits), False, 0, (10,))


@pytest.mark.gpu
@pytest.mark.parametrize("D,eqseg", [(128, 2), (192, 3), (256, 4), (320, 5), (448, 7)])
def test_segments(D, eqseg, tmp_path, monkeypatch):
    _check(tmp_path, monkeypatch, D, 4.0, True, eqseg, (1, 10))


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 64, 127, 128, 129, 400])
def test_pool_sizes(k, tmp_path, monkeypatch):
    _check(tmp_path, monkeypatch, 128, 3.0, True, 2, (k,))


@pytest.mark.gpu
@pytest.mark.parametrize("seg,eqseg", [(False, 0), (True, 2), (True, 3)])
def test_tied_distances(seg, eqseg, tmp_path, monkeypatch):
    _check(tmp_path, monkeypatch, 192, 4.0, seg, eqseg, (3, 10, 40), grid=True)
