"""IVF.estimate where its tiles have their edges: clusters of one tile of 16 blocks, one
vector more or less, many tiles, and none; one and several segments.  Ids and the
three distances equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O

SIZES = (0, 1, 31, 33, 511, 512, 513, 1025, 4200)


@pytest.mark.gpu
@pytest.mark.parametrize("seg,eqseg,bits", [(False, 0, 4.0), (True, 2, 3.0), (False, 0, 1.0)])
def test_estimate_at_tile_edges(seg, eqseg, bits, tmp_path):
    from saq_gb300 import ivf
    rng = np.random.default_rng(5)
    D, K = 192, len(SIZES)
    cids = np.repeat(np.arange(K), SIZES)
    rng.shuffle(cids)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.5 * rng.standard_normal((len(cids), D))).astype(np.float32)
    path = str(tmp_path / "e.index")
    O.build_index(path, x, cent, cids.astype(np.uint32), bits, seg, eqseg, None)
    ref, ix = O.OracleIndex(path), ivf.IVF.load(path)
    for nprobe in (1, 4, K):
        for q in x[:3]:
            for got, want in zip(ix.estimate(q, nprobe), ref.estimate(q, nprobe)):
                assert np.array_equal(np.asarray(got).view(np.uint32), np.asarray(want).view(np.uint32)), nprobe
