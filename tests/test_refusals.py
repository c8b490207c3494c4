"""A call that its sizes make impossible is refused before any of its work is started, so
that nothing still runs on its buffers when the error is returned."""
import numpy as np
import pytest

from saq_gb300 import index_format as F


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["exact", "tc"])
def test_too_wide_for_the_shortlist(form, tmp_path):
    from saq_gb300 import _native as N, ivf
    dim, S, K = 14336, 4, 2
    D = dim * S  # the shortlist keeps a query in shared memory: 220 KB hold 53,248 dimensions
    z = lambda dt: np.zeros(0, dt)
    f = F.IndexFile(0, D, K, np.ones((K, D), np.float32), b"\0" * F.QUANTIZE_CONFIG_BYTES, D, np.ones(D, np.float32),
                    [F.Segment(dim, 1, None, b"\0" * F.QUANT_SINGLE_CONFIG_BYTES) for _ in range(S)])
    f.clusters = [F.Cluster(0, z(np.float32), z(np.uint8), z(np.uint8), np.zeros((0, S, 2), np.float32), z(np.uint32),
                            [np.ones(dim, np.float32)] * S) for _ in range(K)]
    path = str(tmp_path / "w.index")
    F.save(f, path)
    ix = ivf.IVF.load(path)
    q = np.ones((64, D), np.float32)
    before = ix.lib.saqg_kernel_launches()
    with pytest.raises(N.SaqgError, match="shortlist"):
        ix.search(q, 1, 1) if form == "exact" else ix.search_tc(q, 1, 1, shortlist=4)
    assert ix.lib.saqg_kernel_launches() == before
