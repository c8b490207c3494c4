"""The split pass's records on a device short of memory: a call takes what the device
gives, down to nothing, and its answers stay the oracle's; a later call keeps the smaller
space or takes more once there is more, and a captured graph replays what it was given.
Allocations beyond SAQG_TEST_ALLOC_BYTES fail as cudaMalloc on a full device does."""
import ctypes as C

import numpy as np
import pytest

import oracle as O


@pytest.fixture(scope="module")
def problem(tmp_path_factory):
    rng = np.random.default_rng(8)
    n, D, K = 24000, 128, 8
    cids = rng.integers(0, K, n).astype(np.uint32)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.8 * rng.standard_normal((n, D))).astype(np.float32)
    q = (cent[rng.integers(0, K, 40)] + 0.8 * rng.standard_normal((40, D))).astype(np.float32)
    path = str(tmp_path_factory.mktemp("rec") / "r.index")
    O.build_index(path, x, cent, cids, 4.0, True, 2, None)
    oi, od = O.OracleIndex(path).search(q, 10, K, threads=8, with_dists=True)
    return path, q, K, oi, od


def _check(ix, problem, nq):
    _, q, K, oi, od = problem
    ids, d = ix.search(q[:nq], 10, K, return_dists=True)
    assert np.array_equal(ids, oi[:nq]) and np.array_equal(d.view(np.uint32), od[:nq].view(np.uint32))


# 17 MB of records wanted by 40 queries (750 blocks each), 0.43 MB by one
@pytest.mark.gpu
@pytest.mark.parametrize("nq,room", [(40, 8 << 20), (40, 2 << 20), (40, 300_000), (1, 300_000), (1, 100_000)])
def test_less_room_same_answers(problem, nq, room, monkeypatch):
    from saq_gb300 import ivf
    ix = ivf.IVF.load(problem[0])
    monkeypatch.setenv("SAQG_TEST_ALLOC_BYTES", str(room))
    for _ in range(3):
        _check(ix, problem, nq)
    monkeypatch.delenv("SAQG_TEST_ALLOC_BYTES")
    for _ in range(2):
        _check(ix, problem, nq)
    _check(ix, problem, 40)


@pytest.mark.gpu
def test_no_room_at_all_is_an_error(problem, monkeypatch):
    from saq_gb300 import _native as N, ivf
    ix = ivf.IVF.load(problem[0])
    monkeypatch.setenv("SAQG_TEST_ALLOC_BYTES", "1000")
    with pytest.raises(N.SaqgError, match="cudaMalloc"):
        ix.search(problem[1], 10, problem[2])
    monkeypatch.delenv("SAQG_TEST_ALLOC_BYTES")
    _check(ix, problem, 40)


@pytest.mark.gpu
def test_graph_with_less_room(problem, monkeypatch):
    import torch
    from saq_gb300 import _native as N, ivf
    path, q, K, oi, od = problem
    ix = ivf.IVF.load(path)
    qd = torch.from_numpy(q).cuda()
    ids = torch.zeros((40, 10), dtype=torch.int32, device="cuda")
    d = torch.zeros((40, 10), dtype=torch.float32, device="cuda")
    g, cfg = C.c_void_p(), ivf.SearcherConfig().to_c()
    monkeypatch.setenv("SAQG_TEST_ALLOC_BYTES", str(4 << 20))
    N.check(ix.lib.saqg_search_graph_create(ix._h, qd.data_ptr(), 40, 10, K, C.byref(cfg), ids.data_ptr(),
                                            d.data_ptr(), None, C.byref(g)))
    monkeypatch.delenv("SAQG_TEST_ALLOC_BYTES")
    try:
        for _ in range(2):
            ids.zero_()
            N.check(ix.lib.saqg_search_graph_launch(g, None))
            torch.cuda.synchronize()
            assert np.array_equal(ids.cpu().numpy().view(np.uint32), oi)
            assert np.array_equal(d.cpu().numpy().view(np.uint32), od.view(np.uint32))
    finally:
        N.check(ix.lib.saqg_search_graph_free(g))
