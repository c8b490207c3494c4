"""saqg_kernel_launches counts what a search launches: the kernel nodes of the same call
captured into a graph, in every scan form, with and without the GEMM ranking, the split
pass and the tensor-core form's stages."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Driver:
    def __init__(self):
        self.lib = C.CDLL("libcuda.so.1")

    def call(self, name, *args):
        rc = getattr(self.lib, name)(*args)
        assert rc == 0, (name, rc)

    def kernels(self, stream, work):
        """Kernel nodes of `work()` captured on the stream."""
        graph, n = C.c_void_p(), C.c_size_t()
        self.call("cuStreamBeginCapture_v2", C.c_void_p(stream), 1)  # thread-local
        try:
            work()
        finally:
            self.call("cuStreamEndCapture", C.c_void_p(stream), C.byref(graph))
        self.call("cuGraphGetNodes", graph, None, C.byref(n))
        nodes = (C.c_void_p * n.value)()
        self.call("cuGraphGetNodes", graph, nodes, C.byref(n))
        kinds = []
        for node in nodes:
            kind = C.c_int()
            self.call("cuGraphNodeGetType", C.c_void_p(node), C.byref(kind))
            kinds.append(kind.value)
        self.call("cuGraphDestroy", graph)
        return kinds.count(0)


@pytest.fixture(scope="module")
def problem():
    from saq_gb300 import ivf
    rng = np.random.default_rng(4)
    n, D, K = 20000, 128, 64
    cids = rng.integers(0, K, n).astype(np.uint32)
    cent = rng.standard_normal((K, D)).astype(np.float32)
    x = (cent[cids] + 0.8 * rng.standard_normal((n, D))).astype(np.float32)
    q = (cent[rng.integers(0, K, 400)] + 0.8 * rng.standard_normal((400, D))).astype(np.float32)
    ix = ivf.IVF(n, D, K, ivf.QuantizeConfig(avg_bits=4.0, seg_eqseg=2))
    ix.construct(x, cent, cids, seed=2)
    return ix, q


@pytest.mark.parametrize("mode,defer,nq,nprobe", [
    ("", "", 1, 4), ("", "", 12, 32), ("", "", 40, 4), ("", "", 100, 4), ("", "", 100, 64), ("", "20", 300, 16),
    ("", "1", 400, 64), ("split", "", 100, 16), ("split", "", 300, 4), ("ws", "", 70, 8), ("warp", "", 100, 8),
    ("seq", "0", 64, 64)])
def test_exact_forms(problem, mode, defer, nq, nprobe, monkeypatch):
    import torch
    from saq_gb300 import _native as N, ivf
    ix, q = problem
    for name, v in (("SAQG_SCAN_MODE", mode), ("SAQG_DEFER_BLOCKS", defer)):
        if v:
            monkeypatch.setenv(name, v)
    qd = torch.from_numpy(q[:nq]).cuda()
    ids = torch.zeros((nq, 10), dtype=torch.int32, device="cuda")
    d = torch.zeros((nq, 10), dtype=torch.float32, device="cuda")
    cfg, stream = ivf.SearcherConfig().to_c(), torch.cuda.Stream()

    def call():
        N.check(ix.lib.saqg_search(ix._h, qd.data_ptr(), nq, 10, nprobe, C.byref(cfg), ids.data_ptr(), d.data_ptr(),
                                   N.SAQG_MEM_DEVICE, C.c_void_p(stream.cuda_stream)))
    call()  # what is built and allocated once
    torch.cuda.synchronize()
    before = ix.lib.saqg_kernel_launches()
    call()
    counted = ix.lib.saqg_kernel_launches() - before
    torch.cuda.synchronize()
    captured = _Driver().kernels(stream.cuda_stream, call)
    call()  # the context's events recorded outside a capture again
    torch.cuda.synchronize()
    assert counted == captured


def test_static_form(problem):
    import torch
    from saq_gb300 import _native as N, ivf
    ix, q = problem
    cfg, stream = ivf.SearcherConfig().to_c(), torch.cuda.Stream()
    for nq in (1, 300):
        qd = torch.from_numpy(q[:nq]).cuda()
        ids = torch.zeros((nq, 10), dtype=torch.int32, device="cuda")

        def call():
            N.check(ix.lib.saqg_search_static(ix._h, qd.data_ptr(), nq, 10, 4, C.byref(cfg), ids.data_ptr(), None,
                                              C.c_void_p(stream.cuda_stream)))
        call()
        torch.cuda.synchronize()
        before = ix.lib.saqg_kernel_launches()
        call()
        counted = ix.lib.saqg_kernel_launches() - before
        torch.cuda.synchronize()
        assert counted == _Driver().kernels(stream.cuda_stream, call)
