"""The GPU encoder against the oracle, codes and factors bit for bit, where its
comparisons in FP32 with a bound (saq_gb300/csrc/encode.cu, AdjView) or its layouts
could go wrong: magnitudes to and past float range, zeros and denormals, one
dominant dimension, ties, every code width, rows on both sides of a warp and of a
block, and buffers that are not 16-byte aligned."""
import ctypes as C

import numpy as np
import pytest

import oracle as O


def _resid(kind, n, d, rng):
    x = rng.standard_normal((n, d)).astype(np.float32)
    if kind == "scales":  # 1e-38 .. 1e18 by row
        return (x * (10.0 ** np.linspace(-38, 18, n))[:, None]).astype(np.float32)
    if kind == "sparse":
        x[rng.random((n, d)) < 0.7] = 0.0
        x[0] = 0.0
        x[1, 1:] = 0.0
        return x
    if kind == "spike":  # one dimension holds nearly all of the norm
        x *= 1e-4
        x[np.arange(n), rng.integers(0, d, n)] = 3.0
        return x
    if kind == "grid":  # equal magnitudes: comparisons at or near equality
        return rng.integers(-4, 5, (n, d)).astype(np.float32)
    if kind == "decay":
        return (x * np.arange(1, d + 1, dtype=np.float32) ** -1.0).astype(np.float32)
    return x


def _equal(a, b):
    """Bit for bit, NaNs of either sign taken as equal."""
    return bool(np.all((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "scales", "sparse", "spike", "grid", "decay"])
@pytest.mark.parametrize("bits", [1, 2, 4, 5, 6, 7, 9, 13])
def test_encoder_equals_oracle(kind, bits):
    from saq_gb300 import ivf
    rng = np.random.default_rng(bits)
    n, d = [(33, 64), (65, 192), (130, 320)][bits % 3]
    x = _resid(kind, n, d, rng)
    cent = rng.standard_normal(d).astype(np.float32)
    for rd, eps in ((6, 1e-8), (1, 1e-8), (0, 1e-8), (20, 0.0), (6, 1e-3)):
        codes, facs = ivf.caq_encode(x, bits, cent, rd_lmt=rd, eps=eps)
        ocodes, ofacs = O.caq_encode(x, bits, cent, rd, eps)
        assert np.array_equal(codes, ocodes), (rd, eps)
        assert _equal(facs, ofacs), (rd, eps)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_encoder_device_buffers_of_any_alignment(shift):
    import torch
    from saq_gb300 import _native as N
    rng = np.random.default_rng(shift)
    n, d, bits = 70, 128, 4
    x = rng.standard_normal((n, d)).astype(np.float32)
    buf = torch.zeros(n * d + 8, device="cuda")
    buf[shift:shift + n * d] = torch.from_numpy(x.reshape(-1)).cuda()
    codes = torch.zeros(n * d + 8, dtype=torch.int32, device="cuda")
    facs = torch.zeros(n * 4, device="cuda")
    N.check(N.load().saqg_caq_encode(C.c_void_p(buf.data_ptr() + 4 * shift), n, d, bits, None, 6, 1e-8,
                                     C.c_void_p(codes.data_ptr() + 4 * shift), C.c_void_p(facs.data_ptr()),
                                     N.SAQG_MEM_DEVICE, None))
    torch.cuda.synchronize()
    ocodes, ofacs = O.caq_encode(x, bits, None, 6, 1e-8)
    assert np.array_equal(codes[shift:shift + n * d].cpu().numpy().reshape(n, d), ocodes)
    assert _equal(facs.cpu().numpy().reshape(n, 4), ofacs)
