"""The u16 LUT quantiser without a division, checked on the CPU in IEEE float32.

Lut::prepare (saqlib/quantization/fastscan/lut.hpp:60-87) stores trunc(RN(x / delta)).
The GPU (search.cu lut_quant) takes n, the integer nearest to RN(x RN(1 / delta)), and
subtracts one when the remainder RN(x - n delta) of one FMA lies below -delta u / 2, u
the spacing of the floats below n.  The FMA is formed in float64, where n delta (41
bits) and the difference are exact."""
import numpy as np

F = np.float32


def _quant(x, d):
    r = F(F(1.0) / d)
    m = ((x * r).astype(F) + F(8388608.0)).astype(F)
    n = (m - F(8388608.0)).astype(F)
    half = (((n.view(np.uint32) - np.uint32(1)) & np.uint32(0x7F800000)) - np.uint32(24 << 23)).view(F)
    with np.errstate(over="ignore"):
        t = (d * half).astype(F)
    rem = (x.astype(np.float64) - n.astype(np.float64) * np.float64(d)).astype(F)
    return (m.view(np.uint32).astype(np.int64) - (rem < -t)) & 0xFFFF


def _exact(x, d):
    return np.trunc((x / d).astype(F)).astype(np.int64) & 0xFFFF


def _delta(span):
    return F(np.float64(F(span)) / (65536.0 - 0.01))


def test_equals_division_on_random_entries():
    rng = np.random.default_rng(1)
    for scale in (1e-24, 1e-6, 1e-2, 1.0, 37.0, 1e4, 1e24):
        for _ in range(8):
            span = F(scale * (0.01 + abs(rng.standard_normal())))
            d = _delta(span)
            x = np.concatenate([(rng.random(200_000) * np.float64(span)).astype(F), np.array([0, span], F)])
            assert np.array_equal(_quant(x, d), _exact(x, d))


def test_equals_division_beside_every_integer():
    rng = np.random.default_rng(2)
    for scale in (1e-20, 3.0, 1e20):
        for _ in range(4):
            span = F(scale * (0.1 + rng.random()))
            d = _delta(span)
            n = np.arange(0, 65536, dtype=np.float64)
            base = (n * np.float64(d)).astype(F)
            for step in range(-6, 7):  # the floats around n d, through the tie below n
                x = (base.view(np.int32) + step).clip(0).view(F)
                x = x[x <= span]
                assert np.array_equal(_quant(x, d), _exact(x, d)), step
