"""The build's column variance and planner at the edges of their kernels: row counts
around a group of four, a stage and the ring of stages; data that are not 16-byte
aligned; plans of variances with zeros, negatives and values that tie."""
import numpy as np
import pytest

import oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 64, 65, 66, 68, 129, 1023, 1024, 1025, 1026, 2177])
def test_column_variance_equals_oracle(n, tmp_path):
    import torch
    from saq_gb300 import index_format as F, ivf
    rng = np.random.default_rng(n)
    D = 64 if n % 2 else 192
    x = (rng.standard_normal((n, D)) * 10.0 ** rng.uniform(-3, 3, D) + 5).astype(np.float32)
    want = O.colwise_var(x)
    for shift in (0, 1):
        buf = torch.empty(n * D + 4, device="cuda")
        t = buf[shift:shift + n * D].view(n, D)
        t.copy_(torch.from_numpy(x))
        ix = ivf.IVF(n, D, 1, ivf.QuantizeConfig(avg_bits=2.0, enable_segmentation=False, random_rotation=False))
        ix.construct(t, np.zeros((1, D), np.float32), np.zeros(n, np.uint32))
        ix.save(str(tmp_path / "i.index"))
        got = F.load(str(tmp_path / "i.index")).variance
        assert np.array_equal(np.asarray(got, np.float32).view(np.uint32), want.view(np.uint32)), shift


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128, 960, 1536])
@pytest.mark.parametrize("bits", [1.5, 4.0, 13.0])
def test_plans_equal_host_planner(D, bits):
    from saq_gb300 import ivf
    rng = np.random.default_rng(D)
    decay = (np.arange(1, D + 1) ** -1.0).astype(np.float32)
    for v in (decay, np.ones(D, np.float32), np.where(np.arange(D) % 3, decay, 0).astype(np.float32),
              rng.standard_normal(D).astype(np.float32), (decay * 1e-30).astype(np.float32)):
        assert ivf.plan_gpu(v, bits) == ivf.plan(v, bits)
