"""The benchmark's line on standard output: every figure a reader of its end needs, short
enough to survive in a log's last kilobytes whatever the legs measured."""
import json
import os
import sys

from conftest import ROOT


def test_contract_line_is_whole_and_short():
    sys.path.insert(0, ROOT)
    import bench
    many = {str(i): 0.123456789 for i in range(2000)}
    full = dict(metric=bench.METRIC, value=1.3e6, unit="queries/s", n_gpus=1, steps=100, warmup=3, ms_per_step=3.1,
                higher_is_better=True, scaling="weak", vs_baseline=None, dtype="int32+f32", data="synthetic",
                config={"workload": "w" * 100, "plan": [[64, 11]] * 16, "form": "f" * 200},
                e2e={"value": 1.2e6, "unit": "queries/s", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 1},
                gpu_launches=1000, clocks={"sm_mhz": 2070, "sm_max_mhz": 2070, "reasons": []}, p99_ms=3.2,
                batched_over_plain=160.0, wall_s=60.0, plain=dict(qps=8000.0, legs=many), serving=many, c1=many, c2=many,
                roofline=dict(bound="hbm", achieved=1.0, peak=2.0, unit="GB/s", frac=0.5, traffic=None, kernel="k",
                              peak_kind="measured", more=many),
                batched_tc=dict(qps=9e5, more=many), cpu_baseline=dict(value=5e3, unit="queries/s", cores=16,
                                                                       kind="port", more=many))
    line = bench.contract_line(full)
    text = json.dumps(line)
    assert "\n" not in text and len(text) < 4000
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline"):
        assert key in line
    assert json.loads(text)["e2e"] == full["e2e"] and os.path.exists(bench.__file__)
