"""The line bench.py prints on stdout: complete and short, however large the record of all legs is."""

import json

import bench


def test_headline_is_short_and_complete():
    text = "x" * 400
    record = {"metric": "w4a4_fused_linear_effective_tops", "value": 52.854736778201, "unit": "TOPS", "n_gpus": 8, "steps": 100, "warmup": 10,
              "ms_per_step": 0.16812345678, "windows": 3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "s4xs4->s32",
              "data": "synthetic", "gpu_launches": 2400, "clocks": {"sm_mhz": 1965, "sm_max_mhz": 1965, "reasons": ["sw_power_cap"]},
              "config": {"workload": bench.WORKLOAD_DESC["decode"], "l2": "weights rotate through 4 distinct copies (> 2x L2)",
                         "parallelism": "replicated x8", "weights": "packed nibbles", "timing": text},
              "e2e": {"value": 63.41234567, "unit": "TOPS", "h2d_bytes_per_step": 1118208, "d2h_bytes_per_step": 1806336, "schedule": text},
              "roofline": {"bound": "hbm", "frac": 0.51475325, "kernel": "decode_gemm_kernel", "per_shape": {str(i): text for i in range(12)}},
              "cpu_baseline": {"value": 0.0039527, "unit": "TOPS", "cores": 16, "kind": "port", "sample": text},
              "prefill": {str(i): text for i in range(24)}, "stack": {"config": text}, "decode_tok_s": 4974.6676827, "wall_s": 101.5}
    line = bench.headline(record)
    assert len(json.dumps(line)) < 1400
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline", "dtype",
                "data", "config", "e2e", "gpu_launches", "clocks"):
        assert key in line
    assert abs(line["value"] / record["value"] - 1) < 1e-5 and abs(line["ms_per_step"] / record["ms_per_step"] - 1) < 1e-5
    assert line["e2e"]["h2d_bytes_per_step"] == 1118208 and line["e2e"]["d2h_bytes_per_step"] == 1806336
    assert "prefill" not in line and line["clocks"] == record["clocks"]
