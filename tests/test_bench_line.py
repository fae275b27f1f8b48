"""The bench's result line stays short enough for a reader that keeps the last 3000 characters of the output, also with eight ranks'
figures in it, and says what the full-precision record says."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def test_one_line_is_short_and_keeps_seven_digits():
    import bench
    third = 1234.0 / 3
    nested = {f"key_{i}": third for i in range(10)}
    record = {"metric": "gemm_tflops", "value": third, "config": bench.workload_config(bench.DEFAULT_WORKLOAD, "strong", 4), "vs_baseline": None,
              "higher_is_better": True, "gpu_launches": 7960, "ms_per_step_min_median_max": [third] * 3, "roofline": nested, "e2e": nested,
              "clocks": nested, "cpu_baseline": nested, "per_rank": [{"step_ms": third, "kernel_ms": third, "quant_kernel_ms": third}] * 8}
    text = bench.one_line(record)
    assert "\n" not in text and len(text) < 3000
    back = json.loads(text)
    assert back["value"] == 411.3333 and back["gpu_launches"] == 7960 and back["vs_baseline"] is None and back["higher_is_better"] is True
    assert back["config"] == record["config"] and back["per_rank"][7]["kernel_ms"] == 411.3333
