"""bench.py's printed line: every key that its readers take, in one line that a log
cut at 3000 characters still holds (CPU only)."""
import json
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))
import bench  # noqa: E402

NUMBER = 12345678.901234567  # as long as a measured figure prints


def result(n):
    """A result as large as a measured one."""
    acc = {"vs": "x" * 60, "compared": 32768, "max_rel_err": NUMBER, "median_rel_err": NUMBER,
           "count_above_1e-10": 0, "worst": [NUMBER] * 20}
    return {"value": NUMBER, "unit": "dets/s", "ms_per_step": NUMBER, "steps": 20,
            "config": bench.workload_config("lll24", 1),
            "plain_fp64": {k: NUMBER for k in ("dets_per_s_reference_arith", "dets_per_s_fused",
                                               "mixed_over_plain_fused",
                                               "mixed_over_plain_reference_arith")},
            "accuracy": acc, "fallbacks": {"count": 1515, "of": 32768}, "hbm_gbs": NUMBER,
            "kernel_times_ms": {f"a_long_kernel_name_{i}<{n}>": {"launches": 20, "ms": NUMBER,
                                                                 "ms_per_launch": NUMBER}
                                for i in range(6)},
            "roofline": {"kernel": f"lup_mixed_tile_kernel<{n}>", "bound": "hbm", "unit": "GB/s",
                         "peak": NUMBER, "peak_source": "x" * 80, "achieved": NUMBER,
                         "frac": NUMBER, "traffic": NUMBER, "kernel_ms_per_launch": NUMBER,
                         "share_of_step": NUMBER, "plain_fp64": {"kernel": "x" * 200}},
            "gpu_launches": 40}


def test_line_is_short_and_complete():
    class Args:
        warmup = 5
    e2e = {"value": NUMBER, "unit": "dets/s", "ms_per_step": NUMBER, "h2d_bytes_per_step": 301989888,
           "d2h_bytes_per_step": 688128, "call": "x" * 150, "host_link_copy_gbs": NUMBER,
           "fraction_of_link": NUMBER}
    line = bench.base_line(Args, 1) | result(24) | {
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"],
                   "samples": 6},
        "e2e": e2e, "e2e_from_coordinates": dict(e2e),
        "cpu_baseline": {"value": NUMBER, "unit": "dets/s", "cores": 16, "kind": "port",
                         "sample": "x" * 120},
        "configs": {"config1_gauss8": result(8), "config2_gauss16": result(16),
                    "config4_mixedn": result(32) | {"per_n": {str(i): [NUMBER] * 9
                                                              for i in range(7)}},
                    "config5_serving": {"value": NUMBER, "unit": "dets/s", "p50_ms": NUMBER,
                                        "p99_ms": NUMBER, "serving": {"x" * 20: [NUMBER] * 300}}}}
    text = json.dumps(bench.headline(line))
    assert len(text) < 3000 and "\n" not in text, len(text)
    short = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
              "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "clocks",
              "e2e", "gpu_launches", "roofline", "accuracy", "cpu_baseline"):
        assert k in short, k
    assert short["config"] == line["config"] and short["clocks"] == line["clocks"]
    for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert short["e2e"][k] == e2e[k]
    assert set(short["configs"]) == set(line["configs"])
