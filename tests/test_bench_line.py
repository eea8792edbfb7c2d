"""The line bench.py prints: every key a reader relies on, and short enough that
the last 3,000 characters of stdout hold all of it, whatever the variants record."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402

KEYS = {"metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
        "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "roofline", "clocks", "cpu_baseline"}


def _record():
    point = {"probes": 64, "ms_per_call": 17.1234, "value": 557000.1, "recall1": 0.8512, "candidates_mean": 137000.5,
             "scan_kernel": {"ms": 16.1234, "GB/s": 10200.5, "frac_hbm": 1.5612}}
    clocks = {"sm_mhz": 1965.0, "sm_min_mhz": 1702.0, "sm_max_mhz": 1965.0,
              "reasons": ["hw_slowdown", "hw_thermal_slowdown", "sw_power_cap", "sw_thermal_slowdown"], "samples": 99,
              "source": "nvidia-smi"}
    roof = {"bound": "tensor", "kernel": "exact2nn_u8fold_pair_kernel", "achieved": 2245.1, "peak": 4550.0,
            "unit": "TFLOP/s", "frac": 0.4934, "traffic": 2630000000.0, "ops_per_launch": 2.56e12, "kernel_ms": 1.1403,
            "peak_note": "n" * 150, "frac_of_2x_bf16_measured": 0.6612}
    variant = {"value": 1234567890.1, "unit": "queries/s", "ms_per_step": 1.2345, "steps": 20, "workload": "w" * 300,
               "call": "c" * 200, "roofline": roof, "operating_point": point, "clocks": clocks}
    names = ("fp16", "pairs512", "mutual512", "learned_hash", "lsh", "cfg1_1000x10000", "float32_general")
    line = {k: None for k in KEYS}
    line.update({
        "metric": bench.METRIC, "value": 8437563.1, "unit": "queries/s", "n_gpus": 8, "steps": 200, "warmup": 50,
        "ms_per_step": 1.1852, "higher_is_better": True, "scaling": "weak", "dtype": "u8",
        "data": "synthetic (seeded generator standing in for ANN_SIFT1M; base seed 0, queries seed = rank)",
        "config": {"workload": bench.WORKLOAD, "queries_per_gpu": 10000, "base_rows": 1000000, "dim": 128, "ratio": 0.8,
                   "l2_between_steps": "flushed (256 MiB write outside the timed events)",
                   "parallelism": "query-sharded x8, base replicated"},
        "e2e": {"value": 4081632.1, "unit": "queries/s", "h2d_bytes_per_step": 129280000, "d2h_bytes_per_step": 40000,
                "call": "cublas_2nn_sift(type=SIFT_U8_HOST) with pinned host buffers", "h2d_copy_ms": 2.3412,
                "frac_of_h2d_copy": 0.9551, "h2d_note": "n" * 200},
        "gpu_launches": 600, "roofline": roof, "clocks": clocks,
        "cpu_baseline": {"value": 207.1, "unit": "queries/s", "cores": 192, "kind": "port",
                         "sample": "10000 queries x 1000000 base rows (15.0 s)"},
        "variants": {n: dict(variant, grid=[dict(variant, points=[point] * 8)] * 16) for n in names}})
    return line


def test_line_is_whole_in_the_tail_of_stdout():
    line = _record()
    assert len(json.dumps(line)) > 20000
    text = json.dumps(bench.short_line(line))
    assert len(text) <= 2900
    got = json.loads(text)
    assert KEYS <= set(got)
    assert got["value"] == line["value"] and got["e2e"]["value"] == line["e2e"]["value"]
    assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(got["e2e"])
    assert set(got["variants"]) == set(line["variants"])
    assert got["variants"]["lsh"]["recall1"] == 0.8512 and got["variants"]["fp16"]["frac"] == 0.4934


def test_record_without_legs():
    line = {k: v for k, v in _record().items() if k not in ("variants", "roofline", "cpu_baseline")}
    got = bench.short_line(line)
    assert got["value"] == line["value"] and "variants" not in got


def test_reference_arm_without_the_reference_says_so(monkeypatch, capsys):
    import types

    import oracle

    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    bench.reference_arm(types.SimpleNamespace(steps=1, warmup=0), 1, 0)
    got = json.loads(capsys.readouterr().out)
    assert got["impl"] == "reference" and got["unavailable"] and "value" not in got
