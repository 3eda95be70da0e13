"""The benchmark's JSON line stays short enough for a reader that keeps the last few thousand characters of the output."""
import json

import bench
from quactlize_b200 import workloads

# a full run's line without its sub-records, every figure at its usual length
LINE = {"metric": "Q4_K decode GEMV HBM GB/s on weight bytes", "value": 3970.12, "unit": "GB/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 0.79871, "ms_per_step_min": 0.79801, "ms_per_step_max": 0.80101, "timed_batches": 5, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "fp16 codes->HFMA2, fp32 accumulate", "data": "synthetic",
        "config": {"workload": "x" * 190, "parallelism": "column-parallel x1", "l2": "x" * 95}, "parity_max_rel": 0.000512,
        "roofline": {"bound": "hbm", "achieved": 3970.1, "peak": 6538.9, "unit": "GB/s", "frac": 0.6071, "frac_of_nominal_8000": 0.4963,
                     "traffic": 33065536, "traffic_source": "x" * 60, "peak_source": "measured", "kernel": "q4k_gemv1_kernel",
                     "algorithmic_bytes_per_launch": 33084074, "us_per_launch": 8.321},
        "e2e": {"value": 45.432, "unit": "GB/s", "h2d_bytes_per_step": 3171487744, "d2h_bytes_per_step": 4194304, "api": "x" * 50, "steps": 3},
        "gpu_launches": 9600, "launch_mode": "cuda_graph", "commit": "0123abc",
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": [], "samples": 1234, "via": "nvml"},
        "fused_gate_up_step": {"what": "gate and up of a layer in one launch", "ms_per_step": 0.69701, "value": 4550.12, "unit": "GB/s", "frac": 0.6958,
                               "bit_identical_to_per_matrix_launches": True, "gpu_launches": 6400},
        "cpu_baseline": {"value": 0.0537, "unit": "GB/s", "cores": 16, "kind": "reference", "sample": "x" * 110, "matmul_only_gbs": 22.538}}


def _records():
    rec = {"us": 1234.567, "frac": 0.61234, "parity_max_rel": 0.00367, "parity_elementwise_ok": True, "kernel": "x" * 50}
    return {name: dict(rec) for name in workloads.registry()}


def test_line_is_short_and_whole(capsys):
    records = _records()
    records["cfg1"] = {"error": "RuntimeError: x"}
    bench.emit(dict(LINE), records)
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < bench.LINE_LIMIT
    line = json.loads(out)
    assert line["configs"]["failed"] == ["cfg1"] and line["configs"]["us_frac"]["cfg4_gate"] == [1234.57, 0.612]
    assert json.loads(err)["configs"] == records


def test_line_without_sub_records(capsys):
    bench.emit({"metric": "m"})
    out, err = capsys.readouterr()
    assert json.loads(out) == {"metric": "m"} and not err
