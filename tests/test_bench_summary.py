"""The benchmark's printed line: the contract's keys with their values, in a few KB however long the record."""
import json

import bench

ERR = {"pattern_equal": True, "pairs_equal": True, "max_abs": 1e-12, "rel_fro": 4.503174776e-14, "bits_differ": 12345678}


def form(ms):
    return {"ms_per_step": ms, "gflops": 1e5 / ms, "plan_ms": 0.1234567890123, "exec_ms": ms - 0.1, "exec_graph_ms": ms,
            "kernel": "k", "roofline": {"bound": "tensor", "frac": 0.61756889, "note": "x" * 200}, "error_vs_oracle": ERR}


def test_summary_is_short_and_complete():
    phase = {"p50_ms": 1.0, "p99_ms": 2.0, "gflops": 3.0, "mean_batch": 1.5, "mean_plan_ms": 0.3, "completed": 400,
             "failed": 0, "slowest": [{"latency_ms": 1.23456789012345, "template": i} for i in range(40)]}
    served = {"streams": [phase] * 30, "stream": phase, "burst": phase, "mix_equals_alone": {"checked": 6}}
    leg = {"value": 23.2, "unit": "GFLOP/s", "cores": 16, "kind": "port", "sample": "s" * 200}
    full = {"metric": bench.METRIC, "value": 26189.56798779343, "unit": "GFLOP/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 4.144476699829101, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic (seeded)", "config": {"workload": bench.WORKLOADS["c1"]},
            "forms": {f: form(4.0) for f in bench.FORMS}, "ratios": {}, "roofline": {"frac": 0.5}, "peaks": {},
            "cpu_baseline": {**leg, "legs": {str(i): leg for i in range(50)}},
            "e2e": {"value": 897.1, "unit": "GFLOP/s", "h2d_bytes_per_step": 168005504, "d2h_bytes_per_step": 5904210624},
            "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []}, "gpu_launches": 180,
            "kernels_per_step": {"k": {"launches": 2, "us": 3.0}},
            "configs": {c: {"workload": "w" * 300, "forms": {f: form(1.0) for f in bench.FORMS}} for c in ("c0", "c2", "c3")},
            "serving": {"alone_plain": {"gflops": 1.0}, "templates": [{"family": "c0"}] * 500, "batched": served,
                        "split": served}}
    text = json.dumps(bench.summary_line(full))
    assert len(text) < 6000, len(text)
    line = json.loads(text)
    assert set(full) == set(line)
    for k in ("metric", "unit", "n_gpus", "steps", "warmup", "higher_is_better", "scaling", "vs_baseline", "dtype", "data",
              "config", "e2e", "clocks", "gpu_launches"):
        assert line[k] == full[k], k
    assert abs(line["value"] / full["value"] - 1) < 1e-5 and abs(line["ms_per_step"] / full["ms_per_step"] - 1) < 1e-5
    assert line["forms"]["split"]["rel_fro"] == 4.50317e-14 and line["forms"]["split"]["bits_differ"] == 12345678
    assert line["serving"]["split"]["burst"]["mean_plan_ms"] == 0.3 and "legs" not in line["cpu_baseline"]
