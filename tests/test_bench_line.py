"""The benchmark's result line stays short enough to be kept whole."""
import json

import bench


def test_line_holds_the_headline_and_stays_short():
    big = {"final_energies": [-8.0123456789] * 64, "bonds": [{"e": 1.5115818501785988e-11} for _ in range(500)],
           "total_s": 117.9123456789, "note": "x" * 300}
    out = {"metric": bench.METRIC, "value": 63.123456789, "unit": "TFLOP/s", "n_gpus": 1, "steps": 20, "warmup": 5,
           "ms_per_step": 1.4398123, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "tf32x3-split (fp64 in/out)", "data": bench.DATA,
           "config": {"workload": "qc-c2-bond", "W": [712, 862, 1028], "precision": "split", "l2": "y" * 200},
           "gpu_launches": 100,
           "e2e": {"value": 60.0, "unit": "TFLOP/s", "ms_per_step": 1.5, "h2d_bytes_per_step": 8, "d2h_bytes_per_step": 8},
           "roofline": {"bound": "hbm", "frac": 0.25, "tensor": {"achieved": 1.0}}, "sweeps": big, "gradient": big,
           "scan": big, "sigma_tuning": [{"ms": 1.0}] * 6, "bond_step_e2e": big,
           "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 3}}
    line = bench.bench_line(out)
    assert "\n" not in line and len(line) <= 3000
    got = json.loads(line)
    for k in bench.REQUIRED:
        assert k in got
    assert got["value"] == out["value"] and got["e2e"] == out["e2e"] and got["clocks"] == out["clocks"]
    assert got["config"]["workload"] == "qc-c2-bond" and got["config"]["W"] == [712, 862, 1028]
    assert got["roofline"] == {"bound": "hbm", "frac": 0.25}
    assert got["sweeps"] == {"total_s": 117.912, "note": big["note"]}
