"""The benchmark's last line: the headline's keys, whole within the 1500 bytes
that a log's tail may keep, however much the run measured beside it."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def test_headline_is_short_and_complete():
    import bench
    x = 1234.567890123456
    case = {"workload": bench.WORKLOAD, "blocks": 8, "nodes": 851400,
            "grid": "193x129x33 as 8 blocks of 25x129x33 along x, wall spacing 5e-6, ratio 1.1",
            "ma": 0.2, "re": 5.0e6, "nutinf_over_nuinf": 3.0, "cfl": 5.0,
            "scheme": "roe_weno3 + central viscous + spalart-allmaras + lu-sgs (reference path)",
            "l2": "flushed (256 MiB write) before every timed step; the case's arrays exceed L2",
            "execution": "each step replayed from a CUDA graph; launch shapes from the autotuner",
            "parallelism": "replicas x8"}
    line = {"metric": "Mcell-iter/s", "value": x, "unit": "Mcell-iter/s", "n_gpus": 8, "steps": 20, "warmup": 5,
            "ms_per_step": x, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (analytic flat-plate grid, freestream start)", "config": case,
            "gpu_launches": 12345, "tuning": "t" * 300, "device_status": 0,
            "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 1234},
            "kernels": {f"k{i}": {"ms_total": x, "launches": 20, "share": x} for i in range(20)},
            "roofline": {"bound": "hbm", "kernel": "k_lusgs_sweep", "achieved": x, "peak": x, "unit": "GB/s", "frac": x,
                         "peak_kind": "measured", "traffic": x, "alg_bytes_per_launch": 1, "units_per_launch": 1,
                         "bytes_per_unit": 392, "ms_per_launch": x},
            "e2e": {"value": x, "unit": "Mcell-iter/s", "h2d_bytes_per_step": 40867200,
                    "d2h_bytes_per_step": 40867256, "fields": ["q", "nut"]},
            "naca": {"x": "y" * 20000}}
    text = json.dumps(bench.headline(line))
    assert len(text) <= 1500, len(text)
    got = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches"):
        assert got[k] == line[k], k
    assert "naca" not in got and "kernels" not in got
