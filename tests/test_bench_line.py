"""The line that bench.py prints on standard output: every key of its contract
and the summaries of roofline and parity, short enough to be kept whole."""
import json

import bench


def test_short_line():
    line = {"metric": bench.METRIC, "value": 35828462086.9052, "unit": "tuples/s", "n_gpus": 1,
            "steps": 300, "warmup": 3, "ms_per_step": 0.7891229863961537, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic" * 6,
            "config": {"workload": "w" * 150, "n_points": 399949, "l2": "flushed" * 5},
            "e2e": {"value": 18671631862.423058, "unit": "tuples/s", "h2d_bytes_per_step": 12798368,
                    "ms_per_step": 1.5142256021499634, "ms_min_median_max": [1.0384000539779663] * 3,
                    "d2h_bytes_per_step": 38464},
            "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []}, "gpu_launches": 2400,
            "roofline": {"kernel": "k", "frac": 0.1, "binding": "issue", "binding_frac": 0.66,
                         "issue": {"source": "x" * 400}},
            "parity": {"counts_exact": True, "max_rel_catsum": 2.1e-16, "per_bin_max_rel": [0.0] * 600},
            "quad": {"x": "y" * 9000}, "stats": {"probes": 1}}
    out = bench.short_line(line)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e",
                "clocks", "gpu_launches"):
        assert out[key] == line[key]
    assert out["roofline"] == {"kernel": "k", "frac": 0.1, "binding": "issue", "binding_frac": 0.66}
    assert out["parity"] == {"counts_exact": True, "max_rel_catsum": 2.1e-16}
    assert len(json.dumps(out)) < 1500
    # ranks of a larger run print no parity
    assert "parity" not in bench.short_line({k: v for k, v in line.items() if k != "parity"})
