"""bench.py prints one line with the measurement, short enough to survive a reader that keeps the last
1500 bytes of the output; the secondary measurements' objects go to a file."""
import json

import bench
from golikov_2d_gb300 import problems

KEYS = {"metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
        "scaling", "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks", "e2e"}


def test_headline_is_short_and_whole():
    x = 123456789.0123456789
    long = {"value": x, "ms_per_step": x, "frac": x, "ops_per_cell": x, "bound": "hbm",
            "unit": "cell-updates/s", "kind": "port", "cores": 144,
            "rows": [{"case": "y" * 50, "rel": x}] * 500}
    cfg = problems.kelvin_helmholtz(64, 64)[0]
    line = {k: long for k in ("roofline", "fp64", "secondary", "ot_to_t05", "batched", "adjoint",
                              "io", "hancock", "cpu_baseline", "sim")}
    line.update({k: x for k in KEYS})
    line["config"] = bench.workload_config("kh4096", cfg, 8)
    line["clocks"] = {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "samples": 1000,
                      "reasons": ["hw_slowdown", "sw_power_cap"]}
    line["e2e"] = {"value": x, "unit": "cell-updates/s", "h2d_bytes_per_step": 536870912,
                   "d2h_bytes_per_step": 536870912, "path": "z" * 300}
    line["hancock"] = {"unavailable": "w" * 1000}
    line["batched"] = {"unavailable": "w" * 1000}
    out = bench.headline(line)
    assert KEYS <= set(out)
    assert out["e2e"]["h2d_bytes_per_step"] == 536870912 and out["value"] == x
    assert len(json.dumps(out)) < 1400
