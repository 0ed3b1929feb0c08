"""The headline line keeps its contract's keys and stays short, whatever its
objects hold (host only)."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import bench  # noqa: E402


def _full():
    f = 1234.567890123456
    line = {"metric": bench.METRIC, "value": f, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": f, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": bench.workload_config(30, 20), "staging": "threads", "executor": "x" * 64,
            "parallelism": "single-gpu", "gates_per_s": f, "passes_per_step": 76, "gpu_launches": 1540,
            "cpu_baseline": {"value": f, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "s" * 150},
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 482, "active_masks": ["0x0"],
                       "power_w_median": f, "util_pct_median": 100.0, "temp_c_max": 34.0}}
    for key, keep in bench.HEADLINE.items():
        line[key] = {k: f for k in keep}
        line[key].update(note="n" * 300, rows=[{"gate": "H", "target": t, "ms": f} for t in range(300)])
    gates = [f"{g}_{m}" for g in ("H", "RX", "RY", "RZ", "U", "X") for m in ("exact", "lazy")]
    line["sweep30"]["summary"] = {g: {"ms_median": f, "hbm_frac_median": 0.9876543} for g in gates}
    line["sweep33"]["summary"] = {g: {"ms_median": f, "frac_median": 0.9876543} for g in ("H", "RZ", "CX", "MCX3")}
    line["parity"]["vs_oracle"] = {"prefix": "p" * 60, "max_abs_diff_fast_vs_oracle": f, "exact_bit_identical": True,
                                   "max_abs_diff_exact_vs_oracle": 0.0, "bound": 1e-12, "ok": True}
    return line


def test_line_is_short_and_whole():
    full = _full()
    line = bench.headline(full)
    text = json.dumps(line)
    assert len(text) < 4096 and "\n" not in text
    assert json.loads(text) == line
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "clocks", "gpu_launches", "cpu_baseline"):
        assert line[key] == full[key]
    for key in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert line["e2e"][key] == full["e2e"][key]
    assert line["sweep33"]["CX"] == [1234.57, 0.988]
    assert full["sweep30"]["rows"]  # the full objects are left as they are


def test_objects_that_were_not_run():
    full = _full()
    for key in ("sweep30", "sweep33", "batch", "qft20", "measure28", "adjoint", "parity", "e2e"):
        full[key] = None
    assert all(bench.headline(full)[k] is None for k in ("sweep30", "batch", "e2e"))
