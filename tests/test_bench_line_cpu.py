"""bench.py's headline line stays short whatever the number of steps: a reader that
keeps the last few kB of the output gets it whole."""
import importlib.util
import json
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def _bench():
    spec = importlib.util.spec_from_file_location("bench", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_line_is_short():
    steps = 500
    x = 1234.56789012345678
    variant = {"ms_per_step": x, "max_ms": x, "ms": [x] * steps, "iters": [3000] * steps, "timesteps": f"1..{steps}",
               "rel_residual": [9.9e-11] * steps, "loop_ms": [x] * steps, "launches": [18] * steps,
               "ms_per_iteration": x, "algorithmic_gbs_per_iteration": x, "warm": [3] * steps,
               "r0_plain": [x] * steps, "r0_pred": [x] * steps, "warm_coef": [[x] * 8] * steps,
               "refinements": [8] * steps, "final_summary": (x, x, x, x),
               "final_field_vs_fp64": {"u_max_rel_diff": x, "summary_rel_diff": dict.fromkeys("abcd", x)}}
    line = {"metric": "m" * 80, "value": x, "unit": "ms", "n_gpus": 1, "steps": steps, "warmup": 5, "ms_per_step": x,
            "higher_is_better": False, "config": {"workload": "w" * 200, "n": 8192},
            "clocks": {"sm_mhz": 2070.0, "reasons": []},
            "e2e": {"value": x, "unit": "ms", "h2d_bytes_per_step": 1074790656, "d2h_bytes_per_step": 537395328,
                    "ms": [x] * steps, "iters": [3000] * steps, "host_wall_ms": [{"upload": x}] * steps},
            "gpu_launches": 326, "variants": {f"variant_{k}": dict(variant) for k in range(5)},
            "roofline": {"frac": x, "kernels": {"a": {"ms": x, "gbs": x, "frac": x}}}}
    out = _bench().short_line(line)
    text = json.dumps(out)
    assert len(text) < 4096
    d = json.loads(text)
    assert d["clocks"] == {"sm_mhz": 2070.0, "reasons": []}
    assert d["value"] == d["ms_per_step"] == x and d["e2e"]["h2d_bytes_per_step"] == 1074790656
    v = d["variants"]["variant_0"]
    assert v["iters"] == 3000 * steps and v["rel_residual_max"] == 9.9e-11 and abs(v["ms_per_iteration"] - x) < 1e-3
    assert line["variants"]["variant_0"]["iters"] == [3000] * steps  # the whole line is left as it was
