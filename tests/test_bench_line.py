"""The bench's output: one JSON line, the last, short enough for a reader that keeps
the output's tail alone, with the headline fields; every leg's results before it."""

import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))


def test_headline_is_the_one_json_line_and_short(capsys):
    import bench
    rate = 1718281828.4590452
    line = {
        "metric": bench.METRIC, "value": rate, "unit": bench.UNIT, "n_gpus": 1, "steps": 60,
        "warmup": 3, "ms_per_step": 9.876543210123456, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded HIT field; no dataset)",
        "config": bench.config_dict(8, 123.45678901234567),
        "e2e": {"value": rate, "unit": bench.UNIT, "h2d_bytes_per_step": 671088640,
                "d2h_bytes_per_step": 671088640, "steps": 60, "how": "x" * 500,
                "serial": {"value": rate}},
        "gpu_launches": 1080,
        "clocks": {"sm_mhz": 1815.0, "sm_min_mhz": 1665.0, "sm_max_mhz": 1965.0,
                   "power_w_median": 912.34567, "power_w_max": 1001.234, "samples": 1234,
                   "source": "nvml",
                   "reasons": ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown",
                               "sw_power_cap"]},
        "roofline": {"bound": "fp64", "achieved": 21.123456789012345, "peak": 34.2,
                     "unit": "TFLOP/s", "frac": 0.61803398874989, "kernel": "k" * 300},
        "mixed": None, "schemes": {"leg": list(range(4000))}, "cpu_baseline": None,
    }
    bench.report(line)
    out = capsys.readouterr().out.splitlines()
    parsed = []
    for text in out:
        try:
            parsed.append(json.loads(text))
        except ValueError:
            pass
    assert len(parsed) == 1 and parsed[0] == json.loads(out[-1])
    got = parsed[0]
    assert len(out[-1]) < 2048
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config",
                "gpu_launches"):
        assert got[key] == line[key]
    assert {k: got["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step",
                                       "d2h_bytes_per_step")} == \
        {k: line["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step")}
    assert {k: got["clocks"][k] for k in ("sm_mhz", "sm_max_mhz", "reasons")} == \
        {k: line["clocks"][k] for k in ("sm_mhz", "sm_max_mhz", "reasons")}
    # the legs are all there, on the line before
    assert json.loads(out[-2].split(" ", 1)[1])["schemes"] == line["schemes"]


def test_stated_sweep_traffic_is_not_below_the_compulsory_bytes():
    import bench
    # per cell: x reads the state and writes the RHS and six primitives; y and z read
    # the state, u_n, p, c and the RHS and write the RHS
    least = 256 ** 3 * 8 * ((5 + 11) + 2 * (5 + 3 + 5 + 5)) / 3
    assert least <= bench.INV_TRAFFIC_BYTES < 1.25 * least
