"""The benchmark's output: one JSON line, the last, with the headline, the end-to-end value,
clocks and the dominant kernel's roofline, short enough (under 4,000 characters) for a
captured tail of the output to hold it whole; the legs stand before it."""
import json

import bench


def test_last_line_is_short_and_complete(capsys):
    args = type("A", (), {"models": 256, "sim_steps": 500})
    line = {"metric": bench.METRIC, "value": 1.9e5, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 1.0, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64+f32",
            "data": "synthetic", "config": bench.workload_config(args, [(0, 0, 700)] * 256),
            "e2e": {"value": 1.6e5, "unit": bench.UNIT, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2},
            "gpu_launches": 1000, "clocks": {"sm_mhz": 2070, "sm_max_mhz": 2070, "reasons": []},
            "roofline": {"bound": "hbm", "achieved": 1.0, "note": "n" * 400},
            "cpu_baseline": {"value": 1.0, "sample": "s" * 300},
            "served": {"requests": ["r" * 100] * 60}, "superelement_chain": {"workload": "w" * 5000}}
    bench.print_result(line)
    out = capsys.readouterr().out.splitlines()
    assert len(out[-1]) < 4000
    last = json.loads(out[-1])
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert last[key] == line[key]
    assert [o for o in out if o.startswith("{")] == [out[-1]]
    legs = dict(o[4:].split(": ", 1) for o in out[:-1])
    assert {k: json.loads(v) for k, v in legs.items()} == {k: line[k] for k in ("served", "superelement_chain")}
