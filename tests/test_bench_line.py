"""The benchmark's output line: one JSON line of a few KB with the contract's keys
untouched, the whole record on stderr."""
import json

import bench


def test_line_stays_short_and_keeps_the_contract(capsys):
    row = {"n": 16, "order": 2, "rel_l2": 1 / 3, "fp64": {"gdofs": 2 / 3, "runs": [1.0, 2.0]}}
    line = {"metric": bench.METRIC, "value": 100 / 3, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 1 / 3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": bench.config_dict(1), "gpu_launches": 100,
            "e2e": {"value": 1 / 7, "unit": "GDOF/s", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2},
            "roofline": {"frac": 1 / 3, "stage_ms": [1 / 3] * 5}, "cpu_baseline": {"sample": "x" * 200},
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}, "fp64_plain": None,
            "poisson": {"note": "y" * 500, "cases": {"a": {"speedup": 10 / 3, "fp64": {"runs": row}}}},
            "equal_error": {"workload": "w", "rows": [row] * 200, "min_error": {"fp64": 1 / 3}}}
    bench.print_result(line)
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < 4096
    got = json.loads(out)
    assert list(got) == list(line)
    for k, v in line.items():
        if k in bench.WHOLE or not isinstance(v, dict):
            assert got[k] == v, k
    assert got["poisson"] == {"cases": {"a": {"speedup": 3.33333}}}
    assert got["equal_error"] == {"workload": "w", "min_error": {"fp64": 0.333333}}
    assert json.loads(err)["details"] == line
