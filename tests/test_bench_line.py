"""The line that bench.py prints stays short enough to be read from the end of the
output: the long sections go to stderr, their key figures stay in config, and the
fields that a reader asks for stay in the line."""
import importlib.util
import json
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_line", ROOT / "bench.py")
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_long_sections_leave_the_line(bench):
    keep = {"metric": "m", "value": 1.0, "unit": "u", "n_gpus": 1, "steps": 2, "warmup": 3, "ms_per_step": 1.0,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "e2e": {"value": 1.0}, "gpu_launches": 4, "roofline": {"frac": 0.5}, "clocks": {"sm_mhz": 2070.0},
            "speedup_vs_plain": 1.5, "cpu_baseline": {"value": 20.0}}
    table = [["bvh4_f16", k, 1.0, 2.0] for k in range(400)]
    line = dict(keep, config={"workload": "w", **{f"key_{k}": 1.25 for k in range(120)}},
                **{k: {"mrays_s": 1.0, "table": table} for k in bench.DETAIL_SECTIONS})
    assert len(json.dumps(line)) > 50000
    details = bench.detach_details(line)
    assert set(details) == set(bench.DETAIL_SECTIONS) and details["precision"]["table"] == table
    assert set(line) == set(keep) | {"config"} and {k: line[k] for k in keep} == keep
    assert len(json.dumps(line)) < 8000


def test_a_line_without_sections_is_unchanged(bench):
    line = {"value": 1.0, "config": {}}
    assert bench.detach_details(line) == {} and line == {"value": 1.0, "config": {}}


def test_both_are_printed(bench):
    text = (ROOT / "bench.py").read_text()
    at = text.index("details = detach_details(line)")
    assert text.index("summarize(line)\n") < at < text.index("print(json.dumps(line), flush=True)\n    replicas.finish")
