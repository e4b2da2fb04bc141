"""The benchmark's result line stays short; the other workloads' whole lines go to standard error (CPU)."""

from __future__ import annotations

import inspect
import json
import sys

from conftest import ROOT

sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


def test_one_line_on_standard_output(capsys) -> None:
    line = {"metric": bench.METRIC, "value": 1.0}
    details = {"bisect": {"value": 2.0, "worst_cases": ["x" * 4000]}, "lensing": {"value": 3.0}}
    bench.emit(line, details)
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and json.loads(out) == line
    assert json.loads(err) == {"details": details}
    bench.emit(line, {})
    out, err = capsys.readouterr()
    assert json.loads(out) == line and err == ""


def test_long_results_are_details() -> None:
    """The blocks of several KB (3.3 to 4.2 each in a run of the default workload) are none of the line's own."""
    source = inspect.getsource(bench.run_ours)
    for name in ('"bisect"', '"lensing"', 'f"mixed_vs_plain_{name[-4:]}"'):
        assert f"details[{name}] = " in source and f"extra[{name}]" not in source
