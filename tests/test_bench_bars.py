"""bench.py ends with an error when a record in its line misses the bar of its path."""
import copy
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402

GOOD = {
    "fp64": {"backward_error": 3.2e-16, "rel_err_vs_oracle": 6.0e-14},
    "mixed": {"backward_error": 4e-14, "rel_err_vs_oracle": 1.1e-11},
    "c3b": {"mixed": {"backward_error": 8.7e-14, "rel_err_vs_oracle": 1.2e-7},
            "fp64": {"backward_error": 4.1e-18, "rel_err_vs_oracle": 6.3e-14}},
    "e2e": {"last_step_parts": {"backward_error": 4e-14}, "fp64_last_step_parts": {"backward_error": 3e-16}},
    "hex20": {"mixed": {"backward_error": 2e-15}, "fp64": {"backward_error": 4.8e-16}},
    "indefinite": {"inertia_equal": True, "rel_err_vs_oracle": 3e-10},
    "unsymmetric": {"delayed_equal": True, "rel_err_vs_oracle": 1e-12},
    "assembly": {"bit_identical_to_oracle": True},
}


def test_a_right_line_is_printed(capsys):
    bench.finish(copy.deepcopy(GOOD))
    assert json.loads(capsys.readouterr().out) == GOOD


def test_without_the_oracle():
    assert bench.missed_bars({"fp64": {"backward_error": 1e-16, "rel_err_vs_oracle": None}}) == []


@pytest.mark.parametrize("path,value", [
    # an FP64 solution of the graded cube that a run once printed and accepted
    (("c3b", "fp64", "rel_err_vs_oracle"), 2.9207e-03), (("c3b", "fp64", "backward_error"), 3.4421e-06),
    (("c3b", "mixed", "backward_error"), 2e-12), (("fp64", "rel_err_vs_oracle"), float("nan")),
    (("e2e", "fp64_last_step_parts", "backward_error"), float("inf")), (("hex20", "fp64", "backward_error"), 1e-11),
    (("indefinite", "inertia_equal"), False), (("indefinite", "rel_err_vs_oracle"), 2e-9),
    (("unsymmetric", "rel_err_vs_oracle"), 1e-9), (("unsymmetric", "delayed_equal"), False),
    (("assembly", "bit_identical_to_oracle"), False)])
def test_a_missed_bar_ends_with_an_error(capsys, path, value):
    line = copy.deepcopy(GOOD)
    rec = line
    for key in path[:-1]:
        rec = rec[key]
    rec[path[-1]] = value
    with pytest.raises(SystemExit) as e:
        bench.finish(line)
    assert e.value.code not in (0, None) and ".".join(path) in str(e.value.code)
    printed = json.loads(capsys.readouterr().out)
    assert len(printed["missed_bars"]) == 1 and printed["missed_bars"][0].startswith(".".join(path))
