"""The summary of the decode call's time stamps (bench.py --decode-trace), without a GPU."""
import importlib.util
import os

import numpy as np

from conftest import ROOT


def test_points_of_calls_with_and_without_a_merge_pass():
    spec = importlib.util.spec_from_file_location("bench_under_test", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    names = ["entry", "set-up", "first tile"]
    assert bench.trace_points(np.zeros((0, 8), np.int64), names, 0, True) == {}  # one launch of clusters: nothing merges behind it
    stamps = np.zeros((3, 8), np.int64)
    stamps[:, 0] = [5000, 6000, 9000]
    stamps[1, 2] = 7500  # the only CTA with a tile; no CTA passes the second point
    assert bench.trace_points(stamps, names, 5000, True) == {"entry": [0.0, 1.0, 4.0], "first tile": [2.5, 2.5, 2.5]}
    assert bench.trace_points(stamps, names, 5000, False) == {"entry": [1.0, 4.0], "first tile": [2.5, 2.5]}
