"""bench.py's CPU baseline where the reference library is not built: the oracle's
restatement is timed in its place, and says so."""
from __future__ import annotations

import numpy as np

import bench
from oracle import oracle as O
from ultrahigh_ann_b200 import synthetic


class _OracleIndex:
    def __init__(self, rows):
        self.rows = rows

    def query_batch(self, queries, count, output, workspace):
        output[:] = O.exact("l2", self.rows, queries)[0]
        return output


def test_baseline_without_the_reference_library(monkeypatch, oracle_module):
    monkeypatch.setattr(O, "ref_available", lambda: False)
    ds = synthetic.row_dataset(rows=60, classes=5, queries=70, d=500, seed=1)
    line, agreement = bench.cpu_baseline(ds, _OracleIndex(ds.rows), None, 1)
    assert line["kind"] == "restatement" and line["value"] > 0
    assert agreement == 1.0


def test_agreement_counts_wrong_rows(monkeypatch, oracle_module):
    monkeypatch.setattr(O, "ref_available", lambda: False)
    ds = synthetic.row_dataset(rows=60, classes=5, queries=64, d=500, seed=1)
    index = _OracleIndex(np.roll(ds.rows, 1, axis=0))
    _, agreement = bench.cpu_baseline(ds, index, None, 1)
    assert agreement == 0.0
