"""A join's condition columns are waited for before anything reads them: binding a strided column to the
pair predicate copies it, and a column that is still arriving from another stream must not be copied."""
import torch

from tqpk.operators import hashjoin as H
from tqpk.variable import Variable


def test_condition_columns_are_waited_for_before_the_predicate_binds_them(monkeypatch):
    waited, bound = set(), []
    monkeypatch.setattr(H, "wait_ready", lambda *vs: waited.update(id(v) for v in vs))
    real = H.compile_filter

    def compile_filter(tree, cols, *a, **k):
        bound.append({c: id(left.get(c) or right.get(c)) in waited for c in cols})
        return real(tree, cols, *a, **k)

    monkeypatch.setattr(H, "compile_filter", compile_filter)
    left = {1: Variable(torch.arange(12, dtype=torch.int64)[::2], "int")}            # strided
    right = {2: Variable(torch.arange(18, dtype=torch.int64)[::3], "int"), 3: Variable(torch.arange(6), "int")}
    pred, probe_cols = H._pair_predicate(left, right, [["l#1", "=", "r#2"], ["r#3", "<", "5"]])
    assert bound == [{1: True, 2: True, 3: True}]
    assert [c for i, c in enumerate(pred.col_ids) if probe_cols >> i & 1] == [2, 3]
