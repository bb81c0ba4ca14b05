"""Projections write four rows at a time: row counts around a thread's four and output widths of eight, four
and one bytes, against the oracle."""
import numpy as np
import pytest
import torch

from golden_io import assert_f64_close
from oracle import tqp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 1023, 4097, 1_000_003])
def test_row_counts(n):
    from tqpk.operators import tqp_project
    from tqpk.variable import Variable
    rng = np.random.default_rng(n)
    cols = {1: rng.integers(90000, 10495001, n) / 100.0, 2: rng.integers(0, 11, n) / 100.0,
            3: rng.integers(-50, 50, n).astype(np.int32), 4: rng.integers(-2**40, 2**40, n),
            5: rng.integers(0, 60, n).astype(np.uint8)}
    args = {"rename map": {},
            "used expr": [[[["p#1", "*", ["1", "-", "d#2"]], "AS", "a#12"]], [[["q#3", "+", "q#3"], "AS", "b#13"]],
                          [[["w#4", "-", "q#3"], "AS", "c#14"]], [[["u#5", "+", "u#5"], "AS", "e#15"]]],
            "materialized in": [1, 2, 3, 4, 5], "materialized out": [12, 13, 14, 15]}
    tg = {c: Variable(torch.from_numpy(a).cuda(), "float" if a.dtype == np.float64 else "int") for c, a in cols.items()}
    assert tqp_project(True, tg, args, None, None) == -1
    ref = O.tqp_project(cols, args)
    for oid in args["materialized out"]:
        got = tg[oid].tensor.cpu().numpy()
        assert got.dtype == ref[oid].dtype, (oid, got.dtype, ref[oid].dtype)
        (assert_f64_close if ref[oid].dtype == np.float64 else np.testing.assert_array_equal)(got, ref[oid])
