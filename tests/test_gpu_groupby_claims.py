"""Sparse group-bys where many threads reach for the same slots: few groups whose keys lie far apart,
rows in any order and stored by their key, with and without a filter, against numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 2, 50, 1000, 90_000])
@pytest.mark.parametrize("stored", [False, True])
@pytest.mark.parametrize("n", [4096, 250_001])
def test_slots_claimed_by_many_threads(groups, stored, n):
    from tqpk.operators import tqp_hash_aggregate
    from tqpk.variable import Variable
    rng = np.random.default_rng(groups * 31 + n)
    key = rng.integers(0, groups, n)
    if stored:
        key.sort()
    key = key * ((1 << 40) // groups) - (1 << 30)
    val = rng.integers(-1000, 1000, n).astype(np.float64)             # sums are exact in any order
    tg = {1: Variable(torch.from_numpy(key).cuda(), "int"), 2: Variable(torch.from_numpy(val).cuda(), "float")}
    tqp_hash_aggregate(True, tg, {"is partial": False, "keys": ["k#1"], "input ids": [1, 2], "out agg ids": [302, 303],
                                  "results": ["k#1", [[["sum", ["v#2"]], "#", "301"], "AS", "s#302"],
                                              [[["count", ["v#2"]], "#", "304"], "AS", "c#303"]]}, None, None, "a")
    k, inverse = np.unique(key, return_inverse=True)
    np.testing.assert_array_equal(tg[1].tensor.reshape(-1).cpu().numpy(), k)
    np.testing.assert_array_equal(tg[302].tensor.reshape(-1).cpu().numpy(), np.bincount(inverse, val))
    np.testing.assert_array_equal(tg[303].tensor.reshape(-1).cpu().numpy(), np.bincount(inverse, val != -64))  # -64: null
