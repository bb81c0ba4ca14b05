"""Group-bys at the edges of the accumulation and emission tiles (256-row rounds, 4096-row tiles, 512- and
4096-slot tiles) against numpy: sparse (hash) and dense key spaces, filters that pass few, all or no rows."""
import numpy as np
import pytest
import torch

from golden_io import assert_f64_close

pytestmark = pytest.mark.gpu

RESULTS = [[[["sum", ["v#3"]], "#", "101"], "AS", "a#201"], [[["count", ["1"]], "#", "102L"], "AS", "a#202"],
           [[["min", ["w#4"]], "#", "103"], "AS", "a#203"], [[["max", ["v#3"]], "#", "104"], "AS", "a#204"],
           [[["avg", [["v#3", "*", ["1.0", "+", "w#4"]]]], "#", "105"], "AS", "a#205"]]


def _run(keys, v, w, mask):
    from tqpk.operators import tqp_hash_aggregate
    from tqpk.variable import Variable
    cols = {1: keys[0], 2: keys[1], 3: v, 4: w}
    tg = {c: Variable(torch.from_numpy(a).cuda(), "int") for c, a in cols.items()}
    args = {"is partial": False, "keys": ["a#1", "b#2"], "input ids": [1, 2, 3, 4],
            "results": ["a#1", "b#2"] + RESULTS, "out agg ids": [201, 202, 203, 204, 205]}
    if mask is not None:
        tg[900] = Variable(torch.from_numpy(mask).cuda(), "bool")
        args["mask map"] = {c: 900 for c in cols}
    tqp_hash_aggregate(True, tg, args, None, None, "a")
    return [tg[c].tensor.cpu().numpy().reshape(-1) for c in (1, 2, 201, 202, 203, 204, 205)]


def _check(keys, v, w, mask):
    got = _run(keys, v, w, mask)
    m = np.ones(v.size, bool) if mask is None else mask
    k = np.stack([keys[0][m].astype(np.int64), keys[1][m].astype(np.int64)], 1)
    u, inv = np.unique(k, axis=0, return_inverse=True)
    inv = inv.reshape(-1)
    g = len(u)
    np.testing.assert_array_equal(got[0], u[:, 0])
    np.testing.assert_array_equal(got[1], u[:, 1])
    cnt = np.bincount(inv, minlength=g)
    np.testing.assert_array_equal(got[3], cnt)
    mag = np.bincount(inv, np.abs(v[m]), g)
    assert_f64_close(got[2], np.bincount(inv, v[m], g), magnitude=mag)
    mn = np.full(g, np.iinfo(w.dtype).max, np.int64)
    np.minimum.at(mn, inv, w[m].astype(np.int64))
    np.testing.assert_array_equal(got[4], mn)
    mx = np.zeros(g)
    np.maximum.at(mx, inv, v[m])
    np.testing.assert_array_equal(got[5], mx)
    t = v[m] * (1.0 + w[m])
    assert_f64_close(got[6], np.bincount(inv, t, g) / cnt, magnitude=np.bincount(inv, np.abs(t), g) / cnt)


def _masks(rng, n):
    one = np.zeros(n, bool)
    one[n - 1] = True
    return [None, rng.integers(0, 7, n) == 0, one]


@pytest.mark.parametrize("n", [1, 255, 257, 4095, 4096, 4097, 300_001])
def test_sparse_keys(n):
    rng = np.random.default_rng(n)
    a = rng.integers(0, 200, n) * 1_000_003
    b = (a // 7 + rng.integers(0, 4, n) * 2500) % 10_000 + rng.integers(0, 2, n) * 5_000_000
    v, w = rng.integers(-5000, 5000, n) * 0.25, rng.integers(0, 50, n).astype(np.int32)
    for mask in _masks(rng, n):
        _check([a, b], v, w, mask)


@pytest.mark.parametrize("slots_a,slots_b", [(1, 1), (1, 511), (1, 512), (3, 171), (64, 64), (1, 4097), (700, 701)])
@pytest.mark.parametrize("n", [1, 5000, 200_000])
def test_dense_keys(n, slots_a, slots_b):
    rng = np.random.default_rng(n + slots_b)
    a = rng.integers(0, slots_a, n).astype(np.int32) - 3
    b = rng.integers(0, slots_b, n)
    v, w = rng.integers(-5000, 5000, n) * 0.25, rng.integers(0, 50, n).astype(np.int32)
    for mask in _masks(rng, n):
        _check([a, b], v, w, mask)


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 60_000])
@pytest.mark.parametrize("width", [1, 3, 8, 10, 25])
def test_key_codes_of_text(n, width):
    """Codes in key-tuple order of a text key (rows at every alignment) beside a float key, under masks."""
    from tqpk.ops import encode_keys
    rng = np.random.default_rng(n + width)
    words = rng.integers(-128, 128, (40, width)).astype(np.int8)
    words[20:, : width // 2] = words[:20, : width // 2]
    t = words[rng.integers(0, 40, n)]
    f = rng.integers(-2, 3, n) * 0.5
    f[f == 0] = np.where(rng.integers(0, 2, (f == 0).sum()) > 0, 0.0, -0.0)
    dev = [torch.from_numpy(t).cuda().reshape(n, width), torch.from_numpy(f).cuda()]
    for mask in _masks(rng, n):
        m = np.ones(n, bool) if mask is None else mask
        codes, reps, g = encode_keys(dev, torch.from_numpy(mask).cuda() if mask is not None else None)
        rows = np.concatenate([t.astype(np.float64), (f + 0.0)[:, None]], 1)[m]
        u, inv = np.unique(rows, axis=0, return_inverse=True)
        assert g == len(u)
        np.testing.assert_array_equal(codes.cpu().numpy()[m], inv.reshape(-1))
        r = reps.cpu().numpy()
        assert m[r].all()
        np.testing.assert_array_equal(np.concatenate([t.astype(np.float64), (f + 0.0)[:, None]], 1)[r], u)
