"""The radix sort at the edges of its tiles and dispatch rules against numpy's stable lexsort: one CTA
up to 2048 rows, one cluster up to 98304 (four rows a thread, or twelve above 32768), 4096-row tiles up to 1228800 rows, 6144-row tiles above; keys whose varying digits lie
in the low half, the high half, both or nowhere, and more of them than a key is sorted by; several keys
in one call."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 2048, 2049, 4095, 4096, 4097, 32_768, 32_769, 98_304, 98_305, 1_228_800, 1_228_801, 1_234_944, (1 << 21) + 8193]


def _image(a, desc):
    """Order-preserving integers of a key column, one or more per row (most significant first)."""
    if a.ndim == 2:
        cols = [a[:, j].astype(np.int64) for j in range(a.shape[1])]
    elif a.dtype == np.float64:
        b = np.where(a == 0, 0.0, a)
        u = b.view(np.uint64).copy()
        neg = u >> np.uint64(63) == 1
        v = np.where(neg, ~u, u | np.uint64(1 << 63))
        v[np.isnan(a)] = np.uint64(2**64 - 2)
        cols = [(v ^ np.uint64(1 << 63)).view(np.int64)]
    else:
        cols = [a.astype(np.int64)]
    return [~c for c in cols] if desc else cols


def _expected(keys, descs):
    cols = [c for k, d in zip(keys, descs) for c in _image(k, d)]
    return np.lexsort(cols[::-1])


def _check(keys, descs, perm=None):
    from tqpk.ops import argsort_keys
    dev = [torch.from_numpy(k).cuda() for k in keys]
    if perm is None:
        exp = _expected(keys, descs)
        got = argsort_keys(dev, descs)
    else:
        exp = perm[_expected([k[perm] for k in keys], descs)]
        got = argsort_keys(dev, descs, torch.from_numpy(perm).cuda())
    np.testing.assert_array_equal(got.cpu().numpy(), exp)


@pytest.mark.parametrize("n", SIZES)
def test_sizes(n):
    rng = np.random.default_rng(n)
    _check([rng.integers(0, max(2, n // 3), n).astype(np.int64)], [bool(n & 1)])
    f = rng.integers(-3000, 3000, n) * 0.25
    f[: min(n, 4)] = [-0.0, 0.0, np.nan, np.inf][: min(n, 4)]
    _check([f, rng.integers(-5, 5, n).astype(np.int32)], [True, False], rng.permutation(n))


@pytest.mark.parametrize("n", [2000, 5000, 300_001])
@pytest.mark.parametrize("make", [lambda r, n: r.integers(-2**40, 2**40, n) << 20, lambda r, n: r.integers(0, 300, n) << 34,
                                  lambda r, n: np.full(n, -7), lambda r, n: r.integers(-64, 1, n),
                                  lambda r, n: r.integers(-2**63, 2**63 - 1, n)])
def test_varying_digits(make, n):
    rng = np.random.default_rng(7)
    k = make(rng, n).astype(np.int64)
    for desc in (False, True):
        _check([k], [desc])


@pytest.mark.parametrize("n", [1500, 2049, 27_600, 60_000, 150_001])
def test_many_keys(n):
    rng = np.random.default_rng(n)
    words = np.frombuffer(b"BRAND-11BRAND-12BRAND-45LARGE TI", np.int8).reshape(4, 8)
    text = np.zeros((n, 25), np.int8)
    text[:, 3:11] = words[rng.integers(0, 4, n)]
    text[:, 17:25] = words[rng.integers(0, 4, n)]
    raw = rng.integers(0, 256, (n, 3)).astype(np.uint8)
    keys = [rng.integers(0, 5, n).astype(np.int64), text, raw, rng.integers(-100, 100, n).astype(np.int8),
            rng.integers(0, 3, n).astype(np.uint8), rng.integers(0, 9, n).astype(np.int32)]
    _check(keys, [True, False, True, True, False, False])
    _check(keys[1:4], [True, False, False], rng.integers(0, n, n))     # rows may repeat


@pytest.mark.parametrize("n", [5000, 98_305, 1_228_800, 1_228_801])
@pytest.mark.parametrize("make", [
    lambda r, n: r.integers(90000, 10495001, n) / 100.0,                      # decimals: equal rows beside each other
    lambda r, n: r.random(n),                                                 # runs of two or three rows to reorder
    lambda r, n: (1 << 52) * (r.integers(0, 3, n) + 1.0) + r.integers(0, 9, n),   # long runs out of order
    lambda r, n: np.where(r.integers(0, 50, n) > 0, 0.07, r.random(n)),       # a long run of equal rows
])
def test_keys_of_more_digits_than_are_sorted_by(make, n):
    rng = np.random.default_rng(11)
    f = make(rng, n).astype(np.float64)
    _check([f], [True])
    _check([rng.integers(0, 3, n).astype(np.int32), f], [False, False], rng.permutation(n))


@pytest.mark.parametrize("n", [3000, 40_000, 150_001])
@pytest.mark.parametrize("dtype", [np.int8, np.uint8])
def test_text_widths(n, dtype):
    """Words cut short by the row's end, rows at every alignment, every byte value, both orders."""
    rng = np.random.default_rng(n)
    for w in (2, 3, 7, 8, 9, 10, 11, 16, 19, 25):
        t = rng.integers(0, 256, (n, w)).astype(np.uint8).view(dtype)
        t[:, : w // 2] = t[: 3, : w // 2][rng.integers(0, 3, n)]           # few values in front: ties decided behind
        for desc in (False, True):
            _check([t], [desc])
    t = np.zeros((n, 9), dtype)
    t[:, 8] = rng.integers(60, 70, n)
    _check([t], [True])


def test_too_many_words_raise():
    from tqpk.ops import argsort_keys
    wide = torch.zeros((3000, 8 * 33), dtype=torch.int8, device="cuda")
    with pytest.raises(NotImplementedError):
        argsort_keys([wide], [False])


@pytest.mark.parametrize("n", [1, 300, 4096, 4097, 98_305, 300_001])
@pytest.mark.parametrize("limit", [1, 10, 255, 256])
def test_topk_by_several_keys(n, limit):
    """Few ties, ties at the cut, a first key that ties everywhere, text keys, NaN and both zeros."""
    from tqpk.ops import topk_keys
    rng = np.random.default_rng(n + limit)
    price = rng.integers(90000, 10495001, n) / 100.0
    coarse = rng.integers(0, 4, n) * 0.5
    coarse[: min(n, 3)] = [-0.0, np.nan, 0.0][: min(n, 3)]
    text = np.zeros((n, 11), np.int8)
    text[:, 4] = rng.integers(0, 3, n)
    text[:, 10] = rng.integers(-2, 2, n)
    ids = rng.permutation(n).astype(np.int64)
    same = np.full(n, 3, np.int32)
    for keys, descs in (([price, ids], [True, False]), ([coarse, same, price], [False, True, True]),
                        ([same, coarse, text], [True, True, False]), ([text, coarse], [True, False]),
                        ([same, coarse], [False, False])):
        got = topk_keys([torch.from_numpy(k).cuda() for k in keys], descs, limit)
        np.testing.assert_array_equal(got.cpu().numpy(), _expected(keys, descs)[:limit])


@pytest.mark.parametrize("n", [2049, 8193, 32_768, 32_769, 98_304])
@pytest.mark.parametrize("first", ["int", "text"])
def test_rows_that_come_in_order(n, first):
    """The cluster leaves out the keys by which the rows already stand in order: all of them, or those
    behind the first column, here as groups come out of an aggregate.  One pair out of order anywhere
    (inside a CTA's rows, across two CTAs, at the end) is a full sort again."""
    rng = np.random.default_rng(n)
    text = np.zeros((n, 11), np.int8)
    text[:] = np.frombuffer(b"a-c-e-g-i-k", np.int8)
    text[:, 9] = rng.integers(97, 110, n)
    keys = [text, rng.integers(0, 40, n).astype(np.int64), rng.integers(-9, 9, n) * 0.5]
    descs = [True, False, True]
    at = _expected(keys, descs)
    keys = [k[at] for k in keys]
    _check(keys, descs)                                                   # in order already
    if first == "int":
        lead, lead_desc = rng.integers(0, 300, n).astype(np.int64), True
    else:
        lead, lead_desc = rng.integers(97, 101, (n, 17)).astype(np.int8), False
    _check([lead] + keys, [lead_desc] + descs)                            # behind the first column
    rows = (n + 15) // 16                                                 # of one CTA
    for p in (0, rows - 1, 5 * rows - 1, min(rows + 600, n - 2), n - 2):
        other = [k.copy() for k in keys]
        for k in other:
            k[[p, p + 1]] = k[[p + 1, p]]
        _check(other, descs)
        _check([lead] + other, [lead_desc] + descs)
    perm = rng.permutation(n)
    back = [np.empty_like(k) for k in keys]
    for b, k in zip(back, keys):
        b[perm] = k
    _check(back, descs, perm)                                             # in order through the given rows


@pytest.mark.parametrize("n", [2049, 70_003, 2_200_001])
@pytest.mark.parametrize("make", [lambda r, n: r.integers(0, 2557, n).astype(np.int32), lambda r, n: r.integers(0, 3, n).astype(np.uint8),
                                  lambda r, n: np.full(n, 2.5), lambda r, n: np.where(r.integers(0, 900, n) == 0, np.nan, 1.0),
                                  lambda r, n: np.sort(r.integers(0, n // 50 + 1, n)), lambda r, n: -np.arange(n)])
def test_topk_of_few_values(make, n):
    """The k first of a column with many ties are the first rows of the stable order."""
    from tqpk.ops import topk_stable
    rng = np.random.default_rng(n)
    a = make(rng, n)
    d = torch.from_numpy(a).cuda()
    for desc in (False, True):
        exp = _expected([a], [desc])
        for k in (1, 10, 33, 100, 256):
            np.testing.assert_array_equal(topk_stable(d, k, desc).cpu().numpy(), exp[:k], err_msg=str((k, desc)))
