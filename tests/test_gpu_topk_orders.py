"""The stable top-k over columns as tables store them: sorted, reversed, in sorted runs, of few values,
at limits on both sides of its rules (32 and 256) and of a warp's and a CTA's share of them."""
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stored(kind, n, rng):
    i = np.arange(n)
    return {"sorted": i, "reversed": n - i, "halves": np.where(i % 2 == 0, i, n - i),
            "runs": i * 2654435761 % n // 9700 * 9700 + i % 9700, "dates": np.sort(rng.integers(0, 2557, n)),
            "dates reversed": np.sort(rng.integers(0, 2557, n))[::-1].copy(),
            "two values": np.minimum(i // 100, 1), "one value": np.zeros(n, np.int64),
            "parts": i % (n // 62 + 1) * 62 + i // (n // 62 + 1), "parts reversed": -(i % (n // 62 + 1)) * 62 + i // (n // 62 + 1),
            "strided": np.where(i % 1024 < 4, rng.integers(0, 1000, n), 1 << 40),
            "lowest": np.where(i % 1000 == 999, np.iinfo(np.int64).min, i)}[kind].astype(np.int64)


KINDS = ["sorted", "reversed", "halves", "runs", "parts", "parts reversed", "dates", "dates reversed", "two values",
         "one value", "strided", "lowest"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [5, 257, 300_001, 2_200_000])
@pytest.mark.parametrize("k", [1, 10, 32, 33, 100, 256])
def test_topk_of_stored_orders(kind, n, k):
    from tqpk.ops import topk_stable
    rng = np.random.default_rng(n + k)
    key = _stored(kind, n, rng)
    perm = rng.permutation(n)
    dev, dperm = torch.from_numpy(key).cuda(), torch.from_numpy(perm).cuda()
    for desc in (False, True):
        image = ~key if desc else key
        order = np.argsort(image, kind="stable")[:k]
        np.testing.assert_array_equal(topk_stable(dev, k, desc).cpu().numpy(), order)
    order = perm[np.argsort(key[perm], kind="stable")[:k]]
    np.testing.assert_array_equal(topk_stable(dev, k, False, dperm).cpu().numpy(), order)
    if kind != "strided":
        f = torch.from_numpy(key.astype(np.float64)).cuda()
        np.testing.assert_array_equal(topk_stable(f, k).cpu().numpy(), np.argsort(key.astype(np.float64), kind="stable")[:k])


@pytest.mark.parametrize("kind", ["sorted", "reversed", "runs", "parts", "parts reversed", "dates", "dates reversed"])
@pytest.mark.parametrize("k", [10, 100, 256])
def test_a_stored_order_is_not_walked_by_one_cta(kind, k):
    """Two keys and a limit (tqp_sort's route): milliseconds to half a second when the first key's stored
    order puts whole groups under the cut, ~0.15 ms otherwise."""
    from tqpk.ops import topk_keys
    n = 6_000_000
    rng = np.random.default_rng(3)
    key = _stored(kind, n, rng)
    cols = [torch.from_numpy(key).cuda(), torch.from_numpy(rng.permutation(n)).cuda()]
    got = topk_keys(cols, [False, True], k)
    best = 1.0
    for _ in range(5):
        torch.cuda.synchronize()
        t = time.perf_counter()
        topk_keys(cols, [False, True], k)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    assert best < 2e-3
    exp = np.lexsort([-cols[1].cpu().numpy(), key])[:k]
    np.testing.assert_array_equal(got.cpu().numpy(), exp)
