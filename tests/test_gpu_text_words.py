"""Everything that reads text rows by words, at every width up to four words: sort words, the sort's
images in its one-CTA, cluster and tiled forms, key codes, row gathers.  A row's last word holds one to
eight bytes, and the rows lie at every alignment."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(n, w, dtype, rng):
    t = rng.integers(0, 256, (n, w)).astype(np.uint8)
    t[:, : w - 1] = t[:5, : w - 1][rng.integers(0, 5, n)]            # the last byte decides
    return t.view(dtype)


@pytest.mark.parametrize("w", range(2, 34))
@pytest.mark.parametrize("dtype", [np.int8, np.uint8])
def test_every_width(w, dtype):
    from tqpk.ops import argsort_keys, encode_keys, gather_rows, string_words
    rng = np.random.default_rng(w)
    for n in (1500, 20_011, 120_003):
        t = _rows(n, w, dtype, rng)
        dev = torch.from_numpy(t).cuda()
        cols = [t[:, j].astype(np.int64) for j in range(w)]
        order = np.lexsort(cols[::-1])
        for word in range((w + 7) // 8):
            v = np.zeros(n, np.uint64)
            for j in range(8):
                c = word * 8 + j
                b = (t[:, c].view(np.uint8) ^ (0x80 if dtype == np.int8 else 0)) if c < w else np.zeros(n, np.uint8)
                v = (v << np.uint64(8)) | b.astype(np.uint64)
            got = string_words(dev, word).cpu().numpy()
            np.testing.assert_array_equal(got, (v ^ np.uint64(1 << 63)).view(np.int64))
        np.testing.assert_array_equal(argsort_keys([dev], [False]).cpu().numpy(), order)
        idx = rng.integers(0, n, n)
        np.testing.assert_array_equal(gather_rows(dev, torch.from_numpy(idx).cuda()).cpu().numpy(), t[idx])
        codes, reps, groups = encode_keys([dev])
        step = (np.diff(t[order].astype(np.int64), axis=0) != 0).any(axis=1)
        want = np.empty(n, np.int64)
        want[order] = np.concatenate([[0], np.cumsum(step)])
        assert groups == want.max() + 1
        np.testing.assert_array_equal(codes.cpu().numpy(), want)
        np.testing.assert_array_equal(t[reps.cpu().numpy()], t[order][np.concatenate([[True], step])])
