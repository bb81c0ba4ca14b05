"""Row gathers at every width from one byte to beyond the widest rule, from columns at every alignment, with
indices out of range, row counts around a block, and outputs that are not 16-byte aligned."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [*range(1, 36), 47, 48, 49, 63, 64, 65, 96, 100, 127, 128, 129, 160, 161, 255, 1000, 4096, 4097])
@pytest.mark.parametrize("n", [1, 7, 255, 256, 257, 1500])
def test_rows(w, n):
    from tqpk import _lib as L
    lib = L.load()
    rng = np.random.default_rng(w * 1000 + n)
    n_src = 40
    raw = torch.from_numpy(rng.integers(0, 256, n_src * w + 64).astype(np.uint8)).cuda()
    idx = rng.integers(0, n_src, n)
    idx[rng.random(n) < 0.1] = n_src - 1
    idx[rng.random(n) < 0.1] = 0
    bad = rng.random(n) < 0.1
    idx[bad] = rng.choice([-1, -64, n_src, n_src + 5, 1 << 50], bad.sum())
    di = torch.from_numpy(idx).cuda()
    ok = (idx >= 0) & (idx < n_src)
    for start, off in ((0, 0), (1, 0), (2, 16), (3, 0), (16, 5), (13, 1)):
        src = raw[start:start + n_src * w].cpu().numpy().reshape(n_src, w)
        want = np.where(ok[:, None], src[np.where(ok, idx, 0)], 0)
        out = torch.full((n * w + 64,), 77, dtype=torch.uint8, device="cuda")
        L.check(lib.tqpk_gather_rows(raw.data_ptr() + start, n_src, w, di.data_ptr(), n, out.data_ptr() + off, None), "gather")
        got = out.cpu().numpy()
        np.testing.assert_array_equal(got[off:off + n * w].reshape(n, w), want)
        assert (got[:off] == 77).all() and (got[off + n * w:] == 77).all()


def test_a_power_of_two_width_is_no_slower_than_its_neighbours():
    """Rows of 128 bytes once met in one bank of shared memory: 425 us for 750 K of them, 80 bytes 77."""
    from tqpk.ops import gather_rows
    n = 1_500_000
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    best = {}
    for w in (120, 128):
        col = torch.randint(0, 100, (n, w), generator=g, device="cuda").to(torch.int8)
        idx = torch.randint(0, n, (n // 2,), generator=g, device="cuda")
        gather_rows(col, idx)
        best[w] = 1e9
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(4):
                gather_rows(col, idx)
            e1.record()
            torch.cuda.synchronize()
            best[w] = min(best[w], e0.elapsed_time(e1) / 4)
    assert best[128] < 1.4 * best[120]
