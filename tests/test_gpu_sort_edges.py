"""The radix sort's finishing passes and calling forms: rows that four digits leave out of order, at
every place of a warp."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("desc", [False, True])
@pytest.mark.parametrize("run", [2, 3, 5])
@pytest.mark.parametrize("shift", range(5))
def test_out_of_order_neighbours_at_every_lane(shift, run, desc):
    """Runs of rows that agree in the key's four highest varying digits and come in the wrong order by the
    lower ones.  The rows are stored in the order of the high digits, so that a run's place in the table
    is its place in a warp of the check: pairs at lanes 30/31 and 31/0 among them."""
    from tqpk.ops import argsort_keys
    n = 131_072 + 77
    i = np.arange(n, dtype=np.int64)
    group = (i + run - shift % run) // run
    high = group * ((1 << 31) // (n // run + 2))                      # varies in four bytes
    low = (n - i) * 9973 % (1 << 20) if run == 5 else (n - i)
    key = (high << 24) + low
    if desc:
        key = -key
    got = argsort_keys([torch.from_numpy(key).cuda()], [desc]).cpu().numpy()
    np.testing.assert_array_equal(got, np.lexsort([-key if desc else key]))


@pytest.mark.parametrize("n", [7, 2048, 2049, 30_000, 98_304, 98_305, 300_000])
@pytest.mark.parametrize("entry", ["stable", "keys"])
def test_permutation_sorted_in_place(n, entry):
    """The permutation argument of a sort as its result too, as a loop over keys writes it; also shifted by
    some rows, and the key column itself."""
    import ctypes as C

    from tqpk import _lib as L
    lib = L.load()
    rng = np.random.default_rng(n)
    key = rng.integers(-(1 << 40), 1 << 40, n)
    key[rng.integers(0, n, n // 2)] = 17
    perm = rng.permutation(n)
    dev = torch.from_numpy(key).cuda()
    one = lambda t, *v: (t * len(v))(*v)                                                     # noqa: E731

    def sort(perm_in, out):
        if entry == "stable":
            ws = torch.empty(lib.tqpk_sort_workspace_bytes(n), dtype=torch.uint8, device="cuda")
            L.check(lib.tqpk_argsort_stable(dev.data_ptr(), L.I64, 1, perm_in, n, out, ws.data_ptr(), ws.numel(), None),
                    "sort")
        else:
            dt, w = one(C.c_int32, L.I64), one(C.c_int32, 0)
            ws = torch.empty(lib.tqpk_argsort_keys_workspace_bytes(n, 1, dt, w), dtype=torch.uint8, device="cuda")
            L.check(lib.tqpk_argsort_keys(1, one(C.c_void_p, dev.data_ptr()), dt, w, one(C.c_int32, 1), perm_in, n, out,
                                          ws.data_ptr(), ws.numel(), None), "sort")
        torch.cuda.synchronize()

    expected = perm[np.lexsort([-key[perm]])]
    buf = torch.full((n + 64,), -1, dtype=torch.int64, device="cuda")
    for shift in (0, 32):
        torch.cuda.synchronize()
        buf[:n] = torch.from_numpy(perm).cuda()
        torch.cuda.synchronize()
        sort(buf.data_ptr(), buf.data_ptr() + 8 * shift)
        np.testing.assert_array_equal(buf[shift:shift + n].cpu().numpy(), expected)
    sort(None, dev.data_ptr())
    np.testing.assert_array_equal(dev.cpu().numpy(), np.lexsort([-key]))
