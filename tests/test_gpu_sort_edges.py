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
