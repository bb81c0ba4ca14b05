"""Joins at the ends of their forms: a build side whose mask leaves a handful of many rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [1, 1 << 40])
def test_few_repeated_build_keys_out_of_many_rows(spread):
    """The build rows of a repeated key are listed from the mask, whose scan needs scratch for all rows,
    not for the few that pass."""
    from tqpk.ops import join_build, join_probe
    nb = 40_000_000
    keys = torch.arange(nb, dtype=torch.int64 if spread > 1 else torch.int32, device="cuda") // 2 * spread
    rows = [5, 777_776, 777_777, nb - 2, nb - 1]
    mask = torch.zeros(nb, dtype=torch.bool, device="cuda")
    mask[rows] = True
    b = join_build(keys, mask)
    probe = torch.tensor([388_888, 3, 2, (nb - 1) // 2], dtype=torch.int64, device="cuda") * spread
    bi, pi = join_probe(b, probe)
    np.testing.assert_array_equal(pi.cpu().numpy(), [0, 0, 2, 3, 3])
    np.testing.assert_array_equal(bi.cpu().numpy(), [777_776, 777_777, 5, nb - 2, nb - 1])
