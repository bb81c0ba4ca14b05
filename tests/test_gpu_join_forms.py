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


@pytest.mark.parametrize("cmp", [-3, 6, 7, 1 << 20])
def test_a_condition_with_an_unknown_operator_holds_for_no_pair(cmp):
    """As in a filter; the operator is an index into the table that turns a comparison round only when it
    is one of that table's."""
    from tqpk import _lib as L
    from tqpk.ops import join_build, join_pairs
    from tqpk.predicate import compile_filter
    keys = torch.arange(600, device="cuda") // 3
    cols = {1: torch.zeros(600, dtype=torch.int64, device="cuda"), 2: torch.zeros(200, dtype=torch.int64, device="cuda")}
    cond = compile_filter(["b#2", "<", "a#1"], cols)
    cond.struct.insn[0].cmp = cmp
    side = sum(1 << i for i, c in enumerate(cond.col_ids) if c == 2)
    probe = torch.arange(200, device="cuda")
    if cmp == L.ISCLOSE:                              # refused, as the filter refuses it
        with pytest.raises(ValueError):
            join_pairs(join_build(keys), probe, None, cond, side)
        return
    bi, pi = join_pairs(join_build(keys), probe, None, cond, side)
    assert bi.numel() == 0 and pi.numel() == 0
