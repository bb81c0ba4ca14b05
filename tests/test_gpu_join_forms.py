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


@pytest.mark.parametrize("nb,np_,keys", [(300, 1, 1), (3000, 700, 1), (17, 3000, 1), (2500, 5000, 3), (40_000, 40, 2), (5000, 9000, 2500),
                                         (4000, 320_000, 200)])
@pytest.mark.parametrize("conditions", [0, 1, 2])
def test_long_runs_are_shared_by_several_ctas(nb, np_, keys, conditions):
    """Few probe rows, many build rows a key: a tile's pairs are split among CTAs, in the pairs' order."""
    from tqpk.ops import join_build, join_pairs
    from tqpk.predicate import compile_filter
    rng = np.random.default_rng(nb + np_)
    bk, pk = rng.integers(0, keys, nb), rng.integers(-1, keys + 1, np_)
    a, c = rng.integers(0, 400, nb), rng.integers(0, 400, np_)
    e, f = rng.integers(0, 100, nb).astype(np.int32), rng.integers(0, 100, np_).astype(np.int32)
    mask = rng.random(np_) < 0.8
    dev = {i: torch.from_numpy(v).cuda() for i, v in ((1, a), (2, c), (3, e), (4, f))}
    cond, side = None, 0
    if conditions:
        tree = ["x#1", "=", "y#2"]
        if conditions == 2:
            tree = [tree, "OR", [["x#3", "<", "y#4"], "AND", ["y#2", "<", "9"]]]
        cond = compile_filter(tree, dev)
        side = sum(1 << i for i, col in enumerate(cond.col_ids) if col in (2, 4))
    bi, pi = join_pairs(join_build(torch.from_numpy(bk).cuda()), torch.from_numpy(pk).cuda(), torch.from_numpy(mask).cuda(), cond, side)
    order = np.argsort(bk, kind="stable")
    starts = np.searchsorted(bk[order], pk, "left")
    counts = (np.searchsorted(bk[order], pk, "right") - starts) * mask
    want_p = np.repeat(np.arange(np_), counts)
    want_b = order[np.repeat(starts, counts) + np.arange(counts.sum()) - np.repeat(np.cumsum(counts) - counts, counts)]
    if conditions:
        keep = a[want_b] == c[want_p]
        if conditions == 2:
            keep |= (e[want_b] < f[want_p]) & (c[want_p] < 9)
        want_b, want_p = want_b[keep], want_p[keep]
    np.testing.assert_array_equal(pi.cpu().numpy(), want_p)
    np.testing.assert_array_equal(bi.cpu().numpy(), want_b)
