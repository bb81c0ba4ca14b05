"""Join builds and probes at the edges of their tiles (128 rows a warp load, 1024 and 4096 rows a tile)
and on both directories against numpy: unique keys, repeated keys, one key holding most of the build
side, masks, probe keys outside the build side's range, unaligned key columns."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(bk, bm, pk, pm, jtype):
    rows = np.nonzero(bm)[0]
    rows = rows[np.argsort(bk[rows], kind="stable")]
    sk = bk[rows]
    lo, hi = np.searchsorted(sk, pk, "left"), np.searchsorted(sk, pk, "right")
    cnt = np.where(pm, hi - lo, 0)
    lone = np.nonzero(pm & (cnt == 0))[0]
    if jtype == "right-semi":
        return np.zeros(0, np.int64), np.nonzero(cnt > 0)[0]
    if jtype == "right-anti":
        return np.zeros(0, np.int64), lone
    pi = np.repeat(np.arange(pk.size), cnt)
    start = np.cumsum(cnt) - cnt
    bi = rows[np.repeat(lo, cnt) + np.arange(pi.size) - np.repeat(start, cnt)]
    if jtype == "right-outer":
        return np.concatenate([bi, np.full(lone.size, -64)]), np.concatenate([pi, lone])
    return bi, pi


def _keys(kind, rng, nb):
    if kind == "unique":
        return rng.permutation(3 * nb)[:nb].astype(np.int64) - nb
    if kind == "repeated":
        return rng.integers(-5, max(1, nb // 4), nb).astype(np.int32)
    if kind == "one key":
        return np.where(rng.integers(0, 10, nb) > 0, 7, rng.integers(0, 50, nb)).astype(np.int64)
    return rng.integers(0, max(2, nb // 2), nb).astype(np.int64) * 10_000_000_019       # sparse


@pytest.mark.parametrize("kind", ["unique", "repeated", "one key", "sparse"])
@pytest.mark.parametrize("nb,npr", [(1, 1), (300, 127), (300, 1024), (2047, 1025), (40, 4096), (5000, 4097), (900, 70_001)])
def test_pairs(kind, nb, npr):
    from tqpk.ops import join_build, join_directory, join_probe
    rng = np.random.default_rng(nb * 7 + npr)
    bk = _keys(kind, rng, nb)
    pk = np.where(rng.integers(0, 3, npr) > 0, bk[rng.integers(0, nb, npr)], rng.integers(-10**6, 10**6, npr)).astype(np.int64)
    if kind == "one key" and npr > 5000:
        pk = np.where(pk == 7, 8, pk)                   # keep the pairs few
    for masked in (False, True):
        bm = rng.integers(0, 4, nb) > 0 if masked else np.ones(nb, bool)
        pm = rng.integers(0, 2, npr) > 0 if masked else np.ones(npr, bool)
        tb, tp = torch.from_numpy(bk).cuda(), torch.from_numpy(np.concatenate([[0], pk])).cuda()[1:]   # unaligned
        mb = torch.from_numpy(bm).cuda() if masked else None
        mp = torch.from_numpy(np.concatenate([[False], pm])).cuda()[1:] if masked else None
        build = join_directory(tb, mb)
        whole = join_build(tb, mb)
        assert whole.unique in (0, 1)
        tb.zero_()                                      # a complete build side does not read its keys again
        for jtype in ("inner", "right-outer"):
            bi, pi = join_probe(whole, tp, mp, jtype)
            ebi, epi = _expected(bk, bm, pk, pm, jtype)
            np.testing.assert_array_equal(pi.cpu().numpy(), epi, err_msg=jtype)
            np.testing.assert_array_equal(bi.cpu().numpy(), ebi, err_msg=jtype)
        tb.copy_(torch.from_numpy(bk))
        for jtype in ("right-semi", "inner", "right-anti", "right-outer", "inner"):
            bi, pi = join_probe(build, tp, mp, jtype)
            ebi, epi = _expected(bk, bm, pk, pm, jtype)
            np.testing.assert_array_equal(pi.cpu().numpy(), epi, err_msg=jtype)
            if jtype in ("inner", "right-outer"):
                np.testing.assert_array_equal(bi.cpu().numpy(), ebi, err_msg=jtype)


CONDS = [[["#12", "=", "#22"]], [["#12", "<", "#22"], ["f#13", ">=", "100.25"]], [["NOT", [["#12", "=", "#22"]]]],
         [["f#13", "=", "500.5"]], [[["f#23", ">", "f#13"], "OR", ["#22", "IN", ["1", "3"]]]], [["#12", "<=", "1.5"]],
         [["#12", ">", "99"]]]


@pytest.mark.parametrize("conds", CONDS)
@pytest.mark.parametrize("kind,nb,npr", [("unique", 700, 1025), ("repeated", 5000, 4097), ("one key", 300, 90),
                                         ("sparse", 900, 20_001)])
def test_conditions_of_a_join(kind, nb, npr, conds):
    """Conditions evaluated by the probe against the oracle's filter over the key-equal pairs."""
    from oracle import tqp_oracle as O
    from tqpk.operators import join_vortex
    from tqpk.variable import Variable
    rng = np.random.default_rng(nb + npr)
    bk = _keys(kind, rng, nb)
    pk = bk[rng.integers(0, nb, npr)]
    cols = {11: bk, 12: rng.integers(0, 5, nb).astype(np.int32), 13: rng.integers(0, 2001, nb) * 0.5,
            21: pk, 22: rng.integers(0, 5, npr).astype(np.int64), 23: rng.integers(0, 2001, npr) * 0.5}
    bi, pi = _expected(bk, np.ones(nb, bool), pk, np.ones(npr, bool), "inner")
    pairs = {c: cols[c][bi] if c < 20 else cols[c][pi] for c in cols}
    keep = np.ones(bi.size, bool)
    for c in conds:
        keep &= O.eval_filter(c, pairs)
    tg = {c: Variable(torch.from_numpy(a).cuda(), "int") for c, a in cols.items()}
    args = {"left group": [11, 12, 13], "right group": [21, 22, 23], "materialized in": [11, 12, 13, 21, 22, 23]}
    assert join_vortex(True, tg, args, 11, 21, conds, "inner", None, None, "j") == int(keep.sum())
    for c in cols:
        np.testing.assert_array_equal(tg[c].tensor.cpu().numpy(), pairs[c][keep], err_msg=str(c))


def test_staged_build_equals_the_whole_build():
    import ctypes as C
    from tqpk import _lib as L
    from tqpk.ops import join_build, join_probe
    lib = L.load()
    rng = np.random.default_rng(3)
    for bk in (rng.permutation(5000), rng.integers(0, 900, 5000)):
        tb, tp = torch.from_numpy(bk).cuda(), torch.from_numpy(rng.integers(0, 6000, 20_000)).cuda()
        exp = join_probe(join_build(tb), tp)
        plan, scratch = L.JoinPlan(), torch.empty(256, dtype=torch.uint8, device="cuda")
        assert lib.tqpk_join_plan_build(tb.data_ptr(), L.I64, None, 5000, C.byref(plan), scratch.data_ptr(), None) == 0
        ws = torch.empty(plan.ws_bytes, dtype=torch.uint8, device="cuda")
        assert lib.tqpk_join_build(C.byref(plan), tb.data_ptr(), L.I64, None, 5000, ws.data_ptr(), ws.numel(), None) == 0
        assert plan.unique == int(len(set(bk.tolist())) == 5000)
        pws = torch.empty(lib.tqpk_join_probe_workspace_bytes(20_000), dtype=torch.uint8, device="cuda")
        m = exp[0].numel()
        ob, op = torch.zeros(m, dtype=torch.int64, device="cuda"), torch.zeros(m, dtype=torch.int64, device="cuda")
        cnt = C.c_int64()
        assert lib.tqpk_join_probe(C.byref(plan), ws.data_ptr(), tp.data_ptr(), L.I64, None, 20_000, L.JT_INNER,
                                   ob.data_ptr(), op.data_ptr(), m, C.byref(cnt), pws.data_ptr(), pws.numel(), None) == 0
        assert cnt.value == m and torch.equal(ob, exp[0]) and torch.equal(op, exp[1])
