"""The mask and key-range kernels on both sides of their row-count rule (four rows a thread below 2621440
rows, sixteen from there) against numpy: every comparison on every column type, literals outside the
column's range, NaN, infinities and both zeros, two-column comparisons, unaligned columns."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MANY = 5 << 19
OPS = {"LT": np.less, "LE": np.less_equal, "GT": np.greater, "GE": np.greater_equal, "EQ": np.equal, "NE": np.not_equal}


def _mask(n, cols, insns):
    from tqpk import _lib as L
    from tqpk.dtypes import code_of
    from tqpk.ops import filter_mask
    from tqpk.predicate import CompiledPredicate
    p = L.Predicate()
    p.n_insn, p.n_cols = len(insns), len(cols)
    for i, c in enumerate(cols):
        p.cols[i], p.dtypes[i] = c.data_ptr(), code_of(c.dtype)
    for i, x in enumerate(insns):
        p.insn[i] = L.PredInsn(*x)
    mask, count = filter_mask(CompiledPredicate(p, cols, list(range(len(cols)))), n, cols[0].device, with_count=True)
    m = mask.cpu().numpy()
    assert int(count.item()) == int(m.sum())
    return m


def _columns(rng, n):
    f = rng.integers(-40, 40, n) * 0.25
    f[rng.integers(0, n, n // 5 + 1)] = rng.choice([np.nan, np.inf, -np.inf, -0.0, 0.0, 5e-324, -5e-324], n // 5 + 1)
    return [rng.integers(-128, 128, n).astype(np.int8), rng.integers(0, 256, n).astype(np.uint8),
            rng.integers(-9, 9, n).astype(np.int32), rng.integers(-9, 9, n) * (1 << 40), f]


@pytest.mark.parametrize("unaligned", [False, True])
@pytest.mark.parametrize("n", [1, 3, 1023, 1024, 1025, MANY - 1, MANY, MANY + 1029])
def test_comparisons(n, unaligned):
    from tqpk import _lib as L
    rng = np.random.default_rng(n)
    cols = _columns(rng, n)
    dev = [torch.from_numpy(np.concatenate([c[:1], c])).cuda()[1:] if unaligned else torch.from_numpy(c).cuda()
           for c in cols]
    for name, fn in OPS.items():
        op = getattr(L, name)
        for i, c in enumerate(cols[:4]):
            for lit in (0, 7, 127, 128, 255, 256, -129, 3 << 40, -(1 << 62)):
                got = _mask(n, [dev[i]], [(L.P_CMP, 0, op, L.DOM_I64, lit, 0.0, 0.0)])
                np.testing.assert_array_equal(got, fn(c.astype(np.int64), np.int64(lit)), err_msg=f"{name} {c.dtype} {lit}")
                if n > 2000:
                    break
        for lit in (0.0, -0.0, 2.25, np.inf, -np.inf, np.nan, 5e-324):
            got = _mask(n, [dev[4]], [(L.P_CMP, 0, op, L.DOM_F64, 0, lit, 0.0)])
            np.testing.assert_array_equal(got, fn(cols[4], lit), err_msg=f"{name} {lit}")
            if n > 2000 and lit == 0.0:
                break
        got = _mask(n, [dev[2]], [(L.P_CMP, 0, op, L.DOM_F32, 0, 1.5, 0.0)])
        np.testing.assert_array_equal(got, fn(cols[2].astype(np.float32), np.float32(1.5)))
        for a, b in ((2, 2), (3, 3), (2, 3), (0, 1)):
            other = cols[b][::-1].copy()
            got = _mask(n, [dev[a], torch.from_numpy(other).cuda()], [(L.P_CMPCOL, 0, op, L.DOM_I64, 1, 0.0, 0.0)])
            np.testing.assert_array_equal(got, fn(cols[a].astype(np.int64), other.astype(np.int64)))
    # (not (a < 0) and b >= 3) or true-and-false, a deep enough stack
    got = _mask(n, dev, [(L.P_TRUE, 0, 0, 0, 0, 0.0, 0.0), (L.P_FALSE, 0, 0, 0, 0, 0.0, 0.0), (L.P_AND, 0, 0, 0, 0, 0.0, 0.0),
                         (L.P_CMP, 2, L.LT, L.DOM_I64, 0, 0.0, 0.0), (L.P_NOT, 0, 0, 0, 0, 0.0, 0.0),
                         (L.P_CMP, 1, L.GE, L.DOM_I64, 3, 0.0, 0.0), (L.P_AND, 0, 0, 0, 0, 0.0, 0.0),
                         (L.P_MASK, 0, 0, 0, 0, 0.0, 0.0), (L.P_AND, 0, 0, 0, 0, 0.0, 0.0), (L.P_OR, 0, 0, 0, 0, 0.0, 0.0)])
    np.testing.assert_array_equal(got, ~(cols[2] < 0) & (cols[1] >= 3) & (cols[0] != 0))


@pytest.mark.parametrize("n", [1, 1025, MANY - 1, MANY + 5])
def test_key_ranges_under_a_mask(n):
    import ctypes as C
    from tqpk import _lib as L
    from tqpk.dtypes import code_of
    lib = L.load()
    rng = np.random.default_rng(n + 1)
    cols = _columns(rng, n)[:4]
    for m in (None, rng.integers(0, 9, n) == 0, np.arange(n) == n - 1, np.zeros(n, bool)):
        mask = torch.from_numpy(m).cuda() if m is not None else None
        for c in cols:
            t = torch.from_numpy(c).cuda()
            plan, scratch = L.JoinPlan(), torch.empty(256, dtype=torch.uint8, device="cuda")
            assert lib.tqpk_join_plan_build(t.data_ptr(), code_of(t.dtype), mask.data_ptr() if m is not None else None, n,
                                            C.byref(plan), scratch.data_ptr(), None) == 0
            s = c if m is None else c[m]
            assert plan.nb_rows == s.size
            assert (plan.key_min, plan.key_max) == ((int(s.min()), int(s.max())) if s.size else (0, -1))


@pytest.mark.parametrize("n", [1, 255, 257, 1023, 1025, 5000])
@pytest.mark.parametrize("width", [6, 25, 188, 189])
def test_text_programs(n, width):
    """Text staged in shared memory (rows of up to 188 bytes) and in place, beside numeric comparisons."""
    from oracle import tqp_oracle as O
    from tqpk.ops import filter_mask
    from tqpk.predicate import compile_filter
    rng = np.random.default_rng(n + width)
    words = [b"ECONOMY", b"TIN", b"MED", b"AB", b"CANADA", b""]
    t = np.zeros((n, width), np.int8)
    for i in range(n):
        s = b" ".join(words[j] for j in rng.integers(0, 6, 1 + width // 8))[:width]
        t[i, :len(s)] = np.frombuffer(s, np.int8)
    cols = {1: t, 2: rng.integers(0, 9, n), 3: np.ascontiguousarray(t[:, : min(width, 9)])}
    dev = {c: torch.from_numpy(a).cuda() for c, a in cols.items()}
    trees = [["StartsWith", ["t#1", "AB"]], ["t#1", "LIKE", "%MED%TIN%"], ["Contains", ["t#1", "NOM"]],
             [["NOT", [["StartsWith", ["t#1", "MED"]]]], "AND", [["k#2", "<", "5"], "OR", ["Contains", ["s#3", "IN"]]]],
             [["substring", ["t#1", "2", "3"]], "IN", ["CON", "ANA", "IN "]], ["s#3", "=", "CANADA"],
             [["substring", ["t#1", str(width - 1), "2"]], "=", "ED"]]
    for tree in trees:
        if "CANADA" in repr(tree) and min(width, 9) < 6:
            continue
        pred = compile_filter(tree, dev)
        mask, count = filter_mask(pred, n, dev[1].device, with_count=True)
        exp = np.asarray(O.eval_filter(tree, cols), bool).reshape(-1)
        np.testing.assert_array_equal(mask.cpu().numpy(), exp, err_msg=repr(tree))
        assert int(count.item()) == int(exp.sum())


@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000])
@pytest.mark.parametrize("width", [2, 15, 16, 25, 160, 161])
def test_gather_of_text_rows(n, width):
    from tqpk.ops import gather_rows
    rng = np.random.default_rng(n + width)
    t = rng.integers(-128, 128, (700, width)).astype(np.int8)
    idx = rng.integers(0, 700, n)
    idx[0] = 699
    got = gather_rows(torch.from_numpy(t).cuda(), torch.from_numpy(idx).cuda())
    np.testing.assert_array_equal(got.cpu().numpy(), t[idx])


def test_key_ranges_of_several_columns():
    from tqpk.ops import key_range, key_ranges
    rng = np.random.default_rng(2)
    cols = [torch.from_numpy(c).cuda() for n in (1, 5000, MANY + 3) for c in _columns(rng, n)[:4]]
    cols.append(torch.empty(0, dtype=torch.int32, device="cuda"))
    assert key_ranges(cols) == [key_range(c) for c in cols]
