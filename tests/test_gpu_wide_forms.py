"""The forms that only tables of 2^32 rows and more select, on small ones: 64-bit directory entries of a
join (the plan's flag set by the test, with the workspace it takes) and 8-byte positions of a sort."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _wide_build(keys, mask):
    from tqpk import _lib as L
    from tqpk.ops import JoinBuild
    lib = L.load()
    plan = L.JoinPlan()
    scratch = torch.empty(256, dtype=torch.uint8, device="cuda")
    L.check(lib.tqpk_join_plan_build(keys.data_ptr(), L.I64 if keys.dtype == torch.int64 else L.I32,
                                     mask.data_ptr() if mask is not None else None, keys.numel(), C.byref(plan),
                                     scratch.data_ptr(), None), "plan")
    plan.unique |= L.JOIN_WIDE
    plan.ws_bytes += 12 * plan.slots + 4096
    b = JoinBuild(plan, torch.empty(plan.ws_bytes, dtype=torch.uint8, device="cuda"), keys, keys.device, mask)
    return b, lib


@pytest.mark.parametrize("case", ["unique", "repeated", "one key", "long runs", "sparse"])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("lazy", [False, True])
def test_joins_with_64_bit_entries(case, masked, lazy):
    from tqpk.ops import join_build, join_pairs, join_probe
    from tqpk.predicate import compile_filter
    rng = np.random.default_rng(len(case))
    nb, np_ = 9001, 20_003
    keys = {"unique": rng.permutation(nb) * 2, "repeated": rng.integers(0, 3000, nb), "one key": np.full(nb // 100, 7),
            "long runs": rng.integers(0, 90, nb), "sparse": rng.integers(0, 3000, nb) << 30}[case].astype(np.int64)
    probe = torch.from_numpy(rng.choice(np.concatenate([keys, [-5, 1 << 50]]), np_)).cuda()
    keys = torch.from_numpy(keys).cuda()
    nb = keys.numel()
    mask = torch.from_numpy(rng.random(nb) < 0.7).cuda() if masked else None
    pmask = torch.from_numpy(rng.random(np_) < 0.5).cuda() if masked else None
    narrow = join_build(keys, mask)
    cols = {1: torch.from_numpy(rng.integers(0, 4, nb)).cuda(), 2: torch.from_numpy(rng.integers(0, 4, np_)).cuda()}
    cond = compile_filter(["a#1", "=", "b#2"], cols)
    side = sum(1 << i for i, c in enumerate(cond.col_ids) if c == 2)
    for jt in ("right-semi", "right-anti", "inner", "right-outer"):
        wide, lib = _wide_build(keys, mask)
        wide._call(lib.tqpk_join_directory if lazy else lib.tqpk_join_build, "build")
        assert wide.plan.unique & 256
        if jt in ("inner", "right-outer"):
            assert torch.equal(join_probe(wide, probe, pmask, jt)[0], join_probe(narrow, probe, pmask, jt)[0])
        assert torch.equal(join_probe(wide, probe, pmask, jt)[1], join_probe(narrow, probe, pmask, jt)[1])
        assert wide.plan.unique & 256
    wide, lib = _wide_build(keys, mask)
    wide._call(lib.tqpk_join_directory if lazy else lib.tqpk_join_build, "build")
    for c in ((), (cond, side)):
        for g, e in zip(join_pairs(wide, probe, pmask, *c), join_pairs(narrow, probe, pmask, *c)):
            assert torch.equal(g, e)


@pytest.mark.parametrize("n", [98_305, 300_001, 1_228_800, 1_300_007])
@pytest.mark.parametrize("kind", ["int64", "price", "runs", "text", "several", "constant"])
def test_sorts_with_8_byte_positions(n, kind):
    from tqpk import _lib as L
    from tqpk.ops import argsort_keys
    lib = L.load()
    rng = np.random.default_rng(n)
    price = rng.integers(90000, 10495001, n) / 100.0
    price[:: n // 50] = np.nan
    text = rng.choice(np.frombuffer(b"AB c", np.int8), (n, 11))
    cols = {"int64": [rng.integers(-(1 << 62), 1 << 62, n)], "price": [price], "constant": [np.full(n, 3)],
            "runs": [(np.arange(n) // 50 << 30) + rng.integers(0, 1 << 20, n)], "text": [text],
            "several": [rng.integers(0, 50, n).astype(np.int32), price, text]}[kind]
    perm = rng.permutation(n)
    descs = [bool(i & 1) for i in range(len(cols))]
    dev = [torch.from_numpy(c).cuda() for c in cols]
    dt = (C.c_int32 * len(cols))(*[{"int64": L.I64, "int32": L.I32, "float64": L.F64, "int8": L.I8}[str(c.dtype)] for c in cols])
    widths = (C.c_int32 * len(cols))(*[c.shape[1] if c.ndim == 2 else 0 for c in cols])
    ws = torch.empty(lib.tqpk_argsort_keys_workspace_bytes(n, len(cols), dt, widths) + 8 * n + 1024, dtype=torch.uint8,
                     device="cuda")
    for p in (None, torch.from_numpy(perm).cuda()):
        out = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        L.check(lib.tqpk_debug_argsort_wide(len(cols), (C.c_void_p * len(cols))(*[c.data_ptr() for c in dev]), dt, widths,
                                            (C.c_int32 * len(cols))(*descs), p.data_ptr() if p is not None else None, n,
                                            out.data_ptr(), ws.data_ptr(), ws.numel(), None), "sort")
        assert torch.equal(out, argsort_keys(dev, descs, p))
