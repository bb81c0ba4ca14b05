"""compile_filter memoises by tree, literals and column shapes: a repeated filter gets the same program
bound to its own columns; another literal, dtype, width or comparison rule compiles afresh."""
import numpy as np
import pytest
import torch

from tqpk.predicate import _FILTER_MEMO, compile_filter

TREES = [["d#1", "<=", "100"], [[["d#1", ">", "2"], "AND", ["NOT", [["v#2", "<", "0.5"]]]]],
         [["StartsWith", ["t#3", "AB"]], "OR", [["substring", ["t#3", "2", "2"]], "IN", ["BC", "xy"]]],
         ["f#4", "=", "1"], [["d#1", "<", "e#5"]]]


def _cols(n, int_dtype=torch.int32, width=6):
    return {1: torch.arange(n, dtype=int_dtype), 2: torch.rand(n, dtype=torch.float64),
            3: torch.zeros(n, width, dtype=torch.int8), 4: torch.ones(n, 1, dtype=torch.uint8),
            5: torch.arange(n, dtype=int_dtype)}


def _program(p):
    s = type(p.struct).from_buffer_copy(p.struct)
    offsets = [s.cols[i] - t.data_ptr() for i, t in enumerate(p.tensors)]
    for i in range(len(s.cols)):
        s.cols[i] = 0
    return bytes(s), offsets, p.col_ids


@pytest.mark.parametrize("tree", TREES)
def test_repeated_filter_rebinds_its_columns(tree):
    _FILTER_MEMO.clear()
    a, b = _cols(40), _cols(70)
    pa, pb = compile_filter(tree, a), compile_filter(tree, b)
    assert len(_FILTER_MEMO) == 1 and pa.sig == pb.sig
    assert _program(pa) == _program(pb)
    for p, cols in ((pa, a), (pb, b)):
        assert [t.data_ptr() for t in p.tensors] == [cols[c].data_ptr() for c in p.col_ids]
    strided = {c: torch.cat([t, t])[::2] for c, t in b.items()}              # read through contiguous copies
    ps = compile_filter(tree, strided)
    assert _program(ps)[0] == _program(pa)[0] and all(t.is_contiguous() for t in ps.tensors)


def test_changes_compile_afresh():
    _FILTER_MEMO.clear()
    sigs = {compile_filter(["d#1", "<=", "100"], _cols(9)).sig, compile_filter(["d#1", "<=", "101"], _cols(9)).sig,
            compile_filter(["d#1", "<=", "100"], _cols(9, torch.int64)).sig,
            compile_filter(["d#1", "<=", "100"], _cols(9, width=7)).sig,
            compile_filter(["d#1", "<=", "100"], _cols(9), agg=True).sig,
            compile_filter(["d#1", "<=", "Subquery"], _cols(9), 100).sig,
            compile_filter(["d#1", "<=", "Subquery"], _cols(9), 100.0).sig}
    assert len(sigs) == 7 and None not in sigs
    held = len(_FILTER_MEMO)
    assert compile_filter(["d#1", "<=", "Subquery"], _cols(9), np.int64(3)).sig is None
    assert len(_FILTER_MEMO) == held
    with pytest.raises(KeyError):
        compile_filter(["z#9", "<", "1"], _cols(9))
    assert len(_FILTER_MEMO) == held
