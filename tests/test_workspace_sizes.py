"""Workspace queries grow with the rows: a workspace for n rows serves any fewer (the key encoder sorts at
most as many groups as it has rows), across the rules that pick tiles, positions and forms."""
import ctypes as C

import pytest

EDGES = [0, 1, 2048, 2049, 4096, 98_304, 98_305, 1_228_799, 1_228_800, 1_228_801, 1_230_000, 1_843_200, 6_001_215,
         (1 << 32) - 1, 1 << 32]


@pytest.fixture(scope="module")
def lib():
    from tqpk import _lib, build
    build.build()
    return _lib.load()


def _grows(size):
    sizes = [size(n) for n in EDGES]
    assert sizes == sorted(sizes), [(n, s) for n, s in zip(EDGES, sizes)]


@pytest.mark.parametrize("words", [1, 2, 7, 32])
def test_sorts(lib, words):
    one = lambda v: (C.c_int32 * 1)(v)                                                       # noqa: E731
    from tqpk import _lib as L
    _grows(lambda n: lib.tqpk_argsort_keys_workspace_bytes(n, 1, one(L.U8), one(8 * words)))
    _grows(lib.tqpk_sort_workspace_bytes)


@pytest.mark.parametrize("k", [1, 32, 33, 256, 257])
def test_topk(lib, k):
    _grows(lambda n: lib.tqpk_topk_workspace_bytes(n, k))
    _grows(lib.tqpk_topk_ties_workspace_bytes)


def test_encode_compaction_and_join(lib):
    _grows(lib.tqpk_key_encode_workspace_bytes)
    _grows(lib.tqpk_compact_workspace_bytes)
    _grows(lib.tqpk_join_probe_workspace_bytes)
