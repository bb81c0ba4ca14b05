"""Comparisons of two columns: every pair of types, aligned and not, below and above the row count from
which a thread takes sixteen rows, with NaN, infinities and both zeros, against torch."""
import operator

import pytest
import torch

pytestmark = pytest.mark.gpu

TYPES = [torch.int8, torch.uint8, torch.bool, torch.int32, torch.int64, torch.float64]
OPS = {"<": operator.lt, "<=": operator.le, ">": operator.gt, ">=": operator.ge, "=": operator.eq}
MANY = 5 << 19


def _column(dtype, n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    v = torch.randint(0 if dtype in (torch.uint8, torch.bool) else -3, 2 if dtype == torch.bool else 4, (n,), generator=g,
                      device="cuda")
    if dtype != torch.float64:
        return v.to(dtype)
    v = v.double() * 0.5
    odd = torch.tensor([float("nan"), float("inf"), -float("inf"), -0.0, 0.0], dtype=torch.float64, device="cuda")
    at = torch.arange(0, n, 7, device="cuda")
    v[at] = odd[at % 5]
    return v


@pytest.mark.parametrize("a", TYPES)
@pytest.mark.parametrize("b", TYPES)
@pytest.mark.parametrize("n", [3, 1026, MANY - 1, MANY + 5])
def test_two_columns(a, b, n):
    from tqpk.ops import filter_mask
    from tqpk.predicate import compile_filter
    x, y = _column(a, n + 1, 1), _column(b, n + 1, 2)
    for off in (0, 1):                             # the second start is not 16-byte aligned
        cols = {1: x[off:off + n], 2: y[off:off + n]}
        for op, f in OPS.items():
            want = f(cols[1].double(), cols[2].double())
            got, _ = filter_mask(compile_filter(["a#1", op, "b#2"], cols), n, x.device)
            assert torch.equal(got, want), (op, off)
            tree = [["NOT", [["a#1", op, "b#2"]]], "AND", ["b#2", "<=", "a#1"]]
            got, _ = filter_mask(compile_filter(tree, cols), n, x.device)
            assert torch.equal(got, ~want & (cols[2].double() <= cols[1].double())), (op, off)
