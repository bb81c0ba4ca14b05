"""Float equality (|x - literal| within an allowed error, or x == literal) on both sides of the row count
from which a thread takes sixteen rows: values at the error's edge, both zeros, infinities and NaN, as
column values, literals and allowed errors."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1025, (5 << 19) + 3])
@pytest.mark.parametrize("lit", [0.05, -0.0, 0.0, 104949.5, -1e308, math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("allowed", [None, 0.0, -0.0, -1.0, math.inf, math.nan])
def test_isclose(n, lit, allowed):
    from tqpk.ops import filter_mask
    from tqpk.predicate import compile_filter
    edge = 1e-5
    base = np.array([0.05, 0.0, -0.0, 104949.5, 104949.51, -1e308, 1e308, math.inf, -math.inf, math.nan, 5e-324])
    near = [f(lit if math.isfinite(lit) else 0.05, e) for e in (edge, edge * 2, 1.2) for f in (lambda x, e: x + e, lambda x, e: x - e)]
    near += [np.nextafter(v, 9e9) for v in near] + [np.nextafter(v, -9e9) for v in near]
    x = np.resize(np.concatenate([base, near]), n)
    dev = torch.from_numpy(x).cuda()
    p = compile_filter(["v#1", "=", "0.05"], {1: dev})
    p.struct.insn[0].lit_f = lit
    if allowed is not None:
        p.struct.insn[0].lit_aux = allowed
    aux = p.struct.insn[0].lit_aux
    with np.errstate(all="ignore"):
        err = np.abs(x - lit)
        want = (x == lit) | (np.isfinite(err) & (err <= aux))
    got, _ = filter_mask(p, n, dev.device)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
