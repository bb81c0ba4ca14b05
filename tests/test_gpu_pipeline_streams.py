"""A fused pipeline built on one stream and run on another: nothing that its constructor queued may land
on what the run writes (the rows, the error words)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _busy(stream, ms=400):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(int(ms * 1.9e6))           # a bounded wait on the device


@pytest.mark.parametrize("kind", ["join", "star", "star, repeated key"])
def test_the_constructors_stream_may_be_behind_the_runs(kind):
    import bench
    from tqpk.pipeline import JoinAggTopK, StarAggTopK
    dom = lambda a: (int(a.min()), int(a.max()))                                             # noqa: E731
    slow, fast = torch.cuda.Stream(), torch.cuda.Stream()
    if kind == "join":
        rng = np.random.default_rng(2)
        nb, np_ = 5000, 40_000
        c = {11: np.arange(nb), 21: rng.integers(0, nb, np_), 23: rng.integers(1, 1000, np_).astype(np.float64)}
        d = {k: torch.from_numpy(v).cuda() for k, v in c.items()}

        def make():
            return JoinAggTopK(d[11], 0, nb - 1, d[21], {}, None, {23: d[23]}, None, ["p#23"], k=20)
    else:
        w = bench.StarJoin(scale=0.01)
        if kind.endswith("key"):
            w.cols[31][-1] = w.cols[31][0]
            w.cols[32][-1] = w.cols[32][0]
        d = {c: torch.from_numpy(a).cuda() for c, a in w.cols.items()}

        def make():
            return StarAggTopK(d[41], d[42], {43: d[43], 44: d[44]}, None, w.value_tree, d[31], {32: d[32]}, None,
                               dom(w.cols[31]), d[51], d[52], dom(w.cols[51]), d[61], dom(w.cols[61]), k=20)
    make().run()                                      # kernels compiled
    torch.cuda.synchronize()
    _busy(slow)
    with torch.cuda.stream(slow):
        p = make()
    with torch.cuda.stream(fast):
        p.run()
        names = [n for n in ("out_keys", "out_vals", "out_cnts", "err") if hasattr(p, n)]
        wrote = [getattr(p, n).clone() for n in names]
    fast.synchronize()
    assert not slow.query()                           # the constructor's stream is behind
    torch.cuda.synchronize()
    for n, w in zip(names, wrote):
        assert torch.equal(getattr(p, n), w), n
    if "err" in names:
        assert bool(p.err.any()) == kind.endswith("key")
