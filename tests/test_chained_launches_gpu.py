"""The matvec's launches are chained by programmatic dependent launch.  The
same bits come out of them on the handle's own stream, on the legacy default
stream, in a captured graph that is replayed on another vector, and with two
handles at work on two streams at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [("CMPS_FP64", "CMPS_ORDER_FOLDED"), ("CMPS_SPLIT_BF16", "CMPS_ORDER_FOLDED"),
         ("CMPS_SPLIT_TF32", "CMPS_ORDER_FOLDED"), ("CMPS_FP64", "CMPS_ORDER_CANONICAL"),
         ("CMPS_SPLIT_BF16", "CMPS_ORDER_CANONICAL"), ("CMPS_SPLIT_TF32", "CMPS_ORDER_CANONICAL")]


def _handle(ctx, seed, precision, order):
    import chainamps_b200 as ca
    from chainamps_b200 import models
    rng = np.random.default_rng(seed)
    d, D, rules = 3, 4, (0,)
    bond = lambda dims: np.repeat(np.arange(len(dims)), dims).reshape(-1, 1).astype(np.int64)  # noqa: E731
    bl, br, bq = bond([33, 64, 9]), bond([17, 40, 65]), np.zeros((D, 1), np.int64)
    W = rng.standard_normal((d, D, d, D)) + 1j * rng.standard_normal((d, D, d, D))
    L = models.random_environment(rng, rules, bl, bq, list(range(D)), right=False)
    R = models.random_environment(rng, rules, br, bq, list(range(D)), right=True)
    h = ca.TwoVertexComponents(ctx, rules, L, models.mpo_tensor(np.zeros((d, 1), np.int64), W, bq), R)
    h.set_order(getattr(ca, order))
    h.set_precision(getattr(ca, precision))
    return h


@pytest.mark.parametrize("precision,order", FORMS)
def test_streams_and_capture(precision, order):
    import torch
    from chainamps_b200 import Context
    ctx = Context(0)
    hs = [_handle(ctx, seed, precision, order) for seed in (1, 2)]
    gen = torch.Generator("cuda").manual_seed(3)
    xs = [torch.randn(h.n, dtype=torch.complex128, device="cuda", generator=gen) for h in hs]
    want = [torch.as_tensor(h.multiply(x.cpu().numpy()), device="cuda") for h, x in zip(hs, xs)]
    assert all(float(w.abs().max()) > 0 for w in want)

    def apply(h, x, y, stream):
        h.multiply_device(x.data_ptr(), y.data_ptr(), stream)
    y = torch.zeros_like(xs[0])
    torch.cuda.synchronize()
    apply(hs[0], xs[0], y, 0)  # the legacy default stream
    torch.cuda.synchronize()
    assert torch.equal(y, want[0])
    # two handles, two streams, many passes in flight
    streams = [torch.cuda.Stream() for _ in hs]
    ys = [[torch.zeros_like(x) for _ in range(20)] for x in xs]
    torch.cuda.synchronize()
    for i in range(20):
        for h, x, out, s in zip(hs, xs, ys, streams):
            apply(h, x, out[i], s.cuda_stream)
    torch.cuda.synchronize()
    for out, w in zip(ys, want):
        assert all(torch.equal(o, w) for o in out)
    # captured, then replayed on another vector
    x, y, s = xs[1].clone(), torch.zeros_like(xs[1]), streams[1]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        apply(hs[1], x, y, s.cuda_stream)
    x.copy_(xs[1] * 2.0)
    torch.cuda.synchronize()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want[1] * 2.0)
    del graph, hs
    ctx.close()
