"""A context on several streams: its own, streams bound by set_stream, torch's
current stream (pdg_run_on).  Every call follows the context's earlier work on
whatever stream that ran: the first apply, which builds the operator's records
behind a sleep of about 20 ms on the GPU, is followed by one on another stream
that reads them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402

SLEEP = 40_000_000


def setup(seed):
    import torch
    rng = np.random.default_rng(seed)
    go = pdg.GridOperator(3, 2, (12, 11, 10), alpha=3.0)
    go.set_permeability(np.exp(rng.standard_normal(go.ncell)))
    x = torch.tensor(rng.uniform(-1, 1, go.ndof), device="cuda")
    ys = [torch.zeros_like(x), torch.zeros_like(x)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    return torch, go, pdg.OnTheFlyOperator(go), x, ys, streams


def finish(torch, go, op, x, ys):
    torch.cuda.synchronize()
    ref = np.zeros(go.ndof)
    op.apply(x.cpu().numpy(), ref)
    for y in ys:
        assert np.array_equal(y.cpu().numpy(), ref)
    go.close()


def test_bound_stream_follows_torchs():
    torch, go, op, x, ys, s = setup(1)
    with torch.cuda.stream(s[0]):
        torch.cuda._sleep(SLEEP)
        op.apply(x, ys[0])
    go.set_stream(s[1])
    op.apply(x, ys[1])
    torch.cuda.synchronize()
    go.set_stream(None)
    finish(torch, go, op, x, ys)


def test_torchs_stream_follows_a_bound_one():
    torch, go, op, x, ys, s = setup(2)
    go.set_stream(s[0])
    with torch.cuda.stream(s[0]):
        torch.cuda._sleep(SLEEP)
    op.apply(x, ys[0])
    go.set_stream(None)
    with torch.cuda.stream(s[1]):
        op.apply(x, ys[1])
    finish(torch, go, op, x, ys)


def test_bound_stream_follows_another():
    torch, go, op, x, ys, s = setup(3)
    go.set_stream(s[0])
    with torch.cuda.stream(s[0]):
        torch.cuda._sleep(SLEEP)
    op.apply(x, ys[0])
    go.set_stream(s[1])
    op.apply(x, ys[1])
    torch.cuda.synchronize()
    go.set_stream(None)
    finish(torch, go, op, x, ys)


def test_capturing_stream_can_be_bound():
    """Nothing is waited for inside a capture, as before."""
    torch, go, op, x, ys, s = setup(4)
    op.apply(x, ys[0])
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s[0]):
        go.set_stream(s[0])
        op.apply(x, ys[1])
    go.set_stream(None)
    ys[1].zero_()
    g.replay()
    finish(torch, go, op, x, ys)
