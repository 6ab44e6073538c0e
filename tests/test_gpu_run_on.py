"""Single operations run on torch's current stream (pdg_run_on): ordering
against the context's other work, and stream capture."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402


def setup(seed=3):
    import torch
    rng = np.random.default_rng(seed)
    go = pdg.GridOperator(3, 2, (12, 11, 10), alpha=3.0)
    K = np.exp(rng.standard_normal(go.ncell))
    go.set_permeability(K)
    x = torch.tensor(rng.uniform(-1, 1, go.ndof), device="cuda")
    return torch, rng, go, x


def host_apply(go, x):
    y = np.zeros(go.ndof)
    pdg.OnTheFlyOperator(go).apply(x.cpu().numpy(), y)
    return y


def test_parameters_set_behind_a_queued_apply():
    torch, rng, go, x = setup()
    op = pdg.OnTheFlyOperator(go)
    c = rng.uniform(0.5, 2.0, go.ncell)
    ref0 = host_apply(go, x)
    y0, y1 = torch.zeros_like(x), torch.zeros_like(x)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        torch.cuda._sleep(40_000_000)      # about 20 ms
        op.apply(x, y0)
    go.set_reaction(c)                     # on the context's stream, after the apply
    with torch.cuda.stream(s):
        op.apply(x, y1)
    torch.cuda.synchronize()
    assert np.array_equal(y0.cpu().numpy(), ref0)
    assert np.array_equal(y1.cpu().numpy(), host_apply(go, x))
    assert not np.array_equal(y0.cpu().numpy(), y1.cpu().numpy())
    go.close()


def test_first_apply_on_one_stream_second_on_another():
    """The records are built behind a sleep on the first stream."""
    torch, rng, go, x = setup(4)
    op = pdg.OnTheFlyOperator(go)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    ys = [torch.zeros_like(x), torch.zeros_like(x)]
    torch.cuda.synchronize()
    for i, s in enumerate(streams):
        with torch.cuda.stream(s):
            if i == 0:
                torch.cuda._sleep(40_000_000)
            op.apply(x, ys[i])
    torch.cuda.synchronize()
    ref = host_apply(go, x)
    assert np.array_equal(ys[0].cpu().numpy(), ref) and np.array_equal(ys[1].cpu().numpy(), ref)
    go.close()


def test_capture_and_solve_around_it():
    torch, rng, go, x = setup(5)
    op = pdg.OnTheFlyOperator(go)
    y = torch.zeros_like(x)
    op.apply(x, y)
    ref = y.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        op.apply(x, y)
    y.zero_()
    g.replay()
    assert torch.equal(y, ref)
    go.set_source(fc=np.ones(go.ncell))
    u = torch.zeros_like(x)
    ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go)
    slp = pdg.StationaryLinearProblemSolver(go, ls, u, 1e-8)
    slp.apply()
    assert slp.result().converged
    r = torch.zeros_like(x)
    go.residual(u, r)
    assert float(r.norm()) <= 1.1e-8 * slp.result().first_defect
    go.close()


def test_states():
    torch, rng, go, x = setup(6)
    lib, h = pdg.load(), go.handle
    assert lib.pdg_run_done(h) == pdg.PDG_ESTATE
    assert lib.pdg_run_on(h, None) == pdg.PDG_OK
    assert lib.pdg_run_on(h, None) == pdg.PDG_ESTATE
    assert lib.pdg_set_stream(h, ctypes.c_void_p(1)) == pdg.PDG_ESTATE
    assert lib.pdg_run_done(h) == pdg.PDG_OK
    go.set_stream(torch.cuda.Stream())
    assert lib.pdg_run_on(h, None) == pdg.PDG_ESTATE
    go.set_stream(None)
    go.close()
