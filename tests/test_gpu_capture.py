"""Applies captured into a CUDA graph right after a coefficient change: the
records that the first apply builds are then built by the graph's replays, so an
apply outside the graph, before any replay, has to build them itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402

FORMS = {
    "apply": lambda go, op, x, y: op.apply(x, y),
    "transpose": lambda go, op, x, y: go.jacobian_apply_transpose(x, y),
    "residual": lambda go, op, x, y: go.residual(x, y),
    "f32": lambda go, op, x, y: go.apply_f32(x, y),
}


# dimension, degree, basis, tensor per cell, arithmetic: every kind of record
@pytest.mark.parametrize("dim,k,basis,tensor,pair", [
    (3, 1, 0, False, False), (3, 2, 0, False, False), (3, 3, 0, False, False),
    (3, 4, 0, False, False), (3, 3, 2, False, False), (3, 2, 0, True, False),
    (3, 2, 0, False, True), (2, 2, 0, False, False)])
@pytest.mark.parametrize("form", list(FORMS))
def test_capture_after_a_coefficient_change(form, dim, k, basis, tensor, pair):
    import torch
    n = (6, 5, 4)[:dim]
    rng = np.random.default_rng(k)
    go = pdg.GridOperator(dim, k, n, alpha=3.0, basis=basis)
    nc = go.ncell
    G = rng.standard_normal((2, nc, dim, dim))
    A = [np.ascontiguousarray(g @ g.transpose(0, 2, 1) + 0.2 * np.eye(dim)) for g in G]
    K = [np.exp(rng.standard_normal(nc)) for _ in range(2)]

    def coefficients(i):
        if tensor:
            go.set_permeability_tensor(A[i])
        else:
            go.set_permeability(K[i])

    coefficients(0)
    go.set_source(fc=np.ones(nc))
    if pair:
        go.set_f64_arithmetic(pdg.F64_FLOAT_PAIR)
    op = pdg.OnTheFlyOperator(go)
    x = torch.tensor(rng.uniform(-1, 1, go.ndof), device="cuda")
    if form == "f32":
        x = x.float()

    def run(y):
        y.zero_()
        FORMS[form](go, op, x, y)
        return y

    y, out = torch.zeros_like(x), torch.zeros_like(x)
    old = run(y).clone()
    coefficients(1)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        run(out)
    new = run(y).clone()           # before any replay
    assert not torch.equal(new, old)
    coefficients(1)                # the same, built outside any capture
    assert torch.equal(run(y), new)
    g.replay()
    assert torch.equal(out, new)
    assert torch.equal(run(y), new)
    go.close()
