"""The FP32 operator and block Jacobi of degrees 1 and 2, one cell per thread
(pdg_cell32.cu): cell counts around the block's 64, odd row lengths (every
16-byte phase of the staged runs), vectors that are not 16-byte aligned, both
forms, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402
import pdg_oracle as O  # noqa: E402

TOL32 = 2e-5   # the FP32 operator's bound everywhere in these tests


def rel(y, ref):
    return np.max(np.abs(y - ref)) / np.max(np.abs(ref))


def vec(torch, n, offset, data=None):
    buf = torch.zeros(n + 4, dtype=torch.float32, device="cuda")
    v = buf[offset:offset + n]
    if data is not None:
        v.copy_(torch.from_numpy(data.astype(np.float32)))
    return v


@pytest.mark.parametrize("k", [1, 2])
@pytest.mark.parametrize("n", [(1, 1, 1), (63, 1, 1), (64, 1, 1), (13, 5, 1), (5, 3, 9), (6, 7, 4)])
@pytest.mark.parametrize("offset", [0, 1])
def test_apply(k, n, offset):
    import torch
    rng = np.random.default_rng(sum(n) + k)
    nc = int(np.prod(n))
    bct = [1, 1, -1, 1, 1, -1]
    K, c = np.exp(rng.standard_normal(nc)), rng.uniform(0.5, 2.0, nc)
    go = pdg.GridOperator(3, k, n, extent=[1.0, 0.5, 2.0], alpha=3.0, method=pdg.NIPG, bctype=bct)
    P = O.Problem(3, k, n, L=(1.0, 0.5, 2.0), alpha=3.0, method=pdg.NIPG, bctype=bct, K=K, c=c)
    go.set_permeability(K)
    go.set_reaction(c)
    x = rng.uniform(-1, 1, go.ndof).astype(np.float32).astype(np.float64)
    xd, yd = vec(torch, go.ndof, offset, x), vec(torch, go.ndof, offset)
    go.apply_f32(xd, yd)
    assert rel(yd.double().cpu().numpy(), P.jacobian_apply(x)) <= TOL32
    y0 = rng.uniform(-1, 1, go.ndof).astype(np.float32)
    yd = vec(torch, go.ndof, offset, y0)
    go.jacobian_apply_transpose_f32(xd, yd)
    assert rel(yd.double().cpu().numpy(), P.jacobian_apply_transpose(x) + y0) <= TOL32
    go.close()


@pytest.mark.parametrize("k", [1, 2])
@pytest.mark.parametrize("n", [(1, 1, 1), (63, 1, 1), (64, 1, 1), (13, 5, 1), (6, 7, 4)])
def test_fdm_and_mixed_solve(k, n):
    import torch
    rng = np.random.default_rng(7 + sum(n) + k)
    nc = int(np.prod(n))
    K = np.exp(rng.standard_normal(nc))
    go = pdg.GridOperator(3, k, n, alpha=3.0)
    go.set_permeability(K)
    d = rng.uniform(-1, 1, go.ndof).astype(np.float32)
    v32 = [vec(torch, go.ndof, o) for o in (0, 1)]
    p32 = pdg.GridOperatorPreconditioner(go, precision=pdg.F32)
    p32.pre()
    for o in (0, 1):
        p32.apply(v32[o], vec(torch, go.ndof, o, d))
    v = np.zeros(go.ndof)
    p64 = pdg.GridOperatorPreconditioner(go)
    p64.pre()
    p64.apply(v, d.astype(np.float64))
    assert torch.equal(v32[0], v32[1])
    assert rel(v32[0].double().cpu().numpy(), v) <= 1e-4   # condition 1e2 of the factors
    # the fused sums and updates of the inner CG
    go.set_source(fc=np.ones(nc))
    sol = []
    for mixed in (False, True):
        ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go, mixed=mixed, inner_reduction=1e-4)
        u = torch.zeros(go.ndof, dtype=torch.float64, device="cuda")
        slp = pdg.StationaryLinearProblemSolver(go, ls, u, 1e-10)
        slp.apply()
        assert slp.result().converged
        sol.append(u.cpu().numpy())
    assert rel(sol[1], sol[0]) <= 1e-8
    go.close()


@pytest.mark.parametrize("k", [1, 2])
@pytest.mark.parametrize("n", [(8, 8, 3), (16, 8, 5), (9, 14, 4), (64, 1, 2)])
@pytest.mark.parametrize("offset", [0, 1])
def test_stacked_runs(k, n, offset):
    """Planes that (nearly) fill runs of 64 cells, odd and even numbers of them."""
    test_apply(k, n, offset)
    if offset == 0:
        test_fdm_and_mixed_solve(k, n)
