"""The nodal 3D operator with a tensor per cell (pdg_tensor.cu) against the
oracle: non-symmetric tensors, sizes around the block's cell count, and the
cell-diagonal form that the dense block Jacobi is built from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402
import pdg_oracle as O  # noqa: E402


def rel(y, ref):
    return np.max(np.abs(y - ref)) / np.max(np.abs(ref))


# cells per block: 32 (k=1), 14, 8, 5 (k=4)
@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(1, 1, 1), (15, 1, 1), (3, 11, 1), (4, 3, 5)])
@pytest.mark.parametrize("symmetric", [True, False])
def test_sizes(k, n, symmetric):
    rng = np.random.default_rng(k + sum(n))
    nc = int(np.prod(n))
    bct = [pdg.BC_DIRICHLET, pdg.BC_NONE, pdg.BC_NEUMANN, pdg.BC_DIRICHLET, pdg.BC_DIRICHLET,
           pdg.BC_NEUMANN]
    go = pdg.GridOperator(3, k, n, extent=[1.0, 0.7, 2.0], alpha=3.0, method=pdg.NIPG, bctype=bct)
    P = O.Problem(3, k, n, L=(1.0, 0.7, 2.0), alpha=3.0, method=pdg.NIPG, bctype=bct)
    G = rng.standard_normal((nc, 3, 3))
    A = G @ G.transpose(0, 2, 1) + 0.2 * np.eye(3)
    if not symmetric:
        A += 0.3 * (G - G.transpose(0, 2, 1))
    c = rng.uniform(0.5, 2.0, nc)
    go.set_permeability_tensor(A)
    go.set_reaction(c)
    P.set(Acell=A, c=c)
    x = rng.uniform(-1, 1, go.ndof)
    y = np.zeros(go.ndof)
    pdg.OnTheFlyOperator(go).apply(x, y)
    assert rel(y, P.jacobian_apply(x)) <= 1e-12
    y[:] = 0
    go.jacobian_apply_transpose(x, y)
    assert rel(y, P.jacobian_apply_transpose(x)) <= 1e-12
    # v = D^-1 d with the dense cell blocks, built by probing the diagonal
    # form: J restricted to one cell of a block-diagonal vector gives d back
    v = np.zeros(go.ndof)
    pr = pdg.GridOperatorPreconditioner(go, kind=pdg.PREC_BJ_DENSE)
    pr.pre()
    pr.apply(v, x)
    for e in {0, nc // 2, nc - 1}:
        one = np.zeros(go.ndof)
        s = slice(e * go.nbasis, (e + 1) * go.nbasis)
        one[s] = v[s]
        assert rel(P.jacobian_apply(one)[s], x[s]) <= 1e-9
    go.close()
