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


def cells(k, n, seed, scale=1.0, sigma=0.0):
    rng = np.random.default_rng(seed)
    nc = int(np.prod(n))
    G = rng.standard_normal((nc, 3, 3))
    A = G @ G.transpose(0, 2, 1) + 0.2 * np.eye(3)
    A *= scale * np.exp(sigma * rng.standard_normal((nc, 1, 1)))
    go = pdg.GridOperator(3, k, n, alpha=3.0)
    P = O.Problem(3, k, n, alpha=3.0)
    go.set_permeability_tensor(A)
    P.set(Acell=A)
    return go, P, rng


def apply(go, x):
    y = np.zeros(go.ndof)
    pdg.OnTheFlyOperator(go).apply(x, y)
    return y


@pytest.mark.parametrize("k", [1, 2, 3])
def test_fixed_point_ranges(k):
    """Degrees 1 to 3 run in 64-bit fixed point: values over 12 decades and
    tensors over e^+-9 from cell to cell; 57-bit operands leave every cell 1e-12
    of its own largest value."""
    go, P, rng = cells(k, (5, 4, 3), 1, sigma=3.0)
    x = rng.uniform(-1, 1, (go.ncell, go.nbasis)) * 10.0 ** rng.uniform(-6, 6, (go.ncell, 1))
    y = apply(go, x.ravel()).reshape(go.ncell, -1)
    ref = P.jacobian_apply(x.ravel()).reshape(go.ncell, -1)
    for e in range(go.ncell):
        assert np.max(np.abs(y[e] - ref[e])) <= 1e-12 * np.max(np.abs(ref[e])), e
    assert not apply(go, np.zeros(go.ndof)).any()
    go.close()


@pytest.mark.parametrize("factor,scale", [(1e-290, 1.0), (1e200, 1.0), (1.0, 1e60)])
def test_fixed_point_ends_of_the_range(factor, scale):
    """Values and tensors beyond the exponents of the limbs: the FP64 form."""
    go, P, rng = cells(2, (4, 3, 2), 2, scale=scale)
    x = rng.uniform(-1, 1, go.ndof)
    assert rel(apply(go, x * factor) / factor, P.jacobian_apply(x)) <= 1e-12
    go.close()


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_fixed_point_non_finite(value):
    go, P, rng = cells(2, (7, 4, 3), 3)
    x = rng.uniform(-1, 1, (go.ncell, go.nbasis))
    ref = P.jacobian_apply(x.ravel()).reshape(go.ncell, -1)
    e = 2 + 7 * (1 + 4 * 1)
    x[e] = value
    y = apply(go, x.ravel()).reshape(go.ncell, -1)
    hit = {e, e - 1, e + 1, e - 7, e + 7, e - 28, e + 28}
    for c in range(go.ncell):
        if c in hit:
            assert not np.isfinite(y[c]).all()
        else:
            assert np.max(np.abs(y[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref))
    go.close()


def test_fixed_point_follows_the_coefficients():
    """A changed tensor or reaction rebuilds the limb coefficients."""
    go, P, rng = cells(2, (3, 3, 2), 4)
    x = rng.uniform(-1, 1, go.ndof)
    apply(go, x)
    A = np.tile(np.array([[2.0, 0.3, 0.1], [0.3, 1.0, 0.2], [0.1, 0.2, 3.0]]), (go.ncell, 1, 1))
    c = rng.uniform(0.5, 2.0, go.ncell)
    go.set_permeability_tensor(A)
    go.set_reaction(c)
    P.set(Acell=A, c=c)
    assert rel(apply(go, x), P.jacobian_apply(x)) <= 1e-13
    go.close()
