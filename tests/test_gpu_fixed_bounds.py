"""The integer bounds of the fixed-point kernels: every value at the top of its
block's binade, with the signs of a row of J (the largest result that values of
this size can give), of a row of a 1D operator times rows of the 1D mass matrix
(the largest value of one stage), or at random; coefficients over a binade.  An
integer sum that does not fit wraps without a trace and is wrong by more than its
bound, against errors of 1e-14; the oracle's own rounding is below 1e-13.
Cells and tensors stretched over decades follow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402
import pdg_oracle as O  # noqa: E402

N3 = (3, 3, 3)
CENTRE = 13                       # the cell with all six neighbours
TOP = 2.0 - 2.0 ** -52
SCALES = [1.0, 1.3, 1.7, TOP]


def rel(y, ref):
    return np.max(np.abs(y - ref)) / np.max(np.abs(ref))


def signs(a):
    return np.where(a < 0, -1.0, 1.0)


def line_operators(k):
    """1D mass matrix and the 1D operator of an inner cell (K = 1, 3 cells, alpha 3)"""
    N, h = k + 1, 1.0 / 3
    polys = []
    for i in range(N):
        p = np.poly1d([1.0])
        for j in range(N):
            if j != i:
                p = p * np.poly1d([k, -j]) / (i - j)
        polys.append(p)
    M, A = np.zeros((N, N)), np.zeros((N, N))
    for i, p in enumerate(polys):
        for j, q in enumerate(polys):
            M[i, j] = np.polyint(p * q)(1.0)
            A[i, j] = np.polyint(p.deriv() * q.deriv())(1.0) / h
    pen = 3.0 * k * (k + 2) / h
    for end, n in ((0, -1.0), (1, 1.0)):
        v = np.array([p(end) for p in polys])
        d = np.array([p.deriv()(end) for p in polys]) / h
        A += pen * np.outer(v, v) - 0.5 * n * (np.outer(v, d) + np.outer(d, v))
    return M, A


def patterns(k, row, rng, rows=12, stages=12, random=6):
    nb = (k + 1) ** 3
    for i in rng.permutation(nb)[:rows]:
        e = np.zeros(27 * nb)
        e[CENTRE * nb + i] = 1.0
        yield signs(row(e))
    M, A = (signs(m) for m in line_operators(k))
    for _ in range(stages):
        f = [M, M, M]
        f[rng.integers(3)] = A
        z, y, x = (m[rng.integers(k + 1)] for m in f)
        own = (z[:, None, None] * y[None, :, None] * x[None, None, :]).ravel()
        yield (rng.choice([-1.0, 1.0], (27, 1)) * own[None, :]).ravel()
    for _ in range(random):
        yield rng.choice([-1.0, 1.0], 27 * nb)


def pair(k, kind, scale, seed, **kw):
    """the operator of one kind with its coefficients times a scale"""
    rng = np.random.default_rng(seed)
    go = pdg.GridOperator(3, k, N3, alpha=3.0, **kw)
    K = np.full(27, (1e-9 if kind == "convection" else 1.0) * scale)
    P = O.Problem(3, k, N3, alpha=3.0, K=K, **kw)
    go.set_permeability(K)
    if kind == "tensor":
        G = rng.standard_normal((3, 3))
        A = np.tile(scale * (G @ G.T + 0.2 * np.eye(3)), (27, 1, 1))
        go.set_permeability_tensor(A)
        P.set(Acell=A)
    if kind == "convection":             # all of J but 1e-9 of it
        modes = pdg.fourier_velocity_modes(seed)
        modes[:, 4:] *= scale
        go.set_velocity_modes(modes)
        P.set_modes(modes)
    return go, P, rng


@pytest.fixture(scope="module")
def references():
    """(kind, degree) -> vectors and the oracle's results at scale 1"""
    return {}


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["plain", "transpose", "tensor", "convection"])
def test_operator(references, kind, k, scale):
    tr = kind == "transpose"
    kw = dict(method=pdg.NIPG) if tr else {}
    if (kind, k) not in references:
        go, P, rng = pair(k, kind, 1.0, k, **kw)
        go.close()
        apply, row = P.jacobian_apply, P.jacobian_apply_transpose
        if tr:
            apply, row = row, apply
        xs = [s * TOP for s in patterns(k, row, rng)]
        references[kind, k] = [(x, apply(x)) for x in xs]
    go, P, rng = pair(k, kind, scale, k, **kw)
    for x, ref in references[kind, k]:
        y = np.zeros(go.ndof)
        if tr:
            go.jacobian_apply_transpose(x, y)
        else:
            pdg.OnTheFlyOperator(go).apply(x, y)
        assert rel(y, scale * ref) <= 1e-12
    go.close()


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("k", [1, 2, 3])
def test_block_jacobi(k, scale):
    go, P, rng = pair(k, "plain", scale, k)
    nb = go.nbasis
    inv = np.linalg.inv(P.block_diagonal()[CENTRE])
    D = P.block_diagonal()
    pr = pdg.GridOperatorPreconditioner(go)
    pr.pre()
    for i in range(min(nb, 20)):
        d, v = np.tile(signs(inv[i]) * TOP, 27), np.zeros(go.ndof)
        pr.apply(v, d)
        r = np.einsum("eij,ej->ei", D, v.reshape(27, nb)).ravel() - d
        # the blocks' condition numbers reach 1e3: 1e3 roundings of 1e-16
        assert np.max(np.abs(r)) <= 1e-11 * TOP
    go.close()


@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("extent,tensor", [
    ((1.0, 1.0, 1e-2), None), ((1e-4, 1.0, 1.0), None),
    ((1.0, 1.0, 1.0), (1.0, 1e-4, 1.0)), ((1.0, 1.0, 1.0), (1e-8, 1.0, 1.0))])
def test_stretched(k, extent, tensor):
    """Cells and diagonal tensors over decades: the three directions share one
    exponent, so the weak one keeps fewer bits of its own, but no fewer of the
    result's: a constant along the strong directions leaves the weak one's terms
    beside terms that cancel, and those have the size that rounds in FP64 too."""
    n = (5, 4, 3)
    rng = np.random.default_rng(k)
    go = pdg.GridOperator(3, k, n, extent=list(extent), alpha=3.0)
    P = O.Problem(3, k, n, L=extent, alpha=3.0, K=np.ones(60))
    K = np.exp(0.5 * rng.standard_normal(60))
    if tensor:
        A = np.zeros((60, 3, 3))
        for j in range(3):
            A[:, j, j] = K * tensor[j]
        go.set_permeability_tensor(A)
        P.set(Acell=A)
    else:
        go.set_permeability(K)
        P.set(K=K)
    x, y = rng.uniform(-1, 1, go.ndof), np.zeros(go.ndof)
    pdg.OnTheFlyOperator(go).apply(x, y)
    assert rel(y, P.jacobian_apply(x)) <= 1e-12
    y[:] = 0.0
    go.jacobian_apply_transpose(x, y)
    assert rel(y, P.jacobian_apply_transpose(x)) <= 1e-12
    # smooth in one direction: rounding against the size of the terms
    op = pdg.OnTheFlyOperator(go)

    def J(u):
        out = np.zeros(go.ndof)
        op.apply(u, out)
        return out

    N = k + 1
    for d in range(3):
        f = [np.ones((m, N)) for m in n]
        f[d] = np.sin(3.0 * (np.arange(n[d])[:, None] + np.arange(N) / k) / n[d] + 0.1)
        u = (f[2][:, None, None, :, None, None] * f[1][None, :, None, None, :, None]
             * f[0][None, None, :, None, None, :]).reshape(-1).copy()
        terms = np.linalg.norm(J(u * rng.choice([-1.0, 1.0], u.size)))
        noise = np.linalg.norm(J(3 * u) - 3 * J(u))
        assert noise <= 3 * 8 * 2.0 ** -53 * terms
    go.close()
