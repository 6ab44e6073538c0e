"""The 3D FP64 operator in 64-bit fixed point (pdg_apply_i.cu) against the
oracle: sizes around the block's cell count, every degree, both forms, wide
ranges of values and coefficients, and data its exponents cannot hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402
import pdg_oracle as O  # noqa: E402


def problem(k, n, seed=1, sigma=1.0, scale=1.0, **kw):
    rng = np.random.default_rng(seed)
    K = scale * np.exp(sigma * rng.standard_normal(int(np.prod(n))))
    go = pdg.GridOperator(3, k, n, alpha=3.0, **kw)
    go.set_permeability(K)
    return go, O.Problem(3, k, n, alpha=3.0, K=K, **kw), rng


def apply(go, x, transpose=False):
    y = np.zeros(go.ndof)
    if transpose:
        go.jacobian_apply_transpose(x, y)
    else:
        pdg.OnTheFlyOperator(go).apply(x, y)
    return y


def rel(y, ref):
    return np.max(np.abs(y - ref)) / np.max(np.abs(ref))


# cells per block: 32 (k=1), 14, 8, 5 (k=4); one cell, one less, equal, one
# more, and cells with all six neighbours
@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(1, 1, 1), (13, 1, 1), (5, 1, 3), (31, 1, 1), (3, 3, 3), (4, 3, 5)])
def test_sizes(k, n):
    go, P, rng = problem(k, n, method=pdg.NIPG)
    x = rng.uniform(-1, 1, go.ndof)
    # 57-bit operands and one rounding per stage against FP64 sums of the
    # same length: both within a few units of 1e-15 of the largest entry
    assert rel(apply(go, x), P.jacobian_apply(x)) <= 1e-14
    assert rel(apply(go, x, True), P.jacobian_apply_transpose(x)) <= 1e-14
    go.close()


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_wide_ranges(k):
    """Values over 12 decades from cell to cell, K over e^+-12: every cell is
    as accurate as its own terms allow."""
    go, P, rng = problem(k, (5, 4, 3), sigma=4.0)
    x = rng.uniform(-1, 1, (go.ncell, go.nbasis)) * 10.0 ** rng.uniform(-6, 6, (go.ncell, 1))
    y = apply(go, x.ravel()).reshape(go.ncell, -1)
    ref = P.jacobian_apply(x.ravel()).reshape(go.ncell, -1)
    # the sum of the magnitudes of a cell's terms: |J| |x| row sums bounded by
    # the block's largest output for the largest input is what FP64 rounds
    for e in range(go.ncell):
        assert np.max(np.abs(y[e] - ref[e])) <= 1e-12 * np.max(np.abs(ref[e])), e
    go.close()


@pytest.mark.parametrize("factor", [1e-290, 1e-200, 1e200, 1e290])
def test_ends_of_the_range(factor):
    go, P, rng = problem(2, (4, 3, 2))
    x = rng.uniform(-1, 1, go.ndof)
    ref = P.jacobian_apply(x)
    assert rel(apply(go, x * factor) / factor, ref) <= 1e-12
    go.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite(value):
    n = (7, 4, 3)
    go, P, rng = problem(2, n)
    x = rng.uniform(-1, 1, go.ndof)
    ref = P.jacobian_apply(x).reshape(go.ncell, -1)
    e = 2 + 7 * (1 + 4 * 1)
    x[e * go.nbasis:(e + 1) * go.nbasis] = value
    y = apply(go, x).reshape(go.ncell, -1)
    hit = {e, e - 1, e + 1, e - 7, e + 7, e - 28, e + 28}
    for c in range(go.ncell):
        if c in hit:
            assert not np.isfinite(y[c]).any()
        else:
            assert np.max(np.abs(y[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref))
    go.close()


def test_zeros_and_one_cell():
    """Zero vectors give zeros; a single non-zero cell reaches itself and its
    neighbours only."""
    n = (4, 4, 4)
    go, P, rng = problem(3, n)
    assert not apply(go, np.zeros(go.ndof)).any()
    x = np.zeros((go.ncell, go.nbasis))
    x[21] = rng.uniform(-1, 1, go.nbasis)
    assert rel(apply(go, x.ravel()), P.jacobian_apply(x.ravel())) <= 1e-14
    y = apply(go, x.ravel()).reshape(go.ncell, -1)
    assert {int(c) for c in np.nonzero(np.abs(y).max(1))[0]} == {21, 20, 22, 17, 25, 5, 37}
    go.close()


def test_extreme_coefficients():
    """K beyond the exponents of the limb records: the FP64 evaluation."""
    go, P, rng = problem(2, (3, 3, 2), scale=1e60)
    x = rng.uniform(-1, 1, go.ndof)
    assert rel(apply(go, x), P.jacobian_apply(x)) <= 1e-12
    go.close()


def block_residual(P, nb, e, v, d):
    """|D_e v_e - d_e| / |d_e| with the oracle's operator on one cell."""
    s = slice(e * nb, (e + 1) * nb)
    one = np.zeros(v.size)
    one[s] = v[s]
    return rel(P.jacobian_apply(one)[s], d[s])


@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(1, 1, 1), (13, 1, 1), (5, 1, 3), (31, 1, 1), (4, 3, 5)])
def test_fdm_sizes(k, n):
    go, P, rng = problem(k, n, sigma=2.0)
    d = rng.uniform(-1, 1, (go.ncell, go.nbasis)) * 10.0 ** rng.uniform(-6, 6, (go.ncell, 1))
    d = d.ravel()
    v = np.zeros(go.ndof)
    pr = pdg.GridOperatorPreconditioner(go)
    pr.pre()
    pr.apply(v, d)
    # the blocks' condition numbers reach 1e3 (k = 4): 1e3 roundings of 1e-16
    for e in range(go.ncell):
        assert block_residual(P, go.nbasis, e, v, d) <= 1e-11
    go.close()


def test_fdm_extremes():
    """Infinities stay in their cell; zeros give zeros; values near the ends
    of the range."""
    go, P, rng = problem(2, (7, 4, 3))
    pr = pdg.GridOperatorPreconditioner(go)
    pr.pre()
    d = rng.uniform(-1, 1, go.ndof)
    ref = np.zeros(go.ndof)
    pr.apply(ref, d)
    v = np.zeros(go.ndof)
    pr.apply(v, np.zeros(go.ndof))
    assert not v.any()
    for f in (1e-280, 1e270):
        pr.apply(v, d * f)
        assert rel(v / f, ref) <= 1e-13
    bad = d.copy()
    bad[9 * go.nbasis:10 * go.nbasis] = np.nan
    pr.apply(v, bad)
    hit = np.zeros(go.ndof, bool)
    hit[9 * go.nbasis:10 * go.nbasis] = True
    assert np.isnan(v[hit]).all()
    assert np.max(np.abs(v[~hit] - ref[~hit])) <= 1e-13 * np.max(np.abs(ref))
    go.close()


def convection(k, n, seed=9, sigma=1.0, **kw):
    go, P, rng = problem(k, n, seed=seed, sigma=sigma, **kw)
    modes = pdg.fourier_velocity_modes(seed)
    go.set_velocity_modes(modes)
    P.set_modes(modes)
    return go, P, rng


# cells per block: 32 (k=1), 14, 8, 5 (k=4)
@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(1, 1, 1), (15, 1, 1), (3, 11, 1), (4, 3, 5)])
@pytest.mark.parametrize("basis", [0, 2])
def test_convection_sizes(k, n, basis):
    """Equidistant and Gauss-Lobatto nodes: the 1D tables' scaling differs."""
    kw = dict(basis=basis) if basis else {}
    go, P, rng = convection(k, n, **kw)
    x = rng.uniform(-1, 1, go.ndof)
    assert rel(apply(go, x), P.jacobian_apply(x)) <= 1e-12
    go.close()


@pytest.mark.parametrize("k", [1, 2, 4])
def test_convection_wide_ranges(k):
    """K of 1e-12 leaves convection alone: a cell's result follows its own
    values and its upwind neighbours', however large the others are."""
    go, P, rng = convection(k, (5, 4, 3), scale=1e-12, sigma=0.1)
    x = rng.uniform(-1, 1, (go.ncell, go.nbasis)) * 10.0 ** rng.uniform(-3, 3, (go.ncell, 1))
    y = apply(go, x.ravel()).reshape(go.ncell, -1)
    ref = P.jacobian_apply(x.ravel()).reshape(go.ncell, -1)
    for e in range(go.ncell):
        assert np.max(np.abs(y[e] - ref[e])) <= 1e-12 * np.max(np.abs(ref[e])), e
    for f in (1e-280, 1e270):
        assert rel(apply(go, x.ravel() * f) / f, ref.ravel()) <= 1e-12
    go.close()


def test_convection_non_finite():
    n = (7, 4, 3)
    go, P, rng = convection(2, n)
    x = rng.uniform(-1, 1, go.ndof)
    ref = P.jacobian_apply(x).reshape(go.ncell, -1)
    e = 2 + 7 * (1 + 4 * 1)
    x[e * go.nbasis:(e + 1) * go.nbasis] = np.nan
    y = apply(go, x).reshape(go.ncell, -1)
    hit = {e, e - 1, e + 1, e - 7, e + 7, e - 28, e + 28}
    for c in range(go.ncell):
        if c in hit:
            assert not np.isfinite(y[c]).any()
        else:
            assert np.max(np.abs(y[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref))
    go.close()


@pytest.mark.parametrize("n", [(32, 1, 1), (33, 1, 1), (11, 3, 2), (5, 8, 2), (9, 7, 5)])
def test_degree2_groups(n):
    """Degree 2 works on groups of 32 cells (pdg_apply_p.cu): one more than a
    group, rows and planes that straddle groups, both forms."""
    test_sizes(2, n)


@pytest.mark.parametrize("e", [31, 32, 63])
def test_degree2_non_finite_at_group_ends(e):
    go, P, rng = problem(2, (70, 1, 1))
    x = rng.uniform(-1, 1, (go.ncell, go.nbasis))
    ref = P.jacobian_apply(x.ravel()).reshape(go.ncell, -1)
    x[e] = np.nan
    y = apply(go, x.ravel()).reshape(go.ncell, -1)
    for c in range(go.ncell):
        if abs(c - e) <= 1:
            assert not np.isfinite(y[c]).any()
        else:
            assert np.max(np.abs(y[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref))
    go.close()


def test_degree2_ranges():
    """Host vectors run in slabs that start inside a group: the same bits as
    one launch."""
    import torch
    go, P, rng = problem(2, (33, 31, 33))
    x = rng.uniform(-1, 1, go.ndof)
    xd, yd = torch.from_numpy(x).cuda(), torch.zeros(go.ndof, dtype=torch.float64, device="cuda")
    pdg.OnTheFlyOperator(go).apply(xd, yd)
    assert np.array_equal(apply(go, x), yd.cpu().numpy())
    go.close()


@pytest.mark.parametrize("n", [(33, 1, 1), (11, 3, 2)])
def test_degree2_unaligned_vectors(n):
    """Vectors that start 8 bytes off a 16-byte boundary: the same bits."""
    import torch
    go, P, rng = problem(2, n)
    x = torch.from_numpy(rng.uniform(-1, 1, go.ndof)).cuda()
    y = torch.zeros_like(x)
    pdg.OnTheFlyOperator(go).apply(x, y)
    xo, yo = (torch.zeros(go.ndof + 1, dtype=torch.float64, device="cuda")[1:] for _ in range(2))
    xo.copy_(x)
    pdg.OnTheFlyOperator(go).apply(xo, yo)
    assert torch.equal(y, yo) and rel(y.cpu().numpy(), P.jacobian_apply(x.cpu().numpy())) <= 1e-14
    go.close()


def smooth(k, n):
    """sin sin sin at the nodes: J x is far below the terms it is the sum of."""
    c = (np.arange(n)[:, None] + np.arange(k + 1)[None, :] / k) / n
    f = np.sin(3.0 * c + 0.1)
    u = (f[:, None, None, :, None, None] * f[None, :, None, None, :, None]
         * f[None, None, :, None, None, :])
    return u.reshape(-1).copy()


@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["plain", "transpose", "tensor", "convection"])
def test_odd_and_rounding_of_smooth_data(k, kind):
    """J(-x) = -J(x) to the bit; and on smooth data, where the terms of J x cancel,
    J(3x) - 3 J(x) is rounding of the size that FP64 leaves on those terms: with
    random signs the same values do not cancel, |J(+-x)| is the size of the
    terms, and two evaluations with a handful of roundings of 2^-53 each leave
    no more than 3 * 8 * 2^-53 of it."""
    n = (6, 6, 6)
    go, P, rng = problem(k, n)
    if kind == "tensor":
        G = rng.standard_normal((216, 3, 3))
        go.set_permeability_tensor(G @ G.transpose(0, 2, 1) + 0.2 * np.eye(3))
    if kind == "convection":
        go.set_velocity_modes(pdg.fourier_velocity_modes(1))
    x = rng.uniform(-1, 1, go.ndof)
    tr = kind == "transpose"
    assert np.array_equal(apply(go, -x, tr), -apply(go, x, tr))
    u = smooth(k, n[0])
    terms = np.linalg.norm(apply(go, u * rng.choice([-1.0, 1.0], u.size), tr))
    noise = np.linalg.norm(apply(go, 3 * u, tr) - 3 * apply(go, u, tr))
    assert noise <= 3 * 8 * 2.0 ** -53 * terms
    go.close()


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_rounding_of_convection_alone(k):
    """The bound of the test above where convection is all of J."""
    go, P, rng = problem(k, (6, 6, 6), scale=1e-9)
    go.set_velocity_modes(pdg.fourier_velocity_modes(1))
    u = smooth(k, 6)
    terms = np.linalg.norm(apply(go, u * rng.choice([-1.0, 1.0], u.size)))
    noise = np.linalg.norm(apply(go, 3 * u) - 3 * apply(go, u))
    assert noise <= 3 * 8 * 2.0 ** -53 * terms
    assert not apply(go, np.zeros(go.ndof)).any()
    go.close()
