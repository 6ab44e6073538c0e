"""The work that programs built on this library have it do, as measurable cases.

Every case goes through the public classes of ``dune-pdelab_gb300/pdg.py`` and
``pdg_torch.py``: single operator and preconditioner applies (the kernels of
every Krylov iteration), and whole solves and gradients as a driver calls them.
``exact`` restates the operator in plain torch at the Gauss points, in 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "dune-pdelab_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import pdg  # noqa: E402
import pdg_torch  # noqa: E402

ALPHA = 3.0                       # penalty factor of the workloads (sigma = 3 k (k+d-1))
BMAX = 10.0                       # bound of |b| of the convection workload
METHODS = {"sipg": pdg.SIPG, "nipg": pdg.NIPG, "iipg": pdg.IIPG}
THETA = {"sipg": -1.0, "nipg": 1.0, "iipg": 0.0}
BCS = {"D": pdg.BC_DIRICHLET, "N": pdg.BC_NEUMANN}
DEV = "cuda:0"


def _case(name, kind, dim, degree, cells, **kw):
    c = {"kind": kind, "dim": dim, "degree": degree,
         "nx": cells[0], "ny": cells[1], "nz": cells[2] if dim == 3 else 1,
         "bits": 64, "method": "sipg", "bc": "DDDDDD", "reaction": False,
         "convection": False, "coefficient": "scalar", "host": False, "sigma": 1.0}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one operator apply on a coarse 2D grid (coarse
        # levels, tests, time loops): latency and launches
        _case("apply_q2_2d_31x33", "apply", 2, 2, (31, 33)),
        # the headline apply: FP64 J x, 3D Q2 64^3, log-normal K
        _case("apply_q2_3d_64", "apply", 3, 2, (64, 64, 64)),
        # the adjoint's operator at the highest degree, odd sizes, mixed
        # boundary types, reaction
        _case("transpose_q4_3d_33x29x37", "transpose", 3, 4, (33, 29, 37), method="nipg",
              bc="DNDDND", reaction=True),
        # convection-diffusion-reaction apply (upwind), the operator of the
        # BiCGStab workload
        _case("apply_cdr_q4_3d_32", "apply", 3, 4, (32, 32, 32), reaction=True,
              convection=True),
        # anisotropic media: a full tensor per cell (Gauss-point operator)
        _case("apply_tensor_q2_3d_41x37x39", "apply", 3, 2, (41, 37, 39),
              coefficient="tensor"),
        # the inner operator of the mixed-precision solve at its full size
        _case("apply_f32_q3_3d_96", "apply", 3, 3, (96, 96, 96), bits=32, sigma=1.5),
        # the preconditioner of every FP64 iteration (fast diagonalisation)
        _case("prec_q3_3d_47x53x49", "prec", 3, 3, (47, 53, 49)),
        # an apply on host vectors in pinned memory, the drop-in boundary of a
        # host program
        _case("host_apply_q2_3d_64", "apply", 3, 2, (64, 64, 64), host=True),
        # a whole small solve: 2D Q1 64^2 Poisson, CG to 1e-10
        _case("solve_cg_q1_2d_64", "solve", 2, 1, (64, 64), sigma=0.0, mixed=False),
        # a whole FP64 solve in 3D, CG + block Jacobi
        _case("solve_cg_q2_3d_24", "solve", 3, 2, (24, 24, 24), mixed=False),
        # the mixed-precision solve, FP32 CG inside FP64 defect correction
        _case("solve_mixed_q2_3d_64", "solve", 3, 2, (64, 64, 64), mixed=True),
        # differentiable solve: forward, adjoint solve and gradients (autograd)
        _case("gradient_q2_3d_32", "gradient", 3, 2, (32, 32, 32)),
    ]


def _cells(rng, dim, degree, lo, hi):
    """Cells per direction for a DOF count log-uniform in [lo, hi], odd sizes
    and aspect ratios included."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi))) / (degree + 1) ** dim
    side = max(2.0, n ** (1.0 / dim))
    c = [max(2, int(round(side * math.exp(rng.uniform(-0.3, 0.3))))) for _ in range(dim)]
    while math.prod(c) * (degree + 1) ** dim > hi:
        i = c.index(max(c))
        c[i] -= 1
    return tuple(c)


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "transpose", "prec", "solve", "gradient"])
    dim = rng.choice([2, 3, 3])
    method = "sipg"
    bc = "".join(rng.choice("DDDN") for _ in range(6))
    if "D" not in bc[:2 * dim]:
        bc = "D" + bc[1:]
    if kind in ("apply", "transpose"):
        degree = rng.choice([1, 2, 3, 4])
        method = rng.choice(["sipg", "sipg", "nipg", "iipg"])
        coefficient, convection, bits, host = "scalar", False, 64, False
        hi = 8e6 if dim == 3 else 2e6
        if kind == "apply":
            what = rng.choice(["plain", "plain", "f32", "f32", "host", "convection", "tensor"])
            bits = 32 if what == "f32" else 64
            host = what == "host"
            convection = what == "convection"
            coefficient = "tensor" if what == "tensor" else "scalar"
            if what in ("convection", "tensor"):
                hi = 3e6
        return _case(None, kind, dim, degree, _cells(rng, dim, degree, 5e3, hi), method=method,
                     bc=bc, reaction=rng.random() < 0.3, convection=convection,
                     coefficient=coefficient, bits=bits, host=host)
    if kind == "prec":
        degree = rng.choice([1, 2, 3, 4])
        return _case(None, kind, dim, degree,
                     _cells(rng, dim, degree, 5e3, 8e6 if dim == 3 else 2e6),
                     bc=bc, bits=rng.choice([64, 32]))
    if kind == "solve":
        mixed = dim == 3 and rng.random() < 0.5
        degree = rng.choice([1, 2, 3])
        hi = 3e6 if mixed else (3e5 if dim == 3 else 5e4)
        return _case(None, kind, dim, degree, _cells(rng, dim, degree, 2e3, hi), bc=bc,
                     reaction=rng.random() < 0.3, mixed=mixed)
    degree = rng.choice([1, 2])
    return _case(None, kind, 3, degree, _cells(rng, 3, degree, 5e3, 5e5), bc=bc)


# ---- inputs ----------------------------------------------------------------
def _grid(case):
    cells = [case["nx"], case["ny"], case["nz"]][:case["dim"]]
    return cells, math.prod(cells), (case["degree"] + 1) ** case["dim"]


def _modes(case, seed):
    """Fourier modes (kx ky kz phase cx cy cz) of a divergence-free velocity
    bounded by BMAX."""
    r, d = np.random.default_rng([seed, 7]), case["dim"]
    m = np.zeros((8, 7))
    for row in m:
        k = np.zeros(3)
        while not k[:d].any():
            k[:d] = r.integers(-2, 3, d)
        a = r.standard_normal(3)
        row[:3], row[3] = k, r.uniform(0, 2 * np.pi)
        row[4:] = np.cross(k, a) if d == 3 else [-k[1] * a[0], k[0] * a[0], 0.0]
    m[:, 4:] *= BMAX / np.linalg.norm(m[:, 4:], axis=1).sum()
    return m


def _inputs(case, seed):
    """Coefficients and vectors from the seed alone (tensors on the GPU)."""
    g = torch.Generator(DEV).manual_seed(int(seed) * 1000003 + 17)
    cells, nc, nb = _grid(case)
    d = case["dim"]

    def normal(*s):
        return torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)

    def uniform(*s):
        return 2 * torch.rand(*s, generator=g, device=DEV, dtype=torch.float64) - 1

    v = {"logK": case["sigma"] * normal(nc)}
    if case["coefficient"] == "tensor":
        # symmetric positive definite, not aligned with the axes
        G = normal(nc, d, d)
        v["A"] = G @ G.transpose(1, 2) / d + 0.1 * torch.eye(d, device=DEV, dtype=torch.float64)
        v["A"] = torch.exp(v["logK"])[:, None, None] * 0.5 * (v["A"] + v["A"].transpose(1, 2))
    if case["reaction"]:
        v["c"] = 1.0 + 0.5 * uniform(nc)
    if case["convection"]:
        v["modes"] = _modes(case, seed)
    if case["kind"] in ("solve", "gradient"):
        v["f"] = 1.0 + 0.1 * normal(nc)
        v["w"] = uniform(nc * nb)
    else:
        v["x"] = uniform(nc * nb)
        if case["bits"] == 32:
            v["x"] = v["x"].float()
    return v


def prepare(case, seed):
    cells, nc, nb = _grid(case)
    v = _inputs(case, seed)
    go = pdg.GridOperator(case["dim"], case["degree"], cells, method=METHODS[case["method"]],
                          alpha=ALPHA, bctype=[BCS[b] for b in case["bc"]])
    go.set_permeability(v["logK"], is_log=True)
    if "A" in v:
        go.set_permeability_tensor(v["A"].cpu().numpy())
    if "c" in v:
        go.set_reaction(v["c"].cpu().numpy())
    if "modes" in v:
        go.set_velocity_modes(v["modes"])
    s = {"case": case, "go": go}
    kind = case["kind"]
    if kind in ("apply", "transpose", "prec"):
        s["x"], s["y"] = v["x"], torch.zeros_like(v["x"])
        if case["host"]:
            s["x"] = v["x"].cpu().pin_memory().numpy()
            s["y"] = torch.zeros(nc * nb, dtype=torch.float64, pin_memory=True).numpy()
        s["op"] = pdg.OnTheFlyOperator(go)
        if kind == "prec":
            s["prec"] = pdg.GridOperatorPreconditioner(
                go, precision=pdg.F64 if case["bits"] == 64 else pdg.F32)
            s["prec"].pre()
    elif kind == "solve":
        go.set_source(fc=v["f"].cpu().numpy())
        s["u"] = torch.zeros(nc * nb, dtype=torch.float64, device=DEV)
        ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go, method=pdg.CG, maxiter=20000,
                                                 mixed=case["mixed"], inner_reduction=1e-4)
        s["slp"] = pdg.StationaryLinearProblemSolver(go, ls, s["u"], 1e-10)
    else:
        s["problem"] = pdg_torch.DGProblem(go, reduction=1e-11)
        s["logK"] = v["logK"].requires_grad_()
        s["f"], s["w"] = v["f"].requires_grad_(), v["w"]
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        if case["bits"] == 32:
            state["go"].apply_f32(state["x"], state["y"])
        else:
            state["op"].apply(state["x"], state["y"])
        return state["y"]
    if kind == "transpose":
        state["y"].zero_()
        return state["go"].jacobian_apply_transpose(state["x"], state["y"])
    if kind == "prec":
        state["prec"].apply(state["y"], state["x"])
        return state["y"]
    if kind == "solve":
        state["u"].zero_()
        return state["slp"].apply()
    u = pdg_torch.solve_dg(state["logK"], state["f"], state["problem"])
    gk, gf = torch.autograd.grad(u, [state["logK"], state["f"]], state["w"])
    return {"u": u.detach(), "dlogK": gk, "df": gf}


def work(case):
    """Vectors and coefficients read and written once; multiply-adds of the
    operator in Kronecker form (d 1D operators, the mass matrices and the
    face terms), for solves of one residual evaluation."""
    cells, nc, nb = _grid(case)
    N, d, b = case["degree"] + 1, case["dim"], case["bits"] // 8
    coef = d * d if case["coefficient"] == "tensor" else 1
    coef += 1 if case["reaction"] else 0
    faces = 2 * d * N ** (d - 1) * 3 * N
    mac = {"apply": 2 * d * N ** (d + 1) + faces, "prec": 2 * d * N ** (d + 1) + N ** d}
    mac["transpose"] = mac["solve"] = mac["apply"]
    mac["gradient"] = 2 * mac["apply"]
    vectors = {"apply": 2, "transpose": 2, "prec": 2, "solve": 1, "gradient": 2}
    more = 3 if case["kind"] == "gradient" else 1 if case["kind"] == "solve" else 0
    if case["convection"]:
        mac["apply"] += 2 * d * N ** (d + 1)
    if case["coefficient"] == "tensor":
        mac["apply"] += 4 * d * N ** (d + 1)
    return {"bytes": float(nc * (vectors[case["kind"]] * nb * b + 8 * (coef + more))),
            "flops": 2.0 * mac[case["kind"]] * nc}


# ---- the same in plain torch, 64 bits ---------------------------------------
class _Plain:
    """The bilinear form of the interior penalty method evaluated at its Gauss
    points.  Fields are [cells z,y,x][local z,y,x] (2D: y,x)."""

    def __init__(self, case, v):
        self.case, self.d, self.N = case, case["dim"], case["degree"] + 1
        self.cells = [case["nx"], case["ny"], case["nz"]][:self.d]
        self.h = [1.0 / n for n in self.cells]
        k, N = case["degree"], self.N
        x, w = np.polynomial.legendre.leggauss(N)
        self.xq, self.wq = 0.5 * (x + 1), torch.tensor(0.5 * w, device=DEV)
        polys = [np.poly1d([1.0]) for _ in range(N)]
        for i in range(N):
            for j in range(N):
                if j != i:
                    polys[i] = polys[i] * np.poly1d([k, -j]) / (i - j)

        def table(points, deriv):
            t = [[(p.deriv() if deriv else p)(s) for p in polys] for s in points]
            return torch.tensor(np.array(t), device=DEV)

        self.B, self.D = table(self.xq, False), table(self.xq, True)
        self.e = [table([0.0], False), table([1.0], False)]
        self.g = [table([0.0], True), table([1.0], True)]
        self.theta = THETA[case["method"]]
        self.pen = ALPHA * k * (k + self.d - 1)
        self.modes = v.get("modes")
        self.c = None if v.get("c") is None else self.per_cell(v["c"])
        self.A = v.get("A")
        if self.A is not None:
            self.A = [[self.per_cell(self.A[:, i, j]) for j in range(self.d)]
                      for i in range(self.d)]

    def per_cell(self, a):
        return a.reshape(self.cells[::-1] + [1] * self.d)

    def tensor(self, K, i, j):
        if self.A is not None:
            return self.A[i][j]
        return K if i == j else None

    def along(self, T, M, j):
        ax = self.d + self.d - 1 - j
        return torch.movedim(torch.tensordot(T, M, dims=([ax], [1])), -1, ax)

    def kron(self, T, mats, transposed=False):
        for j, M in enumerate(mats):
            T = self.along(T, M.t() if transposed else M, j)
        return T

    def weights(self, skip=None):
        W = torch.ones([1] * (2 * self.d), dtype=torch.float64, device=DEV)
        for j in range(self.d):
            if j != skip:
                s = [1] * (2 * self.d)
                s[self.d + self.d - 1 - j] = self.N
                W = W * (self.wq * self.h[j]).reshape(s)
        return W

    def velocity(self, i, skip=None, planes=None):
        """b_i at the volume points, or at the face points of the planes of
        direction `skip`."""
        arg = []
        for j in range(self.d):
            s = [1] * (2 * self.d)
            if j == skip:
                t = torch.tensor(planes, dtype=torch.float64, device=DEV) * self.h[j]
                s[self.d - 1 - j] = len(planes)
            else:
                t = (torch.arange(self.cells[j], device=DEV)[:, None]
                     + torch.tensor(self.xq, device=DEV)) * self.h[j]
                s[self.d - 1 - j], s[self.d + self.d - 1 - j] = self.cells[j], self.N
            arg.append(t.reshape(s))
        b = 0.0
        for m in self.modes:
            b = b + m[4 + i] * torch.sin(2 * math.pi * sum(float(m[j]) * arg[j]
                                                           for j in range(self.d)) + m[3])
        return b

    def grad_mats(self, i, face=None):
        """1D matrices of d/dx_i (i None: of the value) at the volume points,
        or on the face (direction, upper)."""
        mats = []
        for j in range(self.d):
            if face is not None and j == face[0]:
                mats.append(self.g[face[1]] / self.h[j] if j == i else self.e[face[1]])
            else:
                mats.append(self.D / self.h[j] if j == i else self.B)
        return mats

    def traces(self, U, K, j, hi, cut):
        """value and (A e_j).grad on a face, and A e_j's entries"""
        a = [self.tensor(K, i, j) for i in range(self.d)]
        a = [None if t is None else cut(t) for t in a]
        val = self.kron(U, self.grad_mats(None, (j, hi)))
        flux = sum(a[i] * self.kron(U, self.grad_mats(i, (j, hi)))
                   for i in range(self.d) if a[i] is not None)
        return val, flux, a

    def test(self, j, hi, a, v, s):
        """int v psi + s (A e_j).grad psi over a face"""
        W = self.weights(j)
        y = self.kron(W * v, self.grad_mats(None, (j, hi)), True)
        for i in range(self.d):
            if a[i] is not None:
                y = y + self.kron(W * s * a[i], self.grad_mats(i, (j, hi)), True)
        return y

    def apply(self, x, K, coupled=True):
        """J x; coupled False: its cell-diagonal blocks only"""
        d = self.d
        U = x.reshape(self.cells[::-1] + [self.N] * d)
        K = self.per_cell(K)
        W = self.weights()
        grads = [self.kron(U, self.grad_mats(i)) for i in range(d)]
        uq = self.kron(U, self.grad_mats(None)) if self.c is not None or self.modes is not None \
            else None
        Y = torch.zeros_like(U)
        for i in range(d):
            flux = sum(self.tensor(K, i, j) * grads[j] for j in range(d)
                       if self.tensor(K, i, j) is not None)
            if self.modes is not None:
                flux = flux - self.velocity(i) * uq
            Y = Y + self.kron(W * flux, self.grad_mats(i), True)
        if self.c is not None:
            Y = Y + self.kron(W * self.c * uq, self.grad_mats(None), True)
        for j in range(d):
            n, ax = self.cells[j], d - 1 - j
            sl = [slice(None)] * (2 * d)

            def cut(lo, hi):
                s = list(sl)
                s[ax] = slice(lo, hi)
                return lambda t: t[tuple(s)] if t.shape[ax] == n else t

            def add(y, lo, hi):
                shape = list(Y.shape)
                pads = []
                for q in (lo, n - hi):
                    shape[ax] = q
                    pads.append(torch.zeros(shape, dtype=Y.dtype, device=DEV))
                return torch.cat([pads[0], y, pads[1]], dim=ax)

            if n > 1:
                lo, up = cut(0, n - 1), cut(1, n)
                vs, fs, As = self.traces(lo(U), K, j, 1, lo)
                vn, fn, An = self.traces(up(U), K, j, 0, up)
                ds, dn = As[j], An[j]
                S = ds + dn + 1e-20
                ws, wn = dn / S, ds / S
                gam = self.pen / self.h[j] * 2 * ds * dn / S
                bn = None
                if self.modes is not None:
                    bn = self.velocity(j, j, list(range(1, n)))

                def rows(vs, fs, vn, fn):
                    jump, avg = vs - vn, ws * fs + wn * fn
                    t = gam * jump - avg
                    if bn is not None:
                        t = t + bn * torch.where(bn >= 0, vs, vn)
                    return t, self.theta * jump

                if coupled:
                    t, q = rows(vs, fs, vn, fn)
                    ts, qs, tn, qn = t, q, t, q
                else:
                    z, zf = torch.zeros_like(vn), torch.zeros_like(fn)
                    ts, qs = rows(vs, fs, z, zf)
                    tn, qn = rows(z, zf, vn, fn)
                Y = Y + add(self.test(j, 1, As, ts, ws * qs), 0, n - 1)
                Y = Y + add(self.test(j, 0, An, -tn, wn * qn), 1, n)
            for hi in (0, 1):
                if self.case["bc"][2 * j + hi] != "D":
                    continue      # Neumann: no term in u (convection: see below)
                at = cut(n - 1, n) if hi else cut(0, 1)
                val, flux, a = self.traces(at(U), K, j, hi, at)
                sg = 1.0 if hi else -1.0
                t = self.pen / self.h[j] * a[j] * val - sg * flux
                if self.modes is not None:
                    bn = sg * self.velocity(j, j, [n if hi else 0])
                    t = t + torch.clamp(bn, min=0.0) * val
                Y = Y + add(self.test(j, hi, a, t, sg * self.theta * val),
                            n - 1 if hi else 0, n if hi else 1)
        return Y.reshape(-1)

    def blocks(self, K):
        """cell-diagonal blocks [cells][n][n]"""
        n = self.N ** self.d
        nc = math.prod(self.cells)
        out = torch.empty(nc, n, n, dtype=torch.float64, device=DEV)
        for j in range(n):
            e = torch.zeros(nc, n, dtype=torch.float64, device=DEV)
            e[:, j] = 1.0
            out[:, :, j] = self.apply(e.reshape(-1), K, coupled=False).reshape(nc, n)
        return out

    def source(self, f):
        """int f psi"""
        F = self.per_cell(f) * self.weights()
        return self.kron(F, self.grad_mats(None), True).reshape(-1)

    def solve(self, K, b, reduction=1e-14, maxit=6000):
        """CG with the cell blocks as preconditioner"""
        inv = torch.linalg.inv(self.blocks(K))
        nc, n = inv.shape[0], inv.shape[1]

        def prec(r):
            return torch.bmm(inv, r.reshape(nc, n, 1)).reshape(-1)

        x, best = torch.zeros_like(b), None
        r = b.clone()
        z = prec(r)
        p, rho, stop = z.clone(), torch.dot(r, z), reduction * float(torch.linalg.norm(b))
        for it in range(maxit):
            q = self.apply(p, K)
            lam = rho / torch.dot(p, q)
            x, r = x + lam * p, r - lam * q
            if it % 50 == 49 or it + 1 == maxit:
                t = float(torch.linalg.norm(r))
                if t < stop:
                    return x
            z = prec(r)
            new = torch.dot(r, z)
            p, rho = z + (new / rho) * p, new
        return best


def exact(case, seed):
    v = _inputs(case, seed)
    P = _Plain(case, v)
    cells, nc, nb = _grid(case)
    K = torch.exp(v["logK"])
    kind = case["kind"]
    with torch.no_grad():
        if kind == "apply":
            y = P.apply(v["x"].double(), K)
            return y.cpu().numpy() if case["host"] else y
        if kind == "prec":
            r = v["x"].double().reshape(nc, nb, 1)
            return torch.linalg.solve(P.blocks(K), r).reshape(-1)
        if kind == "solve":
            if nc * nb > 500_000:
                return None           # minutes in plain torch
            return P.solve(K, P.source(v["f"]))
    if kind == "transpose":
        x = torch.zeros_like(v["x"]).requires_grad_()
        return torch.autograd.grad(P.apply(x, K), x, v["x"])[0]
    if nc * nb > 200_000:
        return None
    with torch.no_grad():
        u = P.solve(K, P.source(v["f"]))
        lam = None if u is None else P.solve(K, v["w"])
    if lam is None:
        return None
    logK, f = v["logK"].requires_grad_(), v["f"].requires_grad_()
    res = torch.dot(lam, P.apply(u, torch.exp(logK)) - P.source(f))
    gk, gf = torch.autograd.grad(res, [logK, f])
    return {"u": u, "dlogK": -gk, "df": -gf}
