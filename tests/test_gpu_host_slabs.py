"""Applies on host vectors, cut into slabs of planes: at least two slabs in every
case, ragged last slabs, slabs of one plane, 2D and 3D, and results that the
kernel stores into pinned memory itself (degree 2 in 3D).  Every cell is computed
by the same arithmetic as on device vectors, so the results are equal to the bit.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402


def slabs(dim, k, cells, copied_out):
    """planes of each slab: at most one slab per 16384 cells, and one (2.5 where the
    result is copied out into pinned memory) per MB under the root"""
    nc, planes = math.prod(cells), cells[-1]
    mb = 8 * nc * (k + 1) ** dim / 1e6
    s = min(nc // 16384, int(math.sqrt(2.5 * mb if copied_out else mb)), 16, planes)
    per = -(-planes // s)
    return [min(per, planes - i) for i in range(0, planes, per)]


# slabs of pageable results (and of pinned ones that the kernel stores), and of
# pinned ones that are copied out
CASES = [((3, 1, (64, 64, 19)), [10, 9], [7, 7, 5]),
         ((3, 2, (64, 64, 22)), [6, 6, 6, 4], [5, 5, 5, 5, 2]),
         ((3, 2, (150, 150, 3)), [1, 1, 1], [1, 1, 1]),
         ((3, 3, (48, 40, 23)), [12, 11], [12, 11]),
         ((3, 4, (41, 40, 30)), [10, 10, 10], [10, 10, 10]),
         ((2, 2, (512, 334)), [112, 112, 110], [67, 67, 67, 67, 66])]


def operator(dim, k, cells, seed=1):
    import torch
    rng = np.random.default_rng(seed)
    go = pdg.GridOperator(dim, k, cells, alpha=3.0)
    go.set_permeability(rng.standard_normal(go.ncell), is_log=True)
    go.set_source(fc=rng.standard_normal(go.ncell))
    return torch, go, pdg.OnTheFlyOperator(go), rng


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("case,planes,planes_pinned", CASES)
def test_slabs_bitwise_equal_device(case, planes, planes_pinned, pinned):
    assert slabs(*case, False) == planes and slabs(*case, True) == planes_pinned
    torch, go, op, rng = operator(*case)

    def host(a):
        t = torch.tensor(a)
        return t.pin_memory() if pinned else t

    x, y0 = rng.uniform(-1, 1, go.ndof), rng.uniform(-1, 1, go.ndof)
    xh, xd = host(x), torch.tensor(x, device="cuda")
    forms = {"apply": lambda a, b: op.apply(a, b),
             "applyscaleadd": lambda a, b: op.applyscaleadd(-0.75, a, b),
             "residual": lambda a, b: go.residual(a, b),
             "transpose": lambda a, b: go.jacobian_apply_transpose(a, b)}
    for name, f in forms.items():
        yd = torch.tensor(y0, device="cuda")
        f(xd, yd)
        ref = yd.cpu()
        for a in (xh, xd):
            y = host(y0)
            f(a, y)
            assert torch.equal(y, ref), name
        yd = torch.tensor(y0, device="cuda")
        f(xh, yd)
        assert torch.equal(yd.cpu(), ref), name
    go.close()


# 16-byte aligned or not; 32 guard values on either side
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("case", [c for c, _, _ in CASES if c[:2] == (3, 2)])
def test_stores_into_pinned_memory(case, shift):
    torch, go, op, rng = operator(*case)
    n, g = go.ndof, 32
    x = torch.tensor(rng.uniform(-1, 1, n))
    xd = x.cuda()
    yd = torch.zeros_like(xd)
    op.apply(xd, yd)
    ref = yd.cpu()
    xp = x.pin_memory()
    buf = torch.empty(n + 2 * g + 1, dtype=torch.float64).pin_memory()
    for a in (xp, x, xd):
        buf.fill_(-7.0)
        y = buf[g + shift:g + shift + n]
        op.apply(a, y)
        assert torch.equal(y, ref)
        assert (buf[:g + shift] == -7.0).all() and (buf[g + shift + n:] == -7.0).all()
    # in place: a plane is stored once the next one has been copied in
    buf[g + shift:g + shift + n] = x
    y = buf[g + shift:g + shift + n]
    op.apply(y, y)
    assert torch.equal(y, ref)
    go.close()
