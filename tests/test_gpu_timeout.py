"""A bounded device wait that ran out.  The kernel that gave up has set a flag
and left part of its result unwritten; the flag is set here from the host
(nothing waits on the device).  The next call that waits for the device reports
it, once, whatever ran in between."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402

CSRC = os.path.join(os.path.dirname(os.path.abspath(pdg.__file__)), "csrc")

POKE = r"""
#include <vector>
#include "pdg_vec.cuh"
extern "C" void timeout_set(pdg_context *ctx) { *ctx->h_wait = 1; }
// the counts that a launch with a block that gave up leaves behind: one each
extern "C" int counts_set(pdg_context *ctx) {
  const int n = (int)((ctx->ncell / 4 + 2 + pdg::kFuseGroup - 1) / pdg::kFuseGroup);
  const std::vector<int> one(n, 1);
  return ctx->fuse_cnt ? (int)cudaMemcpy(ctx->fuse_cnt, one.data(), sizeof(int) * n,
                                         cudaMemcpyHostToDevice) : -1;
}
"""


@pytest.fixture(scope="module")
def poke(tmp_path_factory):
    import build_lib
    d = tmp_path_factory.mktemp("poke")
    (d / "poke.cu").write_text(POKE)
    r = subprocess.run([build_lib.nvcc(), *build_lib.ARCH, "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC", "-I", CSRC, "-o", str(d / "poke.so"), str(d / "poke.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(str(d / "poke.so"))
    lib.timeout_set.argtypes = lib.counts_set.argtypes = [ctypes.c_void_p]
    return lib


def operator(n):
    import torch
    rng = np.random.default_rng(1)
    go = pdg.GridOperator(3, 2, n, alpha=3.0)
    go.set_permeability(np.exp(rng.standard_normal(go.ncell)))
    go.set_source(fc=np.ones(go.ncell))
    return torch, go, rng.uniform(-1, 1, go.ndof)


# staged through device buffers, and pipelined over slabs
@pytest.mark.parametrize("n", [(6, 5, 4), (64, 64, 16)])
def test_host_apply_reports(poke, n):
    torch, go, x = operator(n)
    op = pdg.OnTheFlyOperator(go)
    ref, y = np.zeros(go.ndof), np.zeros(go.ndof)
    op.apply(x, ref)
    poke.timeout_set(go.handle)
    with pytest.raises(pdg.PDGError) as e:
        op.apply(x, y)
    assert e.value.status == pdg.PDG_ETIMEOUT
    y[:] = 0.0
    op.apply(x, y)                  # reported once
    assert np.array_equal(y, ref)
    go.close()


def test_kept_for_the_next_call_that_waits(poke):
    torch, go, x = operator((6, 5, 4))
    xd = torch.tensor(x, device="cuda")
    y = torch.zeros_like(xd)
    u = torch.zeros_like(xd)
    ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go)
    slp = pdg.StationaryLinearProblemSolver(go, ls, u, 1e-8)
    poke.timeout_set(go.handle)
    pdg.OnTheFlyOperator(go).apply(xd, y)      # asynchronous
    with pytest.raises(pdg.PDGError) as e:
        slp.apply()
    assert e.value.status == pdg.PDG_ETIMEOUT
    u.zero_()
    slp.apply()
    assert slp.result().converged
    go.close()


@pytest.mark.parametrize("mixed", [False, True])
def test_solve_after_a_launch_that_gave_up(poke, mixed):
    """The block counts of the fused sums start from zero in every solve."""
    torch, go, x = operator((12, 11, 10))
    u = torch.zeros(go.ndof, dtype=torch.float64, device="cuda")
    ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go, mixed=mixed)
    slp = pdg.StationaryLinearProblemSolver(go, ls, u, 1e-8)
    slp.apply()
    first, its = u.clone(), slp.result().iterations
    assert poke.counts_set(go.handle) == 0
    u.zero_()
    slp.apply()
    assert torch.equal(u, first) and slp.result().iterations == its
    go.close()
