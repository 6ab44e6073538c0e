"""The warp sums of the fused CG kernels (pdg_vec.cuh) against exact sums."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import pdg  # noqa: E402

CSRC = os.path.join(os.path.dirname(os.path.abspath(pdg.__file__)), "csrc")

KERNELS = r"""
#include "pdg_vec.cuh"
using namespace pdg;
// one warp per row of n values (n <= 32)
__global__ void k_fixed(const double *v, int n, double *out) {
  if (threadIdx.x < n) {
    const double s = warp_sum_fixed(v[blockIdx.x * n + threadIdx.x], n);
    out[blockIdx.x * n + threadIdx.x] = s;
  }
}
__global__ void k_two(const float *v, double *out) {
  const int i = 32 * blockIdx.x + threadIdx.x;
  out[i] = warp_sum_two(TwoFloat{v[2 * i], v[2 * i + 1]});
}
extern "C" int sum_two(const float *v, int rows, double *out) {
  k_two<<<rows, 32>>>(v, out);
  return (int)cudaDeviceSynchronize();
}
extern "C" int sum_fixed(const double *v, int rows, int n, double *out) {
  k_fixed<<<rows, n>>>(v, n, out);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import build_lib
    d = tmp_path_factory.mktemp("sums")
    (d / "sums.cu").write_text(KERNELS)
    r = subprocess.run([build_lib.nvcc(), *build_lib.ARCH, "-std=c++17", "-O3", "-shared",
                        "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", CSRC, "-o",
                        str(d / "sums.so"), str(d / "sums.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(d / "sums.so"))


def bound(row):
    """lanes rounded to 57 bits under the power of two above the largest, the sum
    rounded to 53 bits"""
    top = 2.0 ** math.frexp(max(abs(v) for v in row))[1]
    s = math.fsum(row)
    return s, len(row) * 2.0 ** -58 * top + 2.0 ** -53 * abs(s)


@pytest.mark.parametrize("n", [32, 17, 1])
def test_warp_sum_fixed(lib, n):
    import torch
    rng = np.random.default_rng(n)
    rows = [rng.uniform(-1, 1, n), rng.uniform(0, 1, n) ** 2,
            rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-12, 12, n), np.zeros(n),
            -np.ones(n) * (2.0 - 2.0 ** -52), np.ones(n) * 1e-290]
    # one large value, the others just below two units of the 57 bits
    low = np.full(n, 1.99 * 2.0 ** -56)
    low[n // 2] = 1.0
    rows += [low, -low, low * 2.0 ** 300]
    v = torch.tensor(np.array(rows), device="cuda")
    out = torch.zeros_like(v)
    torch.cuda.synchronize()
    st = lib.sum_fixed(ctypes.c_void_p(v.data_ptr()), len(rows), n,
                       ctypes.c_void_p(out.data_ptr()))
    assert st == 0
    for row, o in zip(rows, out.cpu().numpy()):
        s, tol = bound(row) if row.any() else (0.0, 0.0)
        assert (o == o[0]).all()
        assert abs(o[0] - s) <= tol


def test_warp_sum_two(lib):
    """Pairs of floats: the sums over a warp keep what FP64 keeps of them."""
    import torch
    rng = np.random.default_rng(5)
    rows = [rng.uniform(-1, 1, 32), rng.uniform(0, 1, 32), rng.uniform(0, 1, 32) ** 8,
            rng.uniform(0, 1, 32) * 1e-30, np.zeros(32), np.ones(32),
            rng.uniform(-1, 1, 32) * 10.0 ** rng.uniform(-8, 8, 32)]
    h = np.array(rows).astype(np.float32)
    low = (np.array(rows) - h.astype(np.float64)).astype(np.float32)
    v = torch.tensor(np.stack([h, low], axis=2), device="cuda")
    out = torch.zeros((len(rows), 32), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.sum_two(ctypes.c_void_p(v.data_ptr()), len(rows),
                       ctypes.c_void_p(out.data_ptr())) == 0
    for hr, lr, o in zip(h, low, out.cpu().numpy()):
        both = [float(x) for x in hr] + [float(x) for x in lr]
        s, tol = bound(both) if hr.any() else (0.0, 0.0)
        assert (o == o[0]).all()
        assert abs(o[0] - s) <= tol
    special = np.zeros((3, 32, 2), np.float32)
    special[0, 3, 0] = np.inf
    special[1, 4, 0] = np.nan
    special[2, :, 0] = 1e-44                     # subnormal in FP32
    v = torch.tensor(special, device="cuda")
    torch.cuda.synchronize()
    assert lib.sum_two(ctypes.c_void_p(v.data_ptr()), 3, ctypes.c_void_p(out.data_ptr())) == 0
    o = out.cpu().numpy()
    assert np.isposinf(o[0]).all() and np.isnan(o[1]).all()
    assert (o[2] == float(np.float32(1e-44)) * 32).all()
