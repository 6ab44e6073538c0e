// pdg_fdm_i.cu -- the FP64 cell-block Jacobi in fast-diagonalisation form on 3D
// grids, v = (Qx (x) Qy (x) Qz) diag(1/(lx+ly+lz)) (Qx (x) Qy (x) Qz)^T d, in
// 64-bit fixed point (pdg_fixed.cuh).
//
// Reference: AssembledBlockJacobiPreconditionerLocalOperator's apply
// (backend/istl/matrixfree/assembledblockjacobipreconditioner.hh:162-233).
// Six contractions with per-cell matrices, 6 N + 1 multiply-adds per DOF: in
// FP64 bound by that pipe (1.8 lane operations per SM and cycle), here three
// IMAD.WIDE each.  FP64 vectors in and out.  47x53x49 Q3: 127 us, in FP64
// arithmetic 374 us; the error against 64 bits is the same (4.8e-15, that of
// the factors).
//
// Scaling.  A cell's input has one exponent Ed.  The eigenvectors of a block
// differ in size by decades (they are orthonormal in the mass matrix), so each
// column of Q_dir is scaled by the power of two that brings its sum of
// magnitudes below 1, and the stored 1/(lx+ly+lz) carry the squares of those
// powers: the modes are then as accurate as they are in FP64.  A forward
// stage stays below 2^Ed; a backward stage grows by the largest row sum of
// magnitudes (exponents EB per cell and direction).  Every stage's result is
// rounded to 59 bits under its bound.  The products with
// 1/(lx+ly+lz) are normalised to the cell's largest before they are cut: the
// spectrum of a block spans decades, and a static bound there cost 8 bits
// (errors of 1e-13 at k = 4).
// Degrees 1 to 3.  At degree 4 smooth data still had three times the rounding of
// FP64 (M(3d) - 3 M(d) at 24^3 9.8e-16 of M d against 2.9e-16; degrees 1 to 3: 2.8e-16,
// 1.4e-16, 1.9e-16 against 4.3e-16, 2.3e-16, 3.2e-16), so it keeps the FP64 kernel
// (k_fdm_apply in pdg_prec.cu).
// Cells with data that is not finite or far from the middle of the range send
// their block to a plain FP64 evaluation.
#include "pdg_fixed.cuh"
#include "pdg_ops.cuh"
#include "pdg_vec.cuh"

namespace pdg {

template <int N>
struct FICfg {
  static constexpr int N2 = N * N, NB = N * N * N, TPC = N * N;
  static constexpr int CPB = (N == 4 ? 64 : 128) / TPC;   // 32, 14, 4 cells
  static constexpr int THREADS = CPB * TPC;
  static constexpr int NEXP = 8;   // EB[3], EL, usable
  // two exchange arrays and the factors; padding with the fewest shared-memory
  // wavefronts, counted on the CPU over paddings 0..15
  static constexpr int PER_CELL =
      2 * NB + 3 * N2 + (N == 3 ? 8 : 0);
};

// exponent E with x < 2^E for a non-negative sum x rounded in FP64
__device__ __forceinline__ int sum_exponent(double x) {
  return (int)((__double2hiint(x * (1.0 + 0x1p-40)) >> 20) & 0x7ff) - 1022;
}

// Limbs of the scaled Q and the exponents, one cell per warp (lane (dir, i):
// column and row i of Q_dir); Linv is scaled in place.
template <int N>
__global__ void k_fdm_record_i(long ncell, const double *__restrict__ Q, double *Linv,
                               int2 *__restrict__ out, int *__restrict__ exps) {
  using C = FICfg<N>;
  const long e = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (e >= ncell) return;
  constexpr unsigned kAll = 0xffffffffu;
  const double *q = Q + e * 3 * C::N2;
  const bool on = lane < 3 * N;
  const int dir = on ? lane / N : 0, i = lane % N;
  double cs = 0.0;
#pragma unroll
  for (int k = 0; k < N; k++) cs += fabs(q[dir * C::N2 + k * N + i]);
  const int ec = sum_exponent(cs);   // column i of Q_dir is scaled by 2^-ec
  bool ok = ec > -150 && ec < 150;
  double rs = 0.0;
#pragma unroll
  for (int c = 0; c < N; c++) {
    const int ecc = __shfl_sync(kAll, ec, dir * N + c);
    if (ok) rs += fabs(q[dir * C::N2 + i * N + c]) * __hiloint2double((1023 - ecc) << 20, 0);
  }
  ok = __all_sync(kAll, ok);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int eb = __reduce_max_sync(kAll, on && dir == d && ok ? sum_exponent(rs) : -2000);
    if (lane == 0) exps[e * C::NEXP + d] = max(eb, 0);
  }
  BlockExp bl;
  unsigned mn = kAll;
  for (int b = 0; b < C::NB; b += 32) {
    const int k = b + lane, kk = k < C::NB ? k : 0;
    const int s = __shfl_sync(kAll, ec, kk % N) + __shfl_sync(kAll, ec, N + (kk / N) % N) +
                  __shfl_sync(kAll, ec, 2 * N + kk / C::N2);
    if (k >= C::NB || !ok) continue;
    const double x = Linv[e * C::NB + k] * __hiloint2double((1023 + 2 * s) << 20, 0);
    Linv[e * C::NB + k] = x;
    bl.add(x);
    mn = min(mn, (unsigned)__double2hiint(x) << 1);
  }
  const unsigned ml = __reduce_max_sync(kAll, bl.m);
  mn = __reduce_min_sync(kAll, mn);
  ok = ok && (mn >> 21) > 1023 - 300 && (ml >> 21) < 1023 + 300;
  if (lane == 0) {
    exps[e * C::NEXP + 3] = (int)(ml >> 21) - 1022;
    exps[e * C::NEXP + 4] = ok;
  }
  for (int b = 0; b < 3 * C::N2; b += 32) {
    const int k = b + lane, kk = k < 3 * C::N2 ? k : 0;
    const int ecc = __shfl_sync(kAll, ec, (kk / C::N2) * N + kk % N);
    if (k < 3 * C::N2)
      out[e * 3 * C::N2 + k] = ok ? fix_limbs(q[k], ecc + 1022) : make_int2(0, 0);
  }
}

// The block's cells in plain FP64: not a fast path (see apply_cells_fp64 in
// pdg_apply_i.cu).  Called by every thread of the block; returns the sum of
// d * v over the thread's column.
template <int N>
__device__ __noinline__ double fdm_cells_fp64(const double *__restrict__ Q,
                                            const double *__restrict__ L, const double *d,
                                            double *v, double *S0, int l, long e, bool active,
                                            double scale) {
  using C = FICfg<N>;
  constexpr int N2 = C::N2, NB = C::NB;
  double *S1 = S0 + NB;
  const int tx = l % N, ty = l / N;
  const double *Qx = Q + e * 3 * N2, *Qy = Qx + N2, *Qz = Qy + N2;
  __syncthreads();
  for (int zp = 0; zp < N; zp++) {
    double s = 0.0;
    for (int z = 0; z < N; z++) s += Qz[z * N + zp] * d[e * NB + z * N2 + l];
    S0[zp * N2 + l] = s;
  }
  __syncthreads();
  for (int z = 0; z < N; z++) {
    double s = 0.0;
    for (int y = 0; y < N; y++) s += Qy[y * N + ty] * S0[z * N2 + y * N + tx];
    S1[z * N2 + l] = s;
  }
  __syncthreads();
  for (int z = 0; z < N; z++) {
    double s = 0.0;
    for (int x = 0; x < N; x++) s += Qx[x * N + tx] * S1[z * N2 + ty * N + x];
    S0[z * N2 + l] = s / (L[e * 3 * N + tx] + L[e * 3 * N + N + ty] + L[e * 3 * N + 2 * N + z]);
  }
  __syncthreads();
  for (int z = 0; z < N; z++) {
    double s = 0.0;
    for (int x = 0; x < N; x++) s += Qx[tx * N + x] * S0[z * N2 + ty * N + x];
    S1[z * N2 + l] = s;
  }
  __syncthreads();
  for (int z = 0; z < N; z++) {
    double s = 0.0;
    for (int y = 0; y < N; y++) s += Qy[ty * N + y] * S1[z * N2 + y * N + tx];
    S0[z * N2 + l] = s;
  }
  double part = 0.0;
  if (!active) return part;
  for (int z = 0; z < N; z++) {
    double s = 0.0;
    for (int zp = 0; zp < N; zp++) s += Qz[z * N + zp] * S0[zp * N2 + l];
    const double dz = d[e * NB + z * N2 + l];
    v[e * NB + z * N2 + l] = scale * s;
    part += dz * (scale * s);
  }
  return part;
}

// contraction of N limb pairs (fb: 59 bits), shifted right by s >= 0, rounded
template <int N, class FA, class FB>
__device__ __forceinline__ long long contract(FA fa, FB fb, int s) {
  long long hh = 0, mid = (1ll << (s + 28)) >> 1;
#pragma unroll
  for (int q = 0; q < N; q++) mac2(hh, mid, fa(q), fb(q));
  return mac2_value_wide(hh, mid) >> s;
}

__device__ __forceinline__ int biased_exponent(double x) {
  return (__double2hiint(x) >> 20) & 0x7ff;
}
// v 2^s, rounded for s < 0 (the caller's bound leaves room for s > 0)
__device__ __forceinline__ long long shift_by(long long v, int s) {
  const int r = min(-s, 62);
  return s >= 0 ? (long long)((unsigned long long)v << s) : (v + ((1ll << r) >> 1)) >> r;
}

// One launch: the operands of the fused CG, or part null.  rq != null: first
// d -= lambda rq (lambda = scal[S_ALPHA]), written back; the sums then carry
// |d|^2 and <d, v>.  d, v and rq may alias element-wise: every entry is read
// and written by one thread, read before it is written.
struct FdmFuse {
  double *part;
  long max_blocks;
  int *cnt;
  double *scal;
  int *flags;
  int fin;
  const double *rq;
};

template <int N, bool kFuse>
__global__ void __launch_bounds__(FICfg<N>::THREADS)
    k_fdm_i(long ncell, const int2 *__restrict__ Qi, const int *__restrict__ exps,
            const double *__restrict__ Linv, const double *__restrict__ Q64,
            const double *__restrict__ L64, double *d, double *v, const int *__restrict__ skip,
            const int *__restrict__ cells, int ncells, double scale, const FdmFuse fuse) {
  using C = FICfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC, CPB = C::CPB;
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int sE[2 * CPB];
  const int t = threadIdx.x, cs = t / TPC, l = t - cs * TPC;
  int2 *S0 = reinterpret_cast<int2 *>(smem_raw) + cs * C::PER_CELL;
  int2 *S1 = S0 + NB;
  int2 *Qs = S1 + NB;   // [3][N2]
  const int li = blockIdx.x * CPB + cs;
  const bool active = cells ? li < ncells : li < ncell;
  const long e = active ? (cells ? cells[li] : li) : 0;
  if (t < CPB) {
    sE[2 * t] = kFixZero;
    sE[2 * t + 1] = 0;
  }
  double col[N], lin[N];
#pragma unroll
  for (int z = 0; z < N; z++) {
    col[z] = d[e * NB + z * TPC + l];
    lin[z] = Linv[e * NB + z * TPC + l];
  }
  for (int i = l; i < 3 * N2; i += TPC) Qs[i] = Qi[e * 3 * N2 + i];
  double part2 = 0.0;
  if (kFuse && fuse.rq) {
    const double lambda = fuse.scal[S_ALPHA];
#pragma unroll
    for (int z = 0; z < N; z++) {
      const size_t i = e * NB + z * TPC + l;
      col[z] -= lambda * fuse.rq[i];
      if (active) {
        d[i] = col[z];
        part2 += col[z] * col[z];
      }
    }
  }
  const int *ex = exps + e * C::NEXP;
  BlockExp b;
#pragma unroll
  for (int z = 0; z < N; z++) b.add(col[z]);
  bool bad = ex[4] == 0 || !b.finite();
  __syncthreads();
  atomicMax(&sE[2 * cs], b.exponent());
  __syncthreads();
  const int Ed = sE[2 * cs];
  // bounds after the scaling and of the result
  const int EL = ex[3], Ev = Ed + EL + ex[0] + ex[1] + ex[2];
  bad |= Ed != kFixZero && (Ed < -500 || Ed > 800 || Ev < -800 || Ev > 900);
  const int eb = Ed == kFixZero ? kFixMinBiased : Ed + 1022;
  const int tx = l % N, ty = l / N;
  const int2 *Qx = Qs, *Qy = Qs + N2, *Qz = Qs + 2 * N2;
  // z: a[z'] = sum_z Qz[z][z'] d[z]
  {
    int2 u[N];
#pragma unroll
    for (int z = 0; z < N; z++) u[z] = fix_limbs<kFixWide>(col[z], eb);
#pragma unroll
    for (int zp = 0; zp < N; zp++)
      S0[zp * N2 + l] = limbs(contract<N>([&](int q) { return Qz[q * N + zp]; },
                                          [&](int q) { return u[q]; }, 0));
  }
  const auto finish = [&](double part) {
    reduce_tail_grouped<C::THREADS>(
        fuse.part, fuse.max_blocks, fuse.cnt, RedCtx{nullptr, fuse.scal, fuse.flags},
        fuse.rq ? part2 : part, fuse.rq ? part : 0.0, fuse.fin);
  };
  if (__syncthreads_or(bad)) {
    const double part = fdm_cells_fp64<N>(Q64, L64, d, v, reinterpret_cast<double *>(S0), l, e,
                                          active, scale);
    if (kFuse) finish(part);
    return;
  }
  // y
  {
    int2 c[N];
#pragma unroll
    for (int q = 0; q < N; q++) c[q] = Qy[q * N + ty];
#pragma unroll
    for (int z = 0; z < N; z++)
      S1[z * N2 + l] = limbs(contract<N>([&](int q) { return c[q]; },
                                         [&](int q) { return S0[z * N2 + q * N + tx]; }, 0));
  }
  __syncthreads();
  // x, then the scaling normalised to the cell's largest value
  long long m[N];
  {
    int2 c[N];
#pragma unroll
    for (int q = 0; q < N; q++) c[q] = Qx[q * N + tx];
    int top = 0;
#pragma unroll
    for (int z = 0; z < N; z++) {
      m[z] = contract<N>([&](int q) { return c[q]; },
                         [&](int q) { return S1[z * N2 + ty * N + q]; }, 0);
      // |m lin| < 2^(bits of m + biased exponent of lin), up to a constant
      if (m[z]) top = max(top, 64 - __clzll(m[z] ^ (m[z] >> 63)) + biased_exponent(lin[z]));
    }
    atomicMax(&sE[2 * cs + 1], top);
  }
  __syncthreads();
  const int top = sE[2 * cs + 1];
#pragma unroll
  for (int z = 0; z < N; z++) {
    const int el = biased_exponent(lin[z]);
    long long hh = 0, mid = 0;
    mac2(hh, mid, fix_limbs(lin[z], el), limbs(m[z]));
    // (hh 2^58 + mid 2^29) 2^-k; units of 2^(Ed + top - 1140)
    const int k = top - el - 2;
    S0[z * N2 + l] = limbs(shift_by(hh, 58 - k) + shift_by(mid, 29 - k));
  }
  __syncthreads();
  // back x
  {
    int2 c[N];
#pragma unroll
    for (int q = 0; q < N; q++) c[q] = Qx[tx * N + q];
    const int s = ex[0];
#pragma unroll
    for (int z = 0; z < N; z++)
      S1[z * N2 + l] = limbs(contract<N>([&](int q) { return c[q]; },
                                         [&](int q) { return S0[z * N2 + ty * N + q]; }, s));
  }
  __syncthreads();
  // back y and z
  {
    int2 c[N], u[N];
#pragma unroll
    for (int q = 0; q < N; q++) c[q] = Qy[ty * N + q];
    const int s = ex[1];
#pragma unroll
    for (int z = 0; z < N; z++)
      u[z] = limbs(contract<N>([&](int q) { return c[q]; },
                               [&](int q) { return S1[z * N2 + q * N + tx]; }, s));
    double part = 0.0;
    if (active) {
      // one unit of the last contraction
      const int E = Ed + top - 1140 + ex[0] + ex[1];
      const double unit =
          Ed == kFixZero || top == 0 ? 0.0 : __hiloint2double((E + 1023) << 20, 0);
#pragma unroll
      for (int z = 0; z < N; z++) {
        long long hh = 0, mid = 0;
#pragma unroll
        for (int q = 0; q < N; q++) mac2(hh, mid, Qz[z * N + q], u[q]);
        const double r = scale * ((double)mac2_value_wide(hh, mid) * unit);
        const size_t i = e * NB + z * N2 + l;
        if (kFuse) part += d[i] * r;
        v[i] = r;
      }
    }
    if (kFuse) finish(part);
  }
}

template <int N>
static int fdm_record_i_n(pdg_context *ctx) {
  using C = FICfg<N>;
  PrecData &pd = ctx->prec[PDG_F64];
  PDG_CUDA_TRY(cudaMalloc(&pd.Qi, sizeof(int2) * 3 * C::N2 * ctx->ncell));
  PDG_CUDA_TRY(cudaMalloc(&pd.Qi_exp, sizeof(int) * C::NEXP * ctx->ncell));
  k_fdm_record_i<N><<<(unsigned)((ctx->ncell + 3) / 4), 128, 0, ctx->stream>>>(
      ctx->ncell, (const double *)pd.Q, pd.Lsum_inv, pd.Qi, pd.Qi_exp);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

int fdm_record_i(pdg_context *ctx) {
  switch (ctx->N) {
    case 2: return fdm_record_i_n<2>(ctx);
    case 3: return fdm_record_i_n<3>(ctx);
    case 4: return fdm_record_i_n<4>(ctx);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}

template <int N>
static int fdm_apply_i_n(pdg_context *ctx, const double *d, double *v, const int *skip,
                         const int *cells, int ncells, double scale) {
  using C = FICfg<N>;
  const PrecData &pd = ctx->prec[PDG_F64];
  const long work = cells ? ncells : ctx->ncell;
  if (work <= 0) return PDG_OK;
  const size_t smem = sizeof(int2) * C::CPB * C::PER_CELL;
  const unsigned blocks = (unsigned)((work + C::CPB - 1) / C::CPB);
  FdmFuse fuse{};
  if (ctx->fuse_fin && !cells)
    fuse = FdmFuse{ctx->fuse_part, ctx->fuse_max_blocks, ctx->fuse_cnt, ctx->red_out, ctx->d_flag,
                   ctx->fuse_fin,
                   ctx->fuse_fin == FIN_CG_DEF_BETA ? (const double *)ctx->fuse_q : nullptr};
  // the fused form is its own instance: its code in the plain one cost 4 %
  auto *kernel = fuse.part ? k_fdm_i<N, true> : k_fdm_i<N, false>;
  kernel<<<blocks, C::THREADS, smem, ctx->stream>>>(
      ctx->ncell, pd.Qi, pd.Qi_exp, pd.Lsum_inv, (const double *)pd.Q, (const double *)pd.L,
      const_cast<double *>(d), v, skip, cells, ncells, scale, fuse);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

int fdm_apply_i(pdg_context *ctx, const double *d, double *v, const int *skip, const int *cells,
                int ncells, double scale) {
  switch (ctx->N) {
    case 2: return fdm_apply_i_n<2>(ctx, d, v, skip, cells, ncells, scale);
    case 3: return fdm_apply_i_n<3>(ctx, d, v, skip, cells, ncells, scale);
    case 4: return fdm_apply_i_n<4>(ctx, d, v, skip, cells, ncells, scale);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}

}  // namespace pdg
