// pdg_apply_i.cu -- the coupled 3D FP64 cell operator in 64-bit fixed point
// (degrees 1, 3 and 4; pdg_apply_p.cu has the kernel of degree 2).
//
// Same operator as k_apply<double, 3, N> (pdg_apply.cu; reference:
// ConvectionDiffusionDG::jacobian_apply_volume / _skeleton / _boundary,
// localoperator/convectiondiffusiondg.hh:191-195, 474-481, 892-899), in the
// same form, y_e = sum_dir (A'_dir (x) M (x) M)_dir u_e + face couplings, with
// FP64 vectors in and out.  GB300 issues 1.8 FP64 lane operations per SM and
// cycle, so the FP64 kernels are bound by that pipe whatever they move; here
// the arithmetic runs as 57-bit block fixed point on the integer pipe
// (pdg_fixed.cuh):
//
// * a cell's values, each neighbour line and each cell's coefficients share
//   an exponent; the directional operators and the neighbour lines are limb
//   contractions (three IMAD.WIDE per multiply-add);
// * the sums of a cell get one exponent, chosen so that they cannot overflow;
//   the mass matrices (small integers over a common denominator, the
//   denominators are in the coefficients) and the face lifts are then exact
//   integer arithmetic up to one rounding shift per stage;
// * a cell whose data is not finite, or whose result would leave the normal
//   range by far, sends its block to a plain FP64 evaluation.
//
// The unfactored form is used although it has five masses instead of three:
// masses are the cheap integer products, and Mhat^-1 A' would lose cond(Mhat).
#include <cmath>

#include "pdg_fixed.cuh"
#include "pdg_ops.cuh"
#include "pdg_vec.cuh"

namespace pdg {

template <int N>
struct ICfg {
  static constexpr int N2 = N * N, NB = N * N * N, TPC = N * N, NF = 6;
  static constexpr int CPB = (N == 4 ? 64 : 128) / TPC;   // 32, 4, 5 cells (k = 1, 3, 4)
  static constexpr int THREADS = CPB * TPC;
  static constexpr int NW = NF * (N + 1);
  static constexpr int RECW = 3 * N2 + 2 * NW;       // the FP64 record (both forms)
  static constexpr int RECI = 3 * N2 + NW;           // limb pairs of one form
  static constexpr int NEXP = 16;                    // exponents per cell, see k_record_i
  // ue, X, Y, Z, face data (12 TPC), record; 8 bytes each.  The padding is the
  // one with the fewest shared-memory wavefronts of the kernel's accesses,
  // counted on the CPU over paddings 0..15 (k = 4: 2352 per block instead of
  // 3128 without the right one)
  static constexpr int PER_CELL =
      4 * NB + 12 * TPC + RECI + (N == 2 ? 6 : N == 5 ? 10 : 0);
  static constexpr int LN = N == 2 ? 1 : N == 5 ? 3 : 2;   // ceil log2 N
  static constexpr int LD = N == 2 ? 0 : N == 4 ? 5 : 6;   // ceil log2 max |d|
  // X, Y, Z are formed below 2^61 and shifted to 2^(61 - SHX) so that the
  // masses (row sums 3, 864, 2988) stay below 2^63: N = 2 modulo 2^64,
  // shifting by SHM after the first; N >= 4 with two sums, shifting by SHM
  // after each
  static constexpr bool WIDE = N > 2;
  static constexpr int SHX = N == 2 ? 2 : 0;
  // s2 carries FB more bits than s1: the derivative of the basis multiplies it,
  // and its rounding, by up to 48 (with FB = 0 smooth data at 24^3 Q4 had 5 times
  // the noise of FP64, with 3 less than that)
  static constexpr int FB = N == 2 ? 0 : 3;
  static constexpr int SHM = N == 2 ? 2 : N == 4 ? 10 : 12;
  // exponent of one unit of the result over the cell's Etot
  static constexpr int OUTE = -61 + SHX + (WIDE ? 2 * SHM : SHM);
};

// place of entry i of cell e in the limb records of n entries per cell: cell by
// cell, for the degree of k_apply_p entry by entry within a group of 32 cells
template <int N>
__device__ __forceinline__ size_t limb_at(long e, int n, int i) {
  return N == 3 ? ((size_t)(e / kGroup) * n + i) * kGroup + e % kGroup : (size_t)e * n + i;
}

// Limb record of one form (operator, or its transpose): A'_dir / den^2, then
// per face the line coefficients W[0..N-1] / den^2 and W[N] / (den^2 dden),
// from the FP64 record (zero without a neighbour).  The quotients are formed to more than FP64 (product
// with the reciprocal and its rest) before they are cut to 57 bits.
// exps[e] = {EA, EW1[6], EW2[6], usable}: exponents of A' (all directions),
// of the W[0..N-1] of each face and of each W[N].  One warp per cell.
template <int N>
__global__ void k_record_i(const OpParams<double> p, const double *__restrict__ rec,
                           int2 *__restrict__ out, int *__restrict__ exps, int transpose, double rd,
                           double rd_lo, double rw, double rw_lo) {
  using C = ICfg<N>;
  constexpr int PER = (C::RECI + 31) / 32;
  const long e = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (e >= p.ncell) return;
  unsigned has = 0;   // faces with a neighbour
  {
    const unsigned q0 = p.div0.div((unsigned)e), q1 = p.div1.div(q0);
    const int ix[3] = {(int)((unsigned)e - q0 * (unsigned)p.nc[0]),
                       (int)(q0 - q1 * (unsigned)p.nc[1]), (int)q1};
#pragma unroll
    for (int d = 0; d < 3; d++)
      has |= (ix[d] > 0 ? 1u << 2 * d : 0u) | (ix[d] + 1 < p.nc[d] ? 2u << 2 * d : 0u);
  }
  const double *r = rec + e * C::RECW;
  double q[PER], q2[PER];
  unsigned m[13];   // group maxima: A', W1 of 6 faces, W2 of 6 faces
#pragma unroll
  for (int g = 0; g < 13; g++) m[g] = 0;
  unsigned any = 0;
#pragma unroll
  for (int s = 0; s < PER; s++) {
    const int i = s * 32 + lane;
    q[s] = q2[s] = 0.0;
    if (i >= C::RECI) continue;
    double v;
    int g = 0;
    bool last = false;
    if (i < 3 * C::N2) {
      const int d = i / C::N2, k = (i / N) % N, c = i % N;
      v = r[d * C::N2 + (transpose ? c * N + k : k * N + c)];
    } else {
      const int w = i - 3 * C::N2, f = w / (N + 1);
      last = w % (N + 1) == N;
      g = last ? 7 + f : 1 + f;
      v = has >> f & 1 ? r[3 * C::N2 + (transpose ? C::NW : 0) + w] : 0.0;
    }
    const double ri = last ? rw : rd, rl = last ? rw_lo : rd_lo;
    q[s] = v * ri;
    q2[s] = fma(v, ri, -q[s]) + v * rl;
    const unsigned hi2 = (unsigned)__double2hiint(q[s]) << 1;
    any |= hi2 >= 0xffe00000u;   // not finite
#pragma unroll
    for (int j = 0; j < 13; j++)
      if (j == g) m[j] = max(m[j], hi2);
  }
#pragma unroll
  for (int g = 0; g < 13; g++) m[g] = __reduce_max_sync(0xffffffffu, m[g]);
  bool ok = !__any_sync(0xffffffffu, any);
  int E[13];
#pragma unroll
  for (int g = 0; g < 13; g++) {
    E[g] = (int)(m[g] >> 21);
    // outside 2^+-150 the FP64 evaluation is used (zero groups are fine)
    if (m[g] != 0 && (E[g] < 1023 - 150 || E[g] > 1023 + 150)) ok = false;
  }
#pragma unroll
  for (int s = 0; s < PER; s++) {
    const int i = s * 32 + lane;
    if (i >= C::RECI) continue;
    int g = 0;
    if (i >= 3 * C::N2) {
      const int w = i - 3 * C::N2;
      g = w % (N + 1) == N ? 7 + w / (N + 1) : 1 + w / (N + 1);
    }
    int eb = 0;
#pragma unroll
    for (int j = 0; j < 13; j++)
      if (j == g) eb = E[j];
    int2 v = make_int2(0, 0);
    if (ok && eb > 0) v = limbs(fix_signed(q[s], eb) + fix_signed(q2[s], eb));
    out[limb_at<N>(e, C::RECI, i)] = v;
  }
  if (lane < C::NEXP) {
    int v = 0;
#pragma unroll
    for (int j = 0; j < 13; j++)
      if (j == lane) v = m[j] ? E[j] - 1022 : kFixZero;
    if (lane == 13) v = ok;
    exps[limb_at<N>(e, C::NEXP, lane)] = v;
  }
}

// The block's cells in plain FP64 (weak form, from the FP64 record): not a
// fast path, it keeps what FP64 gives for infinities, NaN and values near the
// ends of the range.  Called by every thread of the block; returns the sum of
// x * y_out over the thread's column.
template <int N>
__device__ __noinline__ double apply_cells_fp64(const OpParams<double> &p,
                                              const ApplyArgs<double> &a,
                                              const double *__restrict__ rec, double *cell,
                                              int l, int ee, const int *nbr, bool active) {
  using C = ICfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC;
  double *ue = cell, *Xs = ue + NB, *Ys = Xs + NB, *Zs = Ys + NB, *fa = Zs + NB;
  const double *tM = p.tab, *td0 = p.tab + 2 * N2, *td1 = td0 + N;
  const double *r = rec + (size_t)ee * C::RECW;
  const double *W = r + 3 * N2 + (a.transpose ? C::NW : 0);
  const int sk = a.transpose ? 1 : N, sq = a.transpose ? N : 1;
  const int tx = l % N, ty = l / N;
  __syncthreads();
  for (int z = 0; z < N; z++) ue[z * TPC + l] = a.x[(size_t)ee * NB + z * TPC + l];
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    double s1 = 0.0, s2 = 0.0;
    if (nbr[f] >= 0) {
      const double *xn = a.x + (size_t)nbr[f] * NB;
      for (int q = 0; q < N; q++) {
        const int off = dir == 0 ? l * N + q : (dir == 1 ? ty * N2 + q * N + tx : q * N2 + l);
        s1 += W[f * (N + 1) + q] * xn[off];
        if (q == (hi ? 0 : N - 1)) s2 = W[f * (N + 1) + N] * xn[off];
      }
    }
    fa[(2 * f) * TPC + l] = s1;
    fa[(2 * f + 1) * TPC + l] = s2;
  }
  __syncthreads();
  for (int z = 0; z < N; z++) {
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int q = 0; q < N; q++) {
      sx += r[tx * sk + q * sq] * ue[z * N2 + ty * N + q];
      sy += r[N2 + ty * sk + q * sq] * ue[z * N2 + q * N + tx];
      sz += r[2 * N2 + z * sk + q * sq] * ue[q * N2 + l];
    }
    const int lx = z * N + ty, ly = z * N + tx;
    if (tx == 0) sx += fa[lx];
    if (tx == N - 1) sx += fa[2 * TPC + lx];
    sx += td0[tx] * fa[TPC + lx] + td1[tx] * fa[3 * TPC + lx];
    if (ty == 0) sy += fa[4 * TPC + ly];
    if (ty == N - 1) sy += fa[6 * TPC + ly];
    sy += td0[ty] * fa[5 * TPC + ly] + td1[ty] * fa[7 * TPC + ly];
    if (z == 0) sz += fa[8 * TPC + l];
    if (z == N - 1) sz += fa[10 * TPC + l];
    sz += td0[z] * fa[9 * TPC + l] + td1[z] * fa[11 * TPC + l];
    Xs[z * N2 + l] = sx;
    Ys[z * N2 + l] = sy;
    Zs[z * N2 + l] = sz;
  }
  __syncthreads();
  double w[N];
  for (int z = 0; z < N; z++) {
    double s = 0.0, t1 = 0.0;
    for (int q = 0; q < N; q++) {
      s += tM[ty * N + q] * Xs[z * N2 + q * N + tx] + tM[tx * N + q] * Ys[z * N2 + ty * N + q];
      t1 += tM[tx * N + q] * Zs[z * N2 + ty * N + q];
    }
    w[z] = s;
    ue[z * N2 + l] = t1;
  }
  __syncthreads();
  double part = 0.0;
  if (!active) return part;
  for (int z = 0; z < N; z++) {
    double s = 0.0;
    for (int q = 0; q < N; q++)
      s += tM[z * N + q] * w[q] + tM[ty * N + q] * ue[z * N2 + q * N + tx];
    if (a.alpha != 1.0) s *= a.alpha;
    const size_t idx = (size_t)ee * NB + z * TPC + l;
    if (a.accumulate) s += a.y[idx];
    if (a.add) s += a.add[idx];
    part += a.x[idx] * s;
    a.y[idx] = s;
  }
  return part;
}

// 24 or 20 warps per SM.  33x29x37 Q4 183 -> 167 us with five blocks instead of
// the four the register count alone gives, 156 with the results put together on
// the integer pipe, 163 with s2 in finer units.  Degree 2 has its own kernel
// (k_apply_p); the exchanges through shared memory, 12 loads and stores per value
// there, are what it avoids (204 -> 160 us at 64^3 Q2).  At degrees 3 and 4 a plane per thread is 16 or
// 25 values with 96-bit sums, which does not fit the registers.
template <int N>
__global__ void __launch_bounds__(ICfg<N>::THREADS, N == 5 ? 5 : N == 4 ? 12 : 6)
    k_apply_i(const __grid_constant__ OpParams<double> p,
              const __grid_constant__ ApplyArgs<double> a, const int2 *__restrict__ rec,
              const int *__restrict__ exps, const double *__restrict__ rec64) {
  using C = ICfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC, CPB = C::CPB, NF = C::NF;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int sM[N2], sd0[N], sd1[N], sE[2 * CPB];
  const int t = threadIdx.x;
  const int cs = t / TPC;
  const int l = t - cs * TPC;
  int2 *ue = reinterpret_cast<int2 *>(smem_raw) + cs * C::PER_CELL;
  int2 *Xs = ue + NB, *Ys = Xs + NB, *Zs = Ys + NB;
  int2 *fa = Zs + NB;                // [2 NF][TPC]
  int2 *Am = fa + 2 * NF * TPC;      // A'_dir [3][N2], then [NF][N+1]

  if (a.skip && *a.skip) return;
#pragma unroll
  for (int i = 0; i < N2; i++)
    if (t == i) sM[i] = int_m<N>(i);
#pragma unroll
  for (int i = 0; i < N; i++)
    if (t == i) {
      sd0[i] = int_d0<N>(i);
      sd1[i] = int_d1<N>(i);
    }
  if (t < 2 * CPB) sE[t] = 2 * kFixZero;

  const int li = blockIdx.x * CPB + cs;
  const bool ranged = a.ncells > 0;
  const bool active = ranged ? li < a.ncells : li < p.ncell;
  const int e = ranged ? a.cell0 + li : li;
  const int ee = active ? e : 0;
  int ix[3];
  {
    const unsigned q0 = p.div0.div((unsigned)ee);
    const unsigned q1 = p.div1.div(q0);
    ix[0] = (int)((unsigned)ee - q0 * (unsigned)p.nc[0]);
    ix[1] = (int)(q0 - q1 * (unsigned)p.nc[1]);
    ix[2] = (int)q1;
  }
  const int stride[3] = {1, p.nc[0], p.nc[0] * p.nc[1]};
  int nbr[NF];
#pragma unroll
  for (int f = 0; f < NF; f++) {
    const int dir = f >> 1;
    if (f & 1) nbr[f] = ix[dir] + 1 < p.nc[dir] ? ee + stride[dir] : -1;
    else nbr[f] = ix[dir] > 0 ? ee - stride[dir] : -1;
  }

  // ---- all global loads first: own column, neighbour lines, record ----
  double col[N];
  const double *xe = a.x + (size_t)ee * NB;
#pragma unroll
  for (int z = 0; z < N; z++) col[z] = xe[z * TPC + l];
  const int flip = sign_flip(xe[0]);
  double v[NF][N];
#pragma unroll
  for (int f = 0; f < NF; f++) {
    const int dir = f >> 1;
    const double *xn = a.x + (size_t)(nbr[f] >= 0 ? nbr[f] : ee) * NB;
#pragma unroll
    for (int q = 0; q < N; q++) {
      const int off =
          dir == 0 ? l * N + q : (dir == 1 ? (l / N) * N2 + q * N + (l % N) : q * N2 + l);
      v[f][q] = xn[off];
    }
  }
  {
    const int2 *r = rec + (size_t)ee * C::RECI;
    for (int i = l; i < C::RECI; i += TPC) Am[i] = r[i];
  }
  const int *ex = exps + (size_t)ee * C::NEXP;
  const int EA = ex[0];
  __syncthreads();

  // ---- exponents: of the own column, and the bound of the cell's sums ----
  bool bad = ex[13] == 0;
  int eb[NF];   // biased exponent of each neighbour line
  {
    BlockExp own;
#pragma unroll
    for (int z = 0; z < N; z++) own.add(col[z]);
    bad |= !own.finite();
    int cand = 2 * kFixZero;
#pragma unroll
    for (int f = 0; f < NF; f++) {
      BlockExp b;
#pragma unroll
      for (int q = 0; q < N; q++) b.add(v[f][q]);
      eb[f] = b.biased();
      if (nbr[f] >= 0) {
        bad |= !b.finite();
        // |e_i s1 + d_i s2| over the face's two terms
        cand = max(cand, b.exponent() + max(ex[1 + f] + C::LN, ex[7 + f] + C::LD) + 1);
      }
    }
    atomicMax(&sE[2 * cs], own.exponent());
    atomicMax(&sE[2 * cs + 1], cand);
  }
  __syncthreads();
  const int Ex = sE[2 * cs];
  // three terms (volume, two faces) per direction
  const int Etot = max(Ex + EA + C::LN, sE[2 * cs + 1]) + 2;
  bad |= Etot > 900 || (Etot > kFixZero + 1000 && Etot < -780);
  const int ebx = Ex == kFixZero ? kFixMinBiased : Ex + 1022;

  // ---- own column to limbs; neighbour face data, aligned to the cell ----
  int2 uc[N], zf[4];   // own column; the z faces' data is read by this thread only
#pragma unroll
  for (int z = 0; z < N; z++) {
    uc[z] = fix_limbs(col[z], ebx, flip);
    ue[z * TPC + l] = uc[z];
  }
#pragma unroll
  for (int f = 0; f < NF; f++) {
    const int2 *w = Am + 3 * N2 + f * (N + 1);
    const int eu = eb[f] - 1022;
    long long hh = 0, mid = 0, h2 = 0, m2 = 0;
#pragma unroll
    for (int q = 0; q < N; q++) {
      const int2 u = fix_limbs(v[f][q], eb[f], flip);
      mac2(hh, mid, u, w[q]);
      if (q == ((f & 1) ? 0 : N - 1)) mac2(h2, m2, u, w[N]);
    }
    const long long s1 = mac2_value(hh, mid, Etot - eu - ex[1 + f] - 2);
    const long long s2 = mac2_value(h2, m2, Etot - eu - ex[7 + f] - 2 - C::FB);
    if (f < 4) {
      fa[(2 * f) * TPC + l] = split32(s1);
      fa[(2 * f + 1) * TPC + l] = split32(s2);
    } else {
      zf[2 * (f - 4)] = split32(s1);
      zf[2 * (f - 4) + 1] = split32(s2);
    }
  }
  // <x, y_out> of the fused CG
  const auto finish = [&](double part) {
    reduce_tail_grouped<C::THREADS>(a.dot_part, a.dot_max_blocks, a.dot_cnt,
                                    RedCtx{nullptr, a.dot_scal, a.dot_flags}, part, 0.0,
                                    a.dot_fin);
  };
  if (__syncthreads_or(bad)) {
    const double part =
        apply_cells_fp64<N>(p, a, rec64, reinterpret_cast<double *>(ue), l, ee, nbr, active);
    if (a.dot_part) finish(part);
    return;
  }

  // ---- directional operators and face lifts ----
  const int tx = l % N, ty = l / N;
  const int shu = Etot - Ex - EA - 2;
  // rounding constant of line entry i in units of s2: halves of the shifts below,
  // and the half units that cutting took from the volume term, from s1 on the
  // two ends and from the d_i s2 (d: sum of the entry's derivatives)
  const auto cut = [](int i, int d) {
    constexpr int kHalves =
        (C::FB > 0 ? 1 << (C::FB - 1) : 0) + (C::SHX > 0 ? 1 << (C::SHX - 1 + C::FB) : 0);
    return (long long)((((1 + (i == 0) + (i == N - 1)) << C::FB) + d) / 2 + kHalves);
  };
  {
    int2 Ax[N], Ay[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
      Ax[q] = Am[tx * N + q];
      Ay[q] = Am[N2 + ty * N + q];
    }
    const int d0x = sd0[tx], d1x = sd1[tx], d0y = sd0[ty], d1y = sd1[ty];
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int lx = z * N + ty, ly = z * N + tx;
      {
        long long hh = 0, mid = 0;
#pragma unroll
        for (int q = 0; q < N; q++) mac2(hh, mid, Ax[q], ue[z * N2 + ty * N + q]);
        SmallSum<false> s(mac2_value(hh, mid, shu));
        s.add(fa[0 * TPC + lx], tx == 0);
        s.add(fa[2 * TPC + lx], tx == N - 1);
        SmallSum<false> d(cut(tx, d0x + d1x));
        d.add(fa[1 * TPC + lx], d0x);
        d.add(fa[3 * TPC + lx], d1x);
        Xs[z * N2 + l] = split32((s.total() + d.template shifted<C::FB>()) >> C::SHX);
      }
      {
        long long hh = 0, mid = 0;
#pragma unroll
        for (int q = 0; q < N; q++) mac2(hh, mid, Ay[q], ue[z * N2 + q * N + tx]);
        SmallSum<false> s(mac2_value(hh, mid, shu));
        s.add(fa[4 * TPC + ly], ty == 0);
        s.add(fa[6 * TPC + ly], ty == N - 1);
        SmallSum<false> d(cut(ty, d0y + d1y));
        d.add(fa[5 * TPC + ly], d0y);
        d.add(fa[7 * TPC + ly], d1y);
        Ys[z * N2 + l] = split32((s.total() + d.template shifted<C::FB>()) >> C::SHX);
      }
      {
        long long hh = 0, mid = 0;
#pragma unroll
        for (int q = 0; q < N; q++) mac2(hh, mid, Am[2 * N2 + z * N + q], uc[q]);
        SmallSum<false> s(mac2_value(hh, mid, shu));
        if (z == 0) s.add(zf[0], 1);
        if (z == N - 1) s.add(zf[2], 1);
        SmallSum<false> d(cut(z, int_d0<N>(z) + int_d1<N>(z)));
        d.add(zf[1], int_d0<N>(z));
        d.add(zf[3], int_d1<N>(z));
        Zs[z * N2 + l] = split32((s.total() + d.template shifted<C::FB>()) >> C::SHX);
      }
    }
  }
  __syncthreads();
  // ---- W = M_y X + M_x Y ; T1 = M_x Z (into ue: its reads are past) ----
  constexpr long long kHalfM = 1ll << (C::SHM - 1);
  int Mx[N], My[N];
#pragma unroll
  for (int q = 0; q < N; q++) {
    Mx[q] = sM[tx * N + q];
    My[q] = sM[ty * N + q];
  }
  int2 W[N];
#pragma unroll
  for (int z = 0; z < N; z++) {
    SmallSum<C::WIDE> w(kHalfM), t1(kHalfM);
#pragma unroll
    for (int q = 0; q < N; q++) {
      w.add(Xs[z * N2 + q * N + tx], My[q]);
      w.add(Ys[z * N2 + ty * N + q], Mx[q]);
      t1.add(Zs[z * N2 + ty * N + q], Mx[q]);
    }
    W[z] = split32(w.template shifted<C::SHM>());
    ue[z * N2 + l] = split32(t1.template shifted<C::SHM>());
  }
  __syncthreads();
  // ---- out = M_z W + M_y T1 ----
  double part = 0.0;
  if (active) {
    const bool zero = Etot <= kFixZero + 1000;   // no data (but rounding constants)
    double *ye = a.y + (size_t)e * NB;
    const double *ad = a.add ? a.add + (size_t)e * NB : nullptr;
    const bool scale = a.alpha != 1.0;
#pragma unroll
    for (int z = 0; z < N; z++) {
      SmallSum<C::WIDE> s(C::WIDE ? kHalfM : 0);
#pragma unroll
      for (int q = 0; q < N; q++) {
        s.add(W[q], int_m<N>(z * N + q));
        s.add(ue[z * N2 + q * N + tx], My[q]);
      }
      double r = zero ? 0.0
                      : fix_to_double(s.template shifted<C::WIDE ? C::SHM : 0>(), Etot + C::OUTE,
                                      flip);
      if (scale) r *= a.alpha;
      const int idx = z * TPC + l;
      if (a.accumulate) r += ye[idx];
      if (ad) r += ad[idx];
      if (a.dot_part) part += xe[idx] * r;
      ye[idx] = r;
    }
  }
  if (a.dot_part) finish(part);
}

template <int N>
static int record_i_n(pdg_context *ctx, const OpParams<double> &p, int transpose) {
  using C = ICfg<N>;
  int2 *&out = transpose ? ctx->reciT : ctx->reci;
  int *&ex = transpose ? ctx->reciT_exp : ctx->reci_exp;
  const long cells = N == 3 ? (ctx->ncell + kGroup - 1) / kGroup * kGroup : ctx->ncell;
  if (!out) PDG_CUDA_TRY(cudaMalloc(&out, sizeof(int2) * C::RECI * cells));
  if (!ex) PDG_CUDA_TRY(cudaMalloc(&ex, sizeof(int) * C::NEXP * cells));
  const double den = (double)IntTab<N>::den * IntTab<N>::den, denw = den * IntTab<N>::dden;
  const double rd = 1.0 / den, rw = 1.0 / denw;
  const unsigned blocks = (unsigned)((ctx->ncell + 3) / 4);
  k_record_i<N><<<blocks, 128, 0, ctx->stream>>>(p, ctx->rec64, out, ex, transpose, rd,
                                                 std::fma(-rd, den, 1.0) / den, rw,
                                                 std::fma(-rw, denw, 1.0) / denw);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

// the limb records of the operator (transpose 0) or of its transpose (1),
// built once per coefficient field
int prepare_apply_i(pdg_context *ctx, int transpose) {
  int &valid = transpose ? ctx->reciT_valid : ctx->reci_valid;
  if (valid) return PDG_OK;
  if (!ctx->rec64) return set_error(PDG_EINVAL, "limb records need the FP64 records");
  const OpParams<double> p = make_params<double>(ctx, ctx->K64, ctx->c64, ctx->tab64);
  int st;
  switch (ctx->N) {
    case 2: st = record_i_n<2>(ctx, p, transpose); break;
    case 3: st = record_i_n<3>(ctx, p, transpose); break;
    case 4: st = record_i_n<4>(ctx, p, transpose); break;
    case 5: st = record_i_n<5>(ctx, p, transpose); break;
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
  if (st == PDG_OK) mark_built(ctx, &valid);
  return st;
}

// The integer mass tables are those of the equidistant nodes (the Legendre
// basis maps onto them); the Gauss-Lobatto nodes of degree 3 and 4 are
// irrational and keep the FP64 kernel.
bool apply_i_usable(const pdg_context *ctx) {
  return ctx->dim == 3 && (ctx->basis != PDG_BASIS_LOBATTO || ctx->k <= 2);
}

// the fused CG: <p, A p> -> lambda in the same launch
static ApplyArgs<double> fused(const pdg_context *ctx, const ApplyArgs<double> &a) {
  ApplyArgs<double> af = a;
  if (ctx->fuse_fin && a.ncells == 0) {
    af.dot_part = ctx->fuse_part;
    af.dot_max_blocks = ctx->fuse_max_blocks;
    af.dot_cnt = ctx->fuse_cnt;
    af.dot_scal = ctx->red_out;
    af.dot_flags = ctx->d_flag;
    af.dot_fin = ctx->fuse_fin;
  }
  return af;
}

template <int N>
static int launch_i_n(pdg_context *ctx, const ApplyArgs<double> &a, const OpParams<double> &p) {
  using C = ICfg<N>;
  const size_t smem = sizeof(int2) * C::CPB * C::PER_CELL;
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    PDG_CUDA_TRY(cudaFuncSetAttribute(k_apply_i<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    attr_dev = ctx->device;
  }
  const long work = a.ncells > 0 ? a.ncells : ctx->ncell;
  if (work <= 0) return PDG_OK;
  const unsigned blocks = (unsigned)((work + C::CPB - 1) / C::CPB);
  k_apply_i<N><<<blocks, C::THREADS, smem, ctx->stream>>>(
      p, fused(ctx, a), a.transpose ? ctx->reciT : ctx->reci, a.transpose ? ctx->reciT_exp : ctx->reci_exp,
      ctx->rec64);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

int launch_apply_i(pdg_context *ctx, const ApplyArgs<double> &a, const OpParams<double> &p) {
  PDG_TRY(prepare_apply_i(ctx, a.transpose));
  switch (ctx->N) {
    case 2: return launch_i_n<2>(ctx, a, p);
    case 3: return launch_apply_p(ctx, fused(ctx, a), p);
    case 4: return launch_i_n<4>(ctx, a, p);
    case 5: return launch_i_n<5>(ctx, a, p);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}

}  // namespace pdg
