// pdg_conv_i.cu -- the FP64 convection apply (pdg_conv.cu, not transposed) in
// 64-bit fixed point (pdg_fixed.cuh).
//
// Same evaluation as conv_block<double, N> (reference:
// localoperator/convectiondiffusiondg.hh:175-186, 424-443, 796-849): values at
// the Gauss points, times the weighted velocity, tested with the gradients,
// and the upwind fluxes at the face points; 11 N + 3 multiply-adds per DOF in
// the volume and 36 on the faces.  In FP64 that is bound by the FP64 pipe (91 %
// active); as limb contractions it takes three IMAD.WIDE each.  32^3 Q4 with
// the diffusion operator: 421 us, with this part in FP64 993 us; the error
// against 64 bits is the same (1.5e-14 against 1.4e-14), and on smooth data
// J(3u) - 3 J(u) of the convection alone is 1.5e-15, 1.6e-15, 2.7e-15 and 3.8e-15 of
// J u at 24^3, k = 1..4 (FP64: 3.2e-15, 3.6e-15, 8.8e-15, 1.2e-14).
//
// Scaling.  The cell's values, each neighbour's face layer, the cell's volume
// weights and each face's outflow and inflow weights have an exponent each.
// The 1D tables' row and column sums of magnitudes bound every contraction, so
// the exponents of all stages follow from those; B and D (values and
// derivatives at the Gauss points) are scaled so that the two products that
// meet in one sum have the same unit (ConvExp).  The values at the points, after
// the x test, before the z test and the fluxes are brought to 59 bits of their
// largest: the bounds of all stages together cost 10 bits (13 times the rounding
// of FP64 on smooth data at k = 4, at 393 us).  The face fluxes share one
// exponent per cell, formed from what each face can let in or out, so a large
// neighbour downstream costs nothing.  Blocks with data that is not finite or
// far from the middle of the range are evaluated in FP64.
#include <algorithm>
#include <cmath>

#include "pdg_conv.cuh"
#include "pdg_fixed.cuh"

namespace pdg {

// exponents of the tables: |B| < 2^eb, |D| < 2^ed; row sums of |B| < 2^lb, column
// sums of |B| < 2^lbt and of |D| < 2^ldt, with ldt - ed = lbt - eb
struct ConvExp {
  int eb, ed, lb, lbt, ldt;
};

// per cell: exponents of the volume weights (all directions), of each face's
// outflow (F >= 0) and inflow (F < 0) weights, and whether all are in range
constexpr int kConvNexp = 16;
template <int N>
__global__ void k_conv_exps(long ncell, const double *__restrict__ vrec, int *__restrict__ exps) {
  using C = CCfg<N>;
  const long e = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (e >= ncell) return;
  const double *r = vrec + e * (C::VREC + C::FREC);
  BlockExp g;
  for (int i = lane; i < C::VREC; i += 32) g.add(r[i]);
  bool ok = true;
  const auto put = [&](int slot, unsigned m) {
    m = __reduce_max_sync(0xffffffffu, m);
    const int b = (int)(m >> 21);
    ok = ok && (m == 0 || (b > 1023 - 150 && b < 1023 + 150));
    if (lane == 0) exps[e * kConvNexp + slot] = m ? b - 1022 : kFixZero;
  };
  put(0, g.m);
  for (int f = 0; f < 6; f++) {
    BlockExp out, in;
    for (int i = lane; i < C::N2; i += 32) {
      const double v = r[C::VREC + f * C::N2 + i];
      if (v >= 0.0) out.add(v);
      else in.add(v);   // (a NaN too: found by its exponent)
    }
    put(1 + f, out.m);
    put(7 + f, in.m);
  }
  if (lane == 0) exps[e * kConvNexp + 13] = ok;
}

// sum of N limb products (fb: 59 bits), rounded to units 2^s larger
template <int N, class FA, class FB>
__device__ __forceinline__ long long conv_sum(FA fa, FB fb, int s) {
  long long hh = 0, mid = (1ll << (s + 28)) >> 1;
#pragma unroll
  for (int q = 0; q < N; q++) mac2(hh, mid, fa(q), fb(q));
  return mac2_value_wide(hh, mid) >> s;
}

// significant bits of |v|, and v 2^-s, rounded for s > 0
__device__ __forceinline__ int conv_bits(long long v) {
  return v ? 64 - __clzll(v ^ (v >> 63)) : 0;
}
__device__ __forceinline__ long long conv_shift(long long v, int s) {
  const int r = min(s, 62);
  return s > 0 ? (v + ((1ll << r) >> 1)) >> r
               : (long long)((unsigned long long)v << min(-s, 63));
}

template <int N>
__device__ __noinline__ void conv_block_fp64(const OpParams<double> &p, const ApplyArgs<double> &a,
                                             const double *vrec, const double *tabBD,
                                             unsigned char *smem_raw) {
  __syncthreads();
  conv_block<double, N>(p, a, vrec, tabBD, smem_raw);
}

// Five blocks per SM at k = 4 (96 instead of 106 registers) and the records
// prefetched: 32^3 Q4 with the diffusion operator 410 -> 396 -> 389 us when measured (issue
// slots were 40 % busy, a quarter of the stalls waited for the records).
template <int N>
__global__ void __launch_bounds__(CCfg<N>::THREADS, N == 5 ? 5 : N == 4 ? 6 : N == 3 ? 7 : 9)
    k_conv_i(const __grid_constant__ OpParams<double> p,
             const __grid_constant__ ApplyArgs<double> a, const double *__restrict__ vrec,
             const double *__restrict__ tabBD, const int2 *__restrict__ tabi,
             const int *__restrict__ exps, const ConvExp ce) {
  using C = CCfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC, CPB = C::CPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int sE[7 * CPB];
  // bits of the cell's largest value at the points, after the x test, of a flux
  __shared__ int sB[3 * CPB];
  if (a.skip && *a.skip) return;
  int2 *tB = reinterpret_cast<int2 *>(smem_raw);   // B[q][a]
  int2 *tD = tB + N2;                              // D[q][a]
  const int t = threadIdx.x, cs = t / TPC, l = t - cs * TPC;
  int2 *S0 = tB + C::TAB + cs * C::PER_CELL_RAW;
  int2 *S1 = S0 + NB, *S2 = S1 + NB, *S3 = S2 + NB;
  int2 *fl = S3 + NB, *Ue = fl + 6 * N2, *Un = Ue + 6 * N2;
  for (int i = t; i < C::TAB; i += C::THREADS) tB[i] = tabi[i];
  for (int i = t; i < 7 * CPB; i += C::THREADS) sE[i] = kFixZero;
  for (int i = t; i < 3 * CPB; i += C::THREADS) sB[i] = 0;
  const int li = blockIdx.x * CPB + cs;
  const bool ranged = a.ncells > 0;
  const bool active = ranged ? li < a.ncells : li < p.ncell;
  const long e = ranged ? a.cell0 + li : li;
  const long ee = active ? e : 0;
  int ix[3];
  {
    const unsigned q0 = p.div0.div((unsigned)ee);
    const unsigned q1 = p.div1.div(q0);
    ix[0] = (int)((unsigned)ee - q0 * (unsigned)p.nc[0]);
    ix[1] = (int)(q0 - q1 * (unsigned)p.nc[1]);
    ix[2] = (int)q1;
  }
  const long stride[3] = {1, (long)p.nc[0], (long)p.nc[0] * p.nc[1]};
  const double *rec = vrec + ee * (C::VREC + C::FREC);
  const int *ex = exps + ee * kConvNexp;
  const int tx = l % N, ty = l / N;   // also the face node / point (pa, pb)
  // the cells' records to the L2 cache while the trial values are formed
  {
    const long r0 = ranged ? a.cell0 + (long)blockIdx.x * CPB : (long)blockIdx.x * CPB;
    const long r1 = min(r0 + CPB, ranged ? (long)a.cell0 + a.ncells : p.ncell);
    constexpr int RB = (int)sizeof(double) * (C::VREC + C::FREC);
    const uintptr_t b0 = reinterpret_cast<uintptr_t>(vrec) + (uintptr_t)r0 * RB;
    const uintptr_t b1 = (b0 + (uintptr_t)(r1 - r0) * RB) & ~(uintptr_t)15;
    const uintptr_t b = (b0 + 15) & ~(uintptr_t)15;
    if (t == 0 && b < b1)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b), "r"((unsigned)(b1 - b))
                   : "memory");
  }

  // ---- own column, and this thread's node of each neighbour's face layer ----
  double col[N], nl[6];
  const double *xe = a.x + ee * NB;
  const int flip = sign_flip(xe[0]);
#pragma unroll
  for (int z = 0; z < N; z++) col[z] = xe[z * N2 + l];
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    const bool on = hi ? ix[dir] + 1 < p.nc[dir] : ix[dir] > 0;
    nl[f] = 0.0;
    // a face without inflow never reads its neighbour
    if (on && ex[7 + f] != kFixZero) {
      const double *xn = a.x + (ee + (hi ? stride[dir] : -stride[dir])) * NB;
      const int lay = hi ? 0 : N - 1;
      nl[f] = xn[dir == 0 ? l * N + lay : dir == 1 ? ty * N2 + lay * N + tx : lay * N2 + l];
    }
  }
  __syncthreads();
  bool bad = ex[13] == 0;
  {
    BlockExp own;
#pragma unroll
    for (int z = 0; z < N; z++) own.add(col[z]);
    bad |= !own.finite();
    atomicMax(&sE[7 * cs], own.exponent());
#pragma unroll
    for (int f = 0; f < 6; f++) {
      BlockExp b;
      b.add(nl[f]);
      bad |= !b.finite();
      if (b.any) atomicMax(&sE[7 * cs + 1 + f], b.exponent());
    }
  }
  __syncthreads();
  const int Eu = sE[7 * cs], EG = ex[0];
  const int Evol = Eu + 3 * ce.lb + EG;
  int Efl = 3 * kFixZero;
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    const bool on = hi ? ix[dir] + 1 < p.nc[dir] : ix[dir] > 0;
    const int bc = p.bc[f];
    if (on || bc == PDG_BC_DIRICHLET || bc == PDG_BC_OUTFLOW)
      Efl = max(Efl, Eu + 2 * ce.lb + ex[1 + f]);
    if (on) Efl = max(Efl, sE[7 * cs + 1 + f] + 2 * ce.lb + ex[7 + f]);
    else if (bc == PDG_BC_OUTFLOW) Efl = max(Efl, Eu + 2 * ce.lb + ex[7 + f]);
  }
  constexpr int kNone = kFixZero + 2000;   // below: nothing but zeros
  bad |= Evol > 850 || Efl > 850 || (Evol > kNone && Evol < -700) || (Efl > kNone && Efl < -700);
  const int ebu = Eu == kFixZero ? kFixMinBiased : Eu + 1022;
  int2 uc[N];
#pragma unroll
  for (int z = 0; z < N; z++) {
    uc[z] = fix_limbs<kFixWide>(col[z], ebu, flip);
    S3[z * N2 + l] = uc[z];
  }
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int En = sE[7 * cs + 1 + f];
    Un[f * N2 + l] = fix_limbs<kFixWide>(nl[f], En == kFixZero ? kFixMinBiased : En + 1022, flip);
  }
  const int sf = ce.lb - ce.eb, sb = ce.lbt - ce.eb;
  // forward z: S0 = B_z u
#pragma unroll
  for (int q = 0; q < N; q++)
    S0[q * N2 + l] = limbs(conv_sum<N>([&](int k) { return tB[q * N + k]; },
                                       [&](int k) { return uc[k]; }, sf));
  if (__syncthreads_or(bad)) {
    conv_block_fp64<N>(p, a, vrec, tabBD, smem_raw);
    return;
  }
  // ---- volume ----
  long long r[N];
  int up;   // exponent of the unit of r, less Evol
  {
    int2 B[N];
#pragma unroll
    for (int k = 0; k < N; k++) B[k] = tB[ty * N + k];
#pragma unroll
    for (int z = 0; z < N; z++)
      S1[z * N2 + l] = limbs(conv_sum<N>([&](int k) { return B[k]; },
                                         [&](int k) { return S0[z * N2 + k * N + tx]; }, sf));
  }
  __syncthreads();
  {
    int2 B[N], uq[N];
    long long w[N];
    int bits = 0;
#pragma unroll
    for (int k = 0; k < N; k++) B[k] = tB[tx * N + k];
#pragma unroll
    for (int z = 0; z < N; z++) {
      w[z] = conv_sum<N>([&](int k) { return B[k]; },
                         [&](int k) { return S1[z * N2 + ty * N + k]; }, 0);
      bits = max(bits, conv_bits(w[z]));
    }
    atomicMax(&sB[3 * cs], bits);
    __syncthreads();
    const int sq = sB[3 * cs] - kFixWide;
    up = sq - sf - kFixWide;
#pragma unroll
    for (int z = 0; z < N; z++) uq[z] = limbs(conv_shift(w[z], sq));
    // F_dir = G_dir u at the point (tx, ty, z)
    const int ebg = EG == kFixZero ? kFixMinBiased : EG + 1022;
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int q = z * N2 + l;
      S0[q] = limbs(conv_sum<1>([&](int) { return fix_limbs(rec[q], ebg); },
                                [&](int) { return uq[z]; }, 0));
      S1[q] = limbs(conv_sum<1>([&](int) { return fix_limbs(rec[NB + q], ebg); },
                                [&](int) { return uq[z]; }, 0));
      S2[q] = limbs(conv_sum<1>([&](int) { return fix_limbs(rec[2 * NB + q], ebg); },
                                [&](int) { return uq[z]; }, 0));
    }
  }
  __syncthreads();
  {
    // x: Tx = D^t F_x, Ty = B^t F_y, Tz = B^t F_z
    int2 B[N], D[N];
    long long T[3][N];
    int bits = 0;
#pragma unroll
    for (int k = 0; k < N; k++) {
      B[k] = tB[k * N + tx];
      D[k] = tD[k * N + tx];
    }
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int i = z * N2 + ty * N;
      T[0][z] = conv_sum<N>([&](int k) { return D[k]; }, [&](int k) { return S0[i + k]; }, 0);
      T[1][z] = conv_sum<N>([&](int k) { return B[k]; }, [&](int k) { return S1[i + k]; }, 0);
      T[2][z] = conv_sum<N>([&](int k) { return B[k]; }, [&](int k) { return S2[i + k]; }, 0);
#pragma unroll
      for (int d = 0; d < 3; d++) bits = max(bits, conv_bits(T[d][z]));
    }
    atomicMax(&sB[3 * cs + 1], bits);
    __syncthreads();
    const int st = sB[3 * cs + 1] - kFixWide;
    up += st;
#pragma unroll
    for (int z = 0; z < N; z++) {
      S0[z * N2 + l] = limbs(conv_shift(T[0][z], st));
      S1[z * N2 + l] = limbs(conv_shift(T[1][z], st));
      S2[z * N2 + l] = limbs(conv_shift(T[2][z], st));
    }
  }
  __syncthreads();
  {
    // y: Sxy = B^t Tx + D^t Ty, Sz = B^t Tz (same unit, one bit larger)
    int2 B[N], D[N], Sxy[N], Sz[N];
    long long wxy[N], wz[N];
    int bits = 0;
#pragma unroll
    for (int k = 0; k < N; k++) {
      B[k] = tB[k * N + ty];
      D[k] = tD[k * N + ty];
    }
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int i = z * N2 + tx;
      wxy[z] = conv_sum<2 * N>(
          [&](int k) { return k < N ? B[k < N ? k : 0] : D[k < N ? 0 : k - N]; },
          [&](int k) { return k < N ? S0[i + k * N] : S1[i + (k - N) * N]; }, 0);
      wz[z] = conv_sum<N>([&](int k) { return B[k]; }, [&](int k) { return S2[i + k * N]; }, 0);
      bits = max(bits, max(conv_bits(wxy[z]), conv_bits(wz[z])));
    }
    const int sy = bits - kFixWide;   // of this thread's column
    up += sy + ce.ed + 2 * ce.eb;
#pragma unroll
    for (int z = 0; z < N; z++) {
      Sxy[z] = limbs(conv_shift(wxy[z], sy));
      Sz[z] = limbs(conv_shift(wz[z], sy));
    }
    // z: r = B^t Sxy + D^t Sz
#pragma unroll
    for (int z = 0; z < N; z++)
      r[z] = conv_sum<2 * N>(
          [&](int k) { return k < N ? tB[(k < N ? k : 0) * N + z] : tD[(k < N ? 0 : k - N) * N + z]; },
          [&](int k) { return k < N ? Sxy[k < N ? k : 0] : Sz[k < N ? 0 : k - N]; }, 0);
  }

  // ---- faces: rows of the node layers, partial traces (own Ue, neighbour fl) ----
  {
    int2 B[N];
#pragma unroll
    for (int k = 0; k < N; k++) B[k] = tB[tx * N + k];
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const int dir = f >> 1, hi = f & 1;
      const int s0 = dir == 0 ? N : 1, s1 = dir == 2 ? N : N2;   // strides of the layer
      const int sn = dir == 0 ? 1 : dir == 1 ? N : N2;
      const int row = (hi ? N - 1 : 0) * sn + ty * s1;
      Ue[f * N2 + l] = limbs(conv_sum<N>([&](int k) { return B[k]; },
                                         [&](int k) { return S3[row + k * s0]; }, sf));
      fl[f * N2 + l] = limbs(conv_sum<N>([&](int k) { return B[k]; },
                                         [&](int k) { return Un[f * N2 + ty * N + k]; }, sf));
    }
  }
  __syncthreads();
  // ---- upwind flux at the face points (into Un), 59 bits of the largest ----
  int sfl;
  {
    int2 B[N];
    long long w6[6];
    int s6[6], bits = -1000;
#pragma unroll
    for (int k = 0; k < N; k++) B[k] = tB[ty * N + k];
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const int dir = f >> 1, hi = f & 1;
      const bool on = hi ? ix[dir] + 1 < p.nc[dir] : ix[dir] > 0;
      const double bn = rec[C::VREC + f * N2 + l];
      const int bc = p.bc[f];
      const bool out = bn >= 0.0;
      const bool own = out ? on || bc == PDG_BC_DIRICHLET || bc == PDG_BC_OUTFLOW
                           : !on && bc == PDG_BC_OUTFLOW;
      const bool inflow = !out && on && !a.diag_only;
      w6[f] = 0;
      s6[f] = 0;
      if (own || inflow) {
        const int2 *U = own ? Ue : fl;
        const int2 w = limbs(conv_sum<N>([&](int k) { return B[k]; },
                                         [&](int k) { return U[f * N2 + k * N + tx]; }, sf));
        const int EF = out ? ex[1 + f] : ex[7 + f];
        const int Es = own ? Eu : sE[7 * cs + 1 + f];
        long long hh = 0, mid = 0;
        mac2(hh, mid, fix_limbs(bn, EF == kFixZero ? kFixMinBiased : EF + 1022), w);
        w6[f] = mac2_value_wide(hh, mid);
        s6[f] = Efl - (Es + 2 * ce.lb + EF);
        if (w6[f]) bits = max(bits, conv_bits(w6[f]) - s6[f]);
      }
    }
    atomicMax(&sB[3 * cs + 2], bits + 1000);
    __syncthreads();
    const int top = sB[3 * cs + 2];
    sfl = top ? top - 1000 - kFixWide : 0;   // (0: no flux)
#pragma unroll
    for (int f = 0; f < 6; f++) Un[f * N2 + l] = limbs(conv_shift(w6[f], s6[f] + sfl));
  }
  __syncthreads();
  // ---- test with the face basis: rows (into Ue), then columns (into fl) ----
  {
    int2 B[N];
#pragma unroll
    for (int k = 0; k < N; k++) B[k] = tB[k * N + tx];
#pragma unroll
    for (int f = 0; f < 6; f++)
      Ue[f * N2 + l] = limbs(conv_sum<N>([&](int k) { return B[k]; },
                                         [&](int k) { return Un[f * N2 + ty * N + k]; }, sb));
  }
  __syncthreads();
  {
    int2 B[N];
#pragma unroll
    for (int k = 0; k < N; k++) B[k] = tB[k * N + ty];
    // R[n1][n0] of this thread's face node, as plain 64-bit integers
#pragma unroll
    for (int f = 0; f < 6; f++)
      reinterpret_cast<long long *>(fl)[f * N2 + l] =
          conv_sum<N>([&](int k) { return B[k]; },
                      [&](int k) { return Ue[f * N2 + k * N + tx]; }, 0);
  }
  __syncthreads();
  if (!active) return;
  const int sg = flip & (int)0x80000000;
  const double uv =
      Evol > kNone
          ? __hiloint2double(sg | ((Evol + up + 1023) << 20), 0)
          : 0.0;
  const double uf =
      Efl > kNone ? __hiloint2double(sg | ((Efl + ce.lbt + ce.eb + sfl - kFixWide + 1023) << 20), 0) : 0.0;
  const long long *R = reinterpret_cast<const long long *>(fl);
  double *ye = a.y + e * NB;
#pragma unroll
  for (int z = 0; z < N; z++) {
    long long s = 0;
    if (tx == 0) s += R[z * N + ty];
    if (tx == N - 1) s += R[N2 + z * N + ty];
    if (ty == 0) s += R[2 * N2 + z * N + tx];
    if (ty == N - 1) s += R[3 * N2 + z * N + tx];
    if (z == 0) s += R[4 * N2 + l];
    if (z == N - 1) s += R[5 * N2 + l];
    ye[z * N2 + l] += a.alpha * ((double)s * uf - (double)r[z] * uv);
  }
}

static int ceil_log2(double x) {
  int e;
  const double m = std::frexp(x, &e);
  return m == 0.5 ? e - 1 : e;
}

// the limb tables and exponents of the context's 1D basis, and the cells'
// exponents for the current velocity
template <int N>
static int conv_setup_i_n(pdg_context *ctx, const double *tab) {
  using C = CCfg<N>;
  constexpr int N2 = C::N2;
  double maxb = 0, maxd = 0, rb = 0, cb = 0, cd = 0;
  for (int i = 0; i < N; i++) {
    double r = 0, c = 0, d = 0;
    for (int k = 0; k < N; k++) {
      maxb = std::max(maxb, std::fabs(tab[i * N + k]));
      maxd = std::max(maxd, std::fabs(tab[N2 + i * N + k]));
      r += std::fabs(tab[i * N + k]);
      c += std::fabs(tab[k * N + i]);
      d += std::fabs(tab[N2 + k * N + i]);
    }
    rb = std::max(rb, r);
    cb = std::max(cb, c);
    cd = std::max(cd, d);
  }
  int eb, ed0;
  std::frexp(maxb, &eb);
  std::frexp(maxd, &ed0);
  const double slack = 1.0 + 1e-9;
  const int lb = std::max(ceil_log2(rb * slack), eb), lbt = std::max(ceil_log2(cb * slack), eb);
  const int ldt = std::max(ceil_log2(cd * slack), ed0 - eb + lbt);
  const int ed = eb + ldt - lbt;
  int2 h[2 * N2];
  for (int i = 0; i < 2 * N2; i++) {
    const long long X = std::llround(std::ldexp(tab[i], kFixBits - (i < N2 ? eb : ed)));
    const int hi = (int)((X + (1ll << 28)) >> 29);
    h[i] = make_int2(hi, (int)(X - ((long long)hi << 29)));
  }
  const int c[5] = {eb, ed, lb, lbt, ldt};
  for (int i = 0; i < 5; i++) ctx->conv_exp[i] = c[i];
  if (!ctx->convtabi) PDG_CUDA_TRY(cudaMalloc(&ctx->convtabi, sizeof(h)));
  PDG_CUDA_TRY(cudaMemcpy(ctx->convtabi, h, sizeof(h), cudaMemcpyHostToDevice));
  if (!ctx->convexps)
    PDG_CUDA_TRY(cudaMalloc(&ctx->convexps, sizeof(int) * kConvNexp * ctx->ncell));
  k_conv_exps<N><<<(unsigned)((ctx->ncell + 3) / 4), 128, 0, ctx->stream>>>(ctx->ncell, ctx->conv64,
                                                                            ctx->convexps);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

int conv_setup_i(pdg_context *ctx, const double *tab) {
  switch (ctx->N) {
    case 2: return conv_setup_i_n<2>(ctx, tab);
    case 3: return conv_setup_i_n<3>(ctx, tab);
    case 4: return conv_setup_i_n<4>(ctx, tab);
    case 5: return conv_setup_i_n<5>(ctx, tab);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}

template <int N>
static int launch_conv_i_n(pdg_context *ctx, const ApplyArgs<double> &a) {
  using C = CCfg<N>;
  const size_t smem = sizeof(int2) * (C::TAB + C::CPB * C::PER_CELL_RAW);
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    PDG_CUDA_TRY(cudaFuncSetAttribute(k_conv_i<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    attr_dev = ctx->device;
  }
  const OpParams<double> p = make_params<double>(ctx, ctx->K64, nullptr, ctx->tab64);
  const long work = a.ncells > 0 ? a.ncells : ctx->ncell;
  if (work <= 0) return PDG_OK;
  const int *c = ctx->conv_exp;
  k_conv_i<N><<<(unsigned)((work + C::CPB - 1) / C::CPB), C::THREADS, smem, ctx->stream>>>(
      p, a, ctx->conv64, ctx->convtab64, ctx->convtabi, ctx->convexps,
      ConvExp{c[0], c[1], c[2], c[3], c[4]});
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

int launch_conv_i(pdg_context *ctx, const ApplyArgs<double> &a) {
  switch (ctx->N) {
    case 2: return launch_conv_i_n<2>(ctx, a);
    case 3: return launch_conv_i_n<3>(ctx, a);
    case 4: return launch_conv_i_n<4>(ctx, a);
    case 5: return launch_conv_i_n<5>(ctx, a);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}

}  // namespace pdg
