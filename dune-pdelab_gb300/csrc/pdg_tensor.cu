// pdg_tensor.cu -- the 3D cell operator with a full diffusion tensor A per
// cell (and a reaction per cell), in FP64 and FP32.
//
// Reference: ConvectionDiffusionDG::alpha_volume / alpha_skeleton /
// residual_boundary_integral with A at the cell centre
// (localoperator/convectiondiffusiondg.hh:105-188, 270-471, 683-879).
//
// A is constant on the axis-parallel cell, so every integrand is a polynomial
// that the Gauss rule of order 2k integrates exactly and the forms can be
// evaluated on the nodes: with Dn the 1D nodal differentiation matrix
// (derivatives of Q_k functions are nodal fields again), M the 1D mass matrix,
// L = M^-1 Dn^T M and m_0, m_1 = M^-1 e_0, M^-1 e_{N-1},
//
//   y_e = (M (x) M (x) M) [ sum_i L_i F_i + sum_faces m_f t_f + c u ],
//   F_i = sum_j A_ij (g_j + r_j),   g_j = Dn_j u,
//
// t_f the value terms of face f (consistency and penalty: omega-weighted normal
// fluxes and the jump, nodal fields of the face), r_j the lift of theta omega
// jump of the two faces normal to j, which carries the symmetry term
// (A_s n).grad psi through the same divergence as the volume.  All factors of
// the cell sizes are in the scaled tensor A_ij detJ / (h_i h_j).
// Per cell 9 N^4 + 9 N^3 multiply-adds for the volume and masses and about
// 30 N^3 for the faces, against 18 N^4 + 180 N^3 at the Gauss points
// (pdg_general.cu, which remains for tensors and reactions per point and for
// 2D).  FP32 at 15 to 26 thousand cells of degree 1 to 4 takes 16 to 18 us
// against 26 to 38 us.  The FP64 kernel is bound by its FP64 pipe, so its time
// follows the count (41x37x39 Q2 380 us, at the Gauss points 1735 us); the
// operator of degrees 1 to 3 runs in fixed point on the integer pipe instead
// (k_apply_tensor_i below: 100 us).
//
// Thread mapping: N*N threads per cell, thread (tx, ty) owns the z-column;
// face steps: one face node per thread.
#include "pdg_fixed.cuh"
#include "pdg_ops.cuh"

namespace pdg {

template <int N>
struct TCfg {
  static constexpr int N2 = N * N, NB = N * N * N, TPC = N * N;
  static constexpr int CPB = (128 / TPC) > 0 ? (128 / TPC) : 1;
  static constexpr int THREADS = CPB * TPC;
  static constexpr int TAB = 3 * N2 + 4 * N;   // M, Dn, L, m0, m1, d0, d1
  // per cell: u, g_x, g_y, g_z, neighbour face values [6][N2], t [6][N2],
  // r data [6][N2], scaled tensor (9), neighbours' flux columns [6][3], face
  // coefficients [6][3] {omega_s, omega_n, penalty}
  static constexpr int PER_CELL = 4 * NB + 18 * N2 + 9 + 18 + 18;
};

// the cells of a block; called by all its threads
template <typename T, int N>
__device__ __forceinline__ void tensor_block(const OpParams<T> &p, const ApplyArgs<T> &a,
                                             const T *__restrict__ Ac, const T *__restrict__ tab,
                                             unsigned char *smem_raw) {
  using C = TCfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC, CPB = C::CPB;
  T *tM = reinterpret_cast<T *>(smem_raw);
  T *tD = tM + N2, *tL = tD + N2, *tm0 = tL + N2, *tm1 = tm0 + N, *td0 = tm1 + N,
    *td1 = td0 + N;
  const int t = threadIdx.x;
  const int cs = t / TPC;
  const int l = t - cs * TPC;
  T *U = tM + C::TAB + cs * C::PER_CELL;
  T *G = U + NB;                 // [3][NB]: g, then F
  T *Vn = G + 3 * NB;            // [6][N2]
  T *Tf = Vn + 6 * N2;           // [6][N2]
  T *Rf = Tf + 6 * N2;           // [6][N2]
  T *As = Rf + 6 * N2;           // [3][3]
  T *An = As + 9;                // [6][3]: column `dir` of the neighbour's tensor
  T *cf = An + 18;               // [6][3]
  for (int i = t; i < C::TAB; i += blockDim.x) tM[i] = tab[i];

  const int li = blockIdx.x * CPB + cs;
  const bool ranged = !a.cells && a.ncells > 0;
  const bool active = (a.cells || ranged) ? li < a.ncells : li < p.ncell;
  const int e = a.cells ? (active ? a.cells[li] : 0) : (ranged ? a.cell0 + li : li);
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
  int nbr[6];
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1;
    if (f & 1) nbr[f] = ix[dir] + 1 < p.nc[dir] ? ee + stride[dir] : -1;
    else nbr[f] = ix[dir] > 0 ? ee - stride[dir] : -1;
  }
  const bool tr = a.transpose != 0;
  T detJ = T(1);
#pragma unroll
  for (int j = 0; j < 3; j++) detJ *= p.h[j];

  const int tx = l % N, ty = l / N;
  // ---- own column; neighbour lines: face value and normal derivative ----
  T col[N];
  const T *xe = a.x + (size_t)ee * NB;
#pragma unroll
  for (int z = 0; z < N; z++) {
    col[z] = xe[z * TPC + l];
    U[z * TPC + l] = col[z];
  }
  T line[6][N];
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1;
    const bool on = nbr[f] >= 0 && !a.diag_only;
    const T *xn = a.x + (size_t)(on ? nbr[f] : ee) * NB;
#pragma unroll
    for (int q = 0; q < N; q++) {
      const int off = dir == 0 ? l * N + q : (dir == 1 ? ty * N2 + q * N + tx : q * N2 + l);
      line[f][q] = on ? xn[off] : T(0);
    }
    Vn[f * N2 + l] = line[f][(f & 1) ? 0 : N - 1];
  }
  // per-cell data, spread over the cell's threads
  for (int i = l; i < 9; i += TPC)
    As[i] = Ac[(size_t)ee * 9 + i] * detJ / (p.h[i / 3] * p.h[i % 3]);
  for (int f = l; f < 6; f += TPC) {
    const int dir = f >> 1;
    const T delta_s = Ac[(size_t)ee * 9 + dir * 4];
    const int nb = dir == 0 ? ((f & 1) ? (ix[0] + 1 < p.nc[0] ? ee + 1 : -1)
                                       : (ix[0] > 0 ? ee - 1 : -1))
                   : dir == 1 ? ((f & 1) ? (ix[1] + 1 < p.nc[1] ? ee + stride[1] : -1)
                                         : (ix[1] > 0 ? ee - stride[1] : -1))
                              : ((f & 1) ? (ix[2] + 1 < p.nc[2] ? ee + stride[2] : -1)
                                         : (ix[2] > 0 ? ee - stride[2] : -1));
    T om_s = T(0), om_n = T(0), pen = T(0);
    const T scale = p.pen_fac * detJ / (p.h[dir] * p.h[dir]);
    if (nb >= 0) {
      const T *Ab = Ac + (size_t)nb * 9;
      const T delta_n = Ab[dir * 4];
      if (p.weights == PDG_WEIGHTS_ON) {
        // convectiondiffusiondg.hh:326-338
        const T S = delta_s + delta_n + T(1e-20);
        om_s = qdiv(delta_n, S);
        om_n = qdiv(delta_s, S);
        pen = scale * qdiv(T(2) * delta_s * delta_n, S);
      } else {
        om_s = om_n = T(0.5);
        pen = scale;
      }
      for (int j = 0; j < 3; j++) An[f * 3 + j] = Ab[j * 3 + dir] * detJ / (p.h[j] * p.h[dir]);
    } else {
      for (int j = 0; j < 3; j++) An[f * 3 + j] = T(0);
      if (p.bc[f] == PDG_BC_DIRICHLET) {
        om_s = T(1);
        pen = scale * (p.weights == PDG_WEIGHTS_ON ? delta_s : T(1));
      }
    }
    cf[f * 3] = om_s;
    cf[f * 3 + 1] = om_n;
    cf[f * 3 + 2] = pen;
  }
  __syncthreads();

  // ---- g = Dn u in the three directions ----
  {
    T Dx[N], Dy[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
      Dx[q] = tD[tx * N + q];
      Dy[q] = tD[ty * N + q];
    }
#pragma unroll
    for (int z = 0; z < N; z++) {
      T gx = T(0), gy = T(0), gz = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) {
        gx += Dx[q] * U[z * N2 + ty * N + q];
        gy += Dy[q] * U[z * N2 + q * N + tx];
        gz += tD[z * N + q] * col[q];
      }
      G[z * N2 + l] = gx;
      G[NB + z * N2 + l] = gy;
      G[2 * NB + z * N2 + l] = gz;
    }
  }
  __syncthreads();

  // ---- face nodes: t and the lifted jump ----
  const T c1 = tr ? p.theta : T(-1), c2 = tr ? T(-1) : p.theta;
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    const int o1 = dir == 0 ? 1 : 0, o2 = dir == 2 ? 1 : 2;
    const T sgn = hi ? T(1) : T(-1);
    // own node of this thread on the face, and its value
    const int nd = dir == 0 ? l * N + (hi ? N - 1 : 0)
                            : (dir == 1 ? ty * N2 + (hi ? N - 1 : 0) * N + tx
                                        : (hi ? N - 1 : 0) * N2 + l);
    T fs = T(0);
#pragma unroll
    for (int j = 0; j < 3; j++) fs += As[j * 3 + dir] * G[j * NB + nd];
    T dn = T(0), dt1 = T(0), dt2 = T(0);
    const T *dd = hi ? td0 : td1;
#pragma unroll
    for (int q = 0; q < N; q++) {
      dn += dd[q] * line[f][q];
      dt1 += tD[tx * N + q] * Vn[f * N2 + ty * N + q];
      dt2 += tD[ty * N + q] * Vn[f * N2 + q * N + tx];
    }
    const T fn = An[f * 3 + dir] * dn + An[f * 3 + o1] * dt1 + An[f * 3 + o2] * dt2;
    const T jump = U[nd] - line[f][hi ? 0 : N - 1];
    const T om_s = cf[f * 3];
    Tf[f * N2 + l] = c1 * sgn * (om_s * fs + cf[f * 3 + 1] * fn) + cf[f * 3 + 2] * jump;
    Rf[f * N2 + l] = c2 * sgn * om_s * jump;
  }
  __syncthreads();

  // ---- F = A (g + r), at the thread's own column ----
  {
    const T m0x = tm0[tx], m1x = tm1[tx], m0y = tm0[ty], m1y = tm1[ty];
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int lx = z * N + ty, ly = z * N + tx, i = z * N2 + l;
      T g[3] = {G[i], G[NB + i], G[2 * NB + i]};
      const T r[3] = {m0x * Rf[lx] + m1x * Rf[N2 + lx],
                      m0y * Rf[2 * N2 + ly] + m1y * Rf[3 * N2 + ly],
                      tm0[z] * Rf[4 * N2 + l] + tm1[z] * Rf[5 * N2 + l]};
      T F[3] = {T(0), T(0), T(0)};
      if (!tr) {
#pragma unroll
        for (int j = 0; j < 3; j++) g[j] += r[j];
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
          for (int j = 0; j < 3; j++) F[k] += As[k * 3 + j] * g[j];
      } else {
        // A^T for the trial gradient, A for the test gradient's lift
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
          for (int j = 0; j < 3; j++) F[k] += As[j * 3 + k] * g[j] + As[k * 3 + j] * r[j];
      }
#pragma unroll
      for (int k = 0; k < 3; k++) G[k * NB + i] = F[k];
    }
  }
  __syncthreads();

  // ---- S = sum_i L_i F_i + lifted face terms + c u (into U) ----
  {
    T Lx[N], Ly[N], fz[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
      Lx[q] = tL[tx * N + q];
      Ly[q] = tL[ty * N + q];
      fz[q] = G[2 * NB + q * N2 + l];
    }
    const T m0x = tm0[tx], m1x = tm1[tx], m0y = tm0[ty], m1y = tm1[ty];
    const T cc = p.c ? p.c[ee] * detJ : T(0);
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int lx = z * N + ty, ly = z * N + tx;
      T s = cc * col[z];
#pragma unroll
      for (int q = 0; q < N; q++) {
        s += Lx[q] * G[z * N2 + ty * N + q];
        s += Ly[q] * G[NB + z * N2 + q * N + tx];
        s += tL[z * N + q] * fz[q];
      }
      s += m0x * Tf[lx] + m1x * Tf[N2 + lx];
      s += m0y * Tf[2 * N2 + ly] + m1y * Tf[3 * N2 + ly];
      s += tm0[z] * Tf[4 * N2 + l] + tm1[z] * Tf[5 * N2 + l];
      U[z * N2 + l] = s;
    }
  }
  __syncthreads();
  // ---- the three masses ----
  T *S1 = Vn;   // the face data is free now: 18 N2 >= NB values
#pragma unroll
  for (int z = 0; z < N; z++) {
    T s = T(0);
#pragma unroll
    for (int q = 0; q < N; q++) s += tM[tx * N + q] * U[z * N2 + ty * N + q];
    S1[z * N2 + l] = s;
  }
  __syncthreads();
#pragma unroll
  for (int z = 0; z < N; z++) {
    T s = T(0);
#pragma unroll
    for (int q = 0; q < N; q++) s += tM[ty * N + q] * S1[z * N2 + q * N + tx];
    col[z] = s;
  }
  if (active) {
    T *ye = a.y + (size_t)e * NB;
    const T *ad = a.add ? a.add + (size_t)e * NB : nullptr;
    const bool scale = a.alpha != T(1);
#pragma unroll
    for (int z = 0; z < N; z++) {
      T r = T(0);
#pragma unroll
      for (int q = 0; q < N; q++) r += tM[z * N + q] * col[q];
      if (scale) r *= a.alpha;
      const int idx = z * TPC + l;
      if (a.accumulate) r += ye[idx];
      if (ad) r += ad[idx];
      ye[idx] = r;
    }
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(TCfg<N>::THREADS)
    k_apply_tensor(const OpParams<T> p, const ApplyArgs<T> a, const T *__restrict__ Ac,
                   const T *__restrict__ tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.skip && *a.skip) return;
  tensor_block<T, N>(p, a, Ac, tab, smem_raw);
}

// ---------------------------------------------------------------------------
// FP64 in 64-bit block fixed point (pdg_fixed.cuh), degrees 1 to 3: the same
// nodal form, thread mapping and shared arrays.  Dn, L, m_0, m_1 and M of the
// equidistant nodes are small integers over common denominators (dden, q and
// den, which are in the coefficients); products with the cell's coefficients
// are limb products.  Exponents: own values Ex, values of each neighbour's
// side Ef, gradients Ex + LD, the corrected gradient Eh, fluxes and face terms
// Etot, each from bounds; F and t then have 62 bits.  The sum S = sum L F + m t
// is up to 150 (k = 2) times larger in the bound than what the masses leave of
// it, so it is formed exactly (96 bits) and rounded to 61 bits of the cell's
// actual largest value.
// 41x37x39 Q2 375 -> 100 us, 30x31x32 Q3 about 105 us, 80^3 Q1 about 310 us (at
// the Gauss points 1735, 1895, 5238 us); errors against 64 bits 2.4e-16
// (2.7e-16).  With 57 instead of 59 bits for the gradients and their corrected
// form, and a looser bound of the latter, the error was 6.5e-16.
// Degree 4 keeps the FP64 kernel (57-bit values times the derivative table's
// row sum of 128 exceed 64 bits), as do the transpose, which needs twice the
// products, single cells and cell lists.
// ---------------------------------------------------------------------------
template <int N> struct TTab;
// LD, LM: ceil log2 of the largest row sum of dden Dn and of |q m_0| + |q m_1|
template <> struct TTab<2> { static constexpr int dden = 1, q = 1, LD = 1, LM = 3; };
template <> struct TTab<3> { static constexpr int dden = 1, q = 2, LD = 3, LM = 5; };
template <> struct TTab<4> { static constexpr int dden = 2, q = 54, LD = 6, LM = 11; };
template <int N> __host__ __device__ __forceinline__ constexpr int int_dn(int i) {   // dden Dn
  if constexpr (N == 2) {
    constexpr int m[] = {-1, 1, -1, 1};
    return m[i];
  } else if constexpr (N == 3) {
    constexpr int m[] = {-3, 4, -1, -1, 0, 1, 1, -4, 3};
    return m[i];
  } else {
    constexpr int m[] = {-11, 18, -9, 2, -2, -3, 6, -1, 1, -6, 3, 2, -2, 9, -18, 11};
    return m[i];
  }
}
template <int N> __host__ __device__ __forceinline__ constexpr int int_l(int i) {   // q L
  if constexpr (N == 2) {
    constexpr int m[] = {-3, -3, 3, 3};
    return m[i];
  } else if constexpr (N == 3) {
    constexpr int m[] = {-12, -8, 8, 5, 0, -5, -8, 8, 12};
    return m[i];
  } else {
    constexpr int m[] = {-567, -486, 243, -270, 190, 81,  -162, 91,
                         -91,  162,  -81, -190, 270, -243, 486, 567};
    return m[i];
  }
}
template <int N> __host__ __device__ __forceinline__ constexpr int int_m0(int i) {   // q m_0
  if constexpr (N == 2) {
    constexpr int m[] = {4, -2};
    return m[i];
  } else if constexpr (N == 3) {
    constexpr int m[] = {18, -3, 6};
    return m[i];
  } else {
    constexpr int m[] = {864, -136, 64, -216};
    return m[i];
  }
}

template <int N>
struct TICfg : TCfg<N> {
  using B = TCfg<N>;
  // per cell: the scaled tensor (9), per face {own flux (3), neighbour's flux
  // (3), penalty, lift}, the reaction; exponents of these groups and whether
  // they can be held
  static constexpr int FACE = 8, RECI = 9 + 6 * FACE + 1, NEXP = 27;
  static constexpr int X_FACE = 1, X_C = 25, X_OK = 26;   // places among the exponents
  static constexpr int PER = 4 * B::NB + 18 * B::N2 + RECI;
  // gradients have GB bits of Ex + LD: 59 where the exact sum has them (one
  // factor of a limb product may be that wide)
  static constexpr int GS = TTab<N>::LD > 2 ? TTab<N>::LD - 2 : 0, GB = kFixBits + TTab<N>::LD - GS;
  static constexpr int SHM = N == 2 ? 2 : N == 3 ? 5 : 10;   // mass row sums 3, 20, 864
  static constexpr size_t SMEM_FP = sizeof(double) * (B::TAB + B::CPB * B::PER_CELL);
  static constexpr size_t SMEM_FIX = sizeof(int2) * B::CPB * PER;
  static constexpr size_t SMEM = SMEM_FP > SMEM_FIX ? SMEM_FP : SMEM_FIX;
};

// coefficients of a cell as limbs, formed in FP64; one cell per thread, once
// per coefficient field
template <int N>
__global__ void k_record_tensor(const OpParams<double> p, const double *__restrict__ Ac,
                                int2 *__restrict__ out, int *__restrict__ exps) {
  using C = TICfg<N>;
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.ncell) return;
  int ix[3];
  {
    const unsigned q0 = p.div0.div((unsigned)e), q1 = p.div1.div(q0);
    ix[0] = (int)((unsigned)e - q0 * (unsigned)p.nc[0]);
    ix[1] = (int)(q0 - q1 * (unsigned)p.nc[1]);
    ix[2] = (int)q1;
  }
  const long stride[3] = {1, (long)p.nc[0], (long)p.nc[0] * p.nc[1]};
  const double detJ = p.h[0] * p.h[1] * p.h[2];
  const double den3 = (double)IntTab<N>::den * IntTab<N>::den * IntTab<N>::den;
  const double sg = 1.0 / (TTab<N>::dden * den3 * TTab<N>::q), sp = 1.0 / (den3 * TTab<N>::q);
  const double sr = (double)TTab<N>::dden / TTab<N>::q;
  int2 *o = out + e * C::RECI;
  int *x = exps + e * C::NEXP;
  bool ok = true;
  // group of n values v: limbs to o + at, exponent to x[g]
  const auto group = [&](const double *v, int n, int at, int g) {
    BlockExp b;
    for (int i = 0; i < n; i++) b.add(v[i]);
    const int eb = b.biased();
    // outside 2^+-150 the FP64 evaluation is used (zero groups are fine)
    if (!b.finite() || (b.any && (eb < 1023 - 150 || eb > 1023 + 150))) ok = false;
    for (int i = 0; i < n; i++) o[at + i] = ok ? fix_limbs(v[i], eb) : make_int2(0, 0);
    x[g] = b.exponent();
  };
  const double *A = Ac + e * 9;
  double v[9];
  for (int i = 0; i < 9; i++) v[i] = sg * (A[i] * detJ / (p.h[i / 3] * p.h[i % 3]));
  group(v, 9, 0, 0);
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1;
    const double sgn = (f & 1) ? 1.0 : -1.0;
    const double scale = p.pen_fac * detJ / (p.h[dir] * p.h[dir]);
    const bool nb = (f & 1) ? ix[dir] + 1 < p.nc[dir] : ix[dir] > 0;
    const double *An = A + ((f & 1) ? 9 : -9) * stride[dir];
    const double ds = A[dir * 4];
    double os = 0.0, on = 0.0, pen = 0.0;
    if (nb) {
      if (p.weights == PDG_WEIGHTS_ON) {
        const double dn = An[dir * 4], S = ds + dn + 1e-20;   // convectiondiffusiondg.hh:326-338
        os = dn / S;
        on = ds / S;
        pen = scale * (2.0 * ds * dn / S);
      } else {
        os = on = 0.5;
        pen = scale;
      }
    } else if (p.bc[f] == PDG_BC_DIRICHLET) {
      os = 1.0;
      pen = scale * (p.weights == PDG_WEIGHTS_ON ? ds : 1.0);
    }
    double w[3];
    for (int j = 0; j < 3; j++) {
      const double hh = detJ / (p.h[j] * p.h[dir]);
      v[j] = -sgn * sg * os * (A[j * 3 + dir] * hh);
      w[j] = nb ? -sgn * sg * on * (An[j * 3 + dir] * hh) : 0.0;
    }
    const int at = 9 + C::FACE * f, g = C::X_FACE + 4 * f;
    group(v, 3, at, g);
    group(w, 3, at + 3, g + 1);
    v[0] = sp * pen;
    group(v, 1, at + 6, g + 2);
    v[0] = p.theta * sgn * sr * os;
    group(v, 1, at + 7, g + 3);
  }
  v[0] = p.c ? p.c[e] * detJ / den3 : 0.0;
  group(v, 1, C::RECI - 1, C::X_C);
  x[C::X_OK] = ok;
}

template <int N>
__device__ __noinline__ void tensor_block_fp64(const OpParams<double> &p,
                                               const ApplyArgs<double> &a,
                                               const double *__restrict__ Ac,
                                               const double *__restrict__ tab,
                                               unsigned char *smem_raw) {
  tensor_block<double, N>(p, a, Ac, tab, smem_raw);
}

template <int N>
__global__ void __launch_bounds__(TICfg<N>::THREADS, N == 3 ? 6 : 5)
    k_apply_tensor_i(const __grid_constant__ OpParams<double> p,
                     const __grid_constant__ ApplyArgs<double> a, const int2 *__restrict__ rec,
                     const int *__restrict__ exps, const double *__restrict__ Ac,
                     const double *__restrict__ tab) {
  using C = TICfg<N>;
  using B = TTab<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC, CPB = C::CPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int tM[N2], tD[N2], tL[N2], tm0[N];
  __shared__ int sE[CPB][8];   // exponents of the own and the neighbours' values, bits of S
  if (a.skip && *a.skip) return;
  const int t = threadIdx.x;
  const int cs = t / TPC;
  const int l = t - cs * TPC;
  int2 *U = reinterpret_cast<int2 *>(smem_raw) + cs * C::PER;
  int2 *G = U + NB;                 // [3][NB]: gradient (limbs), then F (halves)
  int2 *Vn = G + 3 * NB;            // [6][N2]
  int2 *Tf = Vn + 6 * N2;           // [6][N2]
  int2 *Rf = Tf + 6 * N2;           // [6][N2]
  int2 *Cf = Rf + 6 * N2;           // the record
#pragma unroll
  for (int i = 0; i < N2; i++)
    if (t == i) {
      tM[i] = int_m<N>(i);
      tD[i] = int_dn<N>(i);
      tL[i] = int_l<N>(i);
      if (i < N) tm0[i] = int_m0<N>(i);
    }
  for (int i = t; i < CPB * 8; i += C::THREADS) (&sE[0][0])[i] = (i & 7) == 7 ? 0 : kFixZero;

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
  const int tx = l % N, ty = l / N;
  double col[N], line[6][N];
  const double *xe = a.x + (size_t)ee * NB;
  const int flip = sign_flip(xe[0]);
#pragma unroll
  for (int z = 0; z < N; z++) col[z] = xe[z * TPC + l];
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1;
    const bool on = (f & 1) ? ix[dir] + 1 < p.nc[dir] : ix[dir] > 0;
    const double *xn = xe + (on ? ((f & 1) ? 1 : -1) * (long)stride[dir] * NB : 0);
#pragma unroll
    for (int q = 0; q < N; q++) {
      const int off = dir == 0 ? l * N + q : (dir == 1 ? ty * N2 + q * N + tx : q * N2 + l);
      line[f][q] = on ? xn[off] : 0.0;
    }
  }
  {
    const int2 *r = rec + (size_t)ee * C::RECI;
    for (int i = l; i < C::RECI; i += TPC) Cf[i] = r[i];
  }
  const int *ex = exps + (size_t)ee * C::NEXP;
  __syncthreads();
  bool bad = ex[C::X_OK] == 0;
  {
    BlockExp own;
#pragma unroll
    for (int z = 0; z < N; z++) own.add(col[z]);
    bad |= !own.finite();
    atomicMax(&sE[cs][0], own.exponent());
#pragma unroll
    for (int f = 0; f < 6; f++) {
      BlockExp b;
#pragma unroll
      for (int q = 0; q < N; q++) b.add(line[f][q]);
      bad |= !b.finite();
      atomicMax(&sE[cs][1 + f], b.exponent());
    }
  }
  __syncthreads();
  // ---- exponents ----
  const int Ex = sE[cs][0], Eg = Ex + B::LD, EA = ex[0];
  int Eh = Eg, Et = 2 * kFixZero;
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int *xf = ex + C::X_FACE + 4 * f;
    const int Ef = sE[cs][1 + f], Ej = max(Ex, Ef) + 1;
    Eh = max(Eh, xf[3] + Ej + B::LM);
    Et = max(Et, max(max(xf[0] + Eg, xf[1] + Ef + B::LD) + 2, xf[2] + Ej) + 2);
  }
  Eh += 1;   // the gradient, the lifts of two faces
  const int Etot = max(max(EA + Eh + 2, Et), ex[C::X_C] + Ex + 4);
  bad |= Etot > 850 || (Etot > kFixZero + 1000 && Etot < -700);
  if (__syncthreads_or(bad && active)) {
    tensor_block_fp64<N>(p, a, Ac, tab, smem_raw);
    return;
  }
  const auto biased = [](int E) { return max(E + 1022, kFixMinBiased); };
  const auto shr = [](long long v, int s) { return v >> min((unsigned)s, 63u); };

  constexpr long long kHalfD = C::GS > 0 ? 1ll << (C::GS > 0 ? C::GS - 1 : 0) : 0;
  // ---- values as 57-bit integers; neighbours' normal derivatives ----
  long long uc[N];
  int2 gn[6];   // limbs of the neighbours' normal derivatives, at Ef + LD
#pragma unroll
  for (int z = 0; z < N; z++) {
    uc[z] = fix_signed(col[z], biased(Ex), flip);
    U[z * N2 + l] = split32(uc[z]);
  }
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int eb = biased(sE[cs][1 + f]);
    long long d = 0;
#pragma unroll
    for (int q = 0; q < N; q++) {
      const long long v = fix_signed(line[f][q], eb, flip);
      d += v * int_dn<N>((f & 1) ? q : N2 - N + q);
      if (q == ((f & 1) ? 0 : N - 1)) Vn[f * N2 + l] = split32(v);
    }
    gn[f] = limbs((d + kHalfD) >> C::GS);
  }
  __syncthreads();

  // ---- g = Dn u in the three directions, rounded to GB bits ----
  int Dx[N], Dy[N];
#pragma unroll
  for (int q = 0; q < N; q++) {
    Dx[q] = tD[tx * N + q];
    Dy[q] = tD[ty * N + q];
  }
#pragma unroll
  for (int z = 0; z < N; z++) {
    SmallSum<false> gx(kHalfD), gy(kHalfD);
    long long gz = kHalfD;
#pragma unroll
    for (int q = 0; q < N; q++) {
      gx.add(U[z * N2 + ty * N + q], Dx[q]);
      gy.add(U[z * N2 + q * N + tx], Dy[q]);
      gz += uc[q] * int_dn<N>(z * N + q);
    }
    G[z * N2 + l] = limbs(gx.template shifted<C::GS>());
    G[NB + z * N2 + l] = limbs(gy.template shifted<C::GS>());
    G[2 * NB + z * N2 + l] = limbs(gz >> C::GS);
  }
  __syncthreads();

  // ---- face nodes: t (62 bits of Etot) and the lifted jump (units of 2^(Eh - 61)) ----
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    const int o1 = dir == 0 ? 1 : 0, o2 = dir == 2 ? 1 : 2;
    const int *xf = ex + C::X_FACE + 4 * f;
    const int2 *cf = Cf + 9 + C::FACE * f;
    const int Ef = sE[cs][1 + f], Ej = max(Ex, Ef) + 1;
    const int nd = dir == 0 ? l * N + (hi ? N - 1 : 0)
                            : (dir == 1 ? ty * N2 + (hi ? N - 1 : 0) * N + tx
                                        : (hi ? N - 1 : 0) * N2 + l);
    long long hh = 0, mid = 0;
#pragma unroll
    for (int j = 0; j < 3; j++) mac2(hh, mid, cf[j], G[j * NB + nd]);
    long long s = mac2_round(hh, mid, Etot - xf[0] - Eg + C::GB - 60);
    SmallSum<false> d1(kHalfD), d2(kHalfD);
#pragma unroll
    for (int q = 0; q < N; q++) {
      d1.add(Vn[f * N2 + ty * N + q], Dx[q]);
      d2.add(Vn[f * N2 + q * N + tx], Dy[q]);
    }
    hh = mid = 0;
    mac2(hh, mid, cf[3 + dir], gn[f]);
    mac2(hh, mid, cf[3 + o1], limbs(d1.template shifted<C::GS>()));
    mac2(hh, mid, cf[3 + o2], limbs(d2.template shifted<C::GS>()));
    s += mac2_round(hh, mid, Etot - xf[1] - Ef - B::LD + C::GB - 60);
    const int2 jump =
        limbs(shr(join32(U[nd]) * 4, Ej - Ex) - shr(join32(Vn[f * N2 + l]) * 4, Ej - Ef));   // 59 bits
    hh = mid = 0;
    mac2(hh, mid, cf[6], jump);
    s += mac2_round(hh, mid, Etot - xf[2] - Ej - 1);
    Tf[f * N2 + l] = split32(s);
    hh = mid = 0;
    mac2(hh, mid, cf[7], jump);
    Rf[f * N2 + l] = split32(mac2_round(hh, mid, Eh - xf[3] - Ej));
  }
  __syncthreads();

  // ---- F = A (g + r), at the thread's own column ----
  const int m0x = tm0[tx], m1x = tm0[N - 1 - tx], m0y = tm0[ty], m1y = tm0[N - 1 - ty];
  const int shf = Etot - EA - Eh - 1;
#pragma unroll
  for (int z = 0; z < N; z++) {
    const int lx = z * N + ty, ly = z * N + tx, i = z * N2 + l;
    int2 h[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int2 g = G[j * NB + i];
      // 61 bits, rounded to the 59 that one factor of a limb product may have
      SmallSum<false> s(shr(((long long)g.x * (1ll << 29) + g.y) * (1 << (61 - C::GB)), Eh - Eg) + 2);
      if (j == 0) {
        s.add(Rf[lx], m0x);
        s.add(Rf[N2 + lx], m1x);
      } else if (j == 1) {
        s.add(Rf[2 * N2 + ly], m0y);
        s.add(Rf[3 * N2 + ly], m1y);
      } else {
        s.add(Rf[4 * N2 + l], int_m0<N>(z));
        s.add(Rf[5 * N2 + l], int_m0<N>(N - 1 - z));
      }
      h[j] = limbs(s.total() >> 2);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      long long hh = 0, mid = 0;
#pragma unroll
      for (int j = 0; j < 3; j++) mac2(hh, mid, Cf[k * 3 + j], h[j]);
      G[k * NB + i] = split32(mac2_round(hh, mid, shf));
    }
  }
  __syncthreads();

  // ---- S = sum_i L_i F_i + lifted face terms + c u, exact ----
  long long sl[N], sh[N];   // S = sh 2^32 + sl, 0 <= sl < 2^32
  {
    int Lx[N], Ly[N];
    int2 fz[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
      Lx[q] = tL[tx * N + q];
      Ly[q] = tL[ty * N + q];
      fz[q] = G[2 * NB + q * N2 + l];
    }
    const int2 cc = Cf[C::RECI - 1];
    int bits = 0;
#pragma unroll
    for (int z = 0; z < N; z++) {
      const int lx = z * N + ty, ly = z * N + tx;
      SmallSum<true> s(0);
#pragma unroll
      for (int q = 0; q < N; q++) {
        s.add(G[z * N2 + ty * N + q], Lx[q]);
        s.add(G[NB + z * N2 + q * N + tx], Ly[q]);
        s.add(fz[q], int_l<N>(z * N + q));
      }
      s.add(Tf[lx], m0x);
      s.add(Tf[N2 + lx], m1x);
      s.add(Tf[2 * N2 + ly], m0y);
      s.add(Tf[3 * N2 + ly], m1y);
      s.add(Tf[4 * N2 + l], int_m0<N>(z));
      s.add(Tf[5 * N2 + l], int_m0<N>(N - 1 - z));
      if (p.c) {
        long long hh = 0, mid = 0;
        mac2(hh, mid, cc, limbs(uc[z]));
        s.lo += mac2_round(hh, mid, Etot - ex[C::X_C] - Ex - 3);
      }
      sh[z] = s.hi + (s.lo >> 32);
      sl[z] = (long long)(unsigned)s.lo;
      const long long m = sh[z] ^ (sh[z] >> 63);
      const unsigned lo = (unsigned)sl[z] ^ (unsigned)(sh[z] >> 63);
      bits = max(bits, m ? 96 - __clzll(m) : 32 - __clz(lo));
    }
    atomicMax(&sE[cs][7], bits);
  }
  __syncthreads();
  // 61 bits of the largest
  const int sn = sE[cs][7] - 61;
#pragma unroll
  for (int z = 0; z < N; z++) {
    long long v;
    if (sn > 0) v = (sh[z] << (32 - sn)) + (((sl[z] >> (sn - 1)) + 1) >> 1);
    else v = (long long)((((unsigned long long)sh[z] << 32) + (unsigned long long)sl[z]) << min(-sn, 63));
    U[z * N2 + l] = split32(v);
  }
  __syncthreads();
  // ---- the three masses ----
  constexpr long long kHalfM = 1ll << (C::SHM - 1);
  int2 *S1 = Vn;   // the face data is free now: 18 N2 >= NB values
  int Mx[N], My[N];
#pragma unroll
  for (int q = 0; q < N; q++) {
    Mx[q] = tM[tx * N + q];
    My[q] = tM[ty * N + q];
  }
#pragma unroll
  for (int z = 0; z < N; z++) {
    SmallSum<true> s(kHalfM);
#pragma unroll
    for (int q = 0; q < N; q++) s.add(U[z * N2 + ty * N + q], Mx[q]);
    S1[z * N2 + l] = split32(s.template shifted<C::SHM>());
  }
  __syncthreads();
  int2 w[N];
#pragma unroll
  for (int z = 0; z < N; z++) {
    SmallSum<true> s(kHalfM);
#pragma unroll
    for (int q = 0; q < N; q++) s.add(S1[z * N2 + q * N + tx], My[q]);
    w[z] = split32(s.template shifted<C::SHM>());
  }
  if (!active) return;
  double *ye = a.y + (size_t)e * NB;
  const double *ad = a.add ? a.add + (size_t)e * NB : nullptr;
  const int E = Etot - 62 + sn + 3 * C::SHM;
#pragma unroll
  for (int z = 0; z < N; z++) {
    SmallSum<true> s(kHalfM);
#pragma unroll
    for (int q = 0; q < N; q++) s.add(w[q], int_m<N>(z * N + q));
    double r = fix_to_double(s.template shifted<C::SHM>(), E, flip);
    const int idx = z * TPC + l;
    if (a.alpha != 1.0) r *= a.alpha;
    if (a.accumulate) r += ye[idx];
    if (ad) r += ad[idx];
    ye[idx] = r;
  }
}

template <int N>
static int record_tensor_n(pdg_context *ctx) {
  using C = TICfg<N>;
  if (!ctx->rect) PDG_CUDA_TRY(cudaMalloc(&ctx->rect, sizeof(int2) * C::RECI * ctx->ncell));
  if (!ctx->rect_exp) PDG_CUDA_TRY(cudaMalloc(&ctx->rect_exp, sizeof(int) * C::NEXP * ctx->ncell));
  const OpParams<double> p = make_params<double>(ctx, ctx->K64, ctx->c64, ctx->tab64);
  k_record_tensor<N><<<(unsigned)((ctx->ncell + 127) / 128), 128, 0, ctx->stream>>>(
      p, ctx->Ac64, ctx->rect, ctx->rect_exp);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

// whether the tensor operator has a fixed-point form, and its coefficients,
// built once per coefficient field
bool tensor_i_usable(const pdg_context *ctx) {
  return apply_i_usable(ctx) && ctx->gen_A == 1 && !ctx->cq64 && ctx->N <= 4;
}
int prepare_apply_tensor(pdg_context *ctx) {
  if (ctx->rect_valid) return PDG_OK;
  PDG_TRY(ctx->N == 2 ? record_tensor_n<2>(ctx)
                      : ctx->N == 3 ? record_tensor_n<3>(ctx) : record_tensor_n<4>(ctx));
  mark_built(ctx, &ctx->rect_valid);
  return PDG_OK;
}

template <int N>
static int launch_tensor_i(pdg_context *ctx, const ApplyArgs<double> &a,
                           const OpParams<double> &p) {
  using C = TICfg<N>;
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    PDG_CUDA_TRY(cudaFuncSetAttribute(
        k_apply_tensor_i<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    attr_dev = ctx->device;
  }
  PDG_TRY(prepare_apply_tensor(ctx));
  const long work = a.ncells > 0 ? a.ncells : ctx->ncell;
  const unsigned blocks = (unsigned)((work + C::CPB - 1) / C::CPB);
  k_apply_tensor_i<N><<<blocks, C::THREADS, C::SMEM, ctx->stream>>>(p, a, ctx->rect, ctx->rect_exp,
                                                                   ctx->Ac64, ctx->tabt64);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

template <typename T, int N>
static int launch_tensor_n(pdg_context *ctx, const ApplyArgs<T> &a, const OpParams<T> &p) {
  using C = TCfg<N>;
  const size_t smem = sizeof(T) * (C::TAB + C::CPB * C::PER_CELL);
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    PDG_CUDA_TRY(cudaFuncSetAttribute(k_apply_tensor<T, N>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_dev = ctx->device;
  }
  const long work = (a.cells || a.ncells > 0) ? a.ncells : ctx->ncell;
  if (work <= 0) return PDG_OK;
  const unsigned blocks = (unsigned)((work + C::CPB - 1) / C::CPB);
  const bool dbl = std::is_same<T, double>::value;
  k_apply_tensor<T, N><<<blocks, C::THREADS, smem, ctx->stream>>>(
      p, a, dbl ? (const T *)ctx->Ac64 : (const T *)ctx->Ac32,
      dbl ? (const T *)ctx->tabt64 : (const T *)ctx->tabt32);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

template <typename T>
int launch_apply_tensor(pdg_context *ctx, const ApplyArgs<T> &a, const OpParams<T> &p) {
  if constexpr (std::is_same<T, double>::value) {
    if (tensor_i_usable(ctx) && !a.cells && !a.diag_only && !a.transpose) {
      if (ctx->N == 2) return launch_tensor_i<2>(ctx, a, p);
      if (ctx->N == 3) return launch_tensor_i<3>(ctx, a, p);
      return launch_tensor_i<4>(ctx, a, p);
    }
  }
  switch (ctx->N) {
    case 2: return launch_tensor_n<T, 2>(ctx, a, p);
    case 3: return launch_tensor_n<T, 3>(ctx, a, p);
    case 4: return launch_tensor_n<T, 4>(ctx, a, p);
    case 5: return launch_tensor_n<T, 5>(ctx, a, p);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}
template int launch_apply_tensor<double>(pdg_context *, const ApplyArgs<double> &,
                                         const OpParams<double> &);
template int launch_apply_tensor<float>(pdg_context *, const ApplyArgs<float> &,
                                        const OpParams<float> &);

}  // namespace pdg
