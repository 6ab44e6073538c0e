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
// 2D).  The FP64 kernel is bound by its FP64 pipe, so the time follows the
// count: 41x37x39 Q2 takes 380 us, at the Gauss points 1735 us; FP32 at 15 to
// 26 thousand cells of degree 1 to 4 16 to 18 us against 26 to 38 us.  Errors
// against 64 bits stay at the level of the rounding (3.6e-16 against 2.7e-16).
//
// Thread mapping: N*N threads per cell, thread (tx, ty) owns the z-column;
// face steps: one face node per thread.
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

template <typename T, int N>
__global__ void __launch_bounds__(TCfg<N>::THREADS)
    k_apply_tensor(const OpParams<T> p, const ApplyArgs<T> a, const T *__restrict__ Ac,
                   const T *__restrict__ tab) {
  using C = TCfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, TPC = C::TPC, CPB = C::CPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *tM = reinterpret_cast<T *>(smem_raw);
  T *tD = tM + N2, *tL = tD + N2, *tm0 = tL + N2, *tm1 = tm0 + N, *td0 = tm1 + N,
    *td1 = td0 + N;
  if (a.skip && *a.skip) return;
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
