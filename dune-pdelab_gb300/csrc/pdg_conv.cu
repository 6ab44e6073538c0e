// pdg_conv.cu -- the convection part of ConvectionDiffusionDG:
//   volume   -int u b.grad(psi)                    (convectiondiffusiondg.hh:175-186)
//   faces    upwind flux (b.n >= 0 ? u_s : u_n) b.n psi, once per face with
//            r_s += term1 psi_s, r_n -= term1 psi_n  (:424-443)
//   Dirichlet faces (apply): (b.n >= 0 ? u : 0) b.n psi  (:842-849)
//   outflow faces: u b.n psi                      (:799-820)
// evaluated at the reference's Gauss points (order 2k), 3D.
//
// b is the velocity field b(x) = sum_m c_m sin(2 pi k_m.x + phase_m).  Since
// b does not change during a solve, a set-up kernel stores per cell the
// weighted velocity at every volume point, G_dir(q) = b_dir(x_q) w_q |J| / h_dir,
// and at every point of the six faces, F_f(p) = (b(x_p).n_f) w_p |F|, in FP64
// (and a FP32 copy), so the apply evaluates no trigonometric function.
//
// Apply (N*N threads per cell, z-columns, shared-memory line exchange):
//   volume: u_q = (B (x) B (x) B) u, then
//           y -= (Bt (x) Bt (x) Dt)(G_x u_q) + (Bt (x) Dt (x) Bt)(G_y u_q) + (Dt (x) Bt (x) Bt)(G_z u_q)
//   faces:  traces at face points by direct tensor evaluation of the face
//           node layer, upwind flux per point, tested with the face basis.
// Transposed apply (adjoint): volume -int psi b.grad(u); faces contribute to
// the upwind side only: y_e += int phi (b.n_e) (u_e - u_n) where b.n_e >= 0.
// diag_only (block-Jacobi blocks): neighbour traces are dropped.
#include <cmath>

#include "pdg_conv.cuh"
#include "pdg_ops.cuh"
#include "pdg_vec.cuh"

namespace pdg {

__device__ __forceinline__ void conv_velocity(const Velocity &vel, const double *xg, double *b) {
  b[0] = b[1] = b[2] = 0.0;
  for (int m = 0; m < vel.nmodes; m++) {
    double arg = vel.m[m][3];
    for (int j = 0; j < 3; j++) arg += 2.0 * M_PI * vel.m[m][j] * xg[j];
    const double s = sin(arg);
    for (int j = 0; j < 3; j++) b[j] += vel.m[m][4 + j] * s;
  }
}

// Per-cell velocity record: [3][N^3] volume weights then [6][N^2] face fluxes.
// Flags *bad if an outflow boundary point has inflow (b.n < -1e-30).
template <int N>
__global__ void k_conv_setup(const OpParams<double> p, const Velocity vel, const RhsTables tb,
                             double *__restrict__ rec64, float *__restrict__ rec32,
                             int *__restrict__ bad) {
  using C = CCfg<N>;
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.ncell) return;
  int ix[3];
  {
    long r = e;
    ix[0] = (int)(r % p.nc[0]); r /= p.nc[0];
    ix[1] = (int)(r % p.nc[1]); r /= p.nc[1];
    ix[2] = (int)r;
  }
  const double detJ = p.h[0] * p.h[1] * p.h[2];
  double *r64 = rec64 + e * (C::VREC + C::FREC);
  float *r32 = rec32 + e * (C::VREC + C::FREC);
  for (int q = 0; q < C::NB; q++) {
    const int qa[3] = {q % N, (q / N) % N, q / (N * N)};
    double xg[3], b[3];
    for (int j = 0; j < 3; j++) xg[j] = (ix[j] + tb.x[qa[j]]) * p.h[j];
    conv_velocity(vel, xg, b);
    const double w = tb.w[qa[0]] * tb.w[qa[1]] * tb.w[qa[2]] * detJ;
    for (int d = 0; d < 3; d++) {
      const double g = b[d] * w / p.h[d];
      r64[d * C::NB + q] = g;
      r32[d * C::NB + q] = (float)g;
    }
  }
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    const double area = detJ / p.h[dir];
    const double sgn = hi ? 1.0 : -1.0;
    const bool bnd = hi ? ix[dir] == p.nc[dir] - 1 : ix[dir] == 0;
    for (int q = 0; q < C::N2; q++) {
      const int qt[2] = {q % N, q / N};
      double xg[3], b[3], w = area;
      int t = 0;
      for (int j = 0; j < 3; j++) {
        if (j == dir) { xg[j] = (ix[j] + (hi ? 1.0 : 0.0)) * p.h[j]; continue; }
        xg[j] = (ix[j] + tb.x[qt[t]]) * p.h[j];
        w *= tb.w[qt[t]];
        t++;
      }
      conv_velocity(vel, xg, b);
      const double bn = sgn * b[dir];
      if (bnd && p.bc[f] == PDG_BC_OUTFLOW && bn < -1e-30) atomicExch(bad, 1);
      r64[C::VREC + f * C::N2 + q] = bn * w;
      r32[C::VREC + f * C::N2 + q] = (float)(bn * w);
    }
  }
}

// The same record from velocity point data (pdg_set_velocity_points): b at
// the volume points [ncell][N^3][3] and at the face-lattice points
// [faces][N^2][3], one value per face point for both sides (the reference
// upwinds with b of the inside cell and assumes an H(div) field,
// convectiondiffusiondg.hh:425-426).
template <int N>
__global__ void k_conv_setup_points(const OpParams<double> p, const RhsTables tb,
                                    const double *__restrict__ bqv, const double *__restrict__ bqf,
                                    double *__restrict__ rec64, float *__restrict__ rec32,
                                    int *__restrict__ bad) {
  using C = CCfg<N>;
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.ncell) return;
  int ix[3];
  {
    long r = e;
    ix[0] = (int)(r % p.nc[0]); r /= p.nc[0];
    ix[1] = (int)(r % p.nc[1]); r /= p.nc[1];
    ix[2] = (int)r;
  }
  const double detJ = p.h[0] * p.h[1] * p.h[2];
  double *r64 = rec64 + e * (C::VREC + C::FREC);
  float *r32 = rec32 + e * (C::VREC + C::FREC);
  for (int q = 0; q < C::NB; q++) {
    const int qa[3] = {q % N, (q / N) % N, q / (N * N)};
    const double w = tb.w[qa[0]] * tb.w[qa[1]] * tb.w[qa[2]] * detJ;
    for (int d = 0; d < 3; d++) {
      const double g = bqv[(e * C::NB + q) * 3 + d] * w / p.h[d];
      r64[d * C::NB + q] = g;
      r32[d * C::NB + q] = (float)g;
    }
  }
  for (int f = 0; f < 6; f++) {
    const int dir = f >> 1, hi = f & 1;
    const double area = detJ / p.h[dir];
    const double sgn = hi ? 1.0 : -1.0;
    const bool bnd = hi ? ix[dir] == p.nc[dir] - 1 : ix[dir] == 0;
    const long fi = face_lattice_index(p.nc, 3, dir, ix[dir] + hi, ix);
    for (int q = 0; q < C::N2; q++) {
      const int qt[2] = {q % N, q / N};
      const double w = area * tb.w[qt[0]] * tb.w[qt[1]];
      const double bn = sgn * bqf[(fi * C::N2 + q) * 3 + dir];
      if (bnd && p.bc[f] == PDG_BC_OUTFLOW && bn < -1e-30) atomicExch(bad, 1);
      r64[C::VREC + f * C::N2 + q] = bn * w;
      r32[C::VREC + f * C::N2 + q] = (float)(bn * w);
    }
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(CCfg<N>::THREADS)
    k_conv(const OpParams<T> p, const ApplyArgs<T> a, const T *__restrict__ vrec,
           const T *__restrict__ tabBD) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  conv_block<T, N>(p, a, vrec, tabBD, smem_raw);
}

// ---------------------------------------------------------------------------
template <int N>
static int conv_setup_n(pdg_context *ctx) {
  using C = CCfg<N>;
  const size_t per = (size_t)(C::VREC + C::FREC);
  if (!ctx->conv64) PDG_CUDA_TRY(cudaMalloc(&ctx->conv64, sizeof(double) * per * ctx->ncell));
  if (!ctx->conv32) PDG_CUDA_TRY(cudaMalloc(&ctx->conv32, sizeof(float) * per * ctx->ncell));
  RhsTables tb = make_rhs_tables(ctx);
  double h[2 * N * N];
  // B[q][a] = phi_a(x_q), D[q][a] = phi_a'(x_q)
  for (int q = 0; q < N; q++)
    for (int aa = 0; aa < N; aa++) {
      h[q * N + aa] = tb.B[q * N + aa];
      h[N * N + q * N + aa] = lagrange_derivative(ctx, aa, tb.x[q]);
    }
  if (!ctx->convtab64) {
    float h32[2 * N * N];
    for (int i = 0; i < 2 * N * N; i++) h32[i] = (float)h[i];
    PDG_CUDA_TRY(cudaMalloc(&ctx->convtab64, sizeof(h)));
    PDG_CUDA_TRY(cudaMalloc(&ctx->convtab32, sizeof(h32)));
    PDG_CUDA_TRY(cudaMemcpy(ctx->convtab64, h, sizeof(h), cudaMemcpyHostToDevice));
    PDG_CUDA_TRY(cudaMemcpy(ctx->convtab32, h32, sizeof(h32), cudaMemcpyHostToDevice));
  }
  int *bad = nullptr;
  PDG_CUDA_TRY(cudaMalloc(&bad, sizeof(int)));
  PDG_CUDA_TRY(cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
  OpParams<double> p = make_params<double>(ctx, ctx->K64, ctx->c64, ctx->tab64);
  if (ctx->vel_points)
    k_conv_setup_points<N><<<(unsigned)((ctx->ncell + 127) / 128), 128, 0, ctx->stream>>>(
        p, tb, ctx->bqv64, ctx->bqf64, ctx->conv64, ctx->conv32, bad);
  else
    k_conv_setup<N><<<(unsigned)((ctx->ncell + 127) / 128), 128, 0, ctx->stream>>>(
        p, ctx->vel, tb, ctx->conv64, ctx->conv32, bad);
  PDG_CUDA_TRY(cudaGetLastError());
  int hbad = 0;
  PDG_CUDA_TRY(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  PDG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  cudaFree(bad);
  if (hbad) return set_error(PDG_EOUTFLOW, "outflow boundary condition on inflow");
  return conv_setup_i(ctx, h);
}

int conv_setup(pdg_context *ctx) {
  if (ctx->dim != 3) return set_error(PDG_EUNSUPPORTED, "convection is implemented for 3D grids");
  switch (ctx->N) {
    case 2: return conv_setup_n<2>(ctx);
    case 3: return conv_setup_n<3>(ctx);
    case 4: return conv_setup_n<4>(ctx);
    case 5: return conv_setup_n<5>(ctx);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}

template <typename T, int N>
static int conv_launch_n(pdg_context *ctx, const ApplyArgs<T> &a) {
  using C = CCfg<N>;
  const size_t smem = sizeof(T) * (C::TAB + C::CPB * C::template per_cell<T>());
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    PDG_CUDA_TRY(cudaFuncSetAttribute(k_conv<T, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    attr_dev = ctx->device;
  }
  const bool dbl = std::is_same<T, double>::value;
  OpParams<T> p = make_params<T>(ctx, dbl ? (const T *)ctx->K64 : (const T *)ctx->K32, nullptr,
                                 dbl ? (const T *)ctx->tab64 : (const T *)ctx->tab32);
  const T *rec = dbl ? (const T *)ctx->conv64 : (const T *)ctx->conv32;
  const T *tab = dbl ? (const T *)ctx->convtab64 : (const T *)ctx->convtab32;
  const long work = (a.cells || a.ncells > 0) ? a.ncells : ctx->ncell;
  if (work <= 0) return PDG_OK;
  const unsigned blocks = (unsigned)((work + C::CPB - 1) / C::CPB);
  k_conv<T, N><<<blocks, C::THREADS, smem, ctx->stream>>>(p, a, rec, tab);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

// y += alpha C x (C^T when a.transpose); a.accumulate / a.add are ignored
// (the diffusion launch before it has already produced y).
template <typename T>
int launch_convection(pdg_context *ctx, const ApplyArgs<T> &a) {
  if constexpr (std::is_same<T, double>::value) {
    // off the FP64 pipe (32^3 Q4: 852 us in FP64); cell lists and the transpose
    // keep the FP64 evaluation
    if (!a.transpose && !a.cells && !ctx->f64_pair) return launch_conv_i(ctx, a);
  }
  switch (ctx->N) {
    case 2: return conv_launch_n<T, 2>(ctx, a);
    case 3: return conv_launch_n<T, 3>(ctx, a);
    case 4: return conv_launch_n<T, 4>(ctx, a);
    case 5: return conv_launch_n<T, 5>(ctx, a);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}
template int launch_convection<double>(pdg_context *, const ApplyArgs<double> &);
template int launch_convection<float>(pdg_context *, const ApplyArgs<float> &);

}  // namespace pdg
