// pdg_cell32.cu -- the FP32 operator and the FP32 fast-diagonalisation block
// Jacobi of the mixed-precision inner solve on 3D grids, degrees 1 and 2: one
// cell per thread.
//
// Same operator as k_apply (pdg_apply.cu; reference: ConvectionDiffusionDG::
// jacobian_apply_volume / _skeleton / _boundary, localoperator/
// convectiondiffusiondg.hh:191-195, 474-481, 892-899) and the same block
// Jacobi as k_fdm_apply (pdg_prec.cu; reference: backend/istl/matrixfree/
// assembledblockjacobipreconditioner.hh:162-233).
//
// A cell of degree 2 has 27 values: one thread holds them in registers and
// does all contractions of its cell without exchanging anything, so the only
// shared-memory traffic is the staged input (read once) and the staged output.
// 27 is odd, so the scalar reads of 32 consecutive cells fall on 32 banks.
// The operator takes per cell 22 coefficients (K/h per direction, the reaction
// term, and {kappa_e, kappa_o, penalty} of each face) instead of the assembled
// 1D matrices A'_dir (57 at degree 2): with the shape matrices as constants
// the self terms of a face share the jump and the normal derivatives with its
// neighbour terms.  64^3 Q2 (7.1M DOF) takes 40 us for the operator and 33 us for
// the block Jacobi with the residual update (plane-per-thread kernels with
// exchanges: 81 and 68 us); the bytes need 12 and 22 us.  What is left is the
// latency of load, compute and store within a block at 16 and 18 warps per SM.
// Runs of 64 cells: 32 and 128 are slower on large or small grids (64^3
// mixed CG 252, 252 and 281 ms, 32^3 gradient 69, 80 and 69 ms).
//
// A thread adds its part of the fused dot products in two-float arithmetic; the
// sums over threads are in 57-bit fixed point and FP64 (reduce_tail_two_float).
#include <algorithm>
#include <cstdint>

#include "pdg_ops.cuh"
#include "pdg_stage.cuh"
#include "pdg_vec.cuh"

namespace pdg {

template <int N>
struct C32Cfg {
  static constexpr int N2 = N * N, NB = N * N * N;
  static constexpr int T = 64;                        // cells of a run
  static constexpr int REC = 22;                      // coefficients per cell
  static constexpr int OWN = (T + 2) * NB, RUN = T * NB;
  // staged runs carry up to 3 floats of 16-byte phase of their source
  static constexpr int OWNP = (OWN + 7) / 4 * 4, RUNP = (RUN + 7) / 4 * 4;
  // the operator: two runs (their own cells, four y and two z neighbour runs;
  // two more z neighbour runs unless the runs are each other's), one block of zeros
  static constexpr int THREADS = 2 * T;
  static constexpr int SMEM = (2 * OWNP + 6 * RUNP + NB + 3) / 4 * 4;
  static constexpr int SMEM_SIDE = SMEM + 2 * RUNP;
  static constexpr int SMEM_FDM = 2 * RUNP + (T * 3 * N2 + 7) / 4 * 4 + (T * 3 * N + 7) / 4 * 4;
};

// 1D matrices by value (kernel parameter space)
template <int N>
struct C32Tab {
  float M[N * N], S[N * N], d0[N], d1[N];
};

// {hp K_dir / h_dir (3), hp_x c h_x, per face {hp kappa_e / h, hp kappa_o / h,
// hp penalty}}, formed in FP64 and rounded; [coefficient][cell]
template <int N>
__global__ void k_record_c32(const OpParams<double> p, float *__restrict__ rec) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.ncell) return;
  int ix[3];
  {
    const unsigned q0 = p.div0.div((unsigned)e);
    const unsigned q1 = p.div1.div(q0);
    ix[0] = (int)((unsigned)e - q0 * (unsigned)p.nc[0]);
    ix[1] = (int)(q0 - q1 * (unsigned)p.nc[1]);
    ix[2] = (int)q1;
  }
  const long stride[3] = {1, (long)p.nc[0], (long)p.nc[0] * p.nc[1]};
  const auto put = [&](int k, double v) { rec[k * p.ncell + e] = (float)v; };
  for (int dir = 0; dir < 3; dir++) {
    double hp = 1.0;
    for (int j = 0; j < 3; j++)
      if (j != dir) hp *= p.h[j];
    put(dir, hp * over_h(p, dir, kdir(p, e, dir)));
    if (dir == 0) put(3, p.c ? hp * p.c[e] * p.h[0] : 0.0);
    for (int hi = 0; hi < 2; hi++) {
      const int f = 2 * dir + hi;
      long nb;
      if (hi) nb = ix[dir] + 1 < p.nc[dir] ? e + stride[dir] : -1;
      else nb = ix[dir] > 0 ? e - stride[dir] : -1;
      double raw[3];
      face_coefficients(p, f, kdir(p, e, dir), nb, raw);
      for (int j = 0; j < 3; j++) put(4 + 3 * f + j, hp * raw[j]);
    }
  }
}

// coefficients of a face in the form of this launch: {a1 kappa_e, a1 kappa_o,
// penalty, a2 kappa_e} with (a1, a2) = (1, -theta), transposed (-theta, 1)
struct Face32 {
  float ke, ko, pen, sy;
  __device__ __forceinline__ Face32(const float *r, float a1, float a2)
      : ke(a1 * r[0]), ko(a1 * r[1]), pen(r[2]), sy(a2 * r[0]) {}
};

// one line along the face normal: res = k S u (+ c M u) + the terms of both
// faces; (vl, dl), (vh, dh): the neighbours' face value and derivative
template <int N>
__device__ __forceinline__ void cell_line(const C32Tab<N> &tb, float k, const float (&u)[N],
                                          const Face32 &lo, float vl, float dl, const Face32 &hi,
                                          float vh, float dh, float (&res)[N]) {
  float dul = 0.f, duh = 0.f;
#pragma unroll
  for (int q = 0; q < N; q++) {
    dul += tb.d0[q] * u[q];
    duh += tb.d1[q] * u[q];
  }
  const float jl = u[0] - vl, jh = u[N - 1] - vh;
  const float s2l = lo.sy * jl, s2h = -hi.sy * jh;
#pragma unroll
  for (int i = 0; i < N; i++) {
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < N; q++) s += tb.S[i * N + q] * u[q];
    res[i] = k * s + tb.d0[i] * s2l + tb.d1[i] * s2h;
  }
  res[0] += lo.ke * dul + lo.ko * dl + lo.pen * jl;
  res[N - 1] += hi.pen * jh - hi.ke * duh - hi.ko * dh;
}

// write-back of a run staged in shared memory: element f(O[i], index), by the
// threads i0, i0 + T, ..  f may load from y, so stores wait for the loads of nine
// elements at a time instead of one (y += J x, 64^3 Q2: 56 -> 33 us, 5x4x3 Q2 13.6 ->
// 6.6 us on the device)
template <int T, class F>
__device__ __forceinline__ void write_run(const float *O, float *y, long g0, int count, int i0,
                                          F f) {
  constexpr int U = 9;
  for (int b = i0; b < count; b += U * T) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (b + u * T < count) v[u] = f(O[b + u * T], g0 + b + u * T);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (b + u * T < count) y[g0 + b + u * T] = v[u];
  }
}
// The same unchanged: O has the 16-byte phase of y + g0 (y aligned), whole
// 16-byte chunks are one bulk store by thread i0 = 0, the ends go one by one.
// The caller has fenced the writes of O for the async proxy before its barrier,
// and calls bulk_store_wait in that thread before the block ends.
template <int T>
__device__ __forceinline__ void bulk_store_run(const float *O, float *y, long g0, int count,
                                               int i0) {
  const int head = min((int)((4 - (g0 & 3)) & 3), count), mid = (count - head) & ~3;
  if (i0 == 0 && mid > 0) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(y + g0 + head),
                 "r"(smem_u32(O + head)), "r"(4u * mid)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  if (i0 < head) y[g0 + i0] = O[i0];
  if (i0 < count - head - mid) y[g0 + head + mid + i0] = O[head + mid + i0];
}
__device__ __forceinline__ bool aligned16(const void *p) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}
__device__ __forceinline__ void bulk_store_wait() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void fence_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// A block computes two runs of 64 cells.  kStack: the runs are one plane of the
// slowest direction apart, each is the other's z neighbour; that stages 8.1
// instead of 10.1 cells per computed pair and leaves room for 16 warps per SM
// instead of 12.  Otherwise the runs lie side by side (planes that do not fill
// runs of 64 cells, single planes).  64^3 Q2: one run per block with its
// coefficients staged as well (10 warps per SM) 47 us, stacked runs with
// coefficients read coalesced into registers 40 us.
template <int N, bool kStack>
__global__ void __launch_bounds__(C32Cfg<N>::THREADS)
    k_apply32_cell(const OpParams<float> p, const ApplyArgs<float> a,
                   const float *__restrict__ rec,
                   const __grid_constant__ C32Tab<N> tb, int *tma_err) {
  using C = C32Cfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, T = C::T;
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(8) unsigned long long bar;
  if (a.skip && *a.skip) return;
  const long ndof = p.ncell * NB;
  const long sx = p.nc[0], sxy = (long)p.nc[0] * p.nc[1];
  // first cells of the two runs, and the cells of each
  const int half = threadIdx.x / T, cs = threadIdx.x % T;
  const long dz = kStack ? sxy : T;
  long e0;
  int count;
  if constexpr (kStack) {
    const unsigned chunks = (unsigned)((sxy + T - 1) / T), pair = blockIdx.x / chunks;
    const long in = (long)(blockIdx.x - pair * chunks) * T;
    e0 = (long)pair * 2 * sxy + in;
    count = 2 * (int)pair + half < p.nc[2] ? (int)min((long)T, sxy - in) : 0;
  } else {
    e0 = (long)blockIdx.x * 2 * T;
    count = (int)max(0l, min((long)T, p.ncell - e0 - half * T));
  }
  const long er = e0 + half * dz;
  const bool active = cs < count;
  const long e = er + cs;
  // coefficients first: coalesced, in flight beside the runs' copies
  float R[C::REC];
#pragma unroll
  for (int k = 0; k < C::REC; k++) R[k] = rec[k * p.ncell + (active ? e : 0)];

  Stager<C::THREADS, float> st(&bar);
  float *Y0 = sm + 2 * C::OWNP;
  const float *O0 = st.run(sm, a.x, (e0 - 1) * NB, ndof, C::OWN);
  const float *O1 = st.run(sm + C::OWNP, a.x, (e0 + dz - 1) * NB, ndof, C::OWN);
  const float *ZL = st.run(Y0 + 4 * C::RUNP, a.x, (e0 - sxy) * NB, ndof, C::RUN);
  const float *ZH = st.run(Y0 + 5 * C::RUNP, a.x, (e0 + dz + sxy) * NB, ndof, C::RUN);
  const float *ZL1 = O0 + NB, *ZH0 = O1 + NB;
  if constexpr (!kStack) {
    ZL1 = st.run(sm + C::SMEM, a.x, (e0 + dz - sxy) * NB, ndof, C::RUN);
    ZH0 = st.run(sm + C::SMEM + C::RUNP, a.x, (e0 + sxy) * NB, ndof, C::RUN);
  }
  const float *YL0 = st.run(Y0, a.x, (e0 - sx) * NB, ndof, C::RUN);
  const float *YH0 = st.run(Y0 + 2 * C::RUNP, a.x, (e0 + sx) * NB, ndof, C::RUN);
  const float *YL1 = st.run(Y0 + C::RUNP, a.x, (e0 + dz - sx) * NB, ndof, C::RUN);
  const float *YH1 = st.run(Y0 + 3 * C::RUNP, a.x, (e0 + dz + sx) * NB, ndof, C::RUN);
  float *zero = Y0 + 6 * C::RUNP;   // stands in for an absent neighbour
  if (threadIdx.x < NB) zero[threadIdx.x] = 0.f;
  int ix[3];
  {
    const unsigned ee = active ? (unsigned)e : 0u;
    const unsigned q0 = p.div0.div(ee);
    const unsigned q1 = p.div1.div(q0);
    ix[0] = (int)(ee - q0 * (unsigned)p.nc[0]);
    ix[1] = (int)(q0 - q1 * (unsigned)p.nc[1]);
    ix[2] = (int)q1;
  }
  const bool cp = !a.diag_only;
  const float *U = (half ? O1 : O0) + (cs + 1) * NB;
  const float *xl = cp && ix[0] > 0 ? U - NB : zero;
  const float *xh = cp && ix[0] + 1 < p.nc[0] ? U + NB : zero;
  const float *yl = cp && ix[1] > 0 ? (half ? YL1 : YL0) + cs * NB : zero;
  const float *yh = cp && ix[1] + 1 < p.nc[1] ? (half ? YH1 : YH0) + cs * NB : zero;
  const float *zl = cp && ix[2] > 0 ? (half ? ZL1 : ZL) + cs * NB : zero;
  const float *zh = cp && ix[2] + 1 < p.nc[2] ? (half ? ZH : ZH0) + cs * NB : zero;
  if (!st.wait()) {
    if (threadIdx.x == 0) raise_timeout(tma_err);
    return;
  }
  const float a1 = a.transpose ? -p.theta : 1.f, a2 = a.transpose ? 1.f : -p.theta;

  float out[N][N][N];   // [z][y][x]
  // ---- z operator, then Mhat_x and Mhat_y ----
  {
    const Face32 lo(R + 16, a1, a2), hi(R + 19, a1, a2);
    const float k = R[2];
#pragma unroll
    for (int y = 0; y < N; y++)
#pragma unroll
      for (int x = 0; x < N; x++) {
        const int o = y * N + x;
        float u[N], r[N], dl = 0.f, dh = 0.f, vl = 0.f, vh = 0.f;
#pragma unroll
        for (int q = 0; q < N; q++) {
          u[q] = U[q * N2 + o];
          const float l = zl[q * N2 + o], h = zh[q * N2 + o];
          dl += tb.d1[q] * l;
          dh += tb.d0[q] * h;
          if (q == N - 1) vl = l;
          if (q == 0) vh = h;
        }
        cell_line<N>(tb, k, u, lo, vl, dl, hi, vh, dh, r);
#pragma unroll
        for (int z = 0; z < N; z++) out[z][y][x] = r[z];
      }
#pragma unroll
    for (int z = 0; z < N; z++) {
      float w[N][N];
#pragma unroll
      for (int y = 0; y < N; y++)
#pragma unroll
        for (int x = 0; x < N; x++) {
          float s = 0.f;
#pragma unroll
          for (int q = 0; q < N; q++) s += tb.M[x * N + q] * out[z][y][q];
          w[y][x] = s;
        }
#pragma unroll
      for (int y = 0; y < N; y++)
#pragma unroll
        for (int x = 0; x < N; x++) {
          float s = 0.f;
#pragma unroll
          for (int q = 0; q < N; q++) s += tb.M[y * N + q] * w[q][x];
          out[z][y][x] = s;
        }
    }
  }
  // ---- plane by plane: P = Mhat_y X + Mhat_x Y, out += Mhat_z P ----
  {
    const Face32 xlo(R + 4, a1, a2), xhi(R + 7, a1, a2), ylo(R + 10, a1, a2), yhi(R + 13, a1, a2);
    const float kx = R[0], ky = R[1], kc = R[3];
    // not unrolled: the instruction cache holds one plane's code
#pragma unroll 1
    for (int z = 0; z < N; z++) {
      float u[N][N], P[N][N];
#pragma unroll
      for (int y = 0; y < N; y++)
#pragma unroll
        for (int x = 0; x < N; x++) u[y][x] = U[z * N2 + y * N + x];
      {
        float X[N][N];
#pragma unroll
        for (int y = 0; y < N; y++) {
          float dl = 0.f, dh = 0.f, vl = 0.f, vh = 0.f;
#pragma unroll
          for (int q = 0; q < N; q++) {
            const float l = xl[z * N2 + y * N + q], h = xh[z * N2 + y * N + q];
            dl += tb.d1[q] * l;
            dh += tb.d0[q] * h;
            if (q == N - 1) vl = l;
            if (q == 0) vh = h;
          }
          cell_line<N>(tb, kx, u[y], xlo, vl, dl, xhi, vh, dh, X[y]);
          if (p.c) {
#pragma unroll
            for (int x = 0; x < N; x++) {
              float s = 0.f;
#pragma unroll
              for (int q = 0; q < N; q++) s += tb.M[x * N + q] * u[y][q];
              X[y][x] += kc * s;
            }
          }
        }
#pragma unroll
        for (int y = 0; y < N; y++)
#pragma unroll
          for (int x = 0; x < N; x++) {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < N; q++) s += tb.M[y * N + q] * X[q][x];
            P[y][x] = s;
          }
      }
      {
        float Y[N][N];   // [x][y]
#pragma unroll
        for (int x = 0; x < N; x++) {
          float c[N], dl = 0.f, dh = 0.f, vl = 0.f, vh = 0.f;
#pragma unroll
          for (int q = 0; q < N; q++) {
            c[q] = u[q][x];
            const float l = yl[z * N2 + q * N + x], h = yh[z * N2 + q * N + x];
            dl += tb.d1[q] * l;
            dh += tb.d0[q] * h;
            if (q == N - 1) vl = l;
            if (q == 0) vh = h;
          }
          cell_line<N>(tb, ky, c, ylo, vl, dl, yhi, vh, dh, Y[x]);
        }
#pragma unroll
        for (int y = 0; y < N; y++)
#pragma unroll
          for (int x = 0; x < N; x++) {
            float s = P[y][x];
#pragma unroll
            for (int q = 0; q < N; q++) s += tb.M[x * N + q] * Y[q][y];
            P[y][x] = s;
          }
      }
#pragma unroll
      for (int zz = 0; zz < N; zz++)
#pragma unroll
        for (int y = 0; y < N; y++)
#pragma unroll
          for (int x = 0; x < N; x++) out[zz][y][x] += tb.M[zz * N + z] * P[y][x];
    }
  }
  // <x, y_out> (fused CG: no accumulation), plane sums added exactly
  TwoFloat part{0.f, 0.f};
  if (a.dot_part && active) {
#pragma unroll
    for (int z = 0; z < N; z++) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < N2; i++) s += U[z * N2 + i] * (a.alpha * out[z][i / N][i % N]);
      part = two_add(part, TwoFloat{s, 0.f});
    }
  }
  __syncthreads();   // the y runs are free
  float *O = Y0 + half * C::RUNP + ((er * NB) & 3);
#pragma unroll
  for (int z = 0; z < N; z++)
#pragma unroll
    for (int i = 0; i < N2; i++) O[cs * NB + z * N2 + i] = out[z][i / N][i % N];
  const bool plain = !a.accumulate && !a.add && a.alpha == 1.f && aligned16(a.y);
  if (plain) fence_async();
  __syncthreads();
  if (plain) {
    bulk_store_run<T>(O, a.y, er * NB, count * NB, cs);
    if (cs == 0) bulk_store_wait();
  } else {
    write_run<T>(O, a.y, er * NB, count * NB, cs, [&](float v, long g) {
      float r = a.alpha * v;
      if (a.accumulate) r += a.y[g];
      if (a.add) r += a.add[g];
      return r;
    });
  }
  if (a.dot_part)
    reduce_tail_two_float<C::THREADS>(a.dot_part, a.dot_max_blocks, a.dot_cnt,
                                      RedCtx{nullptr, a.dot_scal, a.dot_flags}, part,
                                      TwoFloat{0.f, 0.f}, a.dot_fin);
}

// v = scale (Qx (x) Qy (x) Qz) diag(1/(lx+ly+lz)) (Qx (x) Qy (x) Qz)^T d;
// rq (fused CG): first d -= lambda rq, written back, and the fused sums carry
// |d|^2 and <d, v>
template <int N>
__global__ void __launch_bounds__(C32Cfg<N>::T, 9)
    k_fdm32_cell(long ncell, const float *__restrict__ Q, const float *__restrict__ L, float *d,
                 float *v, const int *__restrict__ skip, float scale, double *dot_part,
                 long dot_max_blocks, int *dot_cnt, double *dot_scal, int *dot_flags, int dot_fin,
                 const float *rq, int *tma_err) {
  using C = C32Cfg<N>;
  constexpr int N2 = C::N2, NB = C::NB, T = C::T;
  if (skip && *skip) return;
  extern __shared__ __align__(16) float sm[];
  const long e0 = (long)blockIdx.x * T, ndof = ncell * NB;
  float *Q0 = sm + 2 * C::RUNP, *L0 = Q0 + (T * 3 * N2 + 7) / 4 * 4;
  __shared__ __align__(8) unsigned long long bar;
  Stager<T, float> st(&bar);
  // runs start at multiples of 64: no phase
  st.run(sm, d, e0 * NB, ndof, C::RUN);
  if (rq) st.run(sm + C::RUNP, rq, e0 * NB, ndof, C::RUN);
  st.run(Q0, Q, e0 * 3 * N2, ncell * 3 * N2, T * 3 * N2);
  st.run(L0, L, e0 * 3 * N, ncell * 3 * N, T * 3 * N);
  if (!st.wait()) {
    if (threadIdx.x == 0) raise_timeout(tma_err);
    return;
  }
  const int cs = threadIdx.x;
  const bool active = e0 + cs < ncell;
  float *D = sm + cs * NB, *V = sm + C::RUNP + cs * NB;
  const float *Qc = Q0 + cs * 3 * N2, *Lc = L0 + cs * 3 * N;
  float a[N][N][N];
#pragma unroll
  for (int i = 0; i < NB; i++) a[i / N2][(i / N) % N][i % N] = D[i];
  TwoFloat s0{0.f, 0.f}, s1{0.f, 0.f};
  if (rq) {
    const float lambda = (float)dot_scal[S_ALPHA];
#pragma unroll
    for (int z = 0; z < N; z++) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < N2; i++) {
        const float r = a[z][i / N][i % N] - lambda * V[z * N2 + i];
        a[z][i / N][i % N] = r;
        D[z * N2 + i] = r;
        s += r * r;
      }
      s0 = two_add(s0, TwoFloat{s, 0.f});
    }
  }
  float q[N][N], w[N];
  // forward z, y, x
#pragma unroll
  for (int dir = 2; dir >= 0; dir--) {
#pragma unroll
    for (int i = 0; i < N2; i++) q[i / N][i % N] = Qc[dir * N2 + i];
#pragma unroll
    for (int i = 0; i < N2; i++) {
      const int b = i / N, c = i % N;
#pragma unroll
      for (int j = 0; j < N; j++) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < N; k++)
          s += q[k][j] * (dir == 2 ? a[k][b][c] : dir == 1 ? a[b][k][c] : a[b][c][k]);
        w[j] = s;
      }
#pragma unroll
      for (int j = 0; j < N; j++)
        (dir == 2 ? a[j][b][c] : dir == 1 ? a[b][j][c] : a[b][c][j]) = w[j];
    }
  }
#pragma unroll
  for (int z = 0; z < N; z++)
#pragma unroll
    for (int y = 0; y < N; y++)
#pragma unroll
      for (int x = 0; x < N; x++)
        a[z][y][x] = qdiv(a[z][y][x], Lc[x] + Lc[N + y] + Lc[2 * N + z]);
  // back x, y, z (the x factors are still in q)
#pragma unroll
  for (int dir = 0; dir < 3; dir++) {
    if (dir > 0) {
#pragma unroll
      for (int i = 0; i < N2; i++) q[i / N][i % N] = Qc[dir * N2 + i];
    }
#pragma unroll
    for (int i = 0; i < N2; i++) {
      const int b = i / N, c = i % N;
#pragma unroll
      for (int j = 0; j < N; j++) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < N; k++)
          s += q[j][k] * (dir == 2 ? a[k][b][c] : dir == 1 ? a[b][k][c] : a[b][c][k]);
        w[j] = s;
      }
#pragma unroll
      for (int j = 0; j < N; j++)
        (dir == 2 ? a[j][b][c] : dir == 1 ? a[b][j][c] : a[b][c][j]) = w[j];
    }
  }
#pragma unroll
  for (int z = 0; z < N; z++) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < N2; i++) {
      const float r = scale * a[z][i / N][i % N];
      V[z * N2 + i] = r;
      s += D[z * N2 + i] * r;
    }
    s1 = two_add(s1, TwoFloat{s, 0.f});
  }
  if (!active) s0 = s1 = TwoFloat{0.f, 0.f};
  const bool bulk = aligned16(v) && aligned16(d);
  if (bulk) fence_async();
  __syncthreads();
  const int count = (int)min((long)C::RUN, ndof - e0 * NB);
  if (bulk) {
    if (rq) bulk_store_run<T>(sm, d, e0 * NB, count, cs);
    bulk_store_run<T>(sm + C::RUNP, v, e0 * NB, count, cs);
    if (cs == 0) bulk_store_wait();
  } else {
    const auto same = [](float x, long) { return x; };
    if (rq) write_run<T>(sm, d, e0 * NB, count, cs, same);
    write_run<T>(sm + C::RUNP, v, e0 * NB, count, cs, same);
  }
  if (dot_part)
    reduce_tail_two_float<T>(dot_part, dot_max_blocks, dot_cnt,
                             RedCtx{nullptr, dot_scal, dot_flags}, rq ? s0 : s1,
                             rq ? s1 : TwoFloat{0.f, 0.f}, dot_fin);
}

template <int N>
static int launch_apply32_cell_n(pdg_context *ctx, const ApplyArgs<float> &a,
                                 const OpParams<float> &p) {
  using C = C32Cfg<N>;
  static int attr_dev = -1;
  if (attr_dev != ctx->device) {
    PDG_CUDA_TRY(cudaFuncSetAttribute(k_apply32_cell<N, true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(float) * C::SMEM));
    PDG_CUDA_TRY(cudaFuncSetAttribute(k_apply32_cell<N, false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(float) * C::SMEM_SIDE));
    attr_dev = ctx->device;
  }
  if (!ctx->rec32c_valid) {
    if (!ctx->rec32c) PDG_CUDA_TRY(cudaMalloc(&ctx->rec32c, sizeof(float) * C::REC * ctx->ncell));
    const OpParams<double> pd = make_params<double>(ctx, ctx->K64, ctx->c64, ctx->tab64);
    k_record_c32<N><<<(unsigned)((ctx->ncell + 127) / 128), 128, 0, ctx->stream>>>(pd, ctx->rec32c);
    PDG_CUDA_TRY(cudaGetLastError());
    mark_built(ctx, &ctx->rec32c_valid);
  }
  C32Tab<N> tb;
  for (int i = 0; i < C::N2; i++) {
    tb.M[i] = (float)ctx->tab_host[i];
    tb.S[i] = (float)ctx->tab_host[C::N2 + i];
  }
  for (int i = 0; i < N; i++) {
    tb.d0[i] = (float)ctx->tab_host[2 * C::N2 + i];
    tb.d1[i] = (float)ctx->tab_host[2 * C::N2 + N + i];
  }
  const long plane = ctx->ncell / p.nc[2];
  const long stack = (plane + C::T - 1) / C::T * ((p.nc[2] + 1) / 2);
  const long side = (ctx->ncell + 2 * C::T - 1) / (2 * C::T);
  // stacked runs while they take at most a quarter more blocks
  if (4 * stack <= 5 * side)
    k_apply32_cell<N, true><<<(unsigned)stack, C::THREADS, sizeof(float) * C::SMEM, ctx->stream>>>(
        p, a, ctx->rec32c, tb, ctx->h_wait);
  else
    k_apply32_cell<N, false>
        <<<(unsigned)side, C::THREADS, sizeof(float) * C::SMEM_SIDE, ctx->stream>>>(
            p, a, ctx->rec32c, tb, ctx->h_wait);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

int launch_apply32_cell(pdg_context *ctx, const ApplyArgs<float> &a, const OpParams<float> &p) {
  switch (ctx->N) {
    case 2: return launch_apply32_cell_n<2>(ctx, a, p);
    case 3: return launch_apply32_cell_n<3>(ctx, a, p);
    default: return set_error(PDG_EUNSUPPORTED, "one cell per thread: degrees 1 and 2");
  }
}

template <int N>
static int fdm32_cell_n(pdg_context *ctx, const float *d, float *v, const int *skip, float scale) {
  using C = C32Cfg<N>;
  const size_t smem = sizeof(float) * C::SMEM_FDM;
  const bool fuse = ctx->fuse_fin != 0;
  const unsigned blocks = (unsigned)((ctx->ncell + C::T - 1) / C::T);
  k_fdm32_cell<N><<<blocks, C::T, smem, ctx->stream>>>(
      ctx->ncell, (const float *)ctx->prec[PDG_F32].Q, (const float *)ctx->prec[PDG_F32].L,
      const_cast<float *>(d), v, skip, scale, fuse ? ctx->fuse_part : nullptr,
      ctx->fuse_max_blocks, ctx->fuse_cnt, ctx->red_out, ctx->d_flag, ctx->fuse_fin,
      (fuse && ctx->fuse_fin == FIN_CG_DEF_BETA) ? (const float *)ctx->fuse_q : nullptr,
      ctx->h_wait);
  PDG_CUDA_TRY(cudaGetLastError());
  return PDG_OK;
}

int fdm32_cell(pdg_context *ctx, const float *d, float *v, const int *skip, float scale) {
  return ctx->N == 2 ? fdm32_cell_n<2>(ctx, d, v, skip, scale)
                     : fdm32_cell_n<3>(ctx, d, v, skip, scale);
}

}  // namespace pdg
