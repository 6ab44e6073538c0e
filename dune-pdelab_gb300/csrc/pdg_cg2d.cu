// pdg_cg2d.cu -- a whole FP64 CG solve with the FDM cell-block Jacobi on a
// small 2D grid in one cooperative launch.
//
// Reference: dune-istl's CGSolver over OnTheFlyOperator and
// GridOperatorPreconditioner (backend/istl/matrixfree/backends.hh:116-126),
// the recurrence of cg_device (pdg_abi.cu) with the arithmetic of
// k_apply<double, 2, N> and k_fdm_apply<double, 2, N>.
//
// A 2D grid of a few thousand cells gives a launch microseconds of work: with
// three launches per iteration the 2D Q1 64^2 solve took 24 us per iteration,
// nearly all of it launches and reduction tails.  Here every SM owns a run of
// cells for the whole solve.  Their records, factors and vectors stay in shared
// memory; only the search direction and the preconditioned residual are
// written to global memory, for the neighbours' face terms.  An iteration is
// two grid-wide sums:
//
//   p = z + beta p (own cells; a neighbour's p is formed from its z and its
//   previous p), q = A p                                 -- sum <p, q>
//   x += lambda p, r -= lambda q, z = M^-1 r              -- sums <r, r>, <z, r>
//
// A grid-wide sum is two hops: each block publishes its partial sums in its
// slot; block 0 reads the slots, adds them in block order (the same result in
// every run), forms the scalars of the recurrence and publishes those.  Slots
// are released and acquired, so having read the scalars a block is also ordered
// after everything the other blocks wrote before: it is the barrier as well.
// (With every block reading every slot the polling itself took 4 to 5 us.)
// Waits are bounded.
//
// One DOF per thread: a warp-wide FP64 operation occupies its quarter of the SM
// for 64 cycles (measured, dependent or not), so the FP64 operations of a
// thread, not their number per cell, set the time of the two phases, and the
// threads of a block must cover all four quarters.  With one cell per thread
// the 2D Q1 64^2 iteration took 19.5 us.
#include <algorithm>
#include <mutex>

#include "pdg_ops.cuh"
#include "pdg_tma.cuh"
#include "pdg_vec.cuh"

namespace pdg {

template <int N>
struct CG2Cfg {
  static constexpr int N2 = N * N;
  static constexpr int REC = 2 * N2 + 20;              // k_cell_record<double, 2, N>
  // per cell in shared memory: record, Q, 1/(lx+ly); x, r, p, q, z; two
  // exchange arrays and the face data (s1, s2 of N points of 4 faces)
  static constexpr int PER_CELL = REC + 2 * N2 + N2 + 5 * N2 + 2 * N2 + 8 * N;
  static constexpr int TAB = N2 + 2 * N;
};

constexpr int kCg2Sets = 4;              // slot sets in use in turn
// threads per block: one for each of the 2 x 152 slots block 0 polls, so that
// a hop is one L2 round trip; cells go to the first threads
constexpr int kCg2Threads = 320;
constexpr int kCg2Copies = 8;            // copies of the scalars, 128 bytes apart
constexpr int kCg2Polls = 1 << 21;       // bound of one wait (seconds)
// an empty slot: a NaN no arithmetic produces
constexpr unsigned long long kCg2Empty = 0xffffffffffffffffull;

struct Cg2Args {
  const double *rec, *Q, *Linv;
  double *x, *b;          // solution and defect (both updated)
  double *p[2], *z;       // exchanged vectors
  unsigned long long *slots;   // [kCg2Sets][2][grid] partial sums, all empty,
  unsigned long long *result;  // [kCg2Sets][kCg2Copies][16] scalars, all empty
  double *scal;
  int *flags, *timeout;
  int maxit, cells_per_block;
};

__device__ __forceinline__ unsigned long long ld_slot(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_slot(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void st_slot_release(unsigned long long *p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One value read from / written to a slot; an empty slot is never written
__device__ __forceinline__ bool take_slot(const unsigned long long *s, double *v) {
  unsigned long long x = ld_slot(s);
  for (int it = 0; x == kCg2Empty && it < kCg2Polls; it++) x = ld_slot(s);
  *v = __longlong_as_double(x);
  return x != kCg2Empty;
}
__device__ __forceinline__ void put_slot(unsigned long long *s, double v) {
  const unsigned long long x = __double_as_longlong(v);
  st_slot_release(s, x == kCg2Empty ? 0x7ff8000000000000ull : x);
}

// The exchange of one round: sums v0 (and v1, nv = 2) over the first nw warps of
// all blocks; block 0 turns them into nr scalars with `scalars(s, out)`, called
// by its threads 0, 32, .. 32 (nr - 1) (scalar k by thread 32 k); every thread
// gets them in res[0 .. nr).  false: a block or block 0 did not publish in time.
// red: shared scratch of 64 + 2 * gridDim doubles.
template <class F>
__device__ __forceinline__ bool exchange(const Cg2Args &g, unsigned round, int nv, int nr, int nw,
                                         double v0, double v1, double *red, double *res,
                                         F scalars) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nb = gridDim.x;
  const unsigned set = round % kCg2Sets, old = (set + 2) % kCg2Sets;
  if (w < nw) {
    v0 = warp_sum_fixed(v0, 32);
    if (nv > 1) v1 = warp_sum_fixed(v1, 32);
    if (lane == 0) {
      red[2 * w] = v0;
      red[2 * w + 1] = v1;
    }
  }
  __syncthreads();   // every thread's global writes come before the release below
  if (threadIdx.x < 2) {
    const int k = threadIdx.x;
    // free the own slots of the set after next: block 0 has read them (it
    // published the previous round's scalars after that)
    st_slot(g.slots + (2 * (size_t)old + k) * nb + blockIdx.x, kCg2Empty);
    if (k < nv) {
      double v = red[k];
      for (int i = 1; i < nw; i++) v += red[2 * i + k];
      put_slot(g.slots + (2 * (size_t)set + k) * nb + blockIdx.x, v);
    }
  }
  bool ok = true;
  if (blockIdx.x == 0) {
    double *all = red + 64;
    for (int i = threadIdx.x; i < nv * nb; i += kCg2Threads)
      ok = take_slot(g.slots + 2 * (size_t)set * nb + i, all + i) && ok;
    ok = __syncthreads_and(ok);
    if (w < nv) {
      double a = 0.0;
      for (int i = lane; i < nb; i += 32) a += all[w * nb + i];
      a = warp_sum_fixed(a, 32);
      if (lane == 0) red[60 + w] = a;
    }
    __syncthreads();
    if (lane == 0 && w < nr) res[w] = scalars(w, red[60], red[61]);
    __syncthreads();
    if (threadIdx.x < nr * kCg2Copies) {
      const int k = threadIdx.x % nr, c = threadIdx.x / nr;
      // all blocks have read the scalars of the round before last
      for (int j = k; j < 4; j += nr)
        st_slot(g.result + 16 * ((size_t)old * kCg2Copies + c) + j, kCg2Empty);
      // a failed wait is not published: every block then runs out as well
      if (ok) put_slot(g.result + 16 * ((size_t)set * kCg2Copies + c) + k, res[k]);
    }
  } else if (threadIdx.x < nr) {
    ok = take_slot(g.result + 16 * ((size_t)set * kCg2Copies + blockIdx.x % kCg2Copies) +
                       threadIdx.x,
                   res + threadIdx.x);
  }
  return __syncthreads_and(ok);
}

template <int N>
__global__ void __launch_bounds__(kCg2Threads)
    k_cg2d(const OpParams<double> pr, const Cg2Args g) {
  using C = CG2Cfg<N>;
  constexpr int N2 = C::N2, CPP = kCg2Threads / N2;   // cells per pass
  extern __shared__ __align__(16) double sh[];
  __shared__ double sc[4];
  const int t = threadIdx.x;
  const int c0 = blockIdx.x * g.cells_per_block;
  const int c1 = min((int)pr.ncell, c0 + g.cells_per_block);
  const int nc = max(0, c1 - c0), cap = g.cells_per_block;
  const int nw = (min(cap, CPP) * N2 + 31) / 32;      // warps with DOFs
  // records and factors [cell][entry], vectors [cell][N2]
  double *rec = sh, *Q = rec + C::REC * cap, *Li = Q + 2 * N2 * cap, *X = Li + N2 * cap,
         *R = X + N2 * cap, *P = R + N2 * cap, *W = P + N2 * cap, *Z = W + N2 * cap,
         *T0 = Z + N2 * cap, *T1 = T0 + N2 * cap, *F = T1 + N2 * cap, *tM = F + 8 * N * cap,
         *red = tM + C::TAB;
  const double *td0 = tM + N2, *td1 = td0 + N;
  if (g.flags[F_STATE]) return;   // converged before the first iteration
  for (int i = t; i < nc * C::REC; i += kCg2Threads) rec[i] = g.rec[(size_t)c0 * C::REC + i];
  for (int i = t; i < nc * 2 * N2; i += kCg2Threads) Q[i] = g.Q[(size_t)c0 * 2 * N2 + i];
  for (int i = t; i < nc * N2; i += kCg2Threads) {
    const size_t o = (size_t)c0 * N2 + i;
    Li[i] = g.Linv[o];
    X[i] = g.x[o];
    R[i] = g.b[o];
    P[i] = g.p[0][o];   // the first direction p = M^-1 b
  }
  for (int i = t; i < N2; i += kCg2Threads) tM[i] = pr.tab[i];
  for (int i = t; i < 2 * N; i += kCg2Threads) tM[N2 + i] = pr.tab[2 * N2 + i];
  double rho = g.scal[S_RHO], beta = 0.0, def = g.scal[S_DEF];
  const double stop = g.scal[S_DEF0] * g.scal[S_RED];
  __syncthreads();

  const int cl = t / N2, d = t - cl * N2, y = d / N, x = d - y * N;
  int state = 0, it = 0;
  unsigned round = 0;
  double lambda = 0.0;
  while (it < g.maxit && state == 0) {
    // ---- p = z + beta p, q = A p ----
    const double *pold = g.p[it & 1];
    double *pnew = g.p[(it + 1) & 1];
    const bool first = it == 0;
    double s0 = 0.0, s1 = 0.0;
    for (int b = 0; b < nc; b += CPP) {
      const int c = b + cl;
      const bool on = cl < CPP && c < nc;
      const int e = c0 + c;
      double u = 0.0;
      if (on) {
        // neighbour lines: (s1, s2) of the face points, as in k_apply; one or
        // two of the cell's 4 N lines per thread
        const unsigned iy = pr.div0.div((unsigned)e), ix = (unsigned)e - iy * (unsigned)pr.nc[0];
#pragma unroll
        for (int l0 = 0; l0 < 4 * N; l0 += N2) {
          const int l = l0 + d;
          if (l < 4 * N) {
            const int f = l / N, a = l - f * N, hi = f & 1;
            const bool has = f == 0 ? ix > 0 : f == 1 ? (int)ix + 1 < pr.nc[0]
                                             : f == 2 ? iy > 0 : (int)iy + 1 < pr.nc[1];
            double f1 = 0.0, f2 = 0.0;
            if (has) {
              const int st = f < 2 ? 1 : pr.nc[0];
              const size_t o = (size_t)(hi ? e + st : e - st) * N2 + (f < 2 ? a * N : a);
              const int inc = f < 2 ? 1 : N;
              double v[N];
#pragma unroll
              for (int q = 0; q < N; q++) {
                const double po = __ldcg(pold + o + q * inc);
                v[q] = first ? po : fma(beta, po, __ldcg(g.z + o + q * inc));
              }
              const double *td = hi ? td0 : td1;
              double dv = 0.0;
#pragma unroll
              for (int q = 0; q < N; q++) dv += td[q] * v[q];
              const double val = hi ? v[0] : v[N - 1];
              // {hp ke, hp ko, hp pen, th hp ke, th hp ko} of the face
              const double *k5 = rec + c * C::REC + 2 * N2 + 5 * f;
              const double kd = k5[1] * dv, kv = k5[3] * val;
              f1 = (hi ? -kd : kd) - k5[2] * val;
              f2 = hi ? -kv : kv;
            }
            F[c * 8 * N + l] = f1;
            F[c * 8 * N + 4 * N + l] = f2;
          }
        }
        const int i = c * N2 + d;
        u = first ? P[i] : fma(beta, P[i], Z[i]);
        P[i] = u;
        __stcg(pnew + (size_t)c0 * N2 + i, u);
      }
      __syncthreads();
      if (on) {
        const double *Ax = rec + c * C::REC + x * N, *Ay = rec + c * C::REC + N2 + y * N;
        const double *pc = P + c * N2, *f1 = F + c * 8 * N, *f2 = f1 + 4 * N;
        double sx = 0.0, sy = 0.0;
#pragma unroll
        for (int q = 0; q < N; q++) {
          sx += Ax[q] * pc[y * N + q];
          sy += Ay[q] * pc[q * N + x];
        }
        if (x == 0) sx += f1[y];
        sx += td0[x] * f2[y];
        if (x == N - 1) sx += f1[N + y];
        sx += td1[x] * f2[N + y];
        if (y == 0) sy += f1[2 * N + x];
        sy += td0[y] * f2[2 * N + x];
        if (y == N - 1) sy += f1[3 * N + x];
        sy += td1[y] * f2[3 * N + x];
        T0[c * N2 + d] = sx;
        T1[c * N2 + d] = sy;
      }
      __syncthreads();
      if (on) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < N; q++) {
          s += tM[y * N + q] * T0[c * N2 + q * N + x];
          s += tM[x * N + q] * T1[c * N2 + y * N + q];
        }
        W[c * N2 + d] = s;
        s0 += u * s;
      }
    }
    if (!exchange(g, round++, 1, 1, nw, s0, 0.0, red, sc,
                  [&](int, double a, double) { return rho / a; })) {
      state = -1;
      break;
    }
    lambda = sc[0];
    it++;
    // ---- x += lambda p, r -= lambda q, z = M^-1 r ----
    s0 = s1 = 0.0;
    for (int b = 0; b < nc; b += CPP) {
      const int c = b + cl, i = c * N2 + d;
      const bool on = cl < CPP && c < nc;
      const double *Qx = Q + c * 2 * N2, *Qy = Qx + N2, *t0 = T0 + c * N2, *t1 = T1 + c * N2;
      double r = 0.0;
      if (on) {
        r = R[i] - lambda * W[i];
        R[i] = r;
        X[i] += lambda * P[i];
        s0 += r * r;
      }
      __syncthreads();
      if (on) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < N; k++) s += Qy[k * N + y] * R[c * N2 + k * N + x];
        T0[i] = s;
      }
      __syncthreads();
      if (on) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < N; k++) s += Qx[k * N + x] * t0[y * N + k];
        T1[i] = s * Li[i];
      }
      __syncthreads();
      if (on) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < N; k++) s += Qx[x * N + k] * t1[y * N + k];
        T0[i] = s;
      }
      __syncthreads();
      if (on) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < N; k++) s += Qy[y * N + k] * t0[k * N + x];
        Z[i] = s;
        __stcg(g.z + (size_t)c0 * N2 + i, s);
        s1 += r * s;
      }
    }
    // def = |r|, beta = <z, r> / rho, rho = <z, r>
    if (!exchange(g, round++, 2, 3, nw, s0, s1, red, sc, [&](int k, double a, double c) {
          return k == 0 ? sqrt(a) : k == 1 ? c / rho : c;
        })) {
      state = -1;
      break;
    }
    def = sc[0];
    beta = sc[1];
    rho = sc[2];
    if (!isfinite(def)) state = 2;
    else if (def < stop || def < 1e-30) state = 1;
  }
  for (int i = t; i < nc * N2; i += kCg2Threads) {
    const size_t o = (size_t)c0 * N2 + i;
    g.x[o] = X[i];
    g.b[o] = R[i];
  }
  if (blockIdx.x == 0 && t == 0) {
    g.scal[S_DEF] = def;
    g.scal[S_RHO] = rho;
    g.scal[S_ALPHA] = lambda;
    g.scal[S_BETA] = beta;
    g.scal[S_ITER] = it;
    if (state > 0) g.flags[F_STATE] = state;
  }
  if (state < 0 && t == 0) raise_timeout(g.timeout);
}

__global__ void k_cg2d_slots(unsigned long long *s, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) s[i] = kCg2Empty;
}

template <int N>
static int cg2d_n(pdg_context *ctx, double *x, double *b, double *p, double *p2, double *z,
                  int maxit, bool *ran) {
  using C = CG2Cfg<N>;
  *ran = false;
  // the device's limits, shared by the contexts of all host threads
  struct Limits {
    int dev, sms, coop, smem;
  };
  static std::mutex mutex;
  static Limits known{-1, 0, 0, 0};
  Limits lim;
  {
    const std::lock_guard<std::mutex> lock(mutex);
    if (known.dev != ctx->device) {
      lim.dev = ctx->device;
      PDG_CUDA_TRY(cudaDeviceGetAttribute(&lim.sms, cudaDevAttrMultiProcessorCount, lim.dev));
      PDG_CUDA_TRY(cudaDeviceGetAttribute(&lim.coop, cudaDevAttrCooperativeLaunch, lim.dev));
      PDG_CUDA_TRY(
          cudaDeviceGetAttribute(&lim.smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, lim.dev));
      cudaFuncAttributes fa;
      PDG_CUDA_TRY(cudaFuncGetAttributes(&fa, k_cg2d<N>));
      lim.smem -= (int)fa.sharedSizeBytes;
      PDG_CUDA_TRY(cudaFuncSetAttribute(k_cg2d<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        lim.smem));
      known = lim;
    }
    lim = known;
  }
  const int sms = lim.sms;
  if (!lim.coop || sms < 1) return PDG_OK;
  const int grid = (int)std::min<long>(sms, ctx->ncell);
  const int cap = (int)((ctx->ncell + grid - 1) / grid);
  const size_t smem =
      sizeof(double) * ((size_t)C::PER_CELL * cap + C::TAB + 64 + 2 * (size_t)grid);
  // A grid whose cells do not fit on the SMs keeps the launches.  One that fits is
  // faster here at every size: us per iteration with three launches and in one, Q1
  // 64^2 31 and 11, 128^2 36 and 17, 228^2 53 and 44; Q2 48^2 34 and 12, 166^2 59 and
  // 44; Q3 110^2 53 and 32; Q4 90^2 64 and 40 (log-normal K).
  if (smem > (size_t)lim.smem) return PDG_OK;
  const int npart = kCg2Sets * grid * 2, nslots = npart + kCg2Sets * kCg2Copies * 16;
  if (!ctx->cg2_slots)
    PDG_CUDA_TRY(cudaMalloc(&ctx->cg2_slots,
                            sizeof(double) * kCg2Sets * (sms * 2 + kCg2Copies * 16)));
  k_cg2d_slots<<<(nslots + 255) / 256, 256, 0, ctx->stream>>>(ctx->cg2_slots, nslots);
  PDG_CUDA_TRY(cudaGetLastError());
  OpParams<double> pr = make_params<double>(ctx, ctx->K64, ctx->c64, ctx->tab64);
  const PrecData &pd = ctx->prec[PDG_F64];
  Cg2Args g{ctx->rec64, (const double *)pd.Q, pd.Lsum_inv, x, b, {p, p2}, z, ctx->cg2_slots,
            ctx->cg2_slots + npart, ctx->red_out, ctx->d_flag, ctx->h_wait, maxit, cap};
  void *args[] = {&pr, &g};
  PDG_CUDA_TRY(cudaLaunchCooperativeKernel((void *)k_cg2d<N>, dim3(grid), dim3(kCg2Threads), args, smem,
                                           ctx->stream));
  *ran = true;
  return PDG_OK;
}

// The iterations of a CG solve whose scalars are set up (first defect, rho,
// p = M^-1 b); *ran false: not a grid for this kernel, nothing was launched.
int cg2d_solve(pdg_context *ctx, double *x, double *b, double *p, double *p2, double *z, int maxit,
               bool *ran) {
  switch (ctx->N) {
    case 2: return cg2d_n<2>(ctx, x, b, p, p2, z, maxit, ran);
    case 3: return cg2d_n<3>(ctx, x, b, p, p2, z, maxit, ran);
    case 4: return cg2d_n<4>(ctx, x, b, p, p2, z, maxit, ran);
    case 5: return cg2d_n<5>(ctx, x, b, p, p2, z, maxit, ran);
    default: return set_error(PDG_EUNSUPPORTED, "degree not compiled in");
  }
}

}  // namespace pdg
