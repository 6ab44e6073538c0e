// pdg_vec.cuh -- device-resident Krylov scalars and fused vector kernels.
//
// The Krylov recurrences of dune-istl's CGSolver / BiCGSTABSolver keep a
// handful of scalars (rho, alpha, omega, defect ...).  Here they live in a
// small device array so that one iteration is a fixed sequence of kernel
// launches with no host round trip; the convergence test
// (IterativeSolver::Iteration::step: def < def0 * reduction or def < 1e-30,
// non-finite defects abort) is evaluated on the device and raises a flag
// that every later kernel of the solve checks before doing any work.
//
// Dot products are deterministic: each block writes one partial sum (fixed
// grid-stride order, fixed tree), the last block to finish adds the
// partials in block order and runs the "finisher" for the scalars.
#pragma once

#include "pdg_fixed.cuh"
#include "pdg_internal.cuh"

namespace pdg {

// scalar slots
enum Slot {
  S_DEF0 = 0,     // first defect
  S_DEF = 1,      // current defect (two-norm)
  S_RED = 2,      // requested reduction
  S_RHO = 3,      // CG rholast / BiCGStab rho
  S_RHONEW = 4,   // BiCGStab rho_new
  S_ALPHA = 5,    // CG lambda / BiCGStab alpha
  S_BETA = 6,
  S_OMEGA = 7,
  S_H = 8,        // BiCGStab h = <rt, v>
  S_TR = 9,       // BiCGStab <t, r>
  S_TT = 10,      // BiCGStab <t, t>
  S_ITER = 11,    // iteration count (as double; BiCGStab counts halves)
  S_DOT = 12,     // generic dot result
  S_DOT2 = 13,
  S_SCALE = 14,   // mixed precision: scaling of the inner right-hand side
  S_GUARD = 15,   // relative breakdown threshold (0: dune-istl's absolute tests only)
  S_COUNT = 16
};

// flag words (int): [0] state (0 running, 1 converged, 2 non-finite,
// 3 breakdown), [1] reduction counter (last-block detection), [2] the CG
// x update of the stopping iteration is still to be applied
enum { F_STATE = 0, F_COUNTER = 1, F_XPEND = 2, F_COUNT = 3 };

enum Finisher {
  FIN_STORE = 0,        // scal[slot0] = d0 ; scal[slot1] = d1
  FIN_DEF0 = 1,         // def0 = def = sqrt(d0); iteration 0 check
  FIN_DEF = 2,          // def = sqrt(d0); convergence check at scal[S_ITER]
  FIN_CG_LAMBDA = 3,    // lambda = rholast / d0
  FIN_CG_BETA = 4,      // beta = d0 / rholast; rholast = d0
  FIN_BI_RHONEW = 5,    // rho_new = d0; breakdown checks
  FIN_BI_ALPHA = 6,     // h = d0; alpha = rho_new / h
  FIN_BI_OMEGA = 7,     // omega = d0 / d1
  FIN_NORM = 8,         // scal[slot0] = sqrt(d0)
  FIN_CG_DEF_BETA = 9   // def = sqrt(d0) + convergence check; beta = d1 / rholast;
                        // rholast = d1; a stop marks the iteration's x update pending
};

struct RedCtx {
  double *partials;   // [kRedBlocks * 2]
  double *scal;       // [S_COUNT]
  int *flags;         // [F_COUNT]
};

// FIN_CG_DEF_BETA in two independent parts.  CGSolver: the defect check after
// b -= lambda q, then (when it goes on) rho = <M^{-1} b, b>, beta = rho / rholast
__device__ __forceinline__ void finish_cg_def(const RedCtx &rc, double d0) {
  const double def = sqrt(d0);
  int state = 0;
  if (!isfinite(def)) state = 2;
  else if (def < rc.scal[S_DEF0] * rc.scal[S_RED] || def < 1e-30) state = 1;
  rc.scal[S_DEF] = def;
  if (state) {
    rc.flags[F_STATE] = state;
    rc.flags[F_XPEND] = 1;
  }
}
__device__ __forceinline__ void finish_cg_beta(const RedCtx &rc, double d1) {
  rc.scal[S_BETA] = d1 / rc.scal[S_RHO];
  rc.scal[S_RHO] = d1;
}

// Finisher of a reduction: updates the Krylov scalars (dune-istl's
// CGSolver / BiCGSTABSolver recurrences and breakdown tests) from the two
// reduced sums d0, d1.
__device__ inline void run_finisher(const RedCtx &rc, int fin, int slot0, int slot1, double d0,
                             double d1) {
  double *s = rc.scal;
  int *fl = rc.flags;
  switch (fin) {
    case FIN_STORE:
      if (slot0 >= 0) s[slot0] = d0;
      if (slot1 >= 0) s[slot1] = d1;
      break;
    case FIN_NORM:
      s[slot0] = sqrt(d0);
      break;
    case FIN_DEF0: {
      const double def = sqrt(d0);
      s[S_DEF0] = def;
      s[S_DEF] = def;
      if (!isfinite(def)) fl[F_STATE] = 2;
      else if (def < def * s[S_RED] || def < 1e-30) fl[F_STATE] = 1;
      break;
    }
    case FIN_DEF: {
      const double def = sqrt(d0);
      s[S_DEF] = def;
      if (!isfinite(def)) fl[F_STATE] = 2;
      else if (def < s[S_DEF0] * s[S_RED] || def < 1e-30) fl[F_STATE] = 1;
      if (slot0 == S_RHO) s[S_RHO] = s[S_RHONEW];   // BiCGStab: rho = rho_new
      break;
    }
    case FIN_CG_LAMBDA:
      // once per iteration of a running solve: the iteration count advances here
      s[S_ITER] += 1.0;
      s[S_ALPHA] = s[S_RHO] / d0;
      break;
    case FIN_CG_BETA:
      s[S_BETA] = d0 / s[S_RHO];
      s[S_RHO] = d0;
      break;
    // BiCGSTABSolver breakdown tests are absolute (rho, omega <= 1e-80,
    // |h| < 1e-80).  With S_GUARD > 0 (FP32 inner solves, whose dot products
    // carry ~1e-7 relative noise) a relative test is added:
    // |<rt, r>| or |<rt, v>| below S_GUARD |rt| |r| (|rt| |v|) is treated as a
    // breakdown, and the solve stops with the last finite iterate.
    case FIN_BI_RHONEW:
      s[S_RHONEW] = d0;
      if (fabs(s[S_RHO]) <= 1e-80 || fabs(s[S_OMEGA]) <= 1e-80 || !isfinite(d0) ||
          (s[S_GUARD] > 0 && fabs(d0) < s[S_GUARD] * s[S_DEF0] * s[S_DEF]))
        fl[F_STATE] = 3;
      else
        s[S_BETA] = (d0 / s[S_RHO]) * (s[S_ALPHA] / s[S_OMEGA]);
      break;
    case FIN_BI_ALPHA:
      s[S_H] = d0;
      if (fabs(d0) < 1e-80 || !isfinite(d0) ||
          (s[S_GUARD] > 0 && fabs(d0) < s[S_GUARD] * s[S_DEF0] * sqrt(d1)))
        fl[F_STATE] = 3;
      else
        s[S_ALPHA] = s[S_RHONEW] / d0;
      break;
    case FIN_BI_OMEGA:
      s[S_TR] = d0;
      s[S_TT] = d1;
      if (!(d1 > 0.0) || !isfinite(d0 / d1)) fl[F_STATE] = 3;
      else s[S_OMEGA] = d0 / d1;
      break;
    default:
      break;
  }
}


// ---- reductions fused into other kernels ----------------------------------
// A kernel that produces one operand of a dot product (the operator writing
// q = A p, the block preconditioner writing z = M^{-1} r) adds the product of
// its own output with the other operand per block.  Same determinism as the
// dot kernels: block partials in a per-kernel array, the last block adds
// them in block order and runs the finisher.  Blocks of any size <= MAXT.

// sum over the lanes of the mask of integers below 2^58
__device__ __forceinline__ long long warp_sum_i64(unsigned mask, long long x) {
  const unsigned s0 = __reduce_add_sync(mask, (unsigned)x & 0x7ffffffu);
  const unsigned s1 = __reduce_add_sync(mask, (unsigned)(x >> 27) & 0x7ffffffu);
  const int s2 = __reduce_add_sync(mask, (int)(x >> 54));
  return (long long)(((unsigned long long)(unsigned)s2 << 54) + ((unsigned long long)s1 << 27) +
                     s0);
}

// sum of the lanes' values rounded to 57 bits under the power of two above the
// largest (biased exponent b; 128 or more, or all zero), put together on the integer
// pipe (the conversion of a 64-bit integer takes the FP64 pipe 400 cycles)
__device__ __forceinline__ double warp_sum_scaled(unsigned mask, double v, int b) {
  const int eb = max(b, kFixMinBiased);
  return fix_to_double(warp_sum_i64(mask, fix_round(v, eb)), eb - 1022 - kFixBits);
}
// (a call: unrolled in line it costs the kernels' instruction cache)
static __device__ __noinline__ double warp_sum_rare(unsigned mask, double v, int n, int b) {
  if (b != 0x7ff) {   // so small that the unit would be subnormal
    v *= 0x1p512;
    b = (int)(__reduce_max_sync(mask, (unsigned)__double2hiint(v) << 1) >> 21);
    return warp_sum_scaled(mask, v, b) * 0x1p-512;
  }
  double s = 0.0;
#pragma unroll 1
  for (int i = 0; i < n; i++) s += __shfl_sync(mask, v, i);
  return s;
}
// Sum over the first n lanes of a warp (all of which call it; the others do not
// exist), in every one of them, in 57-bit fixed point: a tree of FP64 additions
// takes five steps of about 105 cycles, this about 250 in all.  Every lane is
// rounded to 2^-57 of the power of two above the largest, so a warp is off by at
// most 2^-53 of that, and not to one side (lanes cut toward zero made sums of one
// sign too small).  Values that are not finite are added in FP64.  The result does
// not depend on the order of the lanes.
__device__ __forceinline__ double warp_sum_fixed(double v, int n) {
  const unsigned mask = n >= 32 ? 0xffffffffu : (1u << n) - 1u;
  const unsigned m = __reduce_max_sync(mask, (unsigned)__double2hiint(v) << 1);
  const int b = (int)(m >> 21);
  if (b == 0x7ff || (b < 128 && m != 0)) return warp_sum_rare(mask, v, n, b);
  return warp_sum_scaled(mask, v, b);
}

// Block sums of two values (the second only if `two`): warp sums in sw (at
// least 2 * number of warps), then threads 0 and 1 hold the sums in s0.
__device__ __forceinline__ void block_sum2(double &s0, double s1, bool two, double *sw) {
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const int n = min(32, (int)blockDim.x - 32 * w);
  s0 = warp_sum_fixed(s0, n);
  if (two) s1 = warp_sum_fixed(s1, n);
  if ((threadIdx.x & 31) == 0) {
    sw[2 * w] = s0;
    sw[2 * w + 1] = two ? s1 : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    s0 = sw[threadIdx.x];
    for (int i = 1; i < nw; i++) s0 += sw[2 * i + threadIdx.x];
  }
}

// Two-level tail for grids of many blocks: the last block of each group of
// kFuseGroup blocks adds the group's partials in block order into a group
// partial; the last group to finish adds the group partials in group order
// and runs the finisher.  Up to kFuseOne blocks are one group.  The order of
// every sum is fixed, so the result does not depend on which block finishes
// last.  Layout of `part`: 2 doubles per block, then 2 per group from offset
// 2 * max_blocks; `cnt`: one int per group, zero between launches (each
// group's last block resets its own).
constexpr int kFuseGroup = 256;
constexpr unsigned kFuseOne = 1024;

// publish (s0 of threads 0 and 1) and count; true in the last of `total`
// publishers, which then sees what the others published
__device__ __forceinline__ bool publish_last(double *slot, double s0, int *counter, int total) {
  __shared__ bool last;
  if (threadIdx.x < 32) {
    const double c = __shfl_sync(0xffffffffu, s0, 1);
    if (threadIdx.x == 0) {
      *reinterpret_cast<double2 *>(slot) = make_double2(s0, c);
      int n;
      asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;"
                   : "=r"(n)
                   : "l"(counter)
                   : "memory");
      last = n == total - 1;
    }
  }
  __syncthreads();
  return last;
}

// the block's sums are in s0 of threads 0 and 1; blocks of at least 32 threads
template <int MAXT>
__device__ __forceinline__ void grouped_finish(double *part, long max_blocks, int *cnt,
                                               const RedCtx &rc, double s0, int fin) {
  __shared__ double sw[2 * ((MAXT + 31) / 32)];
  const bool two = fin == FIN_CG_DEF_BETA;
  const int group = gridDim.x <= kFuseOne ? (int)gridDim.x : kFuseGroup;
  const int b = (int)blockIdx.x, g = b / group;
  const int ngroups = (int)((gridDim.x + group - 1) / group);
  const int gsize = min(group, (int)gridDim.x - g * group);
  if (!publish_last(part + 2 * (size_t)b, s0, &cnt[g], gsize)) return;
  const double2 *p2 = reinterpret_cast<const double2 *>(part) + (size_t)g * group;
  const auto sum = [&](const double2 *v, int n) {
    double a = 0.0, c = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double2 x = __ldcg(v + i);
      a += x.x;
      if (two) c += x.y;
    }
    block_sum2(a, c, two, sw);
    return a;
  };
  double a = sum(p2, gsize);
  if (threadIdx.x == 0) cnt[g] = 0;
  if (ngroups > 1) {
    double *gpart = part + 2 * max_blocks;
    if (!publish_last(gpart + 2 * g, a, &rc.flags[F_COUNTER], ngroups)) return;
    a = sum(reinterpret_cast<const double2 *>(gpart), ngroups);
    if (threadIdx.x == 0) rc.flags[F_COUNTER] = 0;
  }
  if (!two) {
    if (threadIdx.x == 0) run_finisher(rc, fin, -1, -1, a, 0.0);
    return;
  }
  // the square root and the quotient of FIN_CG_DEF_BETA by two warps
  if (threadIdx.x < 2) sw[threadIdx.x] = a;
  __syncthreads();
  if (threadIdx.x == 0) finish_cg_def(rc, sw[0]);
  if (threadIdx.x == (blockDim.x > 32 ? 32 : 0)) finish_cg_beta(rc, sw[1]);
}

template <int MAXT>
__device__ __forceinline__ void reduce_tail_grouped(double *part, long max_blocks, int *cnt,
                                                    const RedCtx &rc, double s0, double s1,
                                                    int fin) {
  __shared__ double sw[2 * ((MAXT + 31) / 32)];
  block_sum2(s0, s1, fin == FIN_CG_DEF_BETA, sw);
  grouped_finish<MAXT>(part, max_blocks, cnt, rc, s0, fin);
}

// A thread's sum of FP32 values carried as an unevaluated pair of floats: a few
// additions per thread on the FP32 pipe instead of the FP64 pipe's 17 cycles for each
// warp-wide one.  (48 bits: enough for a handful of terms with 24, not for the sums
// over threads, which warp_sum_two and FP64 do.)
struct TwoFloat {
  float h, l;
};
__device__ __forceinline__ TwoFloat two_add(TwoFloat a, TwoFloat b) {
  const float s = __fadd_rn(a.h, b.h), t = __fsub_rn(s, a.h);
  const float e = __fadd_rn(__fadd_rn(__fsub_rn(a.h, __fsub_rn(s, t)), __fsub_rn(b.h, t)),
                            __fadd_rn(a.l, b.l));
  const float h = __fadd_rn(s, e);
  // a sum that is not finite stays what it is
  return TwoFloat{h, isfinite(h) ? __fsub_rn(e, __fsub_rn(h, s)) : 0.f};
}
// A float x below 2^(E + 1) as a multiple of 2^(E - 21): adding s = 1.5 2^(E + 2), whose
// last place that is, rounds it there, and the sum's bits count it.  x becomes the
// rest, exactly.
__device__ __forceinline__ int take_chunk(float &x, float s) {
  const float t = __fadd_rn(x, s);
  x = __fsub_rn(x, __fsub_rn(t, s));
  return __float_as_int(t) - __float_as_int(s);
}
// sum of the pairs of a whole warp, biased exponent eb of the largest high part in
// 42..251: every pair as three integers of 22 bits, down to 2^-65 of the power of two
// above the largest, summed without rounding; the result has 57 bits before its
// own rounding
__device__ __forceinline__ double warp_sum_chunks(TwoFloat v, int eb) {
  constexpr unsigned kAll = 0xffffffffu;
  const auto magic = [&](int d) { return __int_as_float(((eb + 3 - d) << 23) | 0x400000); };
  const int c1 = take_chunk(v.h, magic(0));
  const float s2 = magic(22);
  const int c2 = take_chunk(v.h, s2) + take_chunk(v.l, s2);
  float rest = __fadd_rn(v.h, v.l);
  const int c3 = take_chunk(rest, magic(44));
  const long long n1 = __reduce_add_sync(kAll, c1), n2 = __reduce_add_sync(kAll, c2);
  const int n3 = __reduce_add_sync(kAll, c3);
  // units of 2^(E - 21), 2^(E - 43) and 2^(E - 65), E = eb - 126
  return fix_to_double(n1 * (1ll << 36) + n2 * (1ll << 14) + ((n3 + 128) >> 8),
                       eb - 126 - kFixBits);
}
// (a call: in line it costs the kernels' instruction cache)
static __device__ __noinline__ double warp_sum_two_rare(TwoFloat v, int eb) {
  constexpr unsigned kAll = 0xffffffffu;
  if (eb == 0xff) return warp_sum_rare(kAll, (double)v.h + (double)v.l, 32, 0x7ff);
  // to the middle of the range and back
  const float up = eb < 42 ? 0x1p100f : 0x1p-8f;
  const TwoFloat w{__fmul_rn(v.h, up), __fmul_rn(v.l, up)};
  const int e = (int)(__reduce_max_sync(kAll, __float_as_uint(w.h) << 1) >> 24);
  if (e == 0) return 0.0;
  return warp_sum_chunks(w, e) * (eb < 42 ? 0x1p-100 : 0x1p8);
}
// Sum of the pairs of a whole warp, in every lane, as exact as warp_sum_fixed, and
// with fewer instructions than a tree of additions of pairs.  Infinities and NaN are
// added in FP64.
__device__ __forceinline__ double warp_sum_two(TwoFloat v) {
  const int eb = (int)(__reduce_max_sync(0xffffffffu, __float_as_uint(v.h) << 1) >> 24);
  if (eb < 42 || eb > 251) return warp_sum_two_rare(v, eb);
  return warp_sum_chunks(v, eb);
}
// reduce_tail_grouped with two-float sums of each thread (blocks of T threads,
// T a multiple of 32)
template <int T>
__device__ __forceinline__ void reduce_tail_two_float(double *part, long max_blocks, int *cnt,
                                                      const RedCtx &rc, TwoFloat s0, TwoFloat s1,
                                                      int fin) {
  __shared__ double sw[2][T / 32];
  const bool two = fin == FIN_CG_DEF_BETA;
  const double a0 = warp_sum_two(s0), a1 = two ? warp_sum_two(s1) : 0.0;
  if ((threadIdx.x & 31) == 0) {
    sw[0][threadIdx.x >> 5] = a0;
    sw[1][threadIdx.x >> 5] = a1;
  }
  __syncthreads();
  // thread 0 adds the first values, thread 1 the second
  double a = 0.0;
  if (threadIdx.x < 2) {
    a = sw[threadIdx.x][0];
#pragma unroll
    for (int i = 1; i < T / 32; i++) a += sw[threadIdx.x][i];
  }
  grouped_finish<T>(part, max_blocks, cnt, rc, a, fin);
}

int red_dot(pdg_context *ctx, const RedCtx &rc, long n, const double *a, const double *b,
            const double *c, const double *d, int fin, int slot0, int slot1, bool respect_flag);
int red_dot_f32(pdg_context *ctx, const RedCtx &rc, long n, const float *a, const float *b,
                const float *c, const float *d, int fin, int slot0, int slot1,
                bool respect_flag);

// fused updates (skip when the flag is raised)
template <typename T>
int cg_update_xr(pdg_context *ctx, const RedCtx &rc, long n, T *x, T *r, const T *p,
                 const T *q);   // x += lambda p; r -= lambda q; def check
template <typename T>
int cg_update_p(pdg_context *ctx, const RedCtx &rc, long n, T *p, const T *z);  // p = z + beta p
// fused CG: x += lambda p ; p = z + beta p (the residual update and defect
// check ran in the preconditioner kernel) and, after the loop, the x update of
// the stopping iteration
template <typename T>
int cg_update_px(pdg_context *ctx, const RedCtx &rc, long n, T *x, T *p, const T *z);
template <typename T>
int cg_finish_x(pdg_context *ctx, const RedCtx &rc, long n, T *x, const T *p);
template <typename T>
int bi_update_p(pdg_context *ctx, const RedCtx &rc, long n, T *p, const T *r, const T *v,
                int first);   // p = r (first) or p = beta (p - omega v) + r
template <typename T>
int bi_update_half(pdg_context *ctx, const RedCtx &rc, long n, T *x, T *r, const T *y,
                   const T *v);   // x += alpha y; r -= alpha v; def check
template <typename T>
int bi_update_full(pdg_context *ctx, const RedCtx &rc, long n, T *x, T *r, const T *y,
                   const T *t);   // x += omega y; r -= omega t; def check; rho = rho_new
int set_iter(pdg_context *ctx, const RedCtx &rc, double it);

// plain vector kernels
template <typename T>
int vec_copy(pdg_context *ctx, long n, const T *src, T *dst);
template <typename T>
int vec_fill(pdg_context *ctx, long n, T *dst, T v);
int vec_axpy(pdg_context *ctx, long n, double alpha, const double *x, double *y);
// y32 = (float)(x64 * s) with s = 1/scal[S_SCALE]
int vec_to_f32_scaled(pdg_context *ctx, long n, const double *x, float *y, const double *scal);
// y64 += scal[S_SCALE] * sign * (double)x32
int vec_add_f32_scaled(pdg_context *ctx, long n, const float *x, double *y, const double *scal,
                       double sign);
int vec_to_f32(pdg_context *ctx, long n, const double *x, float *y);
// skip-aware conversions around an FP32 operator inside an FP64 Krylov solve:
// y32 = (float)x ;  y = (acc ? y : 0) + alpha (double)s32 + (add ? add : 0)
int vec_to_f32_skip(pdg_context *ctx, long n, const double *x, float *y, const int *skip);
int vec_from_f32_combine(pdg_context *ctx, long n, const float *s32, double *y, const double *add,
                         double alpha, int acc, const int *skip);

}  // namespace pdg
