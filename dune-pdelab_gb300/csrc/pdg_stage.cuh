// pdg_stage.cuh -- staging of contiguous runs of a vector in shared memory.
//
// A run of source elements [g0, g0 + count) lands at dst[ph + i], ph = g0 mod
// the elements of 16 bytes, so that source and destination share their 16-byte
// phase (dst is 16-byte aligned and has room for whole 16-byte chunks).  Of an aligned
// source the part inside [0, lim) is one bulk copy of whole chunks by thread 0,
// completing on `bar` (per-thread copies of all runs cost the FP32 operator of
// pdg_cell32.cu about 900 of its 3800 instructions per warp), and at most one chunk's
// rest element-wise.  What lies outside is left as it is: an absent neighbour's values
// and those of inactive cells are not used.  All threads call it, then wait().
//
// Runs that straddle an end go the same way: copied element-wise they are tens of
// loads one after another, and the blocks at the ends of a grid of a few thousand
// cells are its last ones (9x10x11 Q2, device time: FP32 block Jacobi 6.0 us that way,
// 3.7 this, FP32 operator 7.8 and 5.2, FP64 operator 10.6 and 8.7; asynchronous copies
// of the rest: 3.3, 5.0, 8.8, but 64^3 Q2 FP64 159 instead of 158 us).
#pragma once

#include "pdg_tma.cuh"

namespace pdg {

template <int T, typename V>
struct Stager {
  static constexpr int E = 16 / (int)sizeof(V);   // elements of 16 bytes
  unsigned bar;
  __device__ __forceinline__ explicit Stager(unsigned long long *b) : bar(smem_u32(b)) {
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
  }
  __device__ __forceinline__ V *run(V *dst, const V *src, long g0, long lim, int count) {
    const int ph = (int)(((g0 % E) + E) % E);
    const long ga = g0 - ph;
    const int len = (ph + count + E - 1) & ~(E - 1);
    if (ga + len <= 0 || ga >= lim) return dst + ph;
    const bool aligned = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    if (aligned && ga >= 0 && ga + len <= lim) {
      bulk(dst, src + ga, len);
      return dst + ph;
    }
    // the part inside [0, lim); ga is a multiple of E
    const int b = ga < 0 ? (int)-ga : 0, e = lim - ga < len ? (int)(lim - ga) : len;
    int c = b;
    if (aligned) {
      c = e & ~(E - 1);
      if (c > b) bulk(dst + b, src + ga + b, c - b);
      else c = b;
    }
    for (c += threadIdx.x; c < e; c += T) dst[c] = src[ga + c];
    return dst + ph;
  }
  // every copy is announced before it is issued; the phase completes with the
  // arrival in wait()
  __device__ __forceinline__ void bulk(V *dst, const V *src, int n) {
    if (threadIdx.x != 0) return;
    mbar_announce_tx(bar, (unsigned)sizeof(V) * n);
    bulk_load(smem_u32(dst), src, (unsigned)sizeof(V) * n, bar);
  }
  // false: the copies did not arrive within the poll limit.  They may still be
  // in flight then, and a block must not leave its shared memory to the next one
  // while they are: a failed wait gives them the same time once more.
  __device__ __forceinline__ bool wait() {
    if (threadIdx.x == 0) mbar_arrive(bar);
    const bool ok = mbar_wait(bar, 0, kTmaPolls);
    if (!ok) mbar_wait(bar, 0, kTmaPolls);
    return __syncthreads_and(ok);
  }
};

}  // namespace pdg
