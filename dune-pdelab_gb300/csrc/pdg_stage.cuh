// pdg_stage.cuh -- staging of contiguous runs of a vector in shared memory.
//
// A run of source elements [g0, g0 + count) lands at dst[ph + i], ph = g0 mod
// the elements of 16 bytes, so that source and destination share their 16-byte
// phase (dst is 16-byte aligned and has room for whole 16-byte chunks).  Runs
// inside [0, lim) of an aligned source are one bulk copy by thread 0, completing
// on `bar` (per-thread copies of all runs cost the FP32 operator of
// pdg_cell32.cu about 900 of its 3800 instructions per warp); runs that
// straddle an end are copied element-wise with zeros outside, runs outside are
// left out (an absent neighbour's values are not used).  All threads call it,
// then wait().
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
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0 && ga >= 0 && ga + len <= lim) {
      if (threadIdx.x == 0) {
        // every copy is announced before it is issued; the phase completes
        // with the arrival in wait()
        mbar_announce_tx(bar, (unsigned)sizeof(V) * len);
        bulk_load(smem_u32(dst), src + ga, (unsigned)sizeof(V) * len, bar);
      }
    } else {
      for (int c = threadIdx.x; c < len; c += T) {
        const long g = ga + c;
        dst[c] = (g >= 0 && g < lim) ? src[g] : V(0);
      }
    }
    return dst + ph;
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
