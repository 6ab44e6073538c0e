"""The staging helper of pdg_stage.cuh on the CPU: one thread, with the bulk
copies and the barrier of pdg_tma.cuh replaced by a model in which every copy
lands after a given number of polls.  A wait that runs out must not return
while copies into the block's shared memory are still in flight."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dune-pdelab_gb300", "csrc")

TMA = r"""
#pragma once
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#define __device__
#define __forceinline__ inline
struct Dim { unsigned x; };
static Dim threadIdx = {0};
static void __syncthreads() {}
static int __syncthreads_and(int v) { return v; }
constexpr int kTmaPolls = 1000;
// the model: copies queued, polls so far, polls after which they land
static struct { void *dst; const void *src; unsigned n; } queue[8];
static int queued = 0;
static long polls = 0, lands_at = 0;
static unsigned announced = 0;
static bool arrived = false;
template <class T> static uintptr_t smem_u32(T *p) { return (uintptr_t)p; }
static void mbar_init(uintptr_t, unsigned) {}
static void mbar_announce_tx(uintptr_t, unsigned bytes) { announced += bytes; }
static void mbar_arrive(uintptr_t) { arrived = true; }
static void bulk_load(uintptr_t dst, const void *src, unsigned n, uintptr_t) {
  queue[queued].dst = (void *)dst;
  queue[queued].src = src;
  queue[queued++].n = n;
}
static bool mbar_wait(uintptr_t, unsigned, int limit) {
  for (int i = 0; i < limit; i++)
    if (++polls >= lands_at && arrived) {
      for (; queued > 0; queued--) {
        std::memcpy(queue[queued - 1].dst, queue[queued - 1].src, queue[queued - 1].n);
        announced -= queue[queued - 1].n;
      }
      return true;
    }
  return false;
}
"""

MAIN = r"""
#include "pdg_stage.cuh"
alignas(16) static double src[64], dst[64];
static unsigned long long bar;
// every run of a vector of 61 values, by T threads one after another: the values
// inside arrive, nothing is read or written outside
template <int T, typename V>
static int runs() {
  constexpr int E = 16 / (int)sizeof(V), kLim = 61, kMax = 40;
  alignas(16) static V x[kLim + 2 * E], to[kMax + 4 * E];
  lands_at = 1;
  for (int shift = 0; shift < 2; shift++)          // aligned source or not
    for (int g0 = -kMax - 3; g0 < kLim + 3; g0++)
      for (int count = 1; count <= kMax - E; count += 3) {
        for (int i = 0; i < kLim + 2 * E; i++) x[i] = V(-5);
        const V *src = x + E + shift;
        for (int i = 0; i < kLim; i++) x[E + shift + i] = V(i + 1);
        for (V &v : to) v = V(-7);
        V *run = nullptr;
        arrived = false;
        polls = 0;
        for (threadIdx.x = T; threadIdx.x-- > 0;) {
          pdg::Stager<T, V> st(&bar);
          run = st.run(to + E, src, g0, kLim, count);
        }
        threadIdx.x = 0;
        for (int i = 0; i < queued; i++) {
          const V *s = (const V *)queue[i].src;
          if ((uintptr_t)s % 16 || (uintptr_t)queue[i].dst % 16 || queue[i].n % 16 || s < src ||
              s + queue[i].n / sizeof(V) > src + kLim)
            return 1;
        }
        pdg::Stager<T, V> st(&bar);
        if (!st.wait() || queued) return 2;
        for (int i = 0; i < count; i++)
          if (g0 + i >= 0 && g0 + i < kLim && run[i] != V(g0 + i + 1)) return 3;
        const V *end = run + count + E - 1;      // whole chunks
        for (V &v : to)
          if ((&v < to + E || &v >= end) && v != V(-7)) return 4;
        for (V &v : to)
          if (v == V(-5)) return 5;
      }
  return 0;
}
int main(int argc, char **argv) {
  if (argc < 2) {
    const int bad = runs<4, float>() + 10 * runs<2, double>();
    std::printf("%d\n", bad);
    return bad;
  }
  lands_at = std::atol(argv[1]);
  for (int i = 0; i < 64; i++) src[i] = i + 1;
  pdg::Stager<1, double> st(&bar);
  double *run = st.run(dst, src, 5, 64, 20);
  const bool ok = st.wait();
  for (int i = 0; ok && i < 20; i++)
    if (run[i] != src[5 + i]) return 1;
  std::printf("%d %d %u\n", (int)ok, queued, announced);
  return 0;
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("stage")
    shutil.copy(os.path.join(CSRC, "pdg_stage.cuh"), d)
    with open(os.path.join(CSRC, "pdg_stage.cuh")) as f:
        text = f.read()
    # addresses are 64 bits wide here
    (d / "pdg_stage.cuh").write_text(text.replace("unsigned bar;", "uintptr_t bar;"))
    (d / "pdg_tma.cuh").write_text(TMA.replace("constexpr int kTmaPolls",
                                               "namespace pdg {}\nconstexpr int kTmaPolls"))
    (d / "main.cc").write_text(MAIN)
    out = d / "stage"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(d), str(d / "main.cc"), "-o",
                        str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(out)


# (polls until the copies land, in units of one wait's limit): the result, and
# that nothing is in flight when the wait is over
@pytest.mark.parametrize("lands_at,ok", [(1, 1), (1000, 1), (1001, 0), (1999, 0)])
def test_nothing_in_flight_after_a_wait(exe, lands_at, ok):
    r = subprocess.run([exe, str(lands_at)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert [int(v) for v in r.stdout.split()] == [ok, 0, 0]


def test_runs_that_straddle_the_ends(exe):
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
