// pdg_fixed.cuh -- 64-bit block fixed point on the integer pipe.
//
// GB300 multiplies FP64 at about 1.8 lanes per SM and cycle, 32x32 -> 64 bit
// integers (IMAD.WIDE) at about 25 (both measured).  Three of the latter make
// one 57-bit multiply-add, so a contraction whose operands share an exponent
// runs several times faster as integers, and with 57 instead of 53 bits.
//
// A value x with |x| < 2^E (E the exponent of its block: a line, a cell, a
// record) is held as X = x 2^(57 - E), split into two signed limbs,
// X = h 2^29 + l with |h| <= 2^28 and |l| <= 2^28.  A contraction of up to
// 2N <= 10 terms keeps two 64-bit sums, hh = sum h h' and mid = sum h l' + l h'
// (|hh| < 2^60, |mid| < 2^61); the l l' products are below the last place
// kept and are dropped.  Later stages work on plain 64-bit integers with one
// exponent per cell; multiplying those by small integer constants (the
// entries of the 1D mass matrix over their common denominator) is exact.
#pragma once

#include <cstdint>

namespace pdg {

constexpr int kFixBits = 57;        // |X| < 2^kFixBits
constexpr int kGroup = 32;          // cells of a group of the degree-2 limb records
constexpr int kFixZero = -5000;     // exponent of an all-zero block
constexpr int kFixMinBiased = 64;   // smallest biased exponent a block is scaled to

// the 1D mass matrix of the equidistant Lagrange basis (k = 1, 2 also that of
// the Gauss-Lobatto basis) as integers over `den`, and the derivative of the
// basis at 0 as integers over `dden` (at 1: reversed, negated)
template <int N> struct IntTab;
template <> struct IntTab<2> { static constexpr int den = 6, dden = 1; };
template <> struct IntTab<3> { static constexpr int den = 30, dden = 1; };
template <> struct IntTab<4> { static constexpr int den = 1680, dden = 2; };
template <> struct IntTab<5> { static constexpr int den = 5670, dden = 3; };
// entry i of the mass matrix (row-major)
template <int N> __host__ __device__ __forceinline__ constexpr int int_m(int i) {
  if constexpr (N == 2) {
    constexpr int m[] = {2, 1, 1, 2};
    return m[i];
  } else if constexpr (N == 3) {
    constexpr int m[] = {4, 2, -1, 2, 16, 2, -1, 2, 4};
    return m[i];
  } else if constexpr (N == 4) {
    constexpr int m[] = {128, 99, -36, 19, 99, 648, -81, -36, -36, -81, 648, 99, 19, -36, 99, 128};
    return m[i];
  } else {
    constexpr int m[] = {292,  296,  -174, 56,   -29, 296, 1792, -384, 256,  56, -174, -384, 1872,
                         -384, -174, 56,   256,  -384, 1792, 296, -29, 56,   -174, 296, 292};
    return m[i];
  }
}
template <int N> __host__ __device__ __forceinline__ constexpr int int_d0(int i) {
  constexpr int d[4][5] = {{-1, 1}, {-3, 4, -1}, {-11, 18, -9, 2}, {-25, 48, -36, 16, -3}};
  return d[N - 2][i];
}
template <int N> __host__ __device__ __forceinline__ constexpr int int_d1(int i) {
  return -int_d0<N>(N - 1 - i);
}

// largest biased exponent of a block so far (top 11 bits of m) and whether
// any of its values is non-zero
struct BlockExp {
  unsigned m = 0, any = 0;
  __device__ __forceinline__ void add(double x) {
    const unsigned hi2 = (unsigned)__double2hiint(x) << 1;
    m = max(m, hi2);
    any |= hi2 | (unsigned)__double2loint(x);
  }
  __device__ __forceinline__ int biased() const { return max((int)(m >> 21), kFixMinBiased); }
  __device__ __forceinline__ bool finite() const { return (m >> 21) != 0x7ffu; }
  // E with |x| < 2^E (values below 2^(kFixMinBiased - 1023) count as zero
  // beside it), kFixZero for a block of zeros
  __device__ __forceinline__ int exponent() const { return any ? biased() - 1022 : kFixZero; }
};

// magnitude of x in units of 2^(E - F), E = eb - 1022, truncated (x finite,
// biased exponent at most eb; zeros and subnormals give 0, since eb >= 64)
template <int F = kFixBits>
__device__ __forceinline__ unsigned long long fix_mag(double x, int eb) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int sh = min(eb - (int)((hi >> 20) & 0x7ffu), 63);
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const unsigned long long t =
      ((unsigned long long)__funnelshift_l(lo, mh, F - 53) << 32) | (unsigned)(lo << (F - 53));
  return t >> sh;
}
// x rounded to units of 2^(E - 57), E = eb - 1022 (x finite, biased exponent at
// most eb, eb >= 64; halves away from zero, zeros and subnormals give 0)
__device__ __forceinline__ long long fix_round(double x, int eb) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int sh = min(eb - (int)((hi >> 20) & 0x7ffu), 63);
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const unsigned long long t =
      ((unsigned long long)__funnelshift_l(lo, mh, kFixBits - 53) << 32) |
      (unsigned)(lo << (kFixBits - 53));
  const long long r = (long long)((t + ((1ull << sh) >> 1)) >> sh);
  return (int)hi < 0 ? -r : r;
}
// The operators compute a cell with the sign of its first value taken out of all
// its data (flip: 0 or -1, sign_flip of that value): rounding then sees the same
// integers for x and -x, so J(-x) = -J(x) to the bit, as in FP64.
__device__ __forceinline__ int sign_flip(double x) { return __double2hiint(x) >> 31; }
__device__ __forceinline__ long long fix_signed(double x, int eb, int flip = 0) {
  const long long t = (long long)fix_mag(x, eb);
  return (__double2hiint(x) ^ flip) < 0 ? -t : t;
}
// limbs (h, l) of X = h 2^29 + l, l rounded to the nearest multiple's rest
__device__ __forceinline__ int2 limbs(long long X) {
  const int h = (int)((X + (1ll << 28)) >> 29);
  return make_int2(h, (int)((unsigned)X - ((unsigned)h << 29)));
}
template <int F = kFixBits>
__device__ __forceinline__ int2 fix_limbs(double x, int eb, int flip = 0) {
  const int2 r = limbs((long long)fix_mag<F>(x, eb));
  const int s = (__double2hiint(x) ^ flip) >> 31;
  return make_int2((r.x ^ s) - s, (r.y ^ s) - s);
}

// hh and mid of one limb multiply-add
__device__ __forceinline__ void mac2(long long &hh, long long &mid, int2 a, int2 b) {
  hh += (long long)a.x * b.x;
  mid += (long long)a.x * b.y;
  mid += (long long)a.y * b.x;
}
// One of the operands may have kFixWide = 59 bits (|h| <= 2^30): the sums of
// five such products stay below 2^62.
constexpr int kFixWide = 59;
// the contraction of 57-bit operands in units of 2^(Ea + Eb - 59) (one of them
// 59 bits wide: 2^(Ea + Eb - 61)), shifted right by sh, cut: half a unit too small
// on average, which the caller adds where it costs nothing (without that the bias
// of a residual was 1.7e-12 of J x at 24^3 Q4 and smooth data)
__device__ __forceinline__ long long mac2_value(long long hh, long long mid, int sh) {
  return ((hh << 3) + (mid >> 26)) >> (int)min((unsigned)sh, 63u);
}
// the same rounded; beyond 61 bits what is left is at most a few units
__device__ __forceinline__ long long mac2_round(long long hh, long long mid, int sh) {
  const int s = (int)min((unsigned)sh, 61u);
  return ((hh << 3) + ((mid + (1ll << 25)) >> 26) + ((1ll << s) >> 1)) >> s;
}

// the contraction of a 59-bit with a 57-bit operand in units of 2^(Ea + Eb - 59)
__device__ __forceinline__ long long mac2_value_wide(long long hh, long long mid) {
  return (hh << 1) + (mid >> 28);
}

// a 64-bit integer as v = y 2^32 + x with signed 32-bit x and y
__device__ __forceinline__ int2 split32(long long v) {
  const int lo = (int)v;
  return make_int2(lo, (int)(v >> 32) - (lo >> 31));
}
__device__ __forceinline__ long long join32(int2 v) {
  return (long long)(((unsigned long long)(unsigned)v.y << 32)) + (long long)v.x;
}
// sum of c * v over small integer constants c, modulo 2^64 (kWide false; the
// caller's bound keeps the sum below 2^63) or as two 64-bit sums
template <bool kWide> struct SmallSum;
template <> struct SmallSum<false> {
  long long lo;
  unsigned hi;
  __device__ __forceinline__ explicit SmallSum(long long init) : lo(init), hi(0) {}
  __device__ __forceinline__ void add(int2 v, int c) {
    lo += (long long)v.x * c;
    hi += (unsigned)v.y * (unsigned)c;
  }
  __device__ __forceinline__ long long total() const {
    return (long long)((unsigned long long)lo + ((unsigned long long)hi << 32));
  }
  template <int S> __device__ __forceinline__ long long shifted() const { return total() >> S; }
};
template <> struct SmallSum<true> {
  long long lo, hi;
  __device__ __forceinline__ explicit SmallSum(long long init) : lo(init), hi(0) {}
  __device__ __forceinline__ void add(int2 v, int c) {
    lo += (long long)v.x * c;
    hi += (long long)v.y * c;
  }
  template <int S> __device__ __forceinline__ long long shifted() const {
    return (long long)((unsigned long long)hi << (32 - S)) + (lo >> S);
  }
};

// v 2^E rounded to the nearest double (|v| < 2^63, the result in the normal
// range or v = 0), put together on the integer pipe: the conversion of a 64-bit
// integer is six FP64-pipe operations of 64 cycles per warp and sub-partition
__device__ __forceinline__ double fix_to_double(long long v, int E, int flip = 0) {
  unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
  const int lz = __clzll((long long)m);
  m <<= (lz & 63);
  // 1.f 2^(63 - lz + E); the leading one of m >> 11 adds one to the exponent field
  const unsigned long long bits =
      ((unsigned long long)(unsigned)(63 - lz + E + 1022) << 52) + (m >> 11) + ((m >> 10) & 1);
  const int hi = (int)(bits >> 32) | (((int)(v >> 32) ^ flip) & (int)0x80000000);
  return v == 0 ? 0.0 : __hiloint2double(hi, (int)bits);
}

}  // namespace pdg
