// Two-dimensional density sums from exact strip moments (pair body
// PAIR_MOMENT).
//
// The 2-D density at target t is sum_s wx(t,s) wy(t,s) with
// w = max(0, g^2 - d^2) per dimension in scaled units (the reference's
// densities_2d loop, densities_omp.cpp:97-126, and density_2d.cuh). The
// points are strip-major: strips of width h/S along dimension 1, sorted by
// dimension 0 inside each strip. For one target and one strip:
//  * the sources in x-support form one index range [l, r) of the strip,
//    found by two binary searches with the pair kernels' own test
//    fma(-d, d, g^2) > 0 (monotone in |d|);
//  * if the strip's smallest and largest y both pass the y test, every
//    source of the strip does (|fl(y - t_y)| lies between the two), and on
//    [l, r) the sum is a polynomial in the sources' coordinates:
//      sum (G1 - (TX - X)^2)(G2 - (TY - Y)^2)
//        = sum_{a,b <= 2} c_a(TX) d_b(TY) M_ab,   M_ab = sum X^a Y^b,
//    with X = x 2^23, Y = y 2^23 fixed point and G = g^2 2^46. The moments
//    come from prefix sums over the strip-major order taken modulo 2^128;
//    the identity holds in the integers, reduction modulo 2^128 is a ring
//    map and the true value lies in (-2^124, 2^124), so the signed modular
//    result IS the exact integer: no cancellation whatever the offset or
//    spread of the data;
//  * the strips at distance exactly S from the target's own (where the edge
//    of its y-support falls) are summed pair by pair by the symmetric pair
//    kernel, each pair once for both points (the plan gives every strip one
//    tile run: the strip S above it); strips nearer than S whose y extent
//    still crosses the support (rounding at the widened cell edges) are
//    summed pair by pair here.
// Fixed-point rounding of the coordinates (2^-23 g) changes a kernel value
// by less than 2^-21 g^2 per dimension, far below the 1e-5 density bar.
//
// The epilogue (scale, per-point output, log and per-block sums) runs in the
// same kernel; the symmetric kernel's finish skips these instances. The log
// of each target's exact sum is taken in 64-bit fixed point (ilog_fx48) and
// the block sums are exact integer sums.
#include <algorithm>
#include <cmath>

#include "engine.h"
#include "staging.cuh"  // FULL_MASK

namespace ent {
namespace {

typedef unsigned __int128 u128;

constexpr uint32_t M2_TB = 128;               // targets per block
template <bool NARROW> constexpr int M2_BPS = NARROW ? 12 : 10;  // blocks per SM
constexpr uint32_t M2_PT = 256;               // prefix threads per block
constexpr uint32_t M2_E = 8;                  // prefix values per thread
constexpr uint32_t M2_CHUNK = M2_PT * M2_E;   // prefix values per block
// Moments of a row, in the halves that the two lanes of a target read:
// Y, Y^2, X^2, X^2 Y^2 | XY, X Y^2, X^2 Y, X
constexpr int NM = 8;
constexpr int NH = NM / 2;
// A row of prefix sums in 16-byte chunks. Wide rows hold the eight moments in
// 128 bits each. Narrow rows hold each half as one 384-bit integer, the sum of
// its moments at bit offsets
//   half 0:  Y 2^0 + Y^2 2^64 + X^2 2^160 + X^2 Y^2 2^256
//   half 1:  X 2^0 + XY 2^64 + X Y^2 2^160 + X^2 Y 2^272
// modulo 2^384: differences and sums of rows are one carry chain over the half,
// and while each moment of a target's sources fits its field (MOMENT_NARROW and
// MOMENT_NARROW_SUM) the fields come apart again with their signs (X^2 Y^2 is
// needed modulo 2^128 only). 96 instead of 128 bytes per support end read, and 24 instead
// of 32 adds per lane and row pair; 12 registers of sums instead of 16 let 12
// blocks per SM run (40 registers, no spills) instead of 10. Target kernel, wide /
// narrow rows: 64 x 100k MI 20.6 / 17.7 ms (narrow at 10 blocks 19.0, at 16 21.2),
// 32 x 200k TE at 3 lags 47.9 (10 blocks) / 42.1.
template <bool NARROW> constexpr int ROW_CHUNKS = NARROW ? 6 : 8;

// round(v 2^F) modulo 2^128 (two's complement), v finite.
template <int F>
__device__ __forceinline__ u128 quant(float v) {
  const uint32_t b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 0xffu);
  if (e == 0) return 0;  // zero or subnormal
  const uint64_t m = (uint64_t)((b & 0x7fffffu) | 0x800000u);
  const int sh = e - 150 + F;
  u128 q;
  if (sh >= 128) {
    q = 0;
  } else if (sh >= 0) {
    q = (u128)m << sh;
  } else if (sh > -25) {
    q = (u128)((m + (1ull << (-sh - 1))) >> (-sh));
  } else {
    q = 0;
  }
  return (b & 0x80000000u) ? (u128)0 - q : q;
}

// quant<23> of a value below 2^8 in magnitude (|result| < 2^31), with the
// same rounding (half away from zero).
__device__ __forceinline__ int32_t quant23_narrow(float v) {
  const uint32_t b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 0xffu);
  const uint32_t m = (b & 0x7fffffu) | 0x800000u;
  const int sh = e - 127;  // <= 7
  uint32_t q;
  if (e == 0) q = 0;
  else if (sh >= 0) q = m << sh;
  else if (sh > -25) q = (m + (1u << (-sh - 1))) >> (-sh);
  else q = 0;
  return (b & 0x80000000u) ? -(int32_t)q : (int32_t)q;
}

// both coordinates below 2^8 in magnitude (scaled units)
__device__ __forceinline__ bool narrow2(float2 p) {
  return ((__float_as_uint(p.x) >> 23) & 0xffu) < 135u &&
         ((__float_as_uint(p.y) >> 23) & 0xffu) < 135u;
}

__device__ __forceinline__ u128 u128_of(int64_t hi, uint64_t lo) {
  return ((u128)(uint64_t)hi << 64) | lo;
}

// The eight moments of one point modulo 2^128 (NARROW: of a point known to be
// near the origin). Points whose scaled
// coordinates lie below 2^8 in magnitude (all of them for data within a few
// hundred bandwidths of zero) take 32-bit coordinates and 64 x 64 -> 128-bit
// products; the others the general 128-bit form. Both give the same residues.
template <bool NARROW>
__device__ __forceinline__ void moments(float2 p, u128 (&m)[NM]) {
  if (NARROW || narrow2(p)) {
    const int32_t x = quant23_narrow(p.x), y = quant23_narrow(p.y);
    const int64_t X2 = (int64_t)x * x, Y2 = (int64_t)y * y, XY = (int64_t)x * y;
    const int64_t X = x, Y = y;
    m[0] = (u128)(__int128)y;
    m[1] = (u128)(uint64_t)Y2;
    m[2] = (u128)(uint64_t)X2;
    m[3] = u128_of((int64_t)__umul64hi((uint64_t)X2, (uint64_t)Y2),
                   (uint64_t)X2 * (uint64_t)Y2);
    m[4] = (u128)(__int128)XY;
    m[5] = u128_of(__mul64hi(X, Y2), (uint64_t)X * (uint64_t)Y2);
    m[6] = u128_of(__mul64hi(X2, Y), (uint64_t)X2 * (uint64_t)Y);
    m[7] = (u128)(__int128)x;
    return;
  }
  const u128 X = quant<23>(p.x), Y = quant<23>(p.y);
  const u128 X2 = X * X, Y2 = Y * Y;
  m[0] = Y;
  m[1] = Y2;
  m[2] = X2;
  m[3] = X2 * Y2;
  m[4] = X * Y;
  m[5] = X * Y2;
  m[6] = X2 * Y;
  m[7] = X;
}

// The M2_E points of one prefix thread, loaded at once (16-byte loads when
// all are present: pts is 256-byte aligned and k0 a multiple of 8); returns
// how many are present.
__device__ __forceinline__ uint32_t load_points8(const float2* __restrict__ pts, uint64_t k0,
                                                 uint32_t n, float2 (&p)[M2_E]) {
  static_assert(M2_E == 8, "four 16-byte loads per thread");
  if (k0 + M2_E <= n) {
    const float4* q = reinterpret_cast<const float4*>(pts + k0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = q[i];
      p[2 * i] = make_float2(v.x, v.y);
      p[2 * i + 1] = make_float2(v.z, v.w);
    }
    return M2_E;
  }
  const uint32_t ne = k0 < n ? (uint32_t)(n - k0) : 0u;
#pragma unroll
  for (uint32_t e = 0; e < M2_E; ++e) p[e] = e < ne ? pts[k0 + e] : make_float2(0.f, 0.f);
  return ne;
}

// two neighbouring points, k even and below n (the second one may be absent)
__device__ __forceinline__ void load_pair(const float2* __restrict__ pts, uint64_t k,
                                          uint32_t n, float2 (&p)[2]) {
  if (k + 1 < n) {
    const float4 v = *reinterpret_cast<const float4*>(pts + k);
    p[0] = make_float2(v.x, v.y);
    p[1] = make_float2(v.z, v.w);
  } else {
    p[0] = pts[k];
  }
}

__device__ __forceinline__ u128 shfl_up128(u128 v, int o) {
  const unsigned long long lo = __shfl_up_sync(FULL_MASK, (unsigned long long)v, o);
  const unsigned long long hi = __shfl_up_sync(FULL_MASK, (unsigned long long)(v >> 64), o);
  return ((u128)hi << 64) | lo;
}
__device__ __forceinline__ u128 shfl_idx128(u128 v, int l) {
  const unsigned long long lo = __shfl_sync(FULL_MASK, (unsigned long long)v, l);
  const unsigned long long hi = __shfl_sync(FULL_MASK, (unsigned long long)(v >> 64), l);
  return ((u128)hi << 64) | lo;
}

// 32 bytes in one load (256-bit loads, sm_100 and later)
__device__ __forceinline__ void load32(const void* p, uint64_t (&v)[4]) {
  asm("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
      : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
      : "l"(p));
}

// The narrow form of one half row from a row's moments: every field takes the
// borrow of the negative ones below it.
template <int HALF>
__device__ __forceinline__ void pack_half(const u128 (&m)[NM], uint64_t (&w)[6]) {
  w[0] = (uint64_t)(HALF ? m[7] : m[0]);
  const u128 b = (HALF ? m[4] : m[1]) - (w[0] >> 63);
  const uint64_t bh = (uint64_t)(b >> 64);
  const u128 c = (HALF ? m[5] : m[2]) - (bh >> 63);
  const uint64_t cl = (uint64_t)c, ch = (uint64_t)(c >> 64);
  const u128 d = (HALF ? m[6] : m[3]) - (ch >> 63);
  const uint64_t dl = (uint64_t)d, dh = (uint64_t)(d >> 64);
  w[1] = (uint64_t)b;
  w[2] = (uint32_t)bh | cl << 32;
  w[3] = cl >> 32 | ch << 32;
  w[4] = HALF ? (ch >> 32 & 0xffffu) | dl << 16 : dl;
  w[5] = HALF ? dl >> 48 | dh << 16 : dh;
}

// a += v - u over the 384 bits of a half
__device__ __forceinline__ void add_diff384(uint64_t (&a)[6], const uint64_t (&v)[6],
                                            const uint64_t (&u)[6]) {
  asm("add.cc.u64 %0, %0, %6;\n\t"
      "addc.cc.u64 %1, %1, %7;\n\t"
      "addc.cc.u64 %2, %2, %8;\n\t"
      "addc.cc.u64 %3, %3, %9;\n\t"
      "addc.cc.u64 %4, %4, %10;\n\t"
      "addc.u64 %5, %5, %11;"
      : "+&l"(a[0]), "+&l"(a[1]), "+&l"(a[2]), "+&l"(a[3]), "+&l"(a[4]), "+&l"(a[5])
      : "l"(v[0]), "l"(v[1]), "l"(v[2]), "l"(v[3]), "l"(v[4]), "l"(v[5]));
  asm("sub.cc.u64 %0, %0, %6;\n\t"
      "subc.cc.u64 %1, %1, %7;\n\t"
      "subc.cc.u64 %2, %2, %8;\n\t"
      "subc.cc.u64 %3, %3, %9;\n\t"
      "subc.cc.u64 %4, %4, %10;\n\t"
      "subc.u64 %5, %5, %11;"
      : "+&l"(a[0]), "+&l"(a[1]), "+&l"(a[2]), "+&l"(a[3]), "+&l"(a[4]), "+&l"(a[5])
      : "l"(u[0]), "l"(u[1]), "l"(u[2]), "l"(u[3]), "l"(u[4]), "l"(u[5]));
}

// One lane's half of a target's moment sums over the rows [l, r) of its strips
template <bool NARROW>
struct HalfSums {
  u128 mo[NH];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int m = 0; m < NH; ++m) mo[m] = 0;
  }
  __device__ __forceinline__ void add(const void* P, uint32_t l, uint32_t r, bool side) {
    const u128* pl = static_cast<const u128*>(P) + NM * (size_t)l + NH * side;
    const u128* pr = static_cast<const u128*>(P) + NM * (size_t)r + NH * side;
#pragma unroll
    for (int m = 0; m < NH; m += 2) {
      uint64_t u[4], v[4];
      load32(pl + m, u);
      load32(pr + m, v);
      mo[m] += u128_of((int64_t)v[1], v[0]) - u128_of((int64_t)u[1], u[0]);
      mo[m + 1] += u128_of((int64_t)v[3], v[2]) - u128_of((int64_t)u[3], u[2]);
    }
  }
  __device__ __forceinline__ void moments_of(bool, u128 (&m)[NH]) const {
#pragma unroll
    for (int i = 0; i < NH; ++i) m[i] = mo[i];
  }
};
template <>
struct HalfSums<true> {
  uint64_t a[6];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 6; ++i) a[i] = 0;
  }
  // a half is 32 bytes at 32 x half of the row and 16 at 64 + 16 x half
  static __device__ __forceinline__ void load(const char* row, bool side, uint64_t (&w)[6]) {
    uint64_t q[4];
    load32(row + 32 * side, q);
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(row + 64 + 16 * side);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = q[i];
    w[4] = t.x;
    w[5] = t.y;
  }
  __device__ __forceinline__ void add(const void* P, uint32_t l, uint32_t r, bool side) {
    constexpr size_t ROW = 16 * ROW_CHUNKS<true>;
    uint64_t u[6], v[6];
    load(static_cast<const char*>(P) + ROW * l, side, u);
    load(static_cast<const char*>(P) + ROW * r, side, v);
    add_diff384(a, v, u);
  }
  // a negative field borrowed one from the field above it
  __device__ __forceinline__ void moments_of(bool side, u128 (&m)[NH]) const {
    const int cb = side ? 48 : 32;  // bits of the third field above its first 64
    const uint64_t cl = a[2] >> 32 | a[3] << 32, cm = a[3] >> 32 | a[4] << 32;
    const uint64_t dm = a[4] >> 32 | a[5] << 32, dt = a[5] >> 32;
    const int64_t bh = (int32_t)(uint32_t)a[2];
    const int64_t ch = (int64_t)(cm << (64 - cb)) >> (64 - cb);
    const uint64_t dl = cm >> cb | dm << (64 - cb);
    int64_t dh = (int64_t)(dm >> cb | dt << (64 - cb));
    if (side) dh = (int64_t)((uint64_t)dh << 16) >> 16;
    const u128 f0 = (u128)(__int128)(int64_t)a[0];
    const u128 f1 = u128_of(bh, a[1]) + (a[0] >> 63);
    const u128 f2 = u128_of(ch, cl) + ((uint64_t)bh >> 63);
    const u128 f3 = u128_of(dh, dl) + ((uint64_t)ch >> 63);
    m[0] = side ? f1 : f0;
    m[1] = side ? f2 : f1;
    m[2] = side ? f3 : f2;
    m[3] = side ? f0 : f3;
  }
};

// 32 bytes in one store
__device__ __forceinline__ void store32(void* p, uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
  asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};"
               :: "l"(p), "l"(a), "l"(b), "l"(c), "l"(d)
               : "memory");
}

// a b modulo 2^128 for a signed 64-bit or a 128-bit a
__device__ __forceinline__ u128 mul_c(u128 a, u128 b) { return a * b; }
__device__ __forceinline__ u128 mul_c(int64_t a, u128 b) {
  const uint64_t ua = (uint64_t)a, bl = (uint64_t)b;
  const u128 p = (u128)ua * bl;
  const uint64_t hi = (uint64_t)(p >> 64) + ua * (uint64_t)(b >> 64) - (a < 0 ? bl : 0ull);
  return ((u128)hi << 64) | (uint64_t)p;
}

__device__ __forceinline__ u128 shfl_xor128(u128 v, int o) {
  const unsigned long long lo = __shfl_xor_sync(FULL_MASK, (unsigned long long)v, o);
  const unsigned long long hi = __shfl_xor_sync(FULL_MASK, (unsigned long long)(v >> 64), o);
  return ((u128)hi << 64) | lo;
}

// fixed-point image of a coordinate in the arithmetic of the coefficients
template <bool NARROW>
struct Coef {
  typedef u128 T;
  static __device__ __forceinline__ T of(float v) { return quant<23>(v); }
};
template <>
struct Coef<true> {
  typedef int64_t T;
  static __device__ __forceinline__ T of(float v) { return quant23_narrow(v); }
};

__device__ __forceinline__ double s128_to_double(u128 v) {
  const bool neg = (v >> 127) != 0;
  if (neg) v = (u128)0 - v;
  const double d = __ull2double_rn((unsigned long long)(v >> 64)) * 18446744073709551616.0 +
                   __ull2double_rn((unsigned long long)v);
  return neg ? -d : d;
}

// ---------------------------------------------- log of an exact 128-bit sum
// The per-point log of the strip-moment epilogue without the FP64 pipe (it
// runs at a small fraction of the FP32 rate on this GPU): the target's sum is
// one exact nonnegative integer T (units of 2^-92 g^4), and log T is formed in
// 64-bit fixed point with 2^-48 resolution. T = m 2^p with m in [1, 2) taken
// from T's top 48 bits; the top 8 bits of m after the leading one pick a table
// entry {inv ~ 1/c, log(1/inv) in 2^-56 fixed point}, c = 1 + (k + 1/2)/256
// (the table is made on the host with its libm); r = m inv - 1 is formed
// exactly as a float-float pair rh + rl (|r| < 2^-8, |rl| < 2^-22),
// log1p(r) = r - r^2/2 + r^3/3 - r^4/4 + r^5/5 with rh^2 as an exact FP32
// product pair and the rl cross terms to r^3, and
//   log T = p ln 2 + log(1/inv) + log1p(r),
// every part added in fixed point. Error below 2^-45 (2.9e-14) absolute: the
// 48-bit truncation of T, the rounding of rl and of the fixed-point parts.
constexpr int64_t LN2_FX56 = 49946518145322874LL;  // round(ln 2 * 2^56)

// round(x 2^48) of a float with |x| < 1
__device__ __forceinline__ int64_t f32_to_fx48(float x) {
  const uint32_t b = __float_as_uint(x);
  const int e = (int)((b >> 23) & 0xffu);
  if (e == 0) return 0;
  const int64_t m = (int64_t)((b & 0x7fffffu) | 0x800000u);
  const int sh = e - 102;  // x 2^48 = m 2^(e - 150 + 48)
  int64_t q;
  if (sh >= 0) q = m << sh;
  else if (sh > -25) q = (m + (1LL << (-sh - 1))) >> (-sh);
  else q = 0;
  return (b & 0x80000000u) ? -q : q;
}

// (hi, lo) += m 2^sh rounded to an integer, m < 2^53 (the fixed-point image
// of a nonnegative float or double; two 64-bit words, no 128-bit shifts)
__device__ __forceinline__ void add_shifted(uint64_t m, int sh, uint64_t& lo, uint64_t& hi) {
  uint64_t a = 0, b = 0;  // low and high word of the addend
  if (sh >= 64) {
    b = m << (sh - 64);
  } else if (sh > 0) {
    a = m << sh;
    b = m >> (64 - sh);
  } else if (sh == 0) {
    a = m;
  } else if (sh > -54) {
    a = (m + (1ull << (-sh - 1))) >> (-sh);
  }
  lo += a;
  hi += b + (lo < a ? 1ull : 0ull);
}

// += round(v 2^92) for a finite float v >= 0 below 2^30
__device__ __forceinline__ void add_fx92_f32(float v, uint64_t& lo, uint64_t& hi) {
  const uint32_t b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 0xffu);
  if (e == 0 || (b >> 31)) return;
  add_shifted((uint64_t)((b & 0x7fffffu) | 0x800000u), e - 150 + 92, lo, hi);
}

// += round(v 2^92) for a finite double v >= 0 below 2^30
__device__ __forceinline__ void add_fx92_f64(double v, uint64_t& lo, uint64_t& hi) {
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  const int e = (int)((b >> 52) & 0x7ffu);
  if (e == 0 || (b >> 63)) return;
  add_shifted((b & 0xfffffffffffffull) | (1ull << 52), e - 1075 + 92, lo, hi);
}

// log(T) in 2^-48 fixed point of T = hi 2^64 + lo > 0
__device__ __forceinline__ int64_t ilog_fx48(uint64_t lo, uint64_t hi,
                                             const ILogEntry* __restrict__ tab) {
  if ((lo | hi) == 0) return -(1LL << 62);  // never for a density: its own term is > 0
  const int p = hi ? 127 - __clzll((long long)hi) : 63 - __clzll((long long)lo);
  const int s = p - 47;  // m48 = floor(T / 2^s), in [2^47, 2^48)
  uint64_t m48;
  if (s >= 64) m48 = hi >> (s - 64);
  else if (s > 0) m48 = (hi << (64 - s)) | (lo >> s);
  else m48 = lo << (-s);
  const uint32_t k = (uint32_t)(m48 >> 39) & 255u;
  const ILogEntry t = tab[k];
  // m = mh + ml exactly (24 + 24 bits)
  const float mh = __uint_as_float(0x3f800000u | (uint32_t)((m48 >> 24) & 0x7fffffu));
  const float ml = __fmul_rn(__uint2float_rn((uint32_t)(m48 & 0xffffffu)), 0x1p-47f);
  const float p1 = __fmul_rn(mh, t.inv);
  const float e1 = __fmaf_rn(mh, t.inv, -p1);  // mh inv = p1 + e1 exactly
  const float rh = __fsub_rn(p1, 1.0f);        // exact: p1 in [1/2, 2]
  const float rl = __fmaf_rn(ml, t.inv, e1);
  const float qh = __fmul_rn(rh, rh);
  const float qe = __fmaf_rn(rh, rh, -qh);     // rh^2 = qh + qe exactly
  // two-sum of rh and -qh/2
  const float b2 = __fmul_rn(-0.5f, qh);
  const float sh = __fadd_rn(rh, b2);
  const float bb = __fsub_rn(sh, rh);
  const float err = __fadd_rn(__fsub_rn(rh, __fsub_rn(sh, bb)), __fsub_rn(b2, bb));
  const float h3 = __fmul_rn(__fmul_rn(rh, qh),
                             __fmaf_rn(rh, __fmaf_rn(rh, 0.2f, -0.25f), 1.0f / 3.0f));
  // the small rest: rounding of the two-sum and the cross terms of r^2/2 and
  // r^3/3 with rl (-rh rl + rh^2 rl); rl itself is added on its own
  const float rest = __fadd_rn(__fadd_rn(err, __fmaf_rn(-0.5f, qe, h3)),
                               __fmul_rn(rl, __fsub_rn(qh, rh)));
  int64_t fx = ((int64_t)p * LN2_FX56 + 128) >> 8;
  fx += (t.l56 + 128) >> 8;
  fx += f32_to_fx48(sh) + f32_to_fx48(rl) + f32_to_fx48(rest);
  return fx;
}

// y extent (smallest, largest scaled y) of every strip: one warp per strip, and the
// whole block over its strips of more than YB_LONG points, of which crowded data
// has a few of tens of thousands: MI 16 x 100k 3.21 -> 3.13 ms, 12 x 60k 1.177 ->
// 1.151 ms (lines at 1,024 and 4,096 points alike); 64 x 100k reads 1.6 GB in 0.25 ms.
constexpr uint32_t YB_LONG = 1024;
__device__ __forceinline__ void warp_min_max(float& lo, float& hi) {
  for (int o = 16; o; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(FULL_MASK, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(FULL_MASK, hi, o));
  }
}
// over the points a + first, a + first + step, ... below b, eight loads in flight
// (past the end the strip's last point again)
__device__ __forceinline__ void y_extent(const float2* __restrict__ pts, uint32_t a, uint32_t b,
                                         uint32_t first, uint32_t step, float& lo, float& hi) {
  for (uint32_t k = a + first; k < b; k += 8 * step) {
    float y[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) y[u] = pts[min(k + step * u, b - 1)].y;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      lo = fminf(lo, y[u]);
      hi = fmaxf(hi, y[u]);
    }
  }
}
__global__ void __launch_bounds__(256) k_m2_ybounds(const Mom2D* __restrict__ ms) {
  __shared__ float2 part[8];
  const Mom2D& M = ms[blockIdx.y];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t s0 = blockIdx.x * 8;
  for (uint32_t s = s0; s < min(s0 + 8, M.n_strips); ++s) {  // block-uniform
    const uint32_t a = M.strip_start[s], b = M.strip_start[s + 1];
    const bool all = b - a > YB_LONG;
    if (!all && s != s0 + warp) continue;
    float lo = 3.4e38f, hi = -3.4e38f;
    y_extent(M.pts, a, b, all ? threadIdx.x : lane, all ? 256 : 32, lo, hi);
    warp_min_max(lo, hi);
    if (all) {
      if (lane == 0) part[warp] = make_float2(lo, hi);
      __syncthreads();
      if (warp == 0) {
        lo = part[lane & 7].x;
        hi = part[lane & 7].y;
        warp_min_max(lo, hi);
      }
      __syncthreads();
    }
    if (lane == 0 && (all ? warp == 0 : true)) M.ybound[s] = make_float2(lo, hi);
  }
}

// Block scan helper: exclusive prefix of v (per thread) over the block, and
// the block total; sw holds NM u128 per warp.
__device__ __forceinline__ void block_scan8(u128 (&v)[NM], u128 (&excl)[NM],
                                            u128 (*sw)[NM]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u128 inc[NM];
#pragma unroll
  for (int m = 0; m < NM; ++m) inc[m] = v[m];
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      const u128 u = shfl_up128(inc[m], o);
      if (lane >= o) inc[m] += u;
    }
  }
  if (lane == 31)
#pragma unroll
    for (int m = 0; m < NM; ++m) sw[warp][m] = inc[m];
  __syncthreads();
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    u128 base = inc[m] - v[m];
    for (int w = 0; w < warp; ++w) base += sw[w][m];
    excl[m] = base;
  }
}

// chunk totals of the eight moments
template <bool NARROW>
__global__ void __launch_bounds__(M2_PT)
    k_m2_totals(const Mom2D* __restrict__ ms, u128* __restrict__ tot) {
  __shared__ u128 sw[M2_PT / 32][NM];
  const Mom2D& M = ms[blockIdx.y];
  const uint64_t b0 = (uint64_t)blockIdx.x * M2_CHUNK;
  if (b0 >= M.n) return;  // block-uniform
  const uint64_t k0 = b0 + (uint64_t)threadIdx.x * M2_E;
  float2 pt[M2_E];
  const uint32_t ne = load_points8(M.pts, k0, M.n, pt);
  u128 s[NM];
#pragma unroll
  for (int m = 0; m < NM; ++m) s[m] = 0;
#pragma unroll
  for (uint32_t e = 0; e < M2_E; ++e)
    if (e < ne) {
      u128 q[NM];
      moments<NARROW>(pt[e], q);
#pragma unroll
      for (int m = 0; m < NM; ++m) s[m] += q[m];
    }
  // block total: warp sums, then the warps in order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    for (int o = 16; o; o >>= 1) {
      const unsigned long long lo = __shfl_xor_sync(FULL_MASK, (unsigned long long)s[m], o);
      const unsigned long long hi = __shfl_xor_sync(FULL_MASK, (unsigned long long)(s[m] >> 64), o);
      s[m] += ((u128)hi << 64) | lo;
    }
    if (lane == 0) sw[warp][m] = s[m];
  }
  __syncthreads();
  if (threadIdx.x < NM) {
    u128 t = 0;
    for (uint32_t w = 0; w < M2_PT / 32; ++w) t += sw[w][threadIdx.x];
    tot[NM * ((size_t)M.chunk_base + blockIdx.x) + threadIdx.x] = t;
  }
}

// one warp per instance: exclusive scan of its chunk totals, in place
__global__ void k_m2_chunks(const Mom2D* __restrict__ ms, uint32_t n_inst,
                            u128* __restrict__ tot) {
  const uint32_t q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (q >= n_inst) return;  // warp-uniform
  const uint32_t nch = (ms[q].n + M2_CHUNK - 1) / M2_CHUNK;
  u128* t = tot + NM * (size_t)ms[q].chunk_base;
  for (int m = 0; m < NM; ++m) {
    u128 run = 0;
    for (uint32_t b = 0; b < nch; b += 32) {
      const bool in = b + lane < nch;
      const u128 v = in ? t[NM * (b + lane) + m] : (u128)0;
      u128 inc = v;
      for (int o = 1; o < 32; o <<= 1) {
        const u128 u = shfl_up128(inc, o);
        if (lane >= o) inc += u;
      }
      if (in) t[NM * (b + lane) + m] = run + inc - v;
      run += shfl_idx128(inc, 31);
    }
  }
}

// P[k] = sum_{j<k} moments(pts[j]), k = 0..n. Each thread sums M2_E
// consecutive points. Narrow rows are stored by their lane, three 32-byte
// stores; wide rows of one e (point k0 + e of every lane) pass through shared
// memory, so that every store instruction writes four whole 128-byte rows. Wide
// rows are bound by their way to HBM (64 x 100k: 25.8 GB in 4.6 ms at 3 blocks
// per SM, 5.5 ms at 2 or 4), narrow ones by the LSU (79 % busy: every lane writes
// to another line; 19.3 GB in 4.6 ms; staged like the wide ones 4.9 ms).
template <bool NARROW>
__global__ void __launch_bounds__(M2_PT, 3)
    k_m2_write(const Mom2D* __restrict__ ms, const u128* __restrict__ off) {
  __shared__ u128 sw[M2_PT / 32][NM];
  constexpr int RC = ROW_CHUNKS<NARROW>;
  const Mom2D& M = ms[blockIdx.y];
  const uint64_t b0 = (uint64_t)blockIdx.x * M2_CHUNK;
  if (b0 >= M.n) return;  // block-uniform
  const uint64_t k0 = b0 + (uint64_t)threadIdx.x * M2_E;
  u128 s[NM], run[NM];
#pragma unroll
  for (int m = 0; m < NM; ++m) s[m] = 0;
  for (uint32_t e = 0; e < M2_E; ++e)
    if (k0 + e < M.n) {
      u128 q[NM];
      moments<NARROW>(M.pts[k0 + e], q);
#pragma unroll
      for (int m = 0; m < NM; ++m) s[m] += q[m];
    }
  block_scan8(s, run, sw);
  const u128* o = off + NM * ((size_t)M.chunk_base + blockIdx.x);
#pragma unroll
  for (int m = 0; m < NM; ++m) run[m] += o[m];
  u128* P = static_cast<u128*>(M.P);
  if (b0 == 0 && threadIdx.x == 0)
#pragma unroll
    for (int m = 0; m < RC; ++m) P[m] = 0;
  if constexpr (NARROW) {
    float2 p[2];
#pragma unroll
    for (uint32_t e = 0; e < M2_E; ++e) {
      if (k0 + e >= M.n) return;
      if (e % 2 == 0) load_pair(M.pts, k0 + e, M.n, p);
      u128 q[NM];
      moments<true>(p[e % 2], q);
#pragma unroll
      for (int m = 0; m < NM; ++m) run[m] += q[m];
      uint64_t a[6], b[6];
      pack_half<0>(run, a);
      pack_half<1>(run, b);
      u128* row = P + RC * (k0 + e + 1);
      store32(row, a[0], a[1], a[2], a[3]);
      store32(row + 2, b[0], b[1], b[2], b[3]);
      store32(row + 4, a[4], a[5], b[4], b[5]);
    }
  } else {
    __shared__ u128 stage[M2_PT / 32][32 * NM];  // one row per lane, chunks swizzled
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u128* st = stage[warp];
    // the warp's first point; lane r's rows are points wk0 + 8 r + e
    const uint64_t wk0 = b0 + (uint64_t)(warp * 32) * M2_E;
    for (uint32_t e = 0; e < M2_E; ++e) {
      if (k0 + e < M.n) {
        u128 q[NM];
        moments<false>(M.pts[k0 + e], q);
#pragma unroll
        for (int m = 0; m < NM; ++m) {
          run[m] += q[m];
          st[lane * NM + (m ^ (lane & 7))] = run[m];
        }
      }
      __syncwarp();
      // 8 lanes per row: chunk c of row r = 4 i + lane / 8
      const int c = lane & 7;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = 4 * i + (lane >> 3);
        const uint64_t k = wk0 + (uint64_t)r * M2_E + e;
        if (k < M.n) P[NM * (k + 1) + c] = st[r * NM + (c ^ (r & 7))];
      }
      __syncwarp();
    }
  }
}

// In support means fma(-d, d, g^2) > 0, d = fl(a - b), as in the pair kernels: the
// fma rounds a difference whose sign is exact, so it is |d| < sup (Mom2D::sup).

// acc + wx wy for one source p of target t (x inside the support)
__device__ __forceinline__ float pair_term(float2 p, float2 t, float g1, float g2, float acc) {
  const float dx = __fsub_rn(p.x, t.x), dy = __fsub_rn(p.y, t.y);
  const float wy = __saturatef(__fmaf_rn(-dy, dy, g2));
  return __fmaf_rn(__fmaf_rn(-dx, dx, g1), wy, acc);
}

// x-support of a target at tx in the x-sorted points of one strip, searched
// in [lo, hi) with the pair kernels' own test (monotone in the position and
// in tx): the first position not left of the support, or the first one right of
// it. Left of it is d = fl(x - tx) <= -sup, not right of it d < sup; as one
// comparison d < edge, edge = edge_of(sup, right). With the fma and the two cases in
// each of the six or seven steps of every strip, then / now: target kernel 64 x 100k
// MI 17.0 / 16.4 ms, 32 x 200k TE 41.9 / 40.1 ms; the y tests likewise 16.4 / 16.2 and
// 40.1 / 39.9 ms.
__device__ __forceinline__ float edge_of(float sup, bool right) {
  return right ? sup : -__uint_as_float(__float_as_uint(sup) - 1u);  // sup > 0
}
__device__ __forceinline__ uint32_t support_end(const float2* __restrict__ pts, uint32_t lo,
                                                uint32_t hi, float tx, float edge) {
  while (lo < hi) {
    const uint32_t m = lo + ((hi - lo) >> 1);
    if (__fsub_rn(pts[m].x, tx) < edge) lo = m + 1; else hi = m;
  }
  return lo;
}

// Pair-by-pair sums of the lanes' windows [l, r), every other source per lane
// from l + side on. Lanes without a window pass l = ~0, r = 0. Two forms, which add
// the same terms in the same order:
//  * windows of neighbouring targets lie over one another, and the warp stages 32
//    sources at a time, loaded one batch ahead, from the union of the windows: 103 ns
//    per batch (one warp alone on its SM);
//  * where they lie apart (targets of a sparse strip, or of several strips, beside
//    crowded ones) most of that union is in no window, and every lane reads its own
//    sources, eight at a time: 390 ns per sixteen of the longest window.
// They meet where the union is 3.8 times the longest window. 32 targets spread over
// the x-range of 600k sources, windows of 2,250 / 22,500: target kernel 5.4 / 5.4 ms
// staged, 0.16 / 1.1 by lanes; windows of three quarters of 200k sources 1.3 staged.
constexpr uint32_t M2_APART = 4;
__device__ __forceinline__ float scan_windows(const float2* __restrict__ pts, uint32_t l, uint32_t r,
                                              float2 t, float g1, float g2, bool side,
                                              float2* __restrict__ stage) {
  const int lane = threadIdx.x & 31;
  const uint32_t a = __reduce_min_sync(FULL_MASK, l), b = __reduce_max_sync(FULL_MASK, r);
  const uint32_t longest = __reduce_max_sync(FULL_MASK, l < r ? r - l : 0u);
  float own = 0.f;
  if ((b - a) / M2_APART > longest) {  // warp-uniform
#pragma unroll 1
    for (uint32_t k = l + side; k < r; k += 16) {
      float2 p[8];
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) p[u] = pts[min(k + 2 * u, r - 1)];
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) {
        const float v = pair_term(p[u], t, g1, g2, own);
        if (k + 2 * u < r) own = v;
      }
    }
    return own;
  }
  float2 next = pts[min(a + lane, b - 1)];
#pragma unroll 1
  for (uint32_t base = a; base < b; base += 32) {
    stage[lane] = next;
    __syncwarp();
    next = pts[min(base + 32 + lane, b - 1)];
    const uint32_t odd = (l + side - base) & 1;
#pragma unroll
    for (uint32_t i = 0; i < 32; i += 16) {
      float2 p[8];
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) p[u] = stage[odd + i + 2 * u];
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) {
        const float v = pair_term(p[u], t, g1, g2, own);
        if (base + odd + i + 2 * u - l < r - l) own = v;
      }
    }
    __syncwarp();
  }
  return own;
}

constexpr int M2_MAX_IN = 23;  // inside strips per target: 2S - 1, S <= 12

// A warp holds 32 consecutive sorted positions, in two rounds of 16 targets with
// two lanes each. The strips within S - 1 of the target's own strip are inside
// its y-support (checked per strip against the strip's y extent); the two strips
// at distance S, where the support's y edge falls, are summed pair by pair by
// the symmetric pair kernel beforehand (its FP64 sums arrive in M.acc).
//
// Two lanes per target: one searches the left end of its x-support, the other
// the right end, and each adds up four of the eight 128-bit moments, half a row
// in two 32-byte loads. The kernel waits on dependent loads, so it needs many
// warps; eight sums per lane are 32 of the 48 registers that 10 blocks per SM
// leave, and were kept in local memory, whose traffic (85 M of 131 M memory
// requests on 16 x 100k coordinates) held the kernel up as much as the rows.
// Four fit. Kernel times with wide rows, one / two lanes per target: 64 x 100k MI
// 22.9 / 20.5 ms, 32 x 200k TE at 3 lags 72.7 / 54.0 ms. 8 or 9 blocks per SM: 21.8
// ms; all strips' searches stepped together: 22.3 ms.
//
// Searches. When the warp's 32 targets lie in one strip they are x-sorted,
// and the support bounds in any other strip are monotone in the target's x.
// The warp first finds, for every inside strip at once (one bisection per
// lane), the bounds of its first and last target; each lane then searches
// only between them -- a range of about as many points as the warp's x-span
// holds, instead of the whole strip. Other warps (strip boundaries, the end
// of an instance) search each strip in full.
//
// Sums. The moment rows of all inside strips are added first and combined with
// the target's coefficients once,
//   T = c0 (d0 n + d1 M01 - M02) - d0 M20 + M22     (first lane)
//     + c1 (d0 M10 + d1 M11 - M12) - d1 M21         (second lane);
// strips whose y extent crosses the support (rounding at the widened cell
// edges only) are summed pair by pair, by the whole warp: one target next to a
// crowded strip has tens of thousands of sources, and its two lanes alone took
// 0.5 to 1 ms, after every other block had ended. Same terms in the same order.
// Kernel on 16 / 64 x 100k, two lanes / warp: 1.54 / 1.20, 17.7 / 17.1 ms (17.4
// with four instead of eight sources read ahead of a lane's sum). They follow both
// rounds of moment sums, whose registers they take: among the strips, with both
// forms of scan_windows, they spill 80 bytes (16 / 64 x 100k 1.16 / 17.0 ms, after
// each round 1.03 / 16.0, here 1.02 / 15.9).
//
// Epilogue as the other bodies' finish kernel: density = scale x sum,
// written by original index and/or logged (FP64) and summed per block of
// targets in a fixed order into the instance's slots of tile_logsum.
// LOGONLY: the log-sum epilogue alone (mode == DM_LOGSUM, the estimator
// batches), compiled without the FP64 density path of the other modes.
// NARROW: every coordinate of the instances lies below 2^8 in scaled units
// (MOMENT_NARROW), so a target's coefficients fit in 64 bits, and the moments
// come in narrow rows.
template <bool LOGONLY, bool NARROW>
__global__ void __launch_bounds__(M2_TB, M2_BPS<NARROW>)
    k_m2_density(const Mom2D* __restrict__ ms, uint32_t n_inst,
                 const uint32_t* __restrict__ blk_base, uint32_t blk0,
                 const ILogEntry* __restrict__ ilog, double* __restrict__ tile_logsum,
                 uint32_t mode) {
  __shared__ double s_part[M2_TB / 32];
  __shared__ long long s_fx[M2_TB / 32];
  // per warp and inside strip: [side] {lowest, highest} support end of the warp's
  // targets, and the strip's y extent
  __shared__ uint2 s_br[M2_TB / 32][M2_MAX_IN][2];
  __shared__ float2 s_yb[M2_TB / 32][M2_MAX_IN];
  __shared__ float2 s_pts[M2_TB / 32][32];  // sources staged by scan_windows
  __shared__ u128 s_T[M2_TB];   // the targets' exact sums of their inside strips
  __shared__ uint32_t s_cut[M2_TB];  // and the strips that their supports cut
  const uint32_t gb = blk0 + blockIdx.x;
  uint32_t lo = 0, hi = n_inst;
  while (hi - lo > 1) {
    const uint32_t m = (lo + hi) / 2;
    if (blk_base[m] <= gb) lo = m; else hi = m;
  }
  const Mom2D& M = ms[lo];
  const uint32_t blk = gb - M.blk_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool side = lane & 1;
  const uint32_t n = M.n, w0 = blk * M2_TB + warp * 32;  // the warp's first target
  const float2* __restrict__ pts = M.pts;
  const float supx = M.sup[0], supy = M.sup[1], edge = edge_of(supx, side);
  const int S = (int)M.S;
  const int s0 = (int)M.skeys[min(w0, n - 1)];
  const bool uni = w0 + 31 < n && (int)M.skeys[w0 + 31] == s0;  // strip-major order
  if (uni) {
    // bounds of the warp's first and last target in every inside strip
    for (int q = lane; q < 4 * (2 * S - 1); q += 32) {
      const int sp = s0 + q / 4 - (S - 1);
      uint32_t res = 0;
      if (sp >= 0 && sp < (int)M.n_strips) {
        const uint32_t a = M.strip_start[sp], b = M.strip_start[sp + 1];
        if (a < b) res = support_end(pts, a, b, pts[w0 + ((q & 1) ? 31 : 0)].x, edge_of(supx, q & 2));
        if ((q & 3) == 0) s_yb[warp][q / 4] = M.ybound[sp];
      }
      uint32_t* br = reinterpret_cast<uint32_t*>(&s_br[warp][q / 4][(q >> 1) & 1]);
      br[q & 1] = res;
    }
    __syncwarp();
  }
  // the sources [l, r) of target t (at k) in inside strip o, and whether all of its
  // y's are in the support
  auto sources = [&](uint32_t k, float2 t, int o, uint32_t& l, uint32_t& r) {
    // candidates for this lane's end: [a, b)
    uint32_t a = 0, b = 0;
    float2 yb = make_float2(0.f, 0.f);
    if (uni) {
      const uint2 br = s_br[warp][o][side];
      a = br.x;
      b = br.y;
      yb = s_yb[warp][o];
    } else {
      const int sp = (int)M.skeys[k] + o - (S - 1);
      if (sp >= 0 && sp < (int)M.n_strips) {
        a = M.strip_start[sp];
        b = M.strip_start[sp + 1];
        yb = M.ybound[sp];
      }
    }
    const float ylo = __fsub_rn(yb.x, t.y), yhi = __fsub_rn(yb.y, t.y);
    if (ylo >= supy || yhi <= -supy) a = b = 0;  // all out
    const uint32_t e = support_end(pts, a, b, t.x, edge);
    const uint32_t e2 = __shfl_xor_sync(FULL_MASK, e, 1);
    l = side ? e2 : e;
    r = side ? e : e2;
    return ylo > -supy && yhi < supy;
  };
#pragma unroll 1
  for (int round = 0; round < 2; ++round) {
    const uint32_t k = min(w0 + round * 16 + (lane >> 1), n - 1);
    const float2 t = pts[k];
    HalfSums<NARROW> hs;
    hs.zero();
    uint32_t cnt = 0, cut = 0;  // cut: strips that the support cuts
#pragma unroll 1
    for (int o = 0; o < 2 * S - 1; ++o) {
      uint32_t l, r;
      const bool whole = sources(k, t, o, l, r);
      if (l < r && whole) {
        hs.add(M.P, l, r, side);
        cnt += r - l;
      }
      if (l < r && !whole) cut |= 1u << o;
    }
    typedef typename Coef<NARROW>::T C;
    const C TX = Coef<NARROW>::of(t.x), TY = Coef<NARROW>::of(t.y);
    const C d0 = (C)M.G[1] - TY * TY, d1 = TY + TY;
    const C f0 = side ? TX + TX : (C)M.G[0] - TX * TX;  // c1, c0
    u128 m[NH];
    hs.moments_of(side, m);
    u128 part = mul_c(f0, mul_c(d0, side ? m[3] : (u128)cnt) + mul_c(d1, m[0]) - m[1]) -
                mul_c(side ? d1 : d0, m[2]);
    if (!side) part += m[3];
    part += shfl_xor128(part, 1);
    if (!side) {
      s_T[warp * 32 + round * 16 + (lane >> 1)] = part;
      s_cut[warp * 32 + round * 16 + (lane >> 1)] = cut;
    }
  }
  __syncwarp();
  float fs = 0.f;  // the pair-by-pair sum of the strips that the support cuts
  if (__any_sync(FULL_MASK, s_cut[threadIdx.x] != 0)) {
#pragma unroll 1
    for (int round = 0; round < 2; ++round) {
      const uint32_t k = min(w0 + round * 16 + (lane >> 1), n - 1);
      const float2 t = pts[k];
      const uint32_t cut = s_cut[warp * 32 + round * 16 + (lane >> 1)];
      float f = 0.f;
#pragma unroll 1
      for (uint32_t todo = __reduce_or_sync(FULL_MASK, cut); todo; todo &= todo - 1) {
        const int o = __ffs(todo) - 1;
        const bool scan = (cut >> o) & 1u;
        uint32_t l, r;
        sources(k, t, o, l, r);
        const float own = scan_windows(pts, scan ? l : ~0u, scan ? r : 0u, t, M.g2[0], M.g2[1],
                                       side, s_pts[warp]);
        f += own + __shfl_xor_sync(FULL_MASK, own, 1);
      }
      f = __shfl_sync(FULL_MASK, f, 2 * (lane & 15));
      if (lane >> 4 == round) fs = f;
    }
  }
  const uint32_t k = w0 + lane;
  const u128 T = s_T[threadIdx.x];
  double v = 0.0;     // DM_SUMV: this target's density
  long long fx = 0;   // DM_LOGSUM: log of this target's sum, 2^-48 fixed point
  if (k < n) {
    // the whole sum in units of 2^-92 g^4: the exact moment part, the
    // partial strips' and the edge strips' sums in fixed point
    uint64_t tlo = (uint64_t)T, thi = (uint64_t)(T >> 64);
    if (fs != 0.f) add_fx92_f32(fs, tlo, thi);
    if (M.acc) add_fx92_f64(M.acc[k], tlo, thi);
    if (!LOGONLY && (mode & (DM_WRITE_F64 | DM_SUMV))) {
      const double dens = M.scale * (s128_to_double(((u128)thi << 64) | tlo) * 0x1p-92);
      if (mode & DM_WRITE_F64) M.out[M.perm[k]] = dens;
      v = dens;
    }
    if (mode & DM_LOGSUM) fx = ilog_fx48(tlo, thi, ilog);
  }
  if (mode & DM_LOGSUM) {  // block-uniform: exact integer block sum
    for (int o = 16; o; o >>= 1) fx += __shfl_xor_sync(FULL_MASK, fx, o);
    if (lane == 0) s_fx[warp] = fx;
    __syncthreads();
    if (threadIdx.x == 0) {
      long long tsum = 0;
      for (uint32_t w = 0; w < M2_TB / 32; ++w) tsum += s_fx[w];
      const uint32_t nv = min(M2_TB, n - blk * M2_TB);
      // log density = log T + log(scale) - 92 log 2 = log T + M.logc
      tile_logsum[M.slot_base + blk] = (double)tsum * 0x1p-48 + (double)nv * M.logc;
    }
  } else if (!LOGONLY && (mode & DM_SUMV)) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    if (lane == 0) s_part[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double tsum = 0.0;
      for (uint32_t w = 0; w < M2_TB / 32; ++w) tsum += s_part[w];
      tile_logsum[M.slot_base + blk] = tsum;
    }
  }
}

// Self-test of ilog_fx48 on 128-bit inputs given as (low, high) words.
__global__ void k_ilog_test(const unsigned long long* __restrict__ t, size_t n,
                            const ILogEntry* __restrict__ tab, long long* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = ilog_fx48(t[2 * i], t[2 * i + 1], tab);
}

// One block per instance, one warp per sampled target (quantile (2w+1)/64 of
// dimension 0), a lane per sampled point of its window: the two bisections of
// the window and two gathers are all that a warp waits for.
__global__ void __launch_bounds__(1024)
    k_support_est(const SupportEst* __restrict__ in, float* __restrict__ est) {
  __shared__ float sk[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SupportEst& E = in[blockIdx.x];
  const uint32_t n = E.n;
  const uint32_t pos = (uint32_t)(((2ull * warp + 1) * n) / 64);
  const float xt = key_float(E.keys0[pos]);
  const float yt = E.y1[E.perm0[pos]];
  // window [lo, hi) of dimension 0 within h0 of xt: an end per lane parity
  const bool right = lane & 1;
  const float edge = right ? xt + E.h0 : xt - E.h0;
  uint32_t a = 0, b = n;
  while (a < b) {
    const uint32_t m = a + ((b - a) >> 1);
    const float x = key_float(E.keys0[m]);
    if (right ? x < edge : x <= edge) a = m + 1; else b = m;
  }
  const uint32_t lo = __shfl_sync(FULL_MASK, a, 0), hi = max(lo, __shfl_sync(FULL_MASK, a, 1));
  const uint32_t c = hi - lo;
  const uint32_t ns = min(c, 32u);
  bool in_y = false;
  if ((uint32_t)lane < ns) {
    const uint32_t p = lo + (uint32_t)(((uint64_t)lane * c) / ns);
    in_y = fabsf(E.y1[E.perm0[p]] - yt) < E.h1;
  }
  const uint32_t cnt = __popc(__ballot_sync(FULL_MASK, in_y));
  if (lane == 0) sk[warp] = ns ? (float)c * (float)cnt / (float)ns : 0.f;
  __syncthreads();
  if (warp == 0) {
    float k = sk[lane];
    for (int o = 16; o; o >>= 1) k += __shfl_xor_sync(FULL_MASK, k, o);
    if (lane == 0) est[blockIdx.x] = k / 32.f;
  }
}

}  // namespace

cudaError_t launch_support_est(cudaStream_t st, const SupportEst* in, uint32_t n_inst,
                               float* est) {
  if (n_inst == 0) return cudaSuccess;
  k_support_est<<<n_inst, 1024, 0, st>>>(in, est);
  return cudaGetLastError();
}

uint32_t moments2d_chunks(uint32_t n) { return (n + M2_CHUNK - 1) / M2_CHUNK; }
uint32_t moments2d_blocks(uint32_t n) { return (n + M2_TB - 1) / M2_TB; }
float support_edge(float g2) {
  // d d is exact in FP64
  float d = std::sqrt(g2);
  while (d > 0.f && (double)d * d >= (double)g2) d = std::nextafter(d, 0.f);
  while ((double)d * d < (double)g2) d = std::nextafter(d, 2.f);
  return d;
}
size_t moments2d_prefix_bytes(uint32_t n, bool narrow) {
  return 16 * (size_t)(narrow ? ROW_CHUNKS<true> : ROW_CHUNKS<false>) * ((size_t)n + 1);
}

cudaError_t launch_moments2d_prefix(cudaStream_t st, const Mom2D* ms, uint32_t n_inst,
                                    uint32_t n_narrow, uint32_t max_n, uint32_t max_strips,
                                    void* chunk_tot) {
  if (n_inst == 0) return cudaSuccess;
  u128* tot = static_cast<u128*>(chunk_tot);
  k_m2_ybounds<<<dim3((max_strips + 7) / 8, n_inst), 256, 0, st>>>(ms);
  const unsigned gx = moments2d_chunks(std::max(max_n, 1u));
  const dim3 gn(gx, n_narrow), gw(gx, n_inst - n_narrow);
  if (gn.y) k_m2_totals<true><<<gn, M2_PT, 0, st>>>(ms, tot);
  if (gw.y) k_m2_totals<false><<<gw, M2_PT, 0, st>>>(ms + n_narrow, tot);
  k_m2_chunks<<<(n_inst + 3) / 4, 128, 0, st>>>(ms, n_inst, tot);
  if (gn.y) k_m2_write<true><<<gn, M2_PT, 0, st>>>(ms, tot);
  if (gw.y) k_m2_write<false><<<gw, M2_PT, 0, st>>>(ms + n_narrow, tot);
  return cudaGetLastError();
}

cudaError_t launch_moments2d_targets(cudaStream_t st, const Mom2D* ms, uint32_t n_inst,
                                     uint32_t n_narrow, const uint32_t* blk_base,
                                     uint32_t narrow_blocks, uint32_t n_blocks,
                                     const ILogEntry* ilog, double* tile_logsum, uint32_t mode) {
  if (n_inst == 0 || n_blocks == 0) return cudaSuccess;
  const uint32_t nw = n_inst - n_narrow, wide = n_blocks - narrow_blocks;
  const Mom2D* mw = ms + n_narrow;
  const uint32_t* bw = blk_base + n_narrow;
  if (mode == DM_LOGSUM) {
    if (n_narrow)
      k_m2_density<true, true><<<narrow_blocks, M2_TB, 0, st>>>(ms, n_narrow, blk_base, 0, ilog,
                                                                tile_logsum, mode);
    if (nw)
      k_m2_density<true, false><<<wide, M2_TB, 0, st>>>(mw, nw, bw, narrow_blocks, ilog,
                                                        tile_logsum, mode);
  } else {
    if (n_narrow)
      k_m2_density<false, true><<<narrow_blocks, M2_TB, 0, st>>>(ms, n_narrow, blk_base, 0, ilog,
                                                                 tile_logsum, mode);
    if (nw)
      k_m2_density<false, false><<<wide, M2_TB, 0, st>>>(mw, nw, bw, narrow_blocks, ilog,
                                                         tile_logsum, mode);
  }
  return cudaGetLastError();
}

cudaError_t launch_ilog_test(cudaStream_t st, const unsigned long long* t, size_t n,
                             const ILogEntry* tab, long long* out) {
  if (n == 0) return cudaSuccess;
  const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 4096);
  k_ilog_test<<<blocks, 256, 0, st>>>(t, n, tab, out);
  return cudaGetLastError();
}

}  // namespace ent
