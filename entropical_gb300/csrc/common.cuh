// Shared device helpers for the entropical GB300 kernels (sm_103a only).
//
// - mbarrier + cp.async.bulk (TMA bulk copy) wrappers with bounded waits:
//   every wait gives up after ENT_WAIT_NS nanoseconds, raises a bit in the
//   device error word and lets the kernel drain and return, so a stuck copy
//   can never hang the GPU.
// - packed f32x2 arithmetic (add/sub/fma .f32x2, sm_100+ family): two FP32
//   lanes per instruction, used to halve issue slots in the pair loops.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#ifndef __CUDACC__
#error "compile with nvcc"
#endif

namespace ent {

// Device error word bits (read back by the host after each call).
enum : uint32_t {
  EF_TIMEOUT = 1u,     // a bounded mbarrier / queue wait gave up
  EF_NONFINITE = 2u,   // NaN or Inf met in an input coordinate
  EF_CAPACITY = 4u,    // a tile needed more run slots than allocated
};

constexpr unsigned long long ENT_WAIT_NS = 2000000000ull;  // 2 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(count)
               : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar,
                                                      uint32_t bytes) {
  asm volatile(
      "{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], "
      "%1; }" ::"r"(smem_u32(bar)),
      "r"(bytes)
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; "
      "selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for the phase with the given parity to complete, for at most
// ENT_WAIT_NS. Returns false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer();
  for (uint32_t it = 0; it < (1u << 26); ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && globaltimer() - t0 > ENT_WAIT_NS) return false;
  }
  return false;
}

// Bulk (non-tensor) TMA copy global -> shared, completion counted on `bar`.
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src,
                                         uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], "
      "[%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// 16-byte asynchronous copies global -> shared of single threads
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Programmatic dependent launch: a kernel launched by launch_after() may start
// while its predecessor in the stream drains; grid_chain() returns once that one
// has completed and its writes are visible (at once after an ordinary launch).
// Every kernel of such a chain calls it before it touches memory.
__device__ __forceinline__ void grid_chain() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
cudaError_t launch_chain(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class... P, class... A>
cudaError_t launch_after(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block,
                         cudaStream_t st, A... args) {
  return launch_chain(overlap, kernel, grid, block, 0, st, args...);
}

// ---------------------------------------------------------------- f32x2
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0,%1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Kahan-compensated FP32 accumulation of a partial sum x into (s, c).
__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
  const float y = __fsub_rn(x, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(__fsub_rn(t, s), y);
  s = t;
}

// float -> double by re-biasing the IEEE-754 fields on the integer pipes
// (exact for normal floats; zero and subnormals give 0). The FP64 pipe of
// this GPU runs at a small fraction of the FP32 rate, so conversions on the
// hot path avoid it. Inputs must be finite.
__device__ __forceinline__ double f32_to_f64_int(float v) {
  const uint32_t b = __float_as_uint(v);
  const uint32_t e = (b >> 23) & 0xffu;
  if (e == 0) return 0.0;
  const uint64_t r = ((uint64_t)(b & 0x80000000u) << 32) |
                     ((uint64_t)(e + (1023u - 127u)) << 52) |
                     ((uint64_t)(b & 0x7fffffu) << 29);
  return __longlong_as_double((long long)r);
}

// Table entry of the epilogues' logs: inv ~ 1/c, c = 1 + (k + 1/2)/256, and
// log(1/inv) in 2^-56 fixed point (made on the host with its libm).
struct ILogEntry {
  float inv;
  float pad;
  long long l56;
};
constexpr int ILOG_TABLE_ENTRIES = 256;

// log of a positive normal double x = m 2^e, m = M 2^-52 in [1, 2), for the
// per-point epilogues: returns log(m) in 2^-56 fixed point, e in *e. Integer
// arithmetic, because the FP64 pipe of this GPU runs at 1/64 of the FP32 rate:
// the 12 FP64 operations of a table-reduced FP64 log bound the finish kernel.
// The top 8 bits of m pick the table entry (Tang's method); inv = J 2^-24 with a
// 24-bit J, so r = m inv - 1 (|r| < 2^-8.9) is an exact 77-bit integer, kept to
// 2^-63; log1p(r) = r - r^2/2 + r^3/3 in fixed point and r^4 (-1/4 + r/5 - r^2/6
// + r^3/7), below 2^-37, in FP32. Error below 2^-54 (the FP64 form's was 2^-51).
__device__ __forceinline__ long long log_fx56(double x, const ILogEntry* __restrict__ tab, int* e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  *e = (int)(b >> 52) - 1023;
  const unsigned long long M = (b & 0xfffffffffffffull) | (1ull << 52);
  const ILogEntry t = tab[(unsigned)(M >> 44) & 255u];
  const unsigned long long J = (__float_as_uint(t.inv) & 0x7fffffu) | 0x800000u;
  // m inv = M J 2^-76; r in units of 2^-63
  const long long r = (long long)(((__umul64hi(M, J) << 51) | ((M * J) >> 13)) - (1ull << 63));
  const long long r2 = __mul64hi(r, r);   // r^2 2^62
  const long long r3 = __mul64hi(r2, r);  // r^3 2^61
  const float rf = __fmul_rn((float)(int)(r >> 24), 0x1p-39f);
  const float rs = __fmul_rn(rf, rf);
  const float q = __fmul_rn(
      __fmul_rn(rs, rs),
      __fmaf_rn(rf, __fmaf_rn(rf, __fmaf_rn(rf, 1.f / 7.f, -1.f / 6.f), 0.2f), -0.25f));
  // 192153584101141163 = round(2^64 / 96): r^3/3 from 2^-61 to 2^-56 units
  return t.l56 + (r >> 7) - (r2 >> 7) + __mul64hi(r3, 192153584101141163ll) +
         (long long)__float2int_rn(__fmul_rn(q, 0x1p56f));
}

// whether log_fx56 takes x (the self term makes every density positive)
__device__ __forceinline__ bool log_normal(double x) {
  const unsigned ex = (unsigned)((unsigned long long)__double_as_longlong(x) >> 52);
  return ex != 0u && ex < 0x7ffu;
}
constexpr double LN2 = 0.693147180559945309417232;

// Orderable 32-bit key of a float: unsigned compare == float compare
// (-0.0 sorts just before +0.0; NaN never reaches here).
__device__ __forceinline__ uint32_t float_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float key_float(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, sizeof(f));
  return f;
#endif
}

}  // namespace ent
