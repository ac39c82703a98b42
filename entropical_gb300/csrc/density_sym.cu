// Symmetric pair kernel: every unordered (target, source) pair inside the
// candidate runs is evaluated once and added to both points.
//
// The reference sums, for every target i, K(x_i - x_k) over all k
// (densities_omp.cpp:67-159, density_2d.cuh:34-100); the product kernel is
// symmetric, K(x_i - x_k) == K(x_k - x_i) bit for bit (x_i - x_k is the exact
// negation of x_k - x_i), so each pair can serve both sums. The tile plan
// (k_plan with InstDev::sym) keeps, for a tile of targets [tb, tb + tc) in
// strip-major order, only the sources at positions >= tb:
//   * sources in [tb, tb + tc) (the tile itself) are evaluated in both orders
//     and added on the target side only;
//   * sources at >= tb + tc are added to the target (registers) and to the
//     source: each warp stores its per-source sum over its R targets in its
//     own shared-memory row (one float per staged element); once per chunk
//     the four rows are added in a fixed order and flushed into the FP64
//     sums InstDev::acc, so the FP32 part of every sum is deterministic;
//   * a source before tb belongs to an earlier tile, which evaluates the pair.
// Target-side sums are flushed into the same FP64 array once per chunk (warp
// transpose-sum, one FP64 atomic per target), so no per-target compensation
// state is carried and a warp can hold 32 targets. k_sym_finish scales the
// sums and writes densities or per-tile log-sums.
//
// Every mbarrier wait is bounded; on expiry the kernel reports EF_TIMEOUT,
// waits (bounded) for its own copies in flight and returns.
#include <algorithm>

#include "staging.cuh"

namespace ent {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// Staged elements per chunk; shared memory per CTA = chunk buffers x 2 plus
// one float row per warp (NW x CAP floats). 4 warps: 51 KB (d = 1, 2) and
// 38 KB (d = 3), 4 resp. 5 CTAs per SM; 8 warps: 44 / 51 / 34 KB, 3 CTAs.
template <int D, int NW>
struct SymChunk {
  static constexpr int CH = NW == 4 ? (D == 1 ? 2048 : (D == 2 ? 1536 : 768))
                                    : (D == 1 ? 1024 : (D == 2 ? 1024 : 512));
};

// LIST: the slots come from a work list: first its n_list[1] heavy ones, which lie
// from list_end on, in SYM_SHARES shares of every SYM_SHARES-th chunk (a chunk's
// sums do not depend on who takes it), then the n_list[0] before list_end (a
// template, because the
// slot-ordered 3-D kernel took 611 ms instead of 602 on the 32 x 200k TE batch with
// the list behind a runtime test).
template <int D, int R, int MINB, int NW, bool LIST>
__global__ void __launch_bounds__(NW * 32, MINB)
    k_density_sym(const TileDesc* __restrict__ tiles, uint32_t n_slots,
                  const InstDev* __restrict__ insts, uint32_t* work_counter, uint32_t* err,
                  const uint32_t* __restrict__ list_end, const uint32_t* __restrict__ n_list) {
  typedef Cfg<D, R, SymChunk<D, NW>::CH, NW> C;
  typedef typename C::P P;
  static_assert(R <= 32 && (R & (R - 1)) == 0, "R: power of two <= 32");
  extern __shared__ __align__(128) unsigned char dsm[];
  P* bufs = reinterpret_cast<P*>(dsm);
  float* srow = reinterpret_cast<float*>(dsm + C::SMEM);  // C::NW rows of CAP floats
  __shared__ __align__(8) uint64_t full[2];
  __shared__ Piece ptab[2][C::MAXP];
  __shared__ uint32_t npc[2];
  __shared__ uint32_t run_lo[MAX_RUNS], run_pre[MAX_RUNS + 1];
  __shared__ uint32_t s_g, s_nr, s_tb, s_tc, s_inst, s_c0, s_cs;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  float* myrow = srow + (size_t)warp * C::CAP;
  uint32_t q = 0;
  uint32_t n_shares = 0;  // of the heavy slots
  if constexpr (LIST) {
    n_shares = n_list[1] * SYM_SHARES;
    n_slots = n_shares + n_list[0];
  }

  for (;;) {
    if (tid == 0) {
      const uint32_t g = atomicAdd(work_counter, 1u);
      s_g = g;
      if (g < n_slots) {
        const TileDesc* T = tiles + g;
        if constexpr (LIST) {
          const bool heavy = g < n_shares;
          T = tiles + list_end[heavy ? (int64_t)(g / SYM_SHARES) : (int64_t)n_shares - 1 - g];
          s_c0 = heavy ? g % SYM_SHARES : 0;
          s_cs = heavy ? SYM_SHARES : 1;
        }
        const uint32_t nr = T->n_runs;
        s_tb = T->t_begin;
        s_tc = T->t_count;
        s_inst = T->inst;
        s_nr = nr;
        run_pre[0] = 0;
        for (uint32_t r = 0; r < nr; ++r) {
          run_lo[r] = T->lo[r];
          run_pre[r + 1] = run_pre[r] + T->len[r];
        }
      }
    }
    __syncthreads();
    const uint32_t g = s_g;
    if (g >= n_slots) break;
    const uint32_t tc = s_tc;
    if (tc == 0) {
      __syncthreads();
      continue;
    }
    const InstDev* I = insts + s_inst;
    const P* __restrict__ pts = reinterpret_cast<const P*>(I->pts);
    double* __restrict__ acc64 = I->acc;
    const uint32_t nr = s_nr, nsrc = run_pre[nr], tb = s_tb, tend = tb + tc;
    const float g2a = I->g2[0], g2b = I->g2[D > 1 ? 1 : 0], g2c = I->g2[D > 2 ? 2 : 0];
    const uint32_t nch = (nsrc + C::CH - 1) / C::CH;
    const uint32_t c0 = LIST ? s_c0 : 0, cs = LIST ? s_cs : 1;  // this share's chunks
    if (LIST && c0 >= nch) {  // a share without chunks
      __syncthreads();
      continue;
    }
    if (tid == 0 && c0 < nch)
      issue_chunk<C>(c0, q & 1u, nsrc, nr, run_lo, run_pre, pts, bufs, ptab, npc, full);

    // Register-resident targets of this warp; missing ones sit at +inf, where
    // every term is 0.
    const float FAR = __int_as_float(0x7f800000);
    f32x2 T01[D == 1 ? 1 : R];
    float T2[D == 2 ? 1 : R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t li = warp * R + r;
      P p;
      if (li < tc) {
        p = pts[tb + li];
      } else {
        if constexpr (D == 1) p = FAR;
        else if constexpr (D == 2) p = make_float2(FAR, FAR);
        else p = make_float4(FAR, FAR, FAR, 0.f);
      }
      if constexpr (D == 1) {
        T2[r] = p;
      } else if constexpr (D == 2) {
        T01[r] = pk2(p.x, p.y);
      } else {
        T01[r] = pk2(p.x, p.y);
        T2[r] = p.z;
      }
    }
    const int tgt = lane >> (5 - Log2<R>::v);
    const bool writer = (lane & ((32 / R) - 1)) == 0;
    const uint32_t my_li = warp * R + tgt;

    bool aborted = false;
    uint32_t ab_q = 0;
    bool ab_next = false;
    uint32_t qq = q;
    for (uint32_t c = c0; c < nch; c += cs, ++qq) {
      const uint32_t b = qq & 1u;
      if (tid == 0 && c + cs < nch)
        issue_chunk<C>(c + cs, (qq + 1) & 1u, nsrc, nr, run_lo, run_pre, pts, bufs, ptab,
                       npc, full);
      const bool ok = mbar_wait(&full[b], (qq >> 1) & 1u);
      float acc[R];
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = 0.f;
      if (ok) {
        const P* B = bufs + (size_t)b * C::CAP;
        const uint32_t np = npc[b];
        for (uint32_t pi = 0; pi < np; ++pi) {
          const uint32_t s0 = ptab[b][pi].s0, n = ptab[b][pi].n;
          if constexpr (D == 1) {
            f32x2 accp[R / 2];
            f32x2 T[R / 2];
#pragma unroll
            for (int i = 0; i < R / 2; ++i) {
              accp[i] = pk2(0.f, 0.f);
              T[i] = pk2(T2[2 * i], T2[2 * i + 1]);
            }
#pragma unroll 2
            for (uint32_t k = lane; k < n; k += 32) {
              const float s = B[s0 + k];
              const f32x2 S = pk2(s, s);
              f32x2 src0 = pk2(0.f, 0.f), src1 = pk2(0.f, 0.f);
#pragma unroll
              for (int i = 0; i < R / 2; ++i) {
                float da, db;
                upk2(sub2(T[i], S), da, db);
                const f32x2 w = pk2(__saturatef(__fmaf_rn(-da, da, g2a)),
                                    __saturatef(__fmaf_rn(-db, db, g2a)));
                accp[i] = add2(accp[i], w);
                if (i & 1) src1 = add2(src1, w);
                else src0 = add2(src0, w);
              }
              float u0, u1, u2, u3;
              upk2(src0, u0, u1);
              upk2(src1, u2, u3);
              myrow[s0 + k] = (u0 + u1) + (u2 + u3);
            }
#pragma unroll
            for (int i = 0; i < R / 2; ++i) {
              float a0, a1;
              upk2(accp[i], a0, a1);
              acc[2 * i] += a0;
              acc[2 * i + 1] += a1;
            }
          } else {
            // A piece is two to four steps long and R targets fill the pipes, so
            // the loop is not unrolled: the 3-D kernel of TE 6 x 30k takes 860 / 842
            // / 811 us unrolled by 4 / 2 / 1, of TE 32 x 200k - / 602 / 597 ms; with
            // the next source loaded ahead 632 ms.
#pragma unroll 1
            for (uint32_t k = lane; k < n; k += 32) {
              const P s = B[s0 + k];
              const f32x2 S = pk2(s.x, s.y);
              // source-side sum over the warp's R targets in 4 interleaved
              // partials (short rounding and dependency chains)
              float src[4] = {0.f, 0.f, 0.f, 0.f};
              if constexpr (D == 3) {
                // two targets per step, their chains interleaved
#pragma unroll
                for (int r = 0; r < R / 2; ++r) {
                  const int q = r + R / 2;
                  float dxa, dya, dxb, dyb;
                  upk2(sub2(T01[r], S), dxa, dya);
                  upk2(sub2(T01[q], S), dxb, dyb);
                  const float dza = T2[r] - s.z, dzb = T2[q] - s.z;
                  const float wxa = __saturatef(__fmaf_rn(-dxa, dxa, g2a));
                  const float wxb = __saturatef(__fmaf_rn(-dxb, dxb, g2a));
                  const float wya = __saturatef(__fmaf_rn(-dya, dya, g2b));
                  const float wyb = __saturatef(__fmaf_rn(-dyb, dyb, g2b));
                  const float wza = __saturatef(__fmaf_rn(-dza, dza, g2c));
                  const float wzb = __saturatef(__fmaf_rn(-dzb, dzb, g2c));
                  const float pa = wxa * wya, pb = wxb * wyb;
                  acc[r] = __fmaf_rn(pa, wza, acc[r]);
                  acc[q] = __fmaf_rn(pb, wzb, acc[q]);
                  src[r & 3] = __fmaf_rn(pa, wza, src[r & 3]);
                  src[q & 3] = __fmaf_rn(pb, wzb, src[q & 3]);
                }
              }
              if constexpr (D == 2) {
                // two targets per step, their chains interleaved
#pragma unroll
                for (int r = 0; r < R / 2; ++r) {
                  const int q = r + R / 2;
                  float dxa, dya, dxb, dyb;
                  upk2(sub2(T01[r], S), dxa, dya);
                  upk2(sub2(T01[q], S), dxb, dyb);
                  const float wxa = __saturatef(__fmaf_rn(-dxa, dxa, g2a));
                  const float wxb = __saturatef(__fmaf_rn(-dxb, dxb, g2a));
                  const float wya = __saturatef(__fmaf_rn(-dya, dya, g2b));
                  const float wyb = __saturatef(__fmaf_rn(-dyb, dyb, g2b));
                  acc[r] = __fmaf_rn(wxa, wya, acc[r]);
                  acc[q] = __fmaf_rn(wxb, wyb, acc[q]);
                  src[r & 3] = __fmaf_rn(wxa, wya, src[r & 3]);
                  src[q & 3] = __fmaf_rn(wxb, wyb, src[q & 3]);
                }
              }
              myrow[s0 + k] = (src[0] + src[1]) + (src[2] + src[3]);
            }
          }
        }
      }
      if (__syncthreads_or(!ok)) {
        aborted = true;
        ab_q = qq;
        ab_next = c + cs < nch;
        break;
      }
      // Target side of this chunk: lanes combined, one FP64 add per target.
      const float tot = warp_transpose_sum<R>(acc, lane);
      if (writer && my_li < tc && tot != 0.f)
        atomicAdd(acc64 + tb + my_li, f32_to_f64_int(tot));
      // Source side: every warp wrote every staged element of this chunk
      // into its row; the tile's own targets are complete on the target side.
      const uint32_t np = npc[b];
      for (uint32_t pi = 0; pi < np; ++pi) {
        const Piece p = ptab[b][pi];
        const uint32_t a = p.g0 + (p.s0 - p.o);
        for (uint32_t k = tid; k < p.n; k += C::NT) {
          if (a + k < tend) continue;
          const uint32_t e = p.s0 + k;
          float v = srow[e];
#pragma unroll
          for (int w = 1; w < NW; ++w) v += srow[(size_t)w * C::CAP + e];
          if (v != 0.f) atomicAdd(acc64 + a + k, f32_to_f64_int(v));
        }
      }
      __syncthreads();
    }
    if (aborted) {
      if (tid == 0) {
        atomicOr(err, EF_TIMEOUT);
        mbar_wait(&full[ab_q & 1u], (ab_q >> 1) & 1u);
        if (ab_next) mbar_wait(&full[(ab_q + 1) & 1u], ((ab_q + 1) >> 1) & 1u);
      }
      __syncthreads();
      return;
    }
    q = qq;
  }
}

// The 2-D sums with one warp per tile, for the light tiles on a work list: edge
// tiles of the strip moments carry some 200 sources each, over which the CTA
// form spends most of its time fetching the tile, staging and waiting at its
// barriers. Here each warp runs on its own, fetches the next tile's descriptor
// while it works, reads sources straight from L1/L2 one step ahead, and visits
// for each group of 32 targets only the sources inside that group's x-window.
//
// The sums, bit for bit, are the CTA form's: the warp takes the tile's NS groups
// of R targets (one warp's share there) in turn over each chunk of CH sources,
// with the same source-to-lane assignment; a source's sums over the groups are
// added in the same order in its slot of `row`; sources outside a group's
// window would add exactly 0 to both sides.
//
// A lane only ever touches its own slots of `row` (its index modulo 32 from the
// start of a piece), so the row needs no synchronisation. The instruction
// stream bounds it (128 registers, 16 warps per SM).
constexpr int SW_WARPS = 4;
constexpr int SW_CTAS = 4;  // per SM
// Light tiles go to warps in lists of at least SW_MIN_TILES slots per SM: with
// 12k slots (MI 10 x 25k) a warp gets a few tiles and the last ones are waited
// for, 86 us against 66 by blocks; with 35k (MI 12 x 60k) 246 against 219, with 70k
// (TE 12 x 100k) 1.36 against 1.38 ms. Edge kernel times, by blocks / with warps:
// MI 64 x 100k (1.7 M slots) 15.3 / 14.1 ms, TE 32 x 200k x 3 lags (2.5 M) 72.4 /
// 70.1 ms. SW_MAX_SOURCES of 512, 1024, 3072: TE 70.8, 70.1, 72.7 ms, MI 14.1 ms;
// a tile of 45k sources (a crowded strip) would keep one warp for 1 ms.
constexpr uint32_t SW_MIN_TILES = 512;
constexpr uint32_t SW_MAX_SOURCES = 1024;

// The terms of one source with 32 register-resident targets, as in the CTA
// form: added to the targets' sums; returns their sum for the source.
__device__ __forceinline__ float source_terms(float2 s, const f32x2 (&T)[32], float g2a, float g2b,
                                              float (&acc)[32]) {
  const f32x2 S = pk2(s.x, s.y);
  float src[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    const int q = r + 16;
    float dxa, dya, dxb, dyb;
    upk2(sub2(T[r], S), dxa, dya);
    upk2(sub2(T[q], S), dxb, dyb);
    const float wxa = __saturatef(__fmaf_rn(-dxa, dxa, g2a));
    const float wxb = __saturatef(__fmaf_rn(-dxb, dxb, g2a));
    const float wya = __saturatef(__fmaf_rn(-dya, dya, g2b));
    const float wyb = __saturatef(__fmaf_rn(-dyb, dyb, g2b));
    acc[r] = __fmaf_rn(wxa, wya, acc[r]);
    acc[q] = __fmaf_rn(wxb, wyb, acc[q]);
    src[r & 3] = __fmaf_rn(wxa, wya, src[r & 3]);
    src[q & 3] = __fmaf_rn(wxb, wyb, src[q & 3]);
  }
  return (src[0] + src[1]) + (src[2] + src[3]);
}

__global__ void __launch_bounds__(SW_WARPS * 32, SW_CTAS)
    k_sym_warp(const TileDesc* __restrict__ tiles, const uint32_t* __restrict__ list,
               const uint32_t* __restrict__ n_list, const InstDev* __restrict__ insts,
               uint32_t* work_counter) {
  constexpr int R = 32, NS = 4;  // NS groups of R targets per tile
  constexpr int CH = SymChunk<2, 4>::CH;
  constexpr int NR = 9;  // runs: 2S + 1 strips, S <= 4
  static_assert(sizeof(TileDesc) % 16 == 0 && sizeof(TileDesc) / 16 <= 32, "descriptor copy");
  __shared__ __align__(16) TileDesc s_desc[SW_WARPS][2];
  __shared__ uint2 s_win[SW_WARPS][NS][NR];
  __shared__ float s_row[SW_WARPS][CH + 32 * NR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float FAR = __int_as_float(0x7f800000);
  const uint32_t n_work = *n_list;
  float* const row = s_row[warp];

  auto fetch = [&]() { return lane == 0 ? atomicAdd(work_counter, 1u) : 0u; };
  auto stage = [&](uint32_t g, int b) {
    if (g < n_work && lane < (int)(sizeof(TileDesc) / 16))
      cp_async16(reinterpret_cast<char*>(&s_desc[warp][b]) + 16 * lane,
                 reinterpret_cast<const char*>(tiles + list[g]) + 16 * lane);
    cp_async_commit();
  };

  uint32_t g = __shfl_sync(FULL, fetch(), 0);
  stage(g, 0);
  uint32_t g1 = __shfl_sync(FULL, fetch(), 0);
  for (int b = 0; g < n_work; b ^= 1) {
    stage(g1, b ^ 1);
    const uint32_t g2 = fetch();  // read at the end of the tile
    cp_async_wait<1>();
    __syncwarp();
    const TileDesc& td = s_desc[warp][b];
    const uint32_t tc = td.t_count, nr = td.n_runs;
    const InstDev* I = insts + td.inst;
    const float2* __restrict__ pts = reinterpret_cast<const float2*>(I->pts);
    double* __restrict__ acc64 = I->acc;
    const uint32_t tb = td.t_begin, tend = tb + tc;
    const float g2a = I->g2[0], g2b = I->g2[1];
    const uint32_t ns = (tc + R - 1) / R;
    // x-window of every (group, run): two bisections, one lane each. The
    // group's targets are consecutive in one strip, so x-sorted; the margin
    // covers every rounding. A merged run is not sorted: all of it.
    const float gw = sqrtf(g2a);
    for (uint32_t q = lane; q < 2 * ns * nr; q += 32) {
      const uint32_t side = q & 1u, r = (q >> 1) % nr, w = (q >> 1) / nr;
      const float xf = pts[tb + w * R].x, xl = pts[tb + min(w * R + R, tc) - 1].x;
      const float eps = 1e-5f * (gw + fmaxf(fabsf(xf), fabsf(xl)));
      const float v = side ? xl + gw + eps : xf - gw - eps;
      uint32_t lo = td.lo[r], hi = lo + td.len[r];
      if ((td.merged >> r) & 1u) {
        if (side) lo = hi;
      } else {
        while (lo < hi) {  // first position with x >= v, or x > v
          const uint32_t m = lo + ((hi - lo) >> 1);
          const float x = pts[m].x;
          if (side ? x <= v : x < v) lo = m + 1; else hi = m;
        }
      }
      if (side) s_win[warp][w][r].y = lo; else s_win[warp][w][r].x = lo;
    }
    __syncwarp();

    uint32_t nsrc = 0;
    for (uint32_t r = 0; r < nr; ++r) nsrc += td.len[r];
    // calls f(r, first position, sources, first slot of row) for every piece
    // of a run inside the chunk [cb, ce) of the concatenated sources; returns
    // the slots used
    auto pieces = [&](uint32_t cb, uint32_t ce, auto&& f) {
      uint32_t rb = 0, slot = 0;
      for (uint32_t r = 0; r < nr; ++r) {
        const uint32_t re = rb + td.len[r];
        if (re > cb && rb < ce) {
          const uint32_t p0 = max(cb, rb), n = min(ce, re) - p0;
          f(r, td.lo[r] + (p0 - rb), n, slot);
          slot += (n + 31u) & ~31u;  // pieces start on lane 0's slot
        }
        rb = re;
      }
      return slot;
    };
    for (uint32_t cb = 0; cb < nsrc; cb += CH) {
      const uint32_t ce = min(cb + (uint32_t)CH, nsrc);
      const uint32_t used = pieces(cb, ce, [](uint32_t, uint32_t, uint32_t, uint32_t) {});
      for (uint32_t k = lane; k < used; k += 32) row[k] = 0.f;
      for (uint32_t w = 0; w < ns; ++w) {
        // the group's targets; missing ones sit at +inf, where every term is 0
        f32x2 T01[R];
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t li = w * R + r;
          const float2 p = li < tc ? pts[tb + li] : make_float2(FAR, FAR);
          T01[r] = pk2(p.x, p.y);
          acc[r] = 0.f;
        }
        pieces(cb, ce, [&](uint32_t r, uint32_t p0, uint32_t n, uint32_t slot) {
          const uint2 win = s_win[warp][w][r];
          const uint32_t k0 = (max(win.x, p0) - p0) & ~31u;
          const uint32_t k1 = min(max(win.y, p0) - p0, n);
          const float2* __restrict__ src = pts + p0;
          float* const out = row + slot;
          uint32_t k = k0 + lane;
          if (k >= k1) return;
          float2 s = src[k];
          for (;;) {
            const bool more = k + 32 < k1;
            float2 nx = s;
            if (more) nx = src[k + 32];
            out[k] += source_terms(s, T01, g2a, g2b, acc);
            if (!more) break;
            k += 32;
            s = nx;
          }
        });
        __syncwarp();
        // target side of this chunk: lanes combined, one FP64 add per target
        const float tot = warp_transpose_sum<R>(acc, lane);
        const uint32_t li = w * R + lane;
        if (li < tc && tot != 0.f) atomicAdd(acc64 + tb + li, f32_to_f64_int(tot));
      }
      // source side; the tile's own targets are complete on the target side
      pieces(cb, ce, [&](uint32_t, uint32_t p0, uint32_t n, uint32_t slot) {
        for (uint32_t k = lane; k < n; k += 32) {
          const float v = row[slot + k];
          if (p0 + k >= tend && v != 0.f) atomicAdd(acc64 + p0 + k, f32_to_f64_int(v));
        }
      });
    }
    __syncwarp();  // the descriptor buffer is free
    g = g1;
    g1 = __shfl_sync(FULL, g2, 0);
  }
  cp_async_wait<0>();
}

template <int D, int R, int MINB, int NW, bool LIST>
cudaError_t launch_sym_t(cudaStream_t st, const TileDesc* tiles, const SymWork& w,
                         const InstDev* insts, uint32_t* err, int n_sms, int* launched) {
  typedef Cfg<D, R, SymChunk<D, NW>::CH, NW> C;
  auto kern = k_density_sym<D, R, MINB, NW, LIST>;
  const size_t smem = C::SMEM + (size_t)C::NW * C::CAP * sizeof(float);
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::NT, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  uint64_t grid = (uint64_t)per_sm * (uint64_t)n_sms;
  if (grid > w.n_slots) grid = w.n_slots;
  if (grid == 0) grid = 1;
  kern<<<(unsigned)grid, C::NT, smem, st>>>(tiles, w.n_slots, insts, w.next + 1, err,
                                            LIST ? w.list + w.n_slots : nullptr, w.count + 1);
  if (launched) *launched = (int)grid;
  return cudaGetLastError();
}

// Symmetric epilogue: one warp per tile slot turns the FP64 sums of its
// targets into densities (scale), written by original index and/or summed
// (log or value) into the slot's tile_logsum. Logs are summed as integers, the
// mantissas' logs and the exponents apart, and meet FP64 once per tile: the
// three launches of TE 6 x 30k (3.4 M points) took 142 us with an FP64 log per
// point and take 48; MI 64 x 100k 187 and 41 us.
__global__ void __launch_bounds__(256)
    k_sym_finish(const TileDesc* __restrict__ tiles, uint32_t n_slots,
                 const InstDev* __restrict__ insts, const ILogEntry* __restrict__ logtab,
                 double* tile_logsum, uint32_t mode) {
  const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (g >= n_slots) return;  // warp-uniform
  const TileDesc& T = tiles[g];
  const InstDev& I = insts[T.inst];
  // the strip-moment kernel writes the slots of the instances it owns
  if (I.fused) return;  // warp-uniform
  const uint32_t tc = T.part == 0 ? T.t_count : 0u;  // one slot per tile finishes it
  double ls = 0.0;
  if (tc) {
    const double* __restrict__ acc = I.acc + T.t_begin;
    if (mode & (DM_WRITE_F64 | DM_SUMV)) {
      const double scale = I.scale;
      for (uint32_t li = lane; li < tc; li += 32) {
        const double dens = scale * acc[li];
        if (mode & DM_WRITE_F64) I.out[I.perm[T.t_begin + li]] = dens;
        if (!(mode & DM_LOGSUM) && (mode & DM_SUMV)) ls += dens;
      }
    }
    if (mode & DM_LOGSUM) {
      long long fx = 0;
      int ex = 0;
      bool odd = false;
      for (uint32_t li = lane; li < tc; li += 32) {
        const double v = acc[li];
        if (log_normal(v)) {
          int e;
          fx += log_fx56(v, logtab, &e);
          ex += e;
        } else {
          ls += log(v);
          odd = true;
        }
      }
      for (int o = 16; o; o >>= 1) fx += __shfl_xor_sync(FULL, fx, o);
      ex = __reduce_add_sync(FULL, ex);
      odd = __any_sync(FULL, odd);
      if (odd)
        for (int o = 16; o; o >>= 1) ls += __shfl_xor_sync(FULL, ls, o);
      if (lane == 0)
        tile_logsum[g] = ls + ((double)fx * 0x1p-56 + ((double)ex * LN2 + (double)tc * I.log_scale));
      return;
    }
  }
  if (mode & DM_SUMV) {
    for (int o = 16; o; o >>= 1) ls += __shfl_xor_sync(FULL, ls, o);
  }
  if ((mode & (DM_LOGSUM | DM_SUMV)) && lane == 0) tile_logsum[g] = ls;
}

// One bounded wait on an mbarrier whose expected bytes never arrive: the
// wait gives up after ENT_WAIT_NS and the kernel reports EF_TIMEOUT (no copy
// is in flight, so the CTA may exit).
__global__ void k_wait_test(uint32_t* err) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(&bar, 16);
    if (!mbar_wait(&bar, 0)) atomicOr(err, EF_TIMEOUT);
  }
}

__global__ void k_log64_test(const double* __restrict__ x, size_t n,
                             const ILogEntry* __restrict__ logtab, double* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    int e = 0;
    if (log_normal(x[i])) {
      const long long fx = log_fx56(x[i], logtab, &e);
      out[i] = (double)fx * 0x1p-56 + (double)e * LN2;
    } else {
      out[i] = log(x[i]);
    }
  }
}

}  // namespace

// Shapes of the symmetric bodies: PAIR_SYM 4 warps of 32 targets (d = 1, 2;
// 4 CTAs per SM) / 16 (d = 3; 5 CTAs per SM); PAIR_SYM + 1 8 warps of 16 /
// 8 targets, 3 CTAs per SM. Tiles: 128 targets (d = 1, 2), 64 (d = 3).
int sym_tile_r(int d, int v) {
  if (v == PAIR_SYM) return d == 3 ? 16 : 32;
  return d == 3 ? 8 : 16;
}

int sym_tile_targets(int d, int v) { return (v == PAIR_SYM ? 4 : 8) * sym_tile_r(d, v); }

uint32_t sym_light_sources(uint32_t n_slots, int n_sms) {
  return n_slots >= SW_MIN_TILES * (uint32_t)n_sms ? SW_MAX_SOURCES : 0u;
}

// A tile of a crowded strip has tens of thousands of sources, and a CTA takes up to
// 150 us over them while the others run out of work. Its chunks are independent, so
// SYM_SHARES CTAs share them; but a share without a chunk costs a fetch for nothing,
// so with many slots per SM, where one tile weighs less, only tiles of more than
// four chunks are shared. Device time of a call, no shares / more than 1,536 / more
// than 6,144 sources shared: the reference's MI formula over 10 x 25k (81 slots per
// SM) 608 / 517 / 563 us, MI 12 x 60k (230) 1390 / 1183 / 1182, 16 x 100k (630) 3425 /
// - / 3198, TE 12 x 100k (460) 13.66 / 13.72 / 13.66 ms; with 4 shares MI 6 x 100k 665
// instead of 627 us.
uint32_t sym_heavy_sources(uint32_t n_slots, int n_sms) {
  return n_slots < 128u * (uint32_t)n_sms ? 1536u : 6144u;
}

cudaError_t launch_density_sym(cudaStream_t st, int d, int v, const TileDesc* tiles,
                               const SymWork& w, const InstDev* insts, uint32_t* err, int n_sms,
                               int* launched) {
  const int r = sym_tile_r(d, v);
  const int nw = v == PAIR_SYM ? 4 : 8;
  if (w.list) {  // 2-D slots of a batch with strip moments
    if (d != 2 || v != PAIR_SYM) return cudaErrorInvalidValue;
    const cudaError_t e =
        launch_sym_t<2, 32, 4, 4, true>(st, tiles, w, insts, err, n_sms, launched);
    if (e != cudaSuccess || !sym_light_sources(w.n_slots, n_sms)) return e;
    k_sym_warp<<<SW_CTAS * n_sms, SW_WARPS * 32, 0, st>>>(tiles, w.list, w.count, insts, w.next);
    return cudaGetLastError();
  }
#define ENT_SYM(D, R, M, W)        \
  if (d == D && r == R && nw == W) \
    return launch_sym_t<D, R, M, W, false>(st, tiles, w, insts, err, n_sms, launched);
  ENT_SYM(1, 32, 4, 4)
  ENT_SYM(1, 16, 3, 8)
  ENT_SYM(2, 32, 4, 4)
  ENT_SYM(2, 16, 3, 8)
  ENT_SYM(3, 16, 5, 4)
  ENT_SYM(3, 8, 3, 8)
#undef ENT_SYM
  return cudaErrorInvalidValue;
}

cudaError_t launch_sym_finish(cudaStream_t st, const TileDesc* tiles,
                              uint32_t n_slots, const InstDev* insts,
                              const ILogEntry* logtab, double* tile_logsum, uint32_t mode) {
  if (n_slots == 0) return cudaSuccess;
  const uint64_t blocks = ((uint64_t)n_slots * 32 + 255) / 256;
  k_sym_finish<<<(unsigned)blocks, 256, 0, st>>>(tiles, n_slots, insts, logtab, tile_logsum,
                                                  mode);
  return cudaGetLastError();
}

cudaError_t launch_wait_test(cudaStream_t st, uint32_t* err) {
  k_wait_test<<<1, 32, 0, st>>>(err);
  return cudaGetLastError();
}

cudaError_t launch_log64_test(cudaStream_t st, const double* x, size_t n,
                              const ILogEntry* logtab, double* out) {
  if (n == 0) return cudaSuccess;
  const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 4096);
  k_log64_test<<<blocks, 256, 0, st>>>(x, n, logtab, out);
  return cudaGetLastError();
}

}  // namespace ent
