// Segmented, stable LSD radix sort of (uint32 key, uint32 value) pairs.
//
// Used for two things on the density path:
//   * sorting each coordinate column by value (orderable float keys, four
//     8-bit passes) -- the device replacement of Tools::dim1_sorted_coords
//     (tools.hxx:113-150);
//   * partitioning an already value-sorted sequence into strips (cell ids of
//     the remaining dimensions as keys, 1-3 passes). Because every pass is
//     stable, points stay sorted on dimension 0 inside each strip.
//
// One pass = histogram (per block, per digit, one row of 256 counts per block)
// -> exclusive prefix over a segment's blocks -> stable scatter (warp match +
// per-warp digit counts combined in warp order). Deterministic: the output
// order is a pure function of the input.
//
// The first pass's rows are written by the kernel that makes the keys, which
// covers the same chunk of the same segment per block (block_histogram). What
// follows depends on the size of the sort (radix_fused):
//   * segments that fit one block (radix_in_block) take all passes in one
//     kernel, a block per segment, with the elements in shared memory;
//   * a small sort is bound by the latency of its launches, so each pass is one
//     kernel: a scatter block sums the rows of its segment itself, and counts
//     its elements into the next pass's rows by the block they land in;
//   * a large one is bound by memory traffic, and reading every row in every
//     block, or one atomic per element, costs more than two more kernels: a
//     histogram and a prefix kernel run per pass.
#include <utility>

#include "engine.h"

namespace ent {

namespace {

constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_CHUNK = RS_THREADS * RS_ITEMS;  // elements per block
constexpr int RS_WARPS = RS_THREADS / 32;

__global__ void __launch_bounds__(RS_THREADS)
    k_radix_hist(const uint32_t* __restrict__ keys, int shift, SegTableDev t) {
  __shared__ uint32_t cnt[256];
  grid_chain();
  const uint32_t b = blockIdx.x;
  const uint32_t s = t.blk_seg[b];
  const uint64_t base = t.seg_off[s];
  const uint32_t e0 = (b - t.seg_blk0[s]) * RS_CHUNK;
  const uint32_t e1 = min(e0 + RS_CHUNK, t.seg_len[s]);
  cnt[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t e = e0 + threadIdx.x; e < e1; e += RS_THREADS)
    atomicAdd(&cnt[(keys[base + e] >> shift) & 255u], 1u);
  __syncthreads();
  t.hist[(uint64_t)b * 256 + threadIdx.x] = cnt[threadIdx.x];
}

// inclusive scan of one value per thread over the block; tot: 8 words
__device__ __forceinline__ uint32_t block_inclusive(uint32_t v, uint32_t* tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) tot[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; ++w) v += tot[w];
  return v;
}

// One block per segment, thread d: digit d's counts of the segment's blocks
// become the positions in the segment where the blocks' runs of d start.
__global__ void __launch_bounds__(RS_THREADS) k_radix_scan(SegTableDev t) {
  __shared__ uint32_t tot[RS_WARPS];
  grid_chain();
  constexpr uint32_t U = 8;  // rows in flight
  const uint32_t s = blockIdx.x, d = threadIdx.x;
  const uint32_t nb = t.seg_blk0[s + 1] - t.seg_blk0[s];
  uint32_t* h = t.hist + (uint64_t)t.seg_blk0[s] * 256 + d;
  uint32_t sum = 0;
  for (uint32_t j = 0; j < nb; j += U) {
    uint32_t v[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) v[u] = j + u < nb ? h[(uint64_t)(j + u) * 256] : 0u;
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) sum += v[u];
  }
  uint32_t run = block_inclusive(sum, tot) - sum;
  for (uint32_t j = 0; j < nb; j += U) {
    uint32_t v[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) v[u] = j + u < nb ? h[(uint64_t)(j + u) * 256] : 0u;
#pragma unroll
    for (uint32_t u = 0; u < U; ++u)
      if (j + u < nb) {
        h[(uint64_t)(j + u) * 256] = run;
        run += v[u];
      }
  }
}

// Stable scatter of one block's chunk (RS_CHUNK elements; warp w owns the
// RS_ITEMS * 32 consecutive elements from w * RS_ITEMS * 32). Each warp ranks
// its elements per digit with warp matches and warp-private digit counts (in
// element order); one block-wide scan over (digit, warp) turns the counts
// into positions in the chunk sorted by digit; the chunk is reordered in
// shared memory and its digit runs are written out contiguously (coalesced).
// Four block barriers per chunk. SUM: the rows of t.hist are counts (small
// sorts), else the run starts of k_radix_scan. next: rows of the next pass's
// counts, zeroed by the key kernel (null on the last pass and in large sorts). vin null:
// the values are the element indices of the segment; vout null: keys only.
template <bool SUM>
__global__ void __launch_bounds__(RS_THREADS)
    k_radix_scatter(const uint32_t* __restrict__ kin,
                    const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
                    uint32_t* __restrict__ vout, int shift, SegTableDev t,
                    uint32_t* __restrict__ next) {
  __shared__ uint32_t off[256];     // global start of each digit for this block
  __shared__ uint32_t lstart[256];  // start of each digit in the reordered chunk
  __shared__ uint32_t wcnt[RS_WARPS][256];
  __shared__ uint32_t wtot[RS_WARPS], dtot[RS_WARPS];
  __shared__ uint32_t sk[RS_CHUNK], sv[RS_CHUNK];
  grid_chain();
  const uint32_t b = blockIdx.x;
  const uint32_t s = t.blk_seg[b];
  const uint32_t j = b - t.seg_blk0[s];
  const uint32_t nb = t.seg_blk0[s + 1] - t.seg_blk0[s];
  const uint64_t base = t.seg_off[s];
  const uint32_t len = t.seg_len[s];
  const uint32_t e0 = j * RS_CHUNK;
  const uint32_t ne = min((uint32_t)RS_CHUNK, len - e0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the elements are on their way while the rows are summed
  uint32_t key[RS_ITEMS], val[RS_ITEMS], rnk[RS_ITEMS];
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const uint32_t e = (uint32_t)warp * (RS_ITEMS * 32) + it * 32 + lane;
    key[it] = val[it] = 0;
    if (e < ne) {
      key[it] = kin[base + e0 + e];
      if (vout) val[it] = vin ? vin[base + e0 + e] : e0 + e;
    }
  }
  if (SUM) {
    const uint32_t* h = t.hist + (uint64_t)t.seg_blk0[s] * 256 + threadIdx.x;
    uint32_t all = 0, before = 0;
    constexpr uint32_t U = 16;  // rows in flight
    for (uint32_t i = 0; i < nb; i += U) {
      uint32_t v[U];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) v[u] = i + u < nb ? h[(uint64_t)(i + u) * 256] : 0u;
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) {
        all += v[u];
        before += i + u < j ? v[u] : 0u;
      }
    }
    off[threadIdx.x] = block_inclusive(all, dtot) - all + before;
  } else {
    off[threadIdx.x] = t.hist[(uint64_t)b * 256 + threadIdx.x];
  }
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) wcnt[w][threadIdx.x] = 0;
  __syncthreads();
  // 1. per warp: rank of every element among the warp's elements of its digit
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t* myc = wcnt[warp];
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const uint32_t e = (uint32_t)warp * (RS_ITEMS * 32) + it * 32 + lane;
    const bool valid = e < ne;
    const uint32_t digit = valid ? (key[it] >> shift) & 255u : 256u;
    const uint32_t peers = __match_any_sync(0xffffffffu, digit);
    const uint32_t r = __popc(peers & lt_mask);
    const uint32_t prior = valid ? myc[digit] : 0u;
    __syncwarp();
    if (valid && r == 0) myc[digit] = prior + __popc(peers);
    __syncwarp();
    rnk[it] = prior + r;
  }
  __syncthreads();
  // 2. thread d: digit d's total and per-warp starts; block scan over digits
  const uint32_t d = threadIdx.x;
  uint32_t tot = 0;
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) {
    const uint32_t c = wcnt[w][d];
    wcnt[w][d] = tot;
    tot += c;
  }
  uint32_t x = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wtot[warp] = x;
  __syncthreads();
  uint32_t wp = 0;
  for (int w = 0; w < warp; ++w) wp += wtot[w];
  const uint32_t start = wp + x - tot;
  lstart[d] = start;
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) wcnt[w][d] += start;
  __syncthreads();
  // 3. reorder the chunk by digit in shared memory
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const uint32_t e = (uint32_t)warp * (RS_ITEMS * 32) + it * 32 + lane;
    if (e < ne) {
      const uint32_t dg = (key[it] >> shift) & 255u;
      const uint32_t lp = myc[dg] + rnk[it];
      sk[lp] = key[it];
      if (vout) sv[lp] = val[it];
    }
  }
  __syncthreads();
  // 4. digit runs to their global positions, consecutive elements together
  for (uint32_t i = threadIdx.x; i < ne; i += RS_THREADS) {
    const uint32_t k = sk[i];
    const uint32_t dg = (k >> shift) & 255u;
    const uint32_t pos = off[dg] + (i - lstart[dg]);
    kout[base + pos] = k;
    if (vout) vout[base + pos] = sv[i];
    if (SUM && next)
      atomicAdd(next + (uint64_t)(t.seg_blk0[s] + pos / RS_CHUNK) * 256 +
                    ((k >> (shift + 8)) & 255u),
                1u);
  }
}

// All passes over one segment of at most 1,024 ITEMS elements, one block per
// segment (any order of blocks: a block reads its segment whole before it writes,
// so kin == kout is fine). Thread t of warp w holds the elements at w 32 ITEMS +
// 32 i + lane; a pass ranks them as k_radix_scatter does, turns the (digit, warp)
// counts into positions with one scan over the block (thread 4 d + q: digit d,
// eight warps), and moves the elements through shared memory. Bound by the
// latency of its matches and barriers.
template <int ITEMS>
__global__ void __launch_bounds__(1024)
    k_radix_block(const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                  uint32_t* vout, int begin_bit, int end_bit, SegTableDev t) {
  extern __shared__ uint32_t rb_smem[];
  uint32_t* const sk = rb_smem;
  uint32_t* const sv = rb_smem + 1024 * ITEMS;
  __shared__ uint16_t wcnt[32][256];
  __shared__ uint32_t wtot[32];
  grid_chain();
  const uint32_t s = blockIdx.x;
  const uint64_t base = t.seg_off[s];
  const uint32_t len = t.seg_len[s];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u, w0 = warp * 32 * ITEMS + lane;
  uint32_t key[ITEMS], val[ITEMS];
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    const uint32_t e = w0 + 32 * it;
    key[it] = val[it] = 0;
    if (e < len) {
      key[it] = kin[base + e];
      if (vout) val[it] = vin ? vin[base + e] : e;
    }
  }
  uint16_t* const myc = wcnt[warp];
  for (int shift = begin_bit; shift < end_bit; shift += 8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<uint32_t*>(myc)[32 * i + lane] = 0;
    __syncwarp();
    uint32_t rnk[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const bool valid = w0 + 32 * it < len;
      const uint32_t digit = valid ? (key[it] >> shift) & 255u : 256u;
      const uint32_t peers = __match_any_sync(0xffffffffu, digit);
      const uint32_t r = __popc(peers & lt_mask);
      const uint32_t prior = valid ? myc[digit] : 0u;
      __syncwarp();
      if (valid && r == 0) myc[digit] = (uint16_t)(prior + __popc(peers));
      __syncwarp();
      rnk[it] = prior + r;
    }
    __syncthreads();
    const uint32_t d = threadIdx.x >> 2, q = (threadIdx.x & 3) * 8;
    uint32_t c[8], sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      c[i] = wcnt[q + i][d];
      sum += c[i];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wtot[warp] = x;
    __syncthreads();
    uint32_t run = x - sum + __reduce_add_sync(0xffffffffu, lane < warp ? wtot[lane] : 0u);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      wcnt[q + i][d] = (uint16_t)run;
      run += c[i];
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITEMS; ++it)
      if (w0 + 32 * it < len) {
        const uint32_t p = myc[(key[it] >> shift) & 255u] + rnk[it];
        sk[p] = key[it];
        sv[p] = val[it];
      }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const uint32_t e = w0 + 32 * it;
      if (e < len) {
        key[it] = sk[e];
        val[it] = sv[e];
      }
    }
  }
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    const uint32_t e = w0 + 32 * it;
    if (e < len) {
      kout[base + e] = key[it];
      if (vout) vout[base + e] = val[it];
    }
  }
}

// ---------------------------------------------------------------- keys
// Counts of the block's digits (bits 0..7 of its keys) as its row of t.hist;
// the rows of the `later` next passes, `stride` words apart, start at zero.
__device__ __forceinline__ void block_histogram(const uint32_t (&key)[RS_ITEMS], uint32_t ne,
                                                uint32_t* cnt, uint32_t* __restrict__ row,
                                                int later, size_t stride) {
  cnt[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it)
    if (threadIdx.x + it * RS_THREADS < ne) atomicAdd(&cnt[key[it] & 255u], 1u);
  __syncthreads();
  row[threadIdx.x] = cnt[threadIdx.x];
  for (int p = 1; p <= later; ++p) row[p * stride + threadIdx.x] = 0;
}

// Sort keys and statistics of every view: orderable keys, extremes (of the
// finite values) and a flag for values that are not finite. One block per
// radix chunk, so one long column still spreads over the GPU (one block per
// column took 47 us on a column of 100k values).
__global__ void __launch_bounds__(RS_THREADS)
    k_view_keys(const ViewDev* __restrict__ views, SegTableDev t, uint32_t* __restrict__ keys,
                ViewStatsDev* stats, int later, uint32_t n_views, ViewStatsDev* host) {
  __shared__ uint32_t cnt[256];
  __shared__ bool last;
  __shared__ uint32_t smin[RS_WARPS], smax[RS_WARPS], sbad[RS_WARPS];
  grid_chain();
  const uint32_t b = blockIdx.x;
  const uint32_t s = t.blk_seg[b];
  const uint32_t e0 = (b - t.seg_blk0[s]) * RS_CHUNK;
  const uint32_t ne = min((uint32_t)RS_CHUNK, t.seg_len[s] - e0);
  const float* __restrict__ x = views[s].x + e0;
  uint32_t* __restrict__ out = keys + t.seg_off[s] + e0;
  uint32_t key[RS_ITEMS];
  uint32_t inv_min = 0, mx = 0, bad = 0;
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const uint32_t e = threadIdx.x + it * RS_THREADS;
    key[it] = 0;
    if (e < ne) {
      const float f = x[e];
      key[it] = float_key(f);
      out[e] = key[it];
      if (isfinite(f)) {
        inv_min = max(inv_min, ~key[it]);
        mx = max(mx, key[it]);
      } else {
        bad = 1;
      }
    }
  }
  block_histogram(key, ne, cnt, t.hist + (uint64_t)b * 256, later, 256 * (size_t)gridDim.x);
  inv_min = __reduce_max_sync(0xffffffffu, inv_min);
  mx = __reduce_max_sync(0xffffffffu, mx);
  bad = __reduce_or_sync(0xffffffffu, bad);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    smin[warp] = inv_min;
    smax[warp] = mx;
    sbad[warp] = bad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < RS_WARPS; ++w) {
      inv_min = max(inv_min, smin[w]);
      mx = max(mx, smax[w]);
      bad |= sbad[w];
    }
    atomicMax(&stats[s].inv_min_key, inv_min);
    atomicMax(&stats[s].max_key, mx);
    if (bad) atomicOr(&stats[s].nonfinite, 1u);
    if (host) {
      __threadfence();
      last = atomicAdd(&stats[n_views].inv_min_key, 1u) == gridDim.x - 1;
    }
  }
  if (!host) return;  // grid-uniform
  __syncthreads();
  if (!last) return;  // block-uniform
  __threadfence();
  const volatile uint32_t* from = reinterpret_cast<const volatile uint32_t*>(stats);
  uint32_t* to = reinterpret_cast<uint32_t*>(host);
  for (uint32_t i = threadIdx.x; i < n_views * (sizeof(ViewStatsDev) / 4); i += RS_THREADS)
    to[i] = from[i];
}

// Cell index in FP32 (the FP64 pipe of this GPU is slow): a = fl(fl(x - lo)
// inv_w) is within 3 2^-24 a of the exact (x - lo)/w, i.e. within 1.8e-7 ncell
// cells; the host widens the cells by at least 6e-7 ncell / S so that two
// points within h never land more than S cells apart. x >= lo (the view's
// minimum), so a >= 0 and truncation is floor.
__device__ __forceinline__ uint32_t cell_of(float x, float lo, float inv_w, uint32_t ncell) {
  const float a = __fmul_rn(__fsub_rn(x, lo), inv_w);
  if (!(a < (float)ncell)) return ncell - 1;
  return a > 0.f ? (uint32_t)a : 0u;
}

// Strip keys of the value-sorted points, one block per radix chunk; the
// gathers of a thread's RS_ITEMS points are issued together.
__global__ void __launch_bounds__(RS_THREADS)
    k_strip_keys(const InstDev* __restrict__ insts, const uint32_t* __restrict__ inst_ids,
                 SegTableDev t, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                 int later) {
  __shared__ uint32_t cnt[256];
  grid_chain();
  const uint32_t blk = blockIdx.x;
  const uint32_t s = t.blk_seg[blk];
  const InstDev& I = insts[inst_ids[s]];
  const uint32_t e0 = (blk - t.seg_blk0[s]) * RS_CHUNK;
  const uint32_t ne = min((uint32_t)RS_CHUNK, I.n - e0);
  const uint64_t base = t.seg_off[s] + e0;
  const uint32_t* __restrict__ perm0 = I.perm0 + e0;
  const float* __restrict__ x1 = I.x[1];
  const float* __restrict__ x2 = I.x[2];
  const bool d3 = I.d == 3;
  uint32_t j[RS_ITEMS], key[RS_ITEMS];
  float a[RS_ITEMS], b[RS_ITEMS];
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const uint32_t e = threadIdx.x + it * RS_THREADS;
    j[it] = e < ne ? perm0[e] : 0u;
  }
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    a[it] = x1[j[it]];
    b[it] = d3 ? x2[j[it]] : 0.f;
  }
#pragma unroll
  for (int it = 0; it < RS_ITEMS; ++it) {
    const uint32_t e = threadIdx.x + it * RS_THREADS;
    key[it] = cell_of(a[it], I.lo1, I.inv_w1, I.ncell1);
    if (d3) key[it] = key[it] * I.ncell2 + cell_of(b[it], I.lo2, I.inv_w2, I.ncell2);
    if (e < ne) {
      keys[base + e] = key[it];
      vals[base + e] = j[it];
    }
  }
  block_histogram(key, ne, cnt, t.hist + (uint64_t)blk * 256, later, 256 * (size_t)gridDim.x);
}

}  // namespace

uint32_t radix_blocks_for(uint32_t len) {
  return (len + RS_CHUNK - 1) / RS_CHUNK;
}

// Rows read by the scatter blocks of a pass when each sums its segment's rows:
// 1 KB each from L2, so 64 MB at the line, about what the two kernels saved
// cost there. All passes of a sort, kernel times: 6 x 30k TE (102 strip
// segments of 15 blocks, 23k rows) 145 us summed, 166 us with the histogram
// and prefix kernels; one 100k column (2.4k rows) 75 against 134 us. 64 x 100k
// (154k rows) takes the two kernels: 0.11 ms of them in a 52 ms call.
bool radix_fused(uint32_t total_blocks, uint32_t max_blocks) {
  return (uint64_t)total_blocks * max_blocks <= 65536u;
}

size_t radix_hist_words(uint32_t total_blocks, uint32_t max_blocks, int passes) {
  return 256 * (size_t)total_blocks * (radix_fused(total_blocks, max_blocks) ? passes : 1);
}

// Sorts that one block per segment does in one kernel: up to RB_MAX elements per
// segment, more than one pass, and no more segments than run at once. Device time
// of a call, a kernel per pass / one kernel: 1-D density of 1,000 points 63 / 56 us,
// MI 8 x 2000 122 / 116 us, 8 x 4000 153 / 146 us; with 8 elements per thread 8 x
// 8000 202 / 203 us. 64 / 128 / 256 1-D columns of 4,000 115 / 98, 142 / 114, 202 / 190;
// of 2,000 89 / 83, 113 / 101, 143 / 141; of 500, a quarter of the block's, 74 / 77, 85 / 88,
// 122 / 122. 64 / 128 2-D densities of 4,000 178 / 147, 255 / 237.
constexpr uint32_t RB_MAX = 4096, RB_MAX_SEGMENTS = 256;
static bool radix_in_block(uint32_t n_seg, uint32_t max_blocks, int bits) {
  return max_blocks <= RB_MAX / RS_CHUNK && n_seg <= RB_MAX_SEGMENTS && bits > 8;
}

template <int ITEMS>
static cudaError_t radix_block(cudaStream_t st, const SegTableDev& t, uint32_t n_seg,
                               const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                               uint32_t* vout, int begin_bit, int end_bit, bool overlap) {
  constexpr int smem = 8 * 1024 * ITEMS;
  if (smem > 16 * 1024) {  // with the static part above 48 KB
    const cudaError_t e = cudaFuncSetAttribute(
        k_radix_block<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  return launch_chain(overlap, k_radix_block<ITEMS>, n_seg, 1024, smem, st, kin, vin, kout, vout,
                      begin_bit, end_bit, t);
}

cudaError_t seg_radix_sort(cudaStream_t st, SegTableDev t, uint32_t n_seg, uint32_t total_blocks,
                           uint32_t max_blocks, uint32_t*& keys, uint32_t*& vals,
                           uint32_t*& ktmp, uint32_t*& vtmp, int begin_bit, int end_bit,
                           bool index_values, bool overlap, uint32_t* launches) {
  if (total_blocks == 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  if (radix_in_block(n_seg, max_blocks, end_bit - begin_bit)) {
    const bool odd = (end_bit - begin_bit + 7) / 8 % 2;  // the results where passes leave them
    const auto run = max_blocks <= 1 ? radix_block<2> : radix_block<4>;
    e = run(st, t, n_seg, keys, index_values ? nullptr : vals, odd ? ktmp : keys,
            odd ? vtmp : vals, begin_bit, end_bit, overlap);
    if (odd) {
      std::swap(keys, ktmp);
      std::swap(vals, vtmp);
    }
    *launches += 1;
    return e;
  }
  const bool fused = radix_fused(total_blocks, max_blocks);
  const size_t rows = 256 * (size_t)total_blocks;
  for (int shift = begin_bit; shift < end_bit; shift += 8) {
    const uint32_t* vin = index_values && shift == begin_bit ? nullptr : vals;
    if (fused) {
      uint32_t* next = shift + 8 < end_bit ? t.hist + rows : nullptr;
      e = launch_after(overlap, k_radix_scatter<true>, total_blocks, RS_THREADS, st, keys, vin,
                       ktmp, vtmp, shift, t, next);
      t.hist += rows;
      *launches += 1;
    } else {
      if (shift > begin_bit) {
        e = launch_after(overlap, k_radix_hist, total_blocks, RS_THREADS, st, keys, shift, t);
        if (e != cudaSuccess) return e;
        *launches += 1;
      }
      e = launch_after(overlap, k_radix_scan, n_seg, RS_THREADS, st, t);
      if (e == cudaSuccess)
        e = launch_after(overlap, k_radix_scatter<false>, total_blocks, RS_THREADS, st, keys, vin,
                         ktmp, vtmp, shift, t, nullptr);
      *launches += 2;
    }
    if (e != cudaSuccess) return e;
    uint32_t* a = keys;
    keys = ktmp;
    ktmp = a;
    a = vals;
    vals = vtmp;
    vtmp = a;
  }
  return cudaGetLastError();
}

// later passes whose rows the key kernels have to zero
static int later_passes(uint32_t total_blocks, uint32_t max_blocks, int passes) {
  return radix_fused(total_blocks, max_blocks) ? passes - 1 : 0;
}

cudaError_t launch_view_keys(cudaStream_t st, const ViewDev* views, uint32_t n_views,
                             const SegTableDev& t, uint32_t total_blocks, uint32_t max_blocks,
                             uint32_t* keys, ViewStatsDev* stats, ViewStatsDev* host) {
  if (total_blocks == 0) return cudaSuccess;
  k_view_keys<<<total_blocks, RS_THREADS, 0, st>>>(
      views, t, keys, stats, later_passes(total_blocks, max_blocks, 4), n_views, host);
  return cudaGetLastError();
}

cudaError_t launch_strip_keys(cudaStream_t st, const InstDev* insts, const uint32_t* inst_ids,
                              const SegTableDev& t, uint32_t total_blocks, uint32_t max_blocks,
                              int passes, uint32_t* keys, uint32_t* vals) {
  if (total_blocks == 0) return cudaSuccess;
  k_strip_keys<<<total_blocks, RS_THREADS, 0, st>>>(
      insts, inst_ids, t, keys, vals, later_passes(total_blocks, max_blocks, passes));
  return cudaGetLastError();
}

}  // namespace ent
