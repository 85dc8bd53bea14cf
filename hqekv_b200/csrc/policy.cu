// Importance bookkeeping, block ranking and the plan of the flush (evict + tier-assign; csrc/flush.cu builds the tiers) on
// the device (sm_100a).  Integer / fp16 elementwise work on at most a few hundred thousand tokens; the
// quantity that matters is bit-exact agreement with the reference's torch op sequence, so every
// floating-point reduction here runs in a fixed order with one fp32 accumulator.
#include <string.h>

#include <cooperative_groups.h>

#include "common.cuh"

namespace hqkv {

HQKV_DEFINE_CHECK_COUNTER
unsigned policy_check_failures(bool reset) {
#if HQKV_CHECKS_ENABLED
  unsigned v = 0, z = 0;
  if (cudaMemcpyFromSymbol(&v, g_check_failures, sizeof(v)) != cudaSuccess) return ~0u;
  if (reset) cudaMemcpyToSymbol(g_check_failures, &z, sizeof(z));
  return v;
#else
  (void)reset;
  return 0u;
#endif
}

constexpr int D = 128;

// ------------------------------------------------------------------------------------------------
// importance ring
// ------------------------------------------------------------------------------------------------
// 32 positions per CTA, four warps.  The adds run in the reference's order (batch first with one fp32
// accumulator per head, rounded to fp16; then the heads, one fp32 accumulator), but a position's B * nh
// values lie a whole row apart, so a single chain of loads is all latency: warp w sums the batch for heads
// 8w .. 8w+7 of a pass of 32 heads (eight loads in flight per thread, every load a coalesced 64-byte row
// piece), the per-head results meet in shared memory, and warp 0 adds them in head order.
constexpr int HEAD_SUM_THREADS = 128;
__global__ void __launch_bounds__(HEAD_SUM_THREADS) head_sum_kernel(const __half* __restrict__ w, int B, int nh, int64_t L,
                                                                    int64_t bh_stride, __half* __restrict__ out) {
  __shared__ float per_head[32][32];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t l = static_cast<int64_t>(blockIdx.x) * 32 + lane;
  const bool live = l < L;
  float over_heads = 0.f;
  for (int h0 = 0; h0 < nh; h0 += 32) {
    const int hw = h0 + 8 * warp;
    float over_batch[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) over_batch[j] = 0.f;
#pragma unroll 2
    for (int b = 0; b < B; ++b) {
      __half v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = live && hw + j < nh ? w[(static_cast<int64_t>(b) * nh + hw + j) * bh_stride + l] : __float2half_rn(0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) over_batch[j] = __fadd_rn(over_batch[j], __half2float(v[j]));
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) per_head[8 * warp + j][lane] = __half2float(__float2half_rn(over_batch[j]));
    __syncthreads();
    if (warp == 0) {
      const int n = nh - h0 < 32 ? nh - h0 : 32;
      for (int h = 0; h < n; ++h) over_heads = __fadd_rn(over_heads, per_head[h][lane]);
    }
    __syncthreads();
  }
  if (warp == 0 && live) out[l] = __float2half_rn(over_heads);
}

__global__ void __launch_bounds__(256) token_importance_kernel(const __half* __restrict__ ring, int rows,
                                                               int64_t stride, int64_t L, __half* __restrict__ out) {
  const int64_t l = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (l >= L) return;
  float acc = 0.f;
  for (int r0 = 0; r0 < rows; r0 += 10) {  // ten loads in flight (half of the models' twenty rows), adds in row order
    __half v[10];
#pragma unroll
    for (int j = 0; j < 10; ++j) v[j] = ring[min(r0 + j, rows - 1) * stride + l];
#pragma unroll
    for (int j = 0; j < 10; ++j)
      if (r0 + j < rows) acc = __fadd_rn(acc, __half2float(v[j]));
  }
  const int64_t age = L - l;
  const float count = static_cast<float>(age < rows ? age : rows);
  out[l] = h_divf(__float2half_rn(acc), count);
}

// one warp per token: range over D channels per (b,h), summed over b then h
__global__ void __launch_bounds__(128) token_range_kernel(const __half* __restrict__ v, int B, int H, int64_t T,
                                                          int Dd, int64_t b_stride, int64_t h_stride,
                                                          __half* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  float over_heads = 0.f;
  for (int h = 0; h < H; ++h) {
    float over_batch = 0.f;
    for (int b = 0; b < B; ++b) {
      const __half* row = v + b * b_stride + h * h_stride + t * Dd;
      __half lo = row[lane], hi = row[lane];
      for (int d = lane + 32; d < Dd; d += 32) {
        lo = h_min(lo, row[d]);
        hi = h_max(hi, row[d]);
      }
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        lo = h_min(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        hi = h_max(hi, __shfl_xor_sync(0xffffffffu, hi, off));
      }
      over_batch = __fadd_rn(over_batch, __half2float(h_sub(hi, lo)));
    }
    over_heads = __fadd_rn(over_heads, __half2float(__float2half_rn(over_batch)));
  }
  if (lane == 0) out[t] = __float2half_rn(over_heads);
}

// head_dim 128, 16-byte aligned rows.  The rows of a token - a (batch, head) pair each - are independent up to the two sums
// over them, so they are spread over half-warps (16 bytes per lane, four rows in flight, minimum and negated maximum
// reduced together) and only the sums, in the order above, are one thread's.  A warp per token walked the rows eight at
// a time: with 32 tokens of 64 rows each the whole launch was eight warps long (41 us, now 5; 31 us for 32 k tokens of 8
// rows, now 15, of which reading them takes 10).
// CTA = 2^tshift tokens; `old` = the ranges of the tokens before these, copied to the front of `out` by the CTAs behind.
constexpr int RANGE_THREADS = 256;
constexpr int RANGE_MAX_ROWS = 4096;
__global__ void __launch_bounds__(RANGE_THREADS) token_range128_kernel(const __half* __restrict__ v, int B, int n, int64_t T,
                                                                       int64_t b_stride, int64_t h_stride, int tshift,
                                                                       const __half* __restrict__ old, int64_t n_old, int ctas,
                                                                       __half* __restrict__ out) {
  extern __shared__ int64_t row_at[];  // [row = h * B + b] first element, then the ranges [token][row]
  __half* range_s = reinterpret_cast<__half*>(row_at + n);
  const int tid = threadIdx.x;
  if (static_cast<int>(blockIdx.x) >= ctas) {
    const int64_t base = (static_cast<int64_t>(blockIdx.x) - ctas) * RANGE_THREADS * 8 + tid;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (base + j * RANGE_THREADS < n_old) out[base + j * RANGE_THREADS] = old[base + j * RANGE_THREADS];
    return;
  }
  for (int r = tid; r < n; r += RANGE_THREADS) row_at[r] = (r % B) * b_stride + (r / B) * h_stride;
  __syncthreads();
  const int hw = tid >> 4, l16 = tid & 15, tpc = 1 << tshift;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) << tshift;
  const int items = n << tshift;  // token fastest: neighbouring half-warps read neighbouring rows of memory
  for (int base = hw; base - (hw & 1) < items; base += 4 * (RANGE_THREADS / 16)) {  // (both halves of a warp take part)
    uint4 w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int it = min(base + u * (RANGE_THREADS / 16), items - 1);
      const int64_t t = min(t0 + (it & (tpc - 1)), T - 1);
      w[u] = *reinterpret_cast<const uint4*>(v + row_at[it >> tshift] + t * D + 8 * l16);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const __half2* x = reinterpret_cast<const __half2*>(&w[u]);
      const __half2 lo2 = __hmin2_nan(__hmin2_nan(x[0], x[1]), __hmin2_nan(x[2], x[3]));
      const __half2 hi2 = __hmax2_nan(__hmax2_nan(x[0], x[1]), __hmax2_nan(x[2], x[3]));
      __half2 m = __halves2half2(__hmin_nan(__low2half(lo2), __high2half(lo2)), __hneg(__hmax_nan(__low2half(hi2), __high2half(hi2))));
#pragma unroll
      for (int off = 1; off < 16; off <<= 1) m = __hmin2_nan(m, __shfl_xor_sync(0xffffffffu, m, off));
      const int it = base + u * (RANGE_THREADS / 16);
      if (l16 == 0 && it < items) range_s[(it & (tpc - 1)) * n + (it >> tshift)] = h_sub(__hneg(__high2half(m)), __low2half(m));
    }
  }
  __syncthreads();
  if (tid < tpc && t0 + tid < T) {
    float over_heads = 0.f, over_batch = 0.f;
    const __half* r = range_s + tid * n;
    for (int i = 0, b = 0; i < n; ++i) {
      over_batch = __fadd_rn(over_batch, __half2float(r[i]));
      if (++b == B) {  // last batch entry of this head
        over_heads = __fadd_rn(over_heads, __half2float(__float2half_rn(over_batch)));
        over_batch = 0.f;
        b = 0;
      }
    }
    out[n_old + t0 + tid] = __float2half_rn(over_heads);
  }
}

// ------------------------------------------------------------------------------------------------
// block ranking: one thread-block cluster
// ------------------------------------------------------------------------------------------------
// Each CTA of the cluster forms the keys of its share of the blocks (elementwise pass, then one thread per block adds in
// order) and stores them into the shared memory of all CTAs.  The keys - fp16 key, then block id - are all different, so a
// block's place is the number of smaller keys: every warp counts for its own blocks, with no exchange between the
// steps of a sort.  The comparisons grow with the square of the blocks, so beyond RANK_COUNT_MAX a bitonic sort (by every
// CTA for itself) is kept.  us, blocks of 32 tokens, counting / sort: 512: 7.2 / 12.3, 1024: 10.2 / 14.4, 2048: 19.0 / 22.5,
// 3072: 32.8 / 34.8, 4096: 51.2 / 36.9, 8192: 172 / 69.
constexpr int RANK_THREADS = 1024;
constexpr int RANK_CLUSTER = 8;
constexpr int RANK_MAX_BLOCKS = 8192;
constexpr int RANK_COUNT_MAX = 3072;

__global__ void __launch_bounds__(RANK_THREADS) block_rank_kernel(const __half* importance, const __half* __restrict__ range,
                                                                  __half* divided, int block, int nblocks, int npow2,
                                                                  int64_t* __restrict__ sorted_ids) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ uint32_t keys[];  // [npow2]
  auto started = cluster.barrier_arrive();  // (the other CTAs' shared memory may be written once they all run)
  const int crank = static_cast<int>(cluster.block_rank()), lane = threadIdx.x & 31;
  const int share = (nblocks + RANK_CLUSTER - 1) / RANK_CLUSTER, k0 = min(crank * share, nblocks), k1 = min(k0 + share, nblocks);
  const int64_t total = static_cast<int64_t>(nblocks) * block;
  const float fblock = static_cast<float>(block);
  // elementwise: optional product with the range, then the divide
#pragma unroll 4
  for (int64_t i = static_cast<int64_t>(k0) * block + threadIdx.x; i < static_cast<int64_t>(k1) * block; i += RANK_THREADS) {
    __half x = importance[i];
    if (range) x = h_mul(x, range[i]);
    divided[i] = h_divf(x, fblock);
  }
  __syncthreads();
  cluster.barrier_wait(std::move(started));
  const bool vec = block % 8 == 0 && (reinterpret_cast<uintptr_t>(divided) & 15) == 0;
  for (int k = k0 + threadIdx.x; k < k1; k += RANK_THREADS) {
    float acc = 0.f;
    const __half* p = divided + static_cast<int64_t>(k) * block;
    if (vec) {
      for (int i = 0; i < block; i += 8) {
        const uint4 w = *reinterpret_cast<const uint4*>(p + i);
        const __half* e = reinterpret_cast<const __half*>(&w);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = __fadd_rn(acc, __half2float(e[j]));
      }
    } else {
      for (int i = 0; i < block; ++i) acc = __fadd_rn(acc, __half2float(p[i]));
    }
    const __half key = __float2half_rn(acc);
    uint16_t bits = __half_as_ushort(key);
    if ((bits & 0x7FFFu) == 0) bits = 0;                                  // -0 sorts like +0
    const uint16_t asc = (bits & 0x8000u) ? static_cast<uint16_t>(~bits) : static_cast<uint16_t>(bits | 0x8000u);
    const uint16_t desc = static_cast<uint16_t>(0xFFFFu - asc);           // larger key first
    const uint32_t composite = (static_cast<uint32_t>(desc) << 16) | static_cast<uint32_t>(k);  // ties: lower id first
#pragma unroll
    for (int c = 0; c < RANK_CLUSTER; ++c) cluster.map_shared_rank(keys, c)[k] = composite;
  }
  if (nblocks > RANK_COUNT_MAX)
    for (int k = nblocks + threadIdx.x; k < npow2; k += RANK_THREADS) keys[k] = 0xFFFFFFFFu;
  cluster.sync();
  if (nblocks <= RANK_COUNT_MAX) {
    constexpr int WARPS = RANK_THREADS / 32 * RANK_CLUSTER;
    for (int m0 = crank * (RANK_THREADS / 32) + (threadIdx.x >> 5); m0 < nblocks; m0 += 4 * WARPS) {
      uint32_t mine[4], below[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int q = 0; q < 4; ++q) mine[q] = m0 + q * WARPS < nblocks ? keys[m0 + q * WARPS] : 0u;
      for (int j = lane; j < nblocks; j += 32) {
        const uint32_t other = keys[j];
#pragma unroll
        for (int q = 0; q < 4; ++q) below[q] += other < mine[q] ? 1u : 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (m0 + q * WARPS >= nblocks) break;
        const int64_t place = __reduce_add_sync(0xffffffffu, below[q]), blk = m0 + q * WARPS;
        for (int i = lane; i < block; i += 32) sorted_ids[place * block + i] = blk * block + i;
      }
    }
    return;
  }
  // bitonic sort of (inverted key, block id), every CTA for itself
  for (int size = 2; size <= npow2; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < (npow2 >> 1); i += RANK_THREADS) {
        const int lo = 2 * i - (i & (stride - 1));  // index with the `stride` bit clear
        const int hi = lo + stride;
        const bool up = (lo & size) == 0;
        const uint32_t a = keys[lo], b = keys[hi];
        if ((a > b) == up) {
          keys[lo] = b;
          keys[hi] = a;
        }
      }
      __syncthreads();
    }
  }
  for (int64_t i = static_cast<int64_t>(crank) * RANK_THREADS + threadIdx.x; i < total; i += RANK_THREADS * RANK_CLUSTER) {
    const int j = static_cast<int>(i / block);
    const int64_t blk = keys[j] & 0xFFFFu;
    sorted_ids[i] = blk * block + (i - static_cast<int64_t>(j) * block);
  }
}

// ------------------------------------------------------------------------------------------------
// flush plan: one thread-block cluster
// ------------------------------------------------------------------------------------------------
constexpr int PLAN_THREADS = 1024;
constexpr int PLAN_CLUSTER = 8;   // CTAs of the cluster (the portable maximum)

struct PlanSide {
  const int64_t* tier_idx[HQKV_NUM_TIERS];
  int32_t tier_n[HQKV_NUM_TIERS];
  int64_t cum[6];
  const int64_t* sorted_ids;
  int32_t* plan_src;   // [5][total]
  int64_t* plan_ids;   // [5][total]
  int64_t* survivors;  // [total]
  int32_t* counts;     // [8]
  int32_t done;        // what counts[7] says when the others are there (memory of the host: it polls)
  // scratch
  int8_t* tgt;         // [total] by token id, 16-byte aligned
  int8_t* fin;         // [total] by enumeration slot: category
  int32_t* rank;       // [total] by token id: rank among survivors
  int32_t* gcnt;       // [PLAN_CATS][PLAN_CLUSTER * PLAN_WARPS] per-warp category counts of the whole cluster
};
struct PlanArgs {
  PlanSide side;
  int64_t hist, compress;
};

// Enumeration order of every cached token: residual (ascending id), then the 16-, 8-, 4-, 2-, 1-bit
// tier in storage order.  Slot -> (source tier, position, token id).
__device__ __forceinline__ void enum_slot(const PlanArgs& A, const PlanSide& S, int64_t slot, int& src, int32_t& pos, int64_t& id) {
  if (slot < A.compress) {
    src = -1;
    pos = static_cast<int32_t>(slot);
    id = A.hist + slot;
    return;
  }
  int32_t s = static_cast<int32_t>(slot - A.compress);
  src = -2;
  pos = 0;
  id = 0;
#pragma unroll
  for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
    if (src == -2 && s < S.tier_n[t]) {
      src = t;
      pos = s;
      id = S.tier_idx[t][s];
    }
    s -= S.tier_n[t];
  }
}

// One cluster of PLAN_CLUSTER CTAs of 32 warps.  Every pass walks the enumeration (or the token ids) in
// warp-contiguous ranges - warp w of CTA r is range r * 32 + w - PLAN_BATCH iterations at a time so that the
// dependent loads of a batch (index list -> target -> rank) are in flight together; ordered positions come from
// per-warp counts (left in global memory for the other CTAs), one scan over all warps of the cluster, and ballot /
// match prefixes inside a warp.  The passes are separated by cluster barriers, which also order the global-memory
// scratch between the CTAs.  Categories: 2*t = kept member of tier t, 2*t + 1 = arrival in tier t (destination
// order: kept members first, then arrivals, both in enumeration order); 10 = surviving token id.
// What bounds it is the chain of dependent L2 round trips, two or three per pass: survival read off the targets instead
// of a pass of its own, and the scan by one warp per category instead of 256 steps by one thread took the plan of a
// 32 k-token flush from 24.5 us to 17 us.
constexpr int PLAN_WARPS = PLAN_THREADS / 32;
constexpr int PLAN_GWARPS = PLAN_WARPS * PLAN_CLUSTER;
constexpr int PLAN_BATCH = 4;
constexpr int PLAN_CATS = 2 * HQKV_NUM_TIERS + 1;
constexpr int PLAN_NONE = PLAN_CATS;  // no destination: evicted, or residual without a target

__global__ void __launch_bounds__(PLAN_THREADS) flush_plan_kernel(const __grid_constant__ PlanArgs A) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ int cnt[PLAN_CATS + 1][PLAN_WARPS];  // per-warp totals, then their exclusive offsets over the cluster
  __shared__ int tot[PLAN_CATS];
  const PlanSide& S = A.side;
  const int64_t total = A.hist + A.compress;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int crank = static_cast<int>(cluster.block_rank());
  const int gwarp = crank * PLAN_WARPS + warp;
  const int64_t gtid = static_cast<int64_t>(crank) * PLAN_THREADS + tid;
  constexpr int64_t GTHREADS = static_cast<int64_t>(PLAN_THREADS) * PLAN_CLUSTER;
  const unsigned lt = (1u << lane) - 1u;
  // warp gw owns elements [gw * span, (gw + 1) * span), span a multiple of 32
  const int64_t iters = (total + GTHREADS - 1) / GTHREADS;
  const int64_t span = iters * 32, first = gwarp * span;
  const bool any_evict = S.cum[5] > S.cum[4];
  if (tid < (PLAN_CATS + 1) * PLAN_WARPS) (&cnt[0][0])[tid] = 0;
  // 1. targets by token id (-1: not in the ranked list)
  for (int64_t i = gtid; i < (total + 15) / 16; i += GTHREADS)
    reinterpret_cast<uint4*>(S.tgt)[i] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
  cluster.sync();
#pragma unroll 4
  for (int64_t j = gtid; j < S.cum[5]; j += GTHREADS) {
    int t = 0;
#pragma unroll
    for (int k = 0; k < 5; ++k) t += j >= S.cum[k] ? 1 : 0;
    const int64_t id = S.sorted_ids[j];
    if (HQKV_INDEX_OK(id, total)) S.tgt[id] = static_cast<int8_t>(t);
  }
  cluster.sync();
  // 2. category of every enumeration slot; per-warp counts of the categories and of the surviving token ids
  int mine = 0;
  for (int64_t j0 = 0; j0 < iters; j0 += PLAN_BATCH) {
    int src[PLAN_BATCH], tg[PLAN_BATCH], own[PLAN_BATCH];
    int64_t id[PLAN_BATCH];
#pragma unroll
    for (int u = 0; u < PLAN_BATCH; ++u) {
      const int64_t s = first + (j0 + u) * 32 + lane;
      int32_t pos;
      src[u] = -2;
      id[u] = 0;
      own[u] = 5;
      if (j0 + u < iters && s < total) {
        enum_slot(A, S, s, src[u], pos, id[u]);
        own[u] = S.tgt[s];
      }
    }
#pragma unroll
    for (int u = 0; u < PLAN_BATCH; ++u) tg[u] = (src[u] != -2 && HQKV_INDEX_OK(id[u], total)) ? S.tgt[id[u]] : -1;
#pragma unroll
    for (int u = 0; u < PLAN_BATCH; ++u) {
      const int64_t s = first + (j0 + u) * 32 + lane;
      int cat = PLAN_NONE;
      if (src[u] != -2 && tg[u] != 5) {
        const int f = tg[u] > src[u] ? tg[u] : src[u];  // only moves to fewer bits (larger index); tg == -1 stays
        if (f >= 0) cat = 2 * f + (src[u] == f ? 0 : 1);
      }
      if (src[u] != -2) S.fin[s] = static_cast<int8_t>(cat);
      const unsigned same = __match_any_sync(0xffffffffu, cat);
      if ((same & lt) == 0) cnt[cat][warp] += __popc(same);  // (one lane per category; the row is this warp's)
      __syncwarp();
      mine += own[u] != 5 ? 1 : 0;
    }
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) cnt[PLAN_CATS - 1][warp] = mine;
  __syncthreads();
  // this CTA's per-warp totals -> global memory, for the scan over all warps of the cluster
  if (tid < PLAN_CATS * PLAN_WARPS) {
    const int c = tid / PLAN_WARPS, w = tid - c * PLAN_WARPS;
    S.gcnt[c * PLAN_GWARPS + crank * PLAN_WARPS + w] = cnt[c][w];
  }
  cluster.sync();
  // exclusive offsets of every category over the warps of the cluster (every CTA scans for its own warps): warp =
  // category, eight cluster warps per lane
  static_assert(PLAN_GWARPS == 256, "eight counts per lane");
  if (warp < PLAN_CATS) {
    const int4* g = reinterpret_cast<const int4*>(S.gcnt + warp * PLAN_GWARPS) + 2 * lane;
    const int4 a = __ldcg(g), b = __ldcg(g + 1);
    const int v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    int sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) sum += v[i];
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    int run = incl - sum;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int w = 8 * lane + i - crank * PLAN_WARPS;
      if (w >= 0 && w < PLAN_WARPS) cnt[warp][w] = run;
      run += v[i];
    }
    if (lane == 31) tot[warp] = incl;
  }
  __syncthreads();
  if (crank == 0) {
    if (tid == 0) {
      volatile int32_t* c = S.counts;
#pragma unroll
      for (int t = 0; t < HQKV_NUM_TIERS; ++t) c[t] = tot[2 * t] + tot[2 * t + 1];
      c[5] = tot[PLAN_CATS - 1];
      c[6] = any_evict ? 1 : 0;
      __threadfence_system();
      c[7] = S.done;
    }
  }
  // 3. survivor ranks by token id: rank[i] = survivors with a smaller id; survivors[rank] = id
  {
    int running = cnt[PLAN_CATS - 1][warp];
    for (int64_t j0 = 0; j0 < iters; j0 += PLAN_BATCH) {
      int own[PLAN_BATCH];
#pragma unroll
      for (int u = 0; u < PLAN_BATCH; ++u) {
        const int64_t i = first + (j0 + u) * 32 + lane;
        own[u] = (j0 + u < iters && i < total) ? S.tgt[i] : 5;
      }
#pragma unroll
      for (int u = 0; u < PLAN_BATCH; ++u) {
        const unsigned ballot = __ballot_sync(0xffffffffu, own[u] != 5);
        const int64_t i = first + (j0 + u) * 32 + lane;
        const int r = running + __popc(ballot & lt);
        if (any_evict && i < total && j0 + u < iters) S.rank[i] = r;
        if (own[u] != 5) S.survivors[r] = i;
        running += __popc(ballot);
      }
    }
  }
  if (any_evict) cluster.sync();
  // 4. destination lists
  for (int64_t j0 = 0; j0 < iters; j0 += PLAN_BATCH) {
    int src[PLAN_BATCH], cat[PLAN_BATCH];
    int32_t pos[PLAN_BATCH];
    int64_t id[PLAN_BATCH];
#pragma unroll
    for (int u = 0; u < PLAN_BATCH; ++u) {
      const int64_t s = first + (j0 + u) * 32 + lane;
      src[u] = -2;
      pos[u] = 0;
      id[u] = 0;
      cat[u] = PLAN_NONE;
      if (j0 + u < iters && s < total) {
        enum_slot(A, S, s, src[u], pos[u], id[u]);
        cat[u] = S.fin[s];
      }
    }
    if (any_evict) {
#pragma unroll
      for (int u = 0; u < PLAN_BATCH; ++u)
        if (cat[u] != PLAN_NONE) id[u] = __ldcg(S.rank + id[u]);
    }
#pragma unroll
    for (int u = 0; u < PLAN_BATCH; ++u) {
      const unsigned same = __match_any_sync(0xffffffffu, cat[u]);
      const int base = cnt[cat[u]][warp];  // this warp's running offset of the category (only this warp touches it)
      __syncwarp();
      if (cat[u] != PLAN_NONE) {
        const int64_t j = (cat[u] & 1 ? tot[cat[u] - 1] : 0) + base + __popc(same & lt), at = (cat[u] >> 1) * total + j;
        S.plan_src[at] = ((src[u] + 1) << 28) | pos[u];
        S.plan_ids[at] = id[u];
        if ((same & lt) == 0) cnt[cat[u]][warp] = base + __popc(same);
      }
      __syncwarp();
    }
  }
}

__global__ void __launch_bounds__(256) gather_columns_kernel(const __half* __restrict__ in, int64_t in_stride,
                                                             const int64_t* __restrict__ ids, int64_t n,
                                                             __half* __restrict__ out, int64_t out_stride) {
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int r = blockIdx.y;
  out[r * out_stride + j] = in[r * in_stride + ids[j]];
}

}  // namespace hqkv

using namespace hqkv;

extern "C" int hqkv_head_sum(const void* w, int B, int nh, int64_t L, int64_t bh_stride, void* out, void* stream) {
  HQKV_REQUIRE(B > 0 && nh > 0 && L >= 0 && bh_stride >= L, "head_sum: bad sizes");
  if (L == 0) return HQKV_OK;
  HQKV_REQUIRE(w && out, "head_sum: null pointer");
  // may be placed while the V pass before it drains (the wait for it is the kernel's first instruction): 1-2 us a decode step
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ceil_div(L, 32)));
  cfg.blockDim = dim3(HEAD_SUM_THREADS);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HQKV_CUDA(cudaLaunchKernelEx(&cfg, head_sum_kernel, static_cast<const __half*>(w), B, nh, L, bh_stride, static_cast<__half*>(out)));
  HQKV_LAUNCH_CHECK("head_sum");
  return HQKV_OK;
}

extern "C" int hqkv_token_importance(const void* ring, int rows, int64_t ring_stride, int64_t L, void* out,
                                     void* stream) {
  HQKV_REQUIRE(rows > 0 && L >= 0 && ring_stride >= L, "token_importance: bad sizes");
  if (L == 0) return HQKV_OK;
  HQKV_REQUIRE(ring && out, "token_importance: null pointer");
  token_importance_kernel<<<static_cast<unsigned>(ceil_div(L, 256)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __half*>(ring), rows, ring_stride, L, static_cast<__half*>(out));
  HQKV_LAUNCH_CHECK("token_importance");
  return HQKV_OK;
}

// Ranges of T tokens behind the n_old that are copied.
static int launch_range(const void* v, int B, int H, int64_t T, int64_t b_stride, int64_t h_stride, const void* old, int64_t n_old,
                        void* out, void* stream) {
  // tokens per CTA: one until every SM has four CTAs, then up to sixteen, of 4096 rows between
  // them (with RANGE_MAX_ROWS rows to a token: 32 KB of row offsets and 8 KB of ranges)
  const int n = B * H;
  int tshift = 0;
  while (tshift < 4 && T >> (tshift + 1) >= 4 * 148 && (static_cast<int64_t>(n) << (tshift + 1)) <= RANGE_MAX_ROWS) ++tshift;
  const int64_t ctas = ceil_div(T, 1 << tshift), copies = ceil_div(n_old, 8 * RANGE_THREADS);
  token_range128_kernel<<<static_cast<unsigned>(ctas + copies), RANGE_THREADS, n * sizeof(int64_t) + (static_cast<size_t>(n) << tshift) * sizeof(__half),
                          static_cast<cudaStream_t>(stream)>>>(static_cast<const __half*>(v), B, n, T, b_stride, h_stride, tshift,
                                                               static_cast<const __half*>(old), n_old, static_cast<int>(ctas),
                                                               static_cast<__half*>(out));
  HQKV_LAUNCH_CHECK("token_range");
  return HQKV_OK;
}

extern "C" int hqkv_token_range(const void* v, int B, int H, int64_t T, int Dd, int64_t b_stride, int64_t h_stride,
                                void* out, void* stream) {
  HQKV_REQUIRE(B > 0 && H > 0 && T >= 0 && Dd >= 32, "token_range: bad sizes");
  if (T == 0) return HQKV_OK;
  HQKV_REQUIRE(v && out, "token_range: null pointer");
  if (Dd == 128 && aligned(v, 16) && b_stride % 8 == 0 && h_stride % 8 == 0 && static_cast<int64_t>(B) * H <= RANGE_MAX_ROWS)
    return launch_range(v, B, H, T, b_stride, h_stride, nullptr, 0, out, stream);
  token_range_kernel<<<static_cast<unsigned>(ceil_div(T, 4)), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __half*>(v), B, H, T, Dd, b_stride, h_stride, static_cast<__half*>(out));
  HQKV_LAUNCH_CHECK("token_range");
  return HQKV_OK;
}

static cudaLaunchConfig_t cluster_config(cudaLaunchAttribute* attr, int ctas, int rows, int threads, size_t smem, void* stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, rows);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// importance -> (x range) / block -> `divided` (may be importance itself) -> token ids in ranked order
static int launch_rank(const void* importance, const void* range_or_null, void* divided, int block, int nblocks, int64_t* sorted_ids,
                       void* stream) {
  int npow2 = 2;
  while (npow2 < nblocks) npow2 <<= 1;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = cluster_config(attr, RANK_CLUSTER, 1, RANK_THREADS, npow2 * sizeof(uint32_t), stream);
  HQKV_CUDA(cudaLaunchKernelEx(&cfg, block_rank_kernel, static_cast<const __half*>(importance),
                               static_cast<const __half*>(range_or_null), static_cast<__half*>(divided), block, nblocks, npow2,
                               sorted_ids));
  return HQKV_OK;
}

extern "C" int hqkv_block_rank(void* importance, const void* range_or_null, int block, int nblocks,
                               int64_t* sorted_ids, void* stream) {
  HQKV_REQUIRE(block > 0 && nblocks >= 0, "block_rank: bad sizes");
  HQKV_REQUIRE(nblocks <= RANK_MAX_BLOCKS, "block_rank: at most %d blocks (got %d)", RANK_MAX_BLOCKS, nblocks);
  if (nblocks == 0) return HQKV_OK;
  HQKV_REQUIRE(importance && sorted_ids, "block_rank: null pointer");
  return launch_rank(importance, range_or_null, importance, block, nblocks, sorted_ids, stream);
}

extern "C" size_t hqkv_flush_plan_workspace_bytes(int64_t total) {
  if (total < 0) return 0;
  const size_t t = static_cast<size_t>(total);
  // tgt (1 B) + fin (1 B) + rank (4 B) per token, each region rounded to 256 bytes; per-warp counts; and what it takes to
  // start on a 16-byte boundary
  auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  return up(t) + up(t) + up(4 * t) + up(sizeof(int32_t) * PLAN_CATS * PLAN_GWARPS) + 15;
}

static int fill_plan_side(PlanSide& S, const int64_t* const* tier_idx_host, const int32_t* tier_n_host, int64_t hist, int64_t total,
                          const int64_t* sorted_ids, const int64_t* cum_counts_host, int32_t* plan_src, int64_t* plan_ids,
                          int64_t* survivors, int32_t* counts, unsigned char* ws) {
  int64_t in_tiers = 0;
  for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
    HQKV_REQUIRE(tier_n_host[t] >= 0, "flush_plan: negative tier size");
    HQKV_REQUIRE(tier_n_host[t] == 0 || tier_idx_host[t], "flush_plan: tier %d has tokens but no id list", t);
    S.tier_idx[t] = tier_idx_host[t];
    S.tier_n[t] = tier_n_host[t];
    in_tiers += tier_n_host[t];
  }
  HQKV_REQUIRE(in_tiers == hist, "flush_plan: tiers hold %lld tokens but history_length is %lld", (long long)in_tiers,
               (long long)hist);
  int64_t prev = 0;
  for (int k = 0; k < 6; ++k) {
    HQKV_REQUIRE(cum_counts_host[k] >= prev && cum_counts_host[k] <= total,
                 "flush_plan: cumulative counts must be non-decreasing and at most hist+compress");
    S.cum[k] = cum_counts_host[k];
    prev = cum_counts_host[k];
  }
  auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  ws += -reinterpret_cast<uintptr_t>(ws) & 15;
  S.tgt = reinterpret_cast<int8_t*>(ws);
  S.fin = reinterpret_cast<int8_t*>(ws + up(total));
  S.rank = reinterpret_cast<int32_t*>(ws + 2 * up(total));
  S.gcnt = reinterpret_cast<int32_t*>(ws + 2 * up(total) + up(4 * static_cast<size_t>(total)));
  S.sorted_ids = sorted_ids;
  S.plan_src = plan_src;
  S.plan_ids = plan_ids;
  S.survivors = survivors;
  S.counts = counts;
  return HQKV_OK;
}
static int launch_plan(const PlanArgs& A, void* stream) {
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = cluster_config(attr, PLAN_CLUSTER, 1, PLAN_THREADS, 0, stream);
  HQKV_CUDA(cudaLaunchKernelEx(&cfg, flush_plan_kernel, A));
  return HQKV_OK;
}

extern "C" int hqkv_flush_plan(const int64_t* const* tier_idx_host, const int32_t* tier_n_host, int64_t hist,
                               int64_t compress, const int64_t* sorted_ids, const int64_t* cum_counts_host,
                               int32_t* plan_src, int64_t* plan_ids, int64_t* survivors, int32_t* counts,
                               void* workspace, size_t workspace_bytes, void* stream) {
  HQKV_REQUIRE(tier_idx_host && tier_n_host && cum_counts_host, "flush_plan: null host pointer");
  HQKV_REQUIRE(hist >= 0 && compress >= 0, "flush_plan: negative length");
  const int64_t total = hist + compress;
  HQKV_REQUIRE(total > 0 && total < (1ll << 28), "flush_plan: total length out of range");
  HQKV_REQUIRE(sorted_ids && plan_src && plan_ids && survivors && counts && workspace, "flush_plan: null pointer");
  PlanArgs A;
  memset(&A, 0, sizeof(A));
  A.hist = hist;
  A.compress = compress;
  int rc = fill_plan_side(A.side, tier_idx_host, tier_n_host, hist, total, sorted_ids, cum_counts_host, plan_src, plan_ids,
                          survivors, counts, static_cast<unsigned char*>(workspace));
  if (rc) return rc;
  const size_t need = hqkv_flush_plan_workspace_bytes(total) - 15 + (-reinterpret_cast<uintptr_t>(workspace) & 15);
  if (workspace_bytes < need)
    return fail(HQKV_E_WORKSPACE, "flush_plan: workspace holds %zu bytes, %zu needed", workspace_bytes, need);
  return launch_plan(A, stream);
}

// ------------------------------------------------------------------------------------------------
// a whole flush: scratch of both sides in one piece
// ------------------------------------------------------------------------------------------------
namespace hqkv {
struct FlushScratch {
  int32_t* plan_src[2];
  int64_t* plan_ids[2];
  int64_t* survivors[2];
  unsigned char* plan_ws[2];
  int64_t* v_sorted;
  __half* v_keys;
  size_t bytes;
};
static FlushScratch flush_scratch(void* base, int64_t total) {
  auto up = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  const size_t t = static_cast<size_t>(total);
  unsigned char* p = static_cast<unsigned char*>(base);
  FlushScratch s;
  size_t at = 0;
  for (int side = 0; side < 2; ++side) {
    s.plan_src[side] = reinterpret_cast<int32_t*>(p + at), at += up(HQKV_NUM_TIERS * t * 4);
    s.plan_ids[side] = reinterpret_cast<int64_t*>(p + at), at += up(HQKV_NUM_TIERS * t * 8);
    s.survivors[side] = reinterpret_cast<int64_t*>(p + at), at += up(t * 8);
    s.plan_ws[side] = p + at, at += up(hqkv_flush_plan_workspace_bytes(total));
  }
  s.v_sorted = reinterpret_cast<int64_t*>(p + at), at += up(t * 8);
  s.v_keys = reinterpret_cast<__half*>(p + at), at += up(t * 2);
  s.bytes = at;
  return s;
}

// Survivors to the front, ascending ids, in place: ids[j] >= j, so a CTA that owns a row and walks it in order reads only
// what it has not written yet.  The last row is the range vector, which goes to another buffer.
constexpr int EVICT_THREADS = 1024;
constexpr int EVICT_PER = 8;
__global__ void __launch_bounds__(EVICT_THREADS) evict_kernel(__half* ring, int64_t stride, int rows, const int64_t* __restrict__ ids,
                                                              int64_t n, const __half* norm, __half* norm_kept) {
  const bool is_norm = static_cast<int>(blockIdx.x) == rows;
  const __half* in = is_norm ? norm : ring + blockIdx.x * stride;
  __half* out = is_norm ? norm_kept : ring + blockIdx.x * stride;
  for (int64_t base = 0; base < n; base += EVICT_THREADS * EVICT_PER) {
    __half v[EVICT_PER];
#pragma unroll
    for (int i = 0; i < EVICT_PER; ++i) {
      const int64_t j = base + i * EVICT_THREADS + threadIdx.x;
      v[i] = in[ids[j < n ? j : n - 1]];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < EVICT_PER; ++i) {
      const int64_t j = base + i * EVICT_THREADS + threadIdx.x;
      if (j < n) out[j] = v[i];
    }
    __syncthreads();
  }
}
}  // namespace hqkv

namespace hqkv {
// What a thread keeps between its flushes: two streams, six events, and 64 bytes of host memory that the plans write
// the counts to - they are there as soon as the tokens are counted, while the plan still writes its lists, and no copy has
// to be launched.  Made on first use, for one device at a time; given back when the thread ends.
struct FlushLane {
  int dev = -1;
  cudaStream_t side = nullptr, build = nullptr;   // V side; K build
  cudaEvent_t fork = nullptr, join = nullptr;
  cudaEvent_t ready[2] = {}, built[2] = {};       // a side's outputs may be written; are written
  bool building[2] = {};                          // ... and the caller's stream does not wait for that yet
  volatile int32_t* host = nullptr;
  int32_t calls = 0;
  int open() {
    int now = 0;
    HQKV_CUDA(cudaGetDevice(&now));
    if (!host) {
      void* p = nullptr;
      HQKV_CUDA(cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped));
      memset(p, 0, 64);
      host = static_cast<volatile int32_t*>(p);
    }
    if (now == dev) return HQKV_OK;
    close();
    int least = 0, greatest = 0;  // ahead of the K build's CTAs: the V side's clusters need room on eight SMs at once
    HQKV_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    HQKV_CUDA(cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking, greatest));
    HQKV_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    HQKV_CUDA(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
    HQKV_CUDA(cudaStreamCreateWithPriority(&build, cudaStreamNonBlocking, least));
    for (int i = 0; i < 2; ++i) {
      HQKV_CUDA(cudaEventCreateWithFlags(&ready[i], cudaEventDisableTiming));
      HQKV_CUDA(cudaEventCreateWithFlags(&built[i], cudaEventDisableTiming));
    }
    dev = now;
    return HQKV_OK;
  }
  void close() {
    // a plan that nobody waited for (a call that ended early) may still write its counts: not into memory that is given back,
    // nor after those of the next plan
    if (side) cudaStreamSynchronize(side), cudaStreamDestroy(side);
    if (build) cudaStreamSynchronize(build), cudaStreamDestroy(build);
    for (cudaEvent_t* e : {&fork, &join, &ready[0], &ready[1], &built[0], &built[1]}) {
      if (*e) cudaEventDestroy(*e);
      *e = nullptr;
    }
    side = build = nullptr, building[0] = building[1] = false, dev = -1;
  }
  // waits for the counts of a side whose plan is in stream st
  int counts(int v_side, cudaStream_t st, int32_t* out) {
    const volatile int32_t* c = host + 8 * v_side;
    for (int spins = 0; c[7] != calls; ++spins) {
      if ((spins & 0xFFFF) != 0xFFFF) continue;
      const cudaError_t e = cudaStreamQuery(st);  // an error of the stream ends the wait
      if (e == cudaErrorNotReady) continue;
      HQKV_CUDA(e);
      HQKV_REQUIRE(c[7] == calls, "flush: the plan left no counts");
    }
    for (int i = 0; i < 8; ++i) out[i] = c[i];
    return HQKV_OK;
  }
  ~FlushLane() {
    close();
    if (host) cudaFreeHost(const_cast<int32_t*>(host));
  }
};
static thread_local FlushLane flush_lane;
}  // namespace hqkv

extern "C" size_t hqkv_flush_workspace_bytes(int64_t total) { return total < 0 ? 0 : flush_scratch(nullptr, total).bytes; }

extern "C" int hqkv_flush_prepare(const hqkv_flush_t* f, void* workspace, size_t workspace_bytes, int32_t* counts_host, void* stream) {
  HQKV_REQUIRE(f && workspace && counts_host, "flush_prepare: null pointer");
  HQKV_REQUIRE(f->D == D && f->B > 0 && f->H > 0, "flush_prepare: bad sizes");
  HQKV_REQUIRE(f->hist >= 0 && f->compress > 0 && f->rest >= 0, "flush_prepare: negative length");
  const int64_t total = f->hist + f->compress;
  HQKV_REQUIRE(total < (1ll << 28), "flush_prepare: total length out of range");
  HQKV_REQUIRE(f->block > 0 && total % f->block == 0 && total / f->block <= RANK_MAX_BLOCKS,
               "flush_prepare: %lld tokens are not 1..%d blocks of %d", (long long)total, RANK_MAX_BLOCKS, f->block);
  HQKV_REQUIRE(f->importance && f->k_sorted && f->norm_out && f->v.residual && (f->hist == 0 || f->norm_old), "flush_prepare: null pointer");
  HQKV_REQUIRE(aligned(workspace, 256), "flush_prepare: workspace must be 256-byte aligned");
  const FlushScratch s = flush_scratch(workspace, total);
  if (workspace_bytes < s.bytes)
    return fail(HQKV_E_WORKSPACE, "flush_prepare: workspace holds %zu bytes, %zu needed", workspace_bytes, s.bytes);
  HQKV_REQUIRE(aligned(f->v.residual, 16) && f->v.residual_b_stride % 8 == 0 && f->v.residual_h_stride % 8 == 0 &&
                   static_cast<int64_t>(f->B) * f->H <= RANGE_MAX_ROWS,
               "flush_prepare: the residual window must be 16-byte aligned, B*H at most %d", RANGE_MAX_ROWS);
  PlanArgs A[2];
  memset(A, 0, sizeof(A));
  for (int side = 0; side < 2; ++side) {
    A[side].hist = f->hist;
    A[side].compress = f->compress;
    const int rc = fill_plan_side(A[side].side, side ? f->v_idx : f->k_idx, side ? f->v.n : f->k.n, f->hist, total,
                                  side ? s.v_sorted : f->k_sorted, side ? f->v_cum : f->k_cum, s.plan_src[side], s.plan_ids[side],
                                  s.survivors[side], nullptr, s.plan_ws[side]);
    if (rc) return rc;
  }
  FlushLane& lane = flush_lane;
  int rc = lane.open();
  if (rc) return rc;
  void* counts_dev = nullptr;
  HQKV_CUDA(cudaHostGetDevicePointer(&counts_dev, const_cast<int32_t*>(lane.host), 0));
  lane.calls = lane.calls == 0x7FFFFFFF ? 1 : lane.calls + 1;
  for (int side = 0; side < 2; ++side) {
    A[side].side.counts = static_cast<int32_t*>(counts_dev) + 8 * side;
    A[side].side.done = lane.calls;
  }
  // ranges, ranking and plan of the V side beside the plan and the build of the K side, which need none of them
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  HQKV_CUDA(cudaEventRecord(lane.fork, st));
  HQKV_CUDA(cudaStreamWaitEvent(lane.side, lane.fork, 0));
  rc = launch_plan(A[0], st);
  if (!rc)
    rc = launch_range(f->v.residual, f->B, f->H, f->compress, f->v.residual_b_stride, f->v.residual_h_stride, f->norm_old, f->hist,
                      f->norm_out, lane.side);
  if (!rc)
    rc = launch_rank(f->importance, f->times_range ? f->norm_out : nullptr, s.v_keys, f->block, static_cast<int>(total / f->block),
                     s.v_sorted, lane.side);
  if (!rc) rc = launch_plan(A[1], lane.side);
  const int rec = check_cuda(cudaEventRecord(lane.join, lane.side), "flush_prepare: event");
  if (!rc && !rec) rc = lane.counts(0, st, counts_host);
  if (rc || rec) {
    cudaStreamWaitEvent(st, lane.join, 0);
    return rc ? rc : rec;
  }
  return HQKV_OK;
}

extern "C" int hqkv_flush_join(int32_t* counts_host, void* stream) {
  FlushLane& lane = flush_lane;
  HQKV_REQUIRE(lane.side && lane.calls, "flush_join: this thread has prepared no flush");
  HQKV_CUDA(cudaStreamWaitEvent(static_cast<cudaStream_t>(stream), lane.join, 0));
  return counts_host ? lane.counts(1, lane.side, counts_host + 8) : HQKV_OK;
}

extern "C" int hqkv_flush_tiers(const hqkv_flush_t* f, int v_side, const void* workspace, const int32_t* counts_host,
                                void* const* out_data_host, void* const* out_scale_host, void* const* out_zero_host,
                                int64_t* const* out_ids_host, void* rest_out, void* stream) {
  HQKV_REQUIRE(f && workspace && counts_host, "flush_tiers: null pointer");
  const int64_t total = f->hist + f->compress;
  const int side = v_side ? 1 : 0;
  const FlushScratch s = flush_scratch(const_cast<void*>(workspace), total);
  return hqkv_flush_build(side, side ? &f->v : &f->k, f->B, f->H, f->D, side ? f->group : f->block, s.plan_src[side], s.plan_ids[side],
                          total, counts_host + 8 * side, out_data_host, out_scale_host, out_zero_host, out_ids_host, f->compress,
                          f->rest, rest_out, stream);
}

// The builds of the two sides beside each other: each waits for little else than its plan and memory, and neither fills the
// GPU (small flush: 33 and 18 us one after the other).  Neither is put into the caller's stream: what is written to was
// allocated for that stream, so each waits for what the stream holds by then, and that must not be the other.
// Below a line of work (rows that are copied, new ones four times) the six calls for streams and events cost the host more
// than the overlap gives: there both go into the caller's stream.  us, one after the other / beside: 8 planes, 32 tokens into
// 12 k 76 / 82, 24 k 87 / 80; 32 planes, 32 into 3 k 73.8 / 74.6, 5 k 78.6 / 74.8; 64 planes, 32 into 4 k 92 / 76; 8 planes,
// first flush of 4 k 77.7 / 77.4, 8 k 85 / 78, 16 k 114 / 96.
constexpr int64_t FLUSH_BESIDE_WORK = 160 << 10;
extern "C" int hqkv_flush_tiers_beside(const hqkv_flush_t* f, int v_side, const void* workspace, const int32_t* counts_host,
                                       void* const* out_data_host, void* const* out_scale_host, void* const* out_zero_host,
                                       int64_t* const* out_ids_host, void* rest_out, void* stream) {
  HQKV_REQUIRE(f && workspace && counts_host, "flush_tiers_beside: null pointer");
  FlushLane& lane = flush_lane;
  HQKV_REQUIRE(lane.side && lane.calls, "flush_tiers_beside: this thread has prepared no flush");
  const int side = v_side ? 1 : 0;
  if (static_cast<int64_t>(f->B) * f->H * (f->hist + 4 * f->compress) < FLUSH_BESIDE_WORK)
    return hqkv_flush_tiers(f, v_side, workspace, counts_host, out_data_host, out_scale_host, out_zero_host, out_ids_host, rest_out, stream);
  const cudaStream_t own = side ? lane.side : lane.build;
  HQKV_CUDA(cudaEventRecord(lane.ready[side], static_cast<cudaStream_t>(stream)));
  HQKV_CUDA(cudaStreamWaitEvent(own, lane.ready[side], 0));
  const int rc = hqkv_flush_tiers(f, v_side, workspace, counts_host, out_data_host, out_scale_host, out_zero_host, out_ids_host, rest_out, own);
  if (const int failed = check_cuda(cudaEventRecord(lane.built[side], own), "cudaEventRecord")) {
    cudaStreamSynchronize(own);   // (there is no event to wait for, and the caller may let the memory go)
    return failed;
  }
  lane.building[side] = true;
  return rc;
}

extern "C" int hqkv_flush_finish(void* stream) {
  FlushLane& lane = flush_lane;
  int rc = HQKV_OK;
  for (int side = 0; side < 2; ++side)
    if (lane.building[side]) {
      lane.building[side] = false;
      if (const int failed = check_cuda(cudaStreamWaitEvent(static_cast<cudaStream_t>(stream), lane.built[side], 0), "cudaStreamWaitEvent")) {
        cudaEventSynchronize(lane.built[side]);
        rc = failed;
      }
    }
  return rc;
}

extern "C" int hqkv_flush_evict(const hqkv_flush_t* f, const void* workspace, int64_t survivors, void* norm_kept, void* ring,
                                int64_t ring_stride, int ring_rows, void* stream) {
  HQKV_REQUIRE(f && workspace && norm_kept && ring_rows >= 0 && (ring_rows == 0 || ring), "flush_evict: null pointer");
  const int64_t total = f->hist + f->compress;
  HQKV_REQUIRE(survivors >= 0 && survivors <= total && (ring_rows == 0 || ring_stride >= total), "flush_evict: bad sizes");
  if (survivors == 0) return HQKV_OK;
  const FlushScratch s = flush_scratch(const_cast<void*>(workspace), total);
  evict_kernel<<<ring_rows + 1, EVICT_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__half*>(ring), ring_stride, ring_rows, s.survivors[1], survivors, static_cast<const __half*>(f->norm_out),
      static_cast<__half*>(norm_kept));
  HQKV_LAUNCH_CHECK("flush_evict");
  return HQKV_OK;
}

extern "C" int hqkv_gather_columns_f16(const void* in, int64_t in_stride, int rows, const int64_t* ids, int64_t n,
                                       void* out, int64_t out_stride, void* stream) {
  HQKV_REQUIRE(rows >= 0 && n >= 0, "gather_columns: negative size");
  if (rows == 0 || n == 0) return HQKV_OK;
  HQKV_REQUIRE(in && ids && out, "gather_columns: null pointer");
  HQKV_REQUIRE(rows <= 65535, "gather_columns: too many rows");
  gather_columns_kernel<<<dim3(static_cast<unsigned>(ceil_div(n, 256)), rows), 256, 0,
                          static_cast<cudaStream_t>(stream)>>>(static_cast<const __half*>(in), in_stride, ids, n,
                                                               static_cast<__half*>(out), out_stride);
  HQKV_LAUNCH_CHECK("gather_columns");
  return HQKV_OK;
}
