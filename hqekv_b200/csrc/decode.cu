// Fused mixed-precision decode attention over the tiered KV cache (sm_100a).
//
// Two launches per call:
//   k_pass : logits[pos][h] = scale * q_h . K^_pos for every tier (8/4/2/1-bit packed, fp16 tier,
//            fp16 residual), written to an fp32 scratch at the tokens' logical positions,
//            plus one (max, sum-exp) pair per CTA and head.
//   v_pass : every CTA first folds the k_pass pairs into the global (max, sum) of its heads; each
//            warp then writes the normalised probabilities of its own tokens and accumulates
//            sum_t exp(logit_t - max) * V^_t over them; the CTA's part of the output joins pairs of
//            64-bit words, and whoever completes a pair normalises and writes fp16 (weights given by the caller, and
//            outputs that peers get too: fp64 sums, written by the last CTA of each (batch, kv head)).
//
// The roofline is HBM: every packed word, scale and zero is read exactly once per call and is
// shared by the query heads of its kv head (GQA).  At 2-4 bits there are 1.6-2.7 codes per byte;
// four query heads need four FMAs per code, more than the FP32 pipes can issue at HBM speed, so the
// dot products run on the tensor pipe (mma.sync m16n8k16, fp32 accumulation).  Tiles of codes are
// staged in shared memory with 16-byte cp.async and read back with ldmatrix.trans, which delivers the
// two K-neighbours of an A fragment in one register; the codes enter the MMA as fp16 subnormals (one
// AND per pair) and the scale is folded into the B operand, carried exactly as hi + lo.
// Both kernels are chained with programmatic dependent launch: whatever a kernel needs only from the
// cache is requested before it waits for the kernel ahead of it.
//
// A CTA serves up to four query heads.  With eight per kv head the kv head is served by two CTAs ("virtual" kv heads
// of four query heads each, neighbours in the grid, so that the second read of the tile hits L2).
#include <math.h>
#include <string.h>

#include "common.cuh"

namespace hqkv {

HQKV_DEFINE_CHECK_COUNTER

constexpr int D = 128;           // head dim
constexpr int MAX_REP = 8;       // query heads per kv head
constexpr int MAX_R4 = 4;        // query heads per CTA

struct TierDev {
  const void* k_data;
  const __half* k_scale;
  const __half* k_zero;
  const int64_t* k_idx;
  const void* v_data;
  const __half* v_scale;
  const __half* v_zero;
  const int64_t* v_idx;
  int n_k, n_v;
  int bits;
  int normal;  // 1-bit tier in the Gaussian-codebook codec: value = std * (+-C) + mean, scale slots = std, zero = mean
  struct Units {
    int tokens, cost;        // of a unit
    unsigned per_cost;       // 2^32 / cost, rounded up
    int cost0;               // cost of the plane's units before the tier's
    int cta0;                // ... and its CTAs in the list of the plane's, where no CTA has units of two tiers
  } unit[2];                 // K pass, V pass
};

struct DecodeParams {
  TierDev tier[HQKV_NUM_TIERS + 1];  // [5] = fp16 residual window (token-major K and V)
  int B, H, nh_q, L;
  int halves;              // virtual kv heads per kv head: 2 with eight query heads per kv head, else 1
  int r4, r4_shift;        // query heads per virtual kv head: 1, 2, 4
  int gk_shift, gv_shift;
  int nk_ctas, nv_ctas;    // CTAs per plane = grid rows
  // Units per CTA.  more >= 0: equal shares, the first `more` CTAs take one more; -1: no CTA has units of two tiers (in
  // the K pass 8-bit units, which are half as long, count half).
  int k_per, k_more, v_per, v_more;
  int v_pairs, v_warps;    // 32 tokens a warp of the V pass takes at a time: 1, 2; warps per CTA: 8, 4
  float v_limit, v_units, v_unit;  // an output's two words (see v_finish): bound of a share; the high word's units per 1, and back
  int direct;              // the outputs are finished by whoever adds the last share (see v_finish), not by a CTA that reads them back
  float scale;
  const __half* q;
  const __half* mask;      // additive mask on the logits (null: none); element (b, head, pos) at b*bstride + head*hstride + pos
  long long mask_bstride, mask_hstride;
  const __half* probs_in;  // V pass on caller-supplied weights [B*nh_q][L] (null: softmax of the scratch logits)
  __half* head_sum;        // [L] sum of the probabilities over batch and heads, written by the V pass (null: not wanted)
  unsigned* hs_count;      // [nv_ctas] arrival counters of that sum
  __half* weights;
  __half* out;
  float* logits;   // [B][virtual kv head], see logit_at
  float2* k_part;  // [B][virtual kv head][r4][nk_ctas]
  double* v_acc;   // [B][nh_q][D] output accumulators (or high words, see v_finish): cleared by the K pass, summed into by the V pass
  unsigned long long* v_lows;  // ... and the low words (null: the scratch has no room for them)
  __half* peer_out[HQKV_MAX_PEERS];  // copies of `out` in other GPUs' memory (kv-head sharding), n_peers used
  int n_peers;
  int peer_flagged;  // 1: peer_out are flagged 8-byte entries {two fp16 values, call number}, see peer_unpack_kernel
  // cross-GPU barrier run by the last CTA of the V pass (world == 0: none)
  unsigned* pad[HQKV_MAX_PEERS + 1];  // the ranks' signal pads, own one included
  int rank, world;
  unsigned* peer_state;  // call number, status, finished (batch, kv head) count
  long long max_spins;
  unsigned* counters;  // [B][virtual kv head]
};

// The tokens of a (batch, virtual kv head) plane are a list of UNITS, tiers in order, and its CTAs take consecutive shares of
// it of equal COST, for the CTA with the longest share decides (20/40/40 at 24 x 8 x 15360 tokens in shares of equal count:
// the V pass took 94 us, the time of the CTAs with 4 and 2 bits only).  K pass: 256 tokens of a tier (128 at 8 bits, 64 of the
// fp16 tier and of the residual window).  V pass: a tile per warp, so 256 or 512 (64 in fp16).
// us a unit, K pass with four CTAs on every SM: 8 bits 1.9, 4 bits 3.2, 2 bits 2.9, 1 bit 3.3, fp16 tier 4.3, residual window
// 3.2; V pass with two CTAs of eight warps and 512 tokens: 8 bits 6.5, 4 bits 4.1, 2 bits 4.2, 1 bit 4.8 (16 x 8 planes of 16 k: 89,
// 57, 58 and 66 us a launch).
__host__ __device__ constexpr int unit_tokens(int bits) { return bits == 16 ? 64 : bits == 8 ? 128 : 256; }
__host__ __device__ constexpr int unit_cost(int bits) { return bits == 8 ? 5 : 8; }
// This CTA's tokens [t0, t1) of tier ti; false: none.
template <bool V>
__device__ __forceinline__ bool share_of(const DecodeParams& P, int ti, int& t0, int& t1) {
  const TierDev& T = P.tier[ti];
  const TierDev::Units& U = T.unit[V];
  const int i = blockIdx.y, per = V ? P.v_per : P.k_per, more = V ? P.v_more : P.k_more, n = V ? T.n_v : T.n_k;
  if (more < 0) {  // no CTA has units of two tiers
    const int own = max(static_cast<int>(__umulhi(per, U.per_cost)), 1) * U.tokens;
    t0 = (i - U.cta0) * own;
    t1 = min(t0 + own, n);
    return t0 >= 0 && t0 < t1;
  }
  const int c0 = i * per + min(i, more) - U.cost0, c1 = c0 + per + (i < more ? 1 : 0);
  // a unit belongs to the share that its cost starts in
  t0 = __umulhi(max(c0, 0) + U.cost - 1, U.per_cost) * U.tokens;
  t1 = min(static_cast<int>(__umulhi(max(c1, 0) + U.cost - 1, U.per_cost)) * U.tokens, n);
  return t0 < t1;
}
// The same where no CTA has units of two tiers: the tier, too.
template <bool V>
__device__ __forceinline__ int only_share(const DecodeParams& P, int& t0, int& t1) {
  const int i = blockIdx.y;
  int ti = 0;
#pragma unroll
  for (int t = 1; t <= HQKV_NUM_TIERS; ++t)
    if (i >= P.tier[t].unit[V].cta0) ti = t;
  share_of<V>(P, ti, t0, t1);
  return ti;
}

// Scratch logits of a (batch, virtual kv head) plane: [pos / 4][head][4 positions], the last quad with as many positions as it
// has.  A lane of the K pass has four or eight consecutive tokens of one head, a lane of the V pass takes four.
__device__ __forceinline__ int64_t logit_at(int64_t pos, int head, int heads, int L) {
  const int64_t quad = pos & ~static_cast<int64_t>(3);
  return quad * heads + head * (L - quad < 4 ? static_cast<int>(L - quad) : 4) + (pos & 3);
}

// Grid: x = virtual kv head, y = share of the plane's units, z = batch.
struct Where {
  int b, vh;   // batch, virtual kv head
  int bh;      // (batch, kv head) plane of the cache
  int bvh;     // (batch, virtual kv head) plane of the scratch
  int h0;      // first query head
};
__device__ __forceinline__ Where where(const DecodeParams& P) {
  Where w;
  w.b = blockIdx.z;
  w.vh = blockIdx.x;
  w.bh = w.b * P.H + (P.halves == 2 ? w.vh >> 1 : w.vh);
  w.bvh = w.b * gridDim.x + w.vh;
  w.h0 = w.vh * P.r4;
  return w;
}

// ------------------------------------------------------------------------------------------------
// fragments
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) { return h2_as_u32(__hmul2(u32_as_h2(a), u32_as_h2(b))); }
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
  return h2_as_u32(__hfma2(u32_as_h2(a), u32_as_h2(b), u32_as_h2(c)));
}
// a*b - c, with c = fp16(a*b): the exact remainder
__device__ __forceinline__ uint32_t h2_rem(uint32_t a, uint32_t b, uint32_t c) {
  return h2_as_u32(__hfma2(u32_as_h2(a), u32_as_h2(b), __hneg2(u32_as_h2(c))));
}
// 16-bit halves of two words -> one half2 register: low halves, high halves
__device__ __forceinline__ uint32_t pack_lo16(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410); }
__device__ __forceinline__ uint32_t pack_hi16(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }
__device__ __forceinline__ uint32_t pack_hi_lo(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5432); }  // high half of a, low half of b
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) { return h2_as_u32(__floats2half2_rn(lo, hi)); }

// Streaming loads: the cache is read once per call, keep it out of L1.
__device__ __forceinline__ uint2 ld_stream(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// shared memory by 32-bit address: loads with compile-time offsets, no generic-address arithmetic
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts16(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(static_cast<unsigned short>(v)) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// global -> shared copies without a register round trip; completion = wait_group + barrier
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
// the first `valid` bytes are read, the rest is set to 0
__device__ __forceinline__ void cp_async_8_fill(uint32_t dst, const void* src, int valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// four 8x8 matrices of 16-bit elements, transposed: lane (g, tig) gets elements (row 2*tig, col g) and
// (row 2*tig+1, col g) of matrix i in r[i]; lanes 8*i .. 8*i+7 supply the row addresses of matrix i
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t row_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(row_addr) : "memory");
}
// the same without the transposition: lane (g, tig) gets elements 2*tig, 2*tig+1 of row g
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t row_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(row_addr) : "memory");
}

// 2^x on the special-function unit (about 2 ulp; 2^-inf = 0)
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void softmax_merge(float& m, float& l, float m2, float l2) {
  const float mx = fmaxf(m, m2);
  if (mx == -INFINITY) return;  // both empty
  l = l * fast_exp2((m - mx) * LOG2E) + l2 * fast_exp2((m2 - mx) * LOG2E);
  m = mx;
}

// ------------------------------------------------------------------------------------------------
// k_pass
// ------------------------------------------------------------------------------------------------
// Quantised K tier: rows = channels, packed words along tokens.  A CTA of four warps walks a run of CHUNKS of one tier
// and (batch, kv head): 128 channel rows x 128 bytes of codes at 8 / 4 bits (128 / 256 tokens), x 64 / 32 bytes at 2 / 1
// bits (256 tokens).  Codes go global -> shared with 16-byte cp.async into one of two buffers (the next chunk's while
// this one is worked on); each warp works on its quarter of the tokens out of shared memory.  Wide copies in,
// ldmatrix out: the L1 data pipe moves 128 bytes per wavefront both ways.  (Per-lane loads of the 1-4 bytes a
// thread needs - from global or from shared memory - saturate that pipe at a quarter of the HBM bandwidth.)
//
// ldmatrix.trans over 8 channel rows x 16 bytes hands lane (g, tig) the 16-bit block g of channels
// 2*tig and 2*tig+1 in one register: exactly the two K-neighbours of an m16n8k16 A fragment for the
// tokens of block g (2 / 4 / 8 tokens at 8 / 4 / 2 bits).  What bounds the kernel below 8 bits is the number of
// instructions a warp issues per token, so everything here serves that number:
//  * the integer codes enter the tensor pipe as they are: a masked field at bit k < 10 of a 16-bit
//    lane IS the fp16 subnormal code * 2^(k-24), exactly, so one AND per pair of codes builds an A
//    fragment register; the power of two comes back out in the epilogue;
//  * the scale lives in the B operand: logit = sum_c (q_c * scale_c) * code_c + sum_c q_c * zero_c;
//  * q*scale (11 x 11 significant bits) is carried EXACTLY as hi = fp16(q*scale) and lo = q*scale - hi.  (One fp16
//    rounding of it - or of the dequantised K value - costs ~2e-3 on the attention output with x10 outlier
//    channels.)  At 8 and 4 bits the 16 rows of an M-tile are tokens of ONE scale group of 32, and the eight columns
//    of the B operand are (head 0 hi, head 0 lo, head 1 hi, ...): one MMA does both and a lane adds the two
//    accumulators of its head.  A 16-byte piece of 2-bit codes spans two groups: there the columns are (head 0 first
//    group, head 0 second group, ...), a row keeps the column of its own group, and hi and lo are two MMAs;
//  * a lane's accumulators all belong to query head tig, so logits, softmax statistics and stores need no exchange;
//  * the scales of two 16-channel steps are ONE 16-byte shared-memory read: the scale rows are transposed to
//    [group][channel] in shared memory, channels ordered as a lane's B fragment wants them.  They are fetched for 512
//    tokens at a time, a row's (up to) 48 bytes by neighbouring lanes: one 16-byte piece per lane and row cost the L1
//    tag stage a lookup each, more than the codes did;
//  * the zero point enters through Zq[group][head] = sum_c zero_c * q_c: every warp takes the 32 channels it has
//    transposed itself for all sixteen groups of those 512 tokens (two MMAs), the four partial sums meet in shared memory;
//  * blocks of tokens stay together in a tier, so 32 stored tokens have 32 consecutive positions: checked with one
//    vote, after which the logits are stored at constant offsets.  (Any other list takes the general store.)
constexpr int K_MIN_CTAS = 4;  // CTAs per SM the K pass is compiled for (128 registers; shared memory allows four)
constexpr int KWARPS = 4;
constexpr int KTHREADS = KWARPS * 32;
constexpr int K_SPAN = 64;                   // fp16 tier: tokens at a time
constexpr int K_SLOT = 4;                    // fp16 tier: tokens per 8-byte slot
constexpr int K_BLOCK = 512;                 // tokens whose scales are fetched at a time
constexpr int K_GROUPS = K_BLOCK / 32;       // scale groups of those at most
constexpr int K_RAW = 48;                    // bytes of a raw scale row: three aligned 16-byte pieces cover 16 halfs at any alignment
constexpr int K_SROW = D * 2;                // bytes of a transposed scale row
constexpr int K_ZROW = 80;                   // bytes of a warp's transposed zero row (32 channels; ldmatrix rows in different banks)
constexpr int K_TROW = MAX_R4 + 1;           // floats per token row of the logit tile (odd: no bank conflicts)
constexpr int K_CODES = D * 128;             // bytes of a code buffer

template <int BITS>
struct KTile {
  static constexpr int PITCH = BITS == 1 ? 40 : BITS == 2 ? 64 : 128;  // bytes per channel row in shared memory
  static constexpr int TOKENS = BITS == 8 ? 128 : 256;                 // tokens per chunk
  static constexpr int WTOK = TOKENS / KWARPS;                         // tokens per warp: 32, 64, 64, 64
  static constexpr int HALVES = WTOK / 32;                             // 32-token units per warp
  static constexpr bool ONE_GROUP = BITS >= 4;                         // an M-tile's rows are tokens of one unit
  static constexpr int NX = WTOK / 8;                                  // tokens per lane: 4, 8, 8, 8
};
static_assert(KTile<8>::TOKENS == unit_tokens(8) && KTile<4>::TOKENS == unit_tokens(4) && KTile<1>::TOKENS == unit_tokens(1), "a unit is a chunk");

struct KShared {
  union {
    unsigned char codes[2][K_CODES];
    float tile[KWARPS][K_SPAN * K_TROW];  // fp16 tier / residual: logits [token][head] of each warp
  } u;
  union {
    unsigned char raw[2][KWARPS][32 * K_RAW];  // scale and zero rows as in memory, 32 channels per warp
    struct {
      float m[KWARPS][MAX_R4], l[KWARPS][MAX_R4];  // softmax pairs of the warps, after the last chunk
    } red;
  } v;
  unsigned char s[K_GROUPS * K_SROW];          // [group][k_order(channel)]
  unsigned char z[KWARPS][K_GROUPS * K_ZROW];  // [group][channel of the warp]
  float zq[K_GROUPS][MAX_R4][KWARPS];          // the warps' partial Zq
  // B fragments of q per pair of 16-channel steps and lane: channels 16*kt + 2*tig + (0,1 | 8,9) of the even step, then
  // of the odd one; column n = g is head n >> 1
  uint4 q[4][32];
};
constexpr int K_RAW_PLANE = KWARPS * 32 * K_RAW;

// Position of a channel in a transposed scale row: per pair of 16-channel steps and lane quarter tig the eight channels
// of the lane's two B fragments are neighbours, {2tig, +1, +8, +9} of the even step, then of the odd one.
__device__ __forceinline__ int k_order(int ch) {
  return (ch & ~31) | ((ch & 6) << 2) | ((ch & 16) >> 2) | ((ch & 8) >> 2) | (ch & 1);
}

// halfs off .. off+15 of the 24 in (a, b, c)
__device__ __forceinline__ void align_halfs(const uint4& a, const uint4& b, const uint4& c, int off, uint32_t (&o)[8]) {
  uint32_t w[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
#pragma unroll
  for (int i = 0; i < 10; ++i) w[i] = (off & 4) ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < 9; ++i) w[i] = (off & 2) ? w[i + 1] : w[i];
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = __funnelshift_r(w[i], w[i + 1], 16 * (off & 1));
}

// Scale / zero rows of up to 512 tokens, warp = 32 channels.  The groups [g0, g0 + ng) of a channel are ng halfs at any
// 2-byte alignment; the (up to) three aligned 16-byte pieces that cover them are copied as they are and shifted into
// place on the way to the transposed rows.  (The planes hold B*H*128*G halfs, a multiple of 8, and start 16-byte
// aligned, so every aligned piece that begins inside a plane also ends inside it.)
struct KScales {
  int64_t row0;      // index of half 0 of the warp's first channel row
  int G;             // groups per row
  uint32_t raw, s_at, z_at, z_row;
};
__device__ __forceinline__ void k_scales_request(const TierDev& T, const KScales& k, int g0, int ng) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int id = i * 32 + lane, row = id / 3, piece = id - 3 * row;
    const int64_t e = k.row0 + static_cast<int64_t>(row) * k.G + g0;
    if (8 * piece < static_cast<int>(e & 7) + ng) {
      const int64_t a = (e & ~static_cast<int64_t>(7)) + 8 * piece;
      cp_async_16(k.raw + id * 16, T.k_scale + a);
      cp_async_16(k.raw + K_RAW_PLANE + id * 16, T.k_zero + a);
    }
  }
}
__device__ __forceinline__ void k_scales_transpose(const KScales& k, int g0, int ng) {
  const int lane = threadIdx.x & 31;
  const int off = static_cast<int>((k.row0 + static_cast<int64_t>(lane) * k.G + g0) & 7);
  const uint32_t src = k.raw + lane * K_RAW;
#pragma unroll
  for (int plane = 0; plane < 2; ++plane) {
    const uint32_t p = src + plane * (K_RAW_PLANE);
    const uint4 a = lds128(p), b = lds128(p + 16), c = lds128(p + 32);
    uint32_t o[8];
    align_halfs(a, b, c, off, o);
    const uint32_t at = plane ? k.z_at : k.s_at;
    const int pitch = plane ? K_ZROW : K_SROW;
#pragma unroll
    for (int i = 0; i < K_GROUPS / 2; ++i)
      if (2 * i < ng) {  // (an odd count stores one row more: nobody reads it)
        sts16(at + (2 * i) * pitch, o[i] & 0xFFFFu);
        sts16(at + (2 * i + 1) * pitch, o[i] >> 16);
      }
  }
}
// Partial Zq of the warp's 32 channels: rows = groups.  q = the B fragments of those channels.
__device__ __forceinline__ void k_zero_term(const KScales& k, const uint4& q, float (*zq)[MAX_R4][KWARPS], uint32_t other_rows, bool normal) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  uint32_t r[4];
  ldmatrix_x4(r, k.z_row);        // matrices (groups 0-7, channels 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
  mma16816(acc, r[0], r[1], r[2], r[3], q.x, q.y);
  ldmatrix_x4(r, k.z_row + 32);
  mma16816(acc, r[0], r[1], r[2], r[3], q.z, q.w);
  if (normal) {  // a value is std * C * (2 code - 1) + mean: the code-free term is sum_c (mean - C std) q
    float n[4] = {0.f, 0.f, 0.f, 0.f};
    const uint32_t even = other_rows, odd = other_rows + 8;  // this lane's channels in the transposed scale rows
    uint2 x = lds64(even), y = lds64(even + 8 * K_SROW);
    mma16816(n, x.x, y.x, x.y, y.y, q.x, q.y);
    x = lds64(odd), y = lds64(odd + 8 * K_SROW);
    mma16816(n, x.x, y.x, x.y, y.y, q.z, q.w);
    acc[0] = fmaf(-HQKV_NORMAL1_CENTER, n[0], acc[0]);
    acc[2] = fmaf(-HQKV_NORMAL1_CENTER, n[2], acc[2]);
  }
  zq[g][tig][threadIdx.x >> 5] = acc[0];
  zq[g + 8][tig][threadIdx.x >> 5] = acc[2];
}

// Request the codes of a chunk: src / dst = this thread's first piece, valid = bytes per row (a multiple of 32, 16, 8, 4
// at 8, 4, 2, 1 bits).  The rows of the 2-bit tier are only 8-byte aligned unless its token count is a multiple of 64
// (wide2; otherwise the even rows are copied 16 bytes and the odd ones 8 bytes at a time), those of the 1-bit tier 4-byte.
// The piece index is XORed with row bits so that the eight rows of an ldmatrix (same logical piece) and the pieces a
// cp.async instruction writes both spread over all banks.
template <int BITS>
struct KCopy {
  const unsigned char* src;
  uint32_t dst;
  uint32_t step;   // bytes of memory between this thread's rows
  int first;       // first byte of the row that this thread copies
  int64_t odd;     // 2 bits, odd rows off the 16-byte boundaries: their first piece, from src,
  uint32_t odst;   // where it goes
  int ofirst;      // and its first byte of the row
};
template <int BITS>
__device__ __forceinline__ KCopy<BITS> k_copy_init(const TierDev& T, int bh, int t0, uint32_t codes, bool wide2) {
  using TL = KTile<BITS>;
  const int tid = threadIdx.x;
  const int64_t row_bytes = static_cast<int64_t>(T.n_k) * BITS / 8;
  KCopy<BITS> k;
  int c, r0, bytes, rows;
  if constexpr (BITS == 2) {
    c = tid & 3, r0 = wide2 ? tid >> 2 : 2 * (tid >> 2), bytes = 16, rows = 32;
    k.dst = codes + r0 * 64 + ((c ^ ((r0 >> 1) & 3)) << 4);
  } else {
    c = tid & 7, r0 = tid >> 3, bytes = BITS >= 4 ? 16 : 4, rows = 16;
    k.dst = codes + (BITS >= 4 ? r0 * 128 + ((c ^ (r0 & 7)) << 4)
                               : r0 * TL::PITCH + 4 * c);
  }
  k.first = c * bytes;
  k.step = static_cast<uint32_t>(rows * row_bytes);
  k.src = reinterpret_cast<const unsigned char*>(T.k_data) + (static_cast<int64_t>(bh) * D + r0) * row_bytes +
          static_cast<int64_t>(t0) * BITS / 8 + k.first;
  if constexpr (BITS == 2) {
    const int r1 = 2 * (tid >> 3) + 1, c1 = tid & 7;
    k.ofirst = 8 * c1;
    k.odd = (r1 - r0) * row_bytes + k.ofirst - k.first;
    k.odst = codes + r1 * 64 + (((c1 >> 1) ^ ((r1 >> 1) & 3)) << 4) + 8 * (c1 & 1);
  }
  return k;
}
template <int BITS>
__device__ __forceinline__ void k_codes_request(const KCopy<BITS>& k, int chunk, int valid, bool wide2) {
  using TL = KTile<BITS>;
  const unsigned char* s = k.src + static_cast<int64_t>(chunk) * (TL::TOKENS * BITS / 8);
  const uint32_t d = k.dst + (chunk & 1) * K_CODES;
  if constexpr (BITS == 2) {
    if (wide2) {
      if (k.first >= valid) return;
#pragma unroll
      for (int i = 0; i < 4; ++i) cp_async_16(d + i * 32 * TL::PITCH, s + static_cast<uint64_t>(k.step) * i);
    } else {
      if (k.first < valid) {  // (the last piece of a row may reach into the odd row behind it)
#pragma unroll
        for (int i = 0; i < 2; ++i) cp_async_16(d + i * 64 * TL::PITCH, s + static_cast<uint64_t>(k.step) * (2 * i));
      }
      if (k.ofirst < valid) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          cp_async_8(k.odst + (chunk & 1) * K_CODES + i * 32 * TL::PITCH, s + k.odd + static_cast<uint64_t>(k.step) * i);
      }
    }
    return;
  }
  if (k.first >= valid) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const unsigned char* p = s + static_cast<uint64_t>(k.step) * i;
    if (BITS >= 4) cp_async_16(d + i * 16 * TL::PITCH, p);
    else cp_async_4(d + i * 16 * TL::PITCH, p);
  }
}

// Token of a lane's logit j = (unit or M-tile, then row g / g+8) within the warp's tokens: see k_logit_index.
//   8 bits: M-tile i: row g = token 2g + i, row g+8 = 16 + 2g + i;   4 bits, unit u: 32u + 4g + i and 32u + 4g + 2 + i
//   2 bits: 8g + i and 8g + 4 + i;   1 bit: 16(g&3) + 4(g>>2) + i and + 8
// k_lane_base: the part that depends on the lane, within its unit; k_step: the rest, within the unit of logit j.
template <int BITS>
__device__ __forceinline__ int k_lane_unit() {  // (not used at 4 bits, where a lane has tokens of both units)
  const int g = (threadIdx.x & 31) >> 2;
  return BITS == 2 ? g >> 2 : BITS == 1 ? (g & 3) >> 1 : 0;
}
template <int BITS>
__device__ __forceinline__ int k_lane_base() {
  const int g = (threadIdx.x & 31) >> 2;
  return BITS == 8 ? 2 * g : BITS == 4 ? 4 * g : BITS == 2 ? 8 * (g & 3) : 16 * (g & 1) + 4 * (g >> 2);
}
template <int BITS>
__host__ __device__ constexpr int k_step(int j) {
  const int r = j & 1, i = BITS == 4 ? (j >> 1) & 1 : j >> 1;
  return i + r * (BITS == 8 ? 16 : BITS == 4 ? 2 : BITS == 2 ? 4 : 8);
}

// running (max, sum-exp) of a lane; -inf marks "no value"
template <int N>
__device__ __forceinline__ void softmax_push(float& m, float& l, const float (&x)[N]) {
  float mn = m;
#pragma unroll
  for (int j = 0; j < N; ++j) mn = fmaxf(mn, x[j]);
  const float ref = (mn == -INFINITY ? 0.f : mn) * LOG2E;
  l *= fast_exp2(fmaf(m, LOG2E, -ref));
#pragma unroll
  for (int j = 0; j < N; ++j) l += fast_exp2(fmaf(x[j], LOG2E, -ref));
  m = mn;
}

// The lane's logits of one chunk: x[j], j = NX logits of head tig.  zq = zero terms of the chunk's first group on, scale =
// softmax scale (pscale: that of the code term).  codes = address of the chunk's
// codes, srow0 = scale row of the chunk's first group, qrow = this lane's B fragments of q.
// WG: groups of 64 or 128, whose scales serve all of the warp's 64 tokens.
template <int BITS, bool WG>
__device__ __forceinline__ void k_chunk_logits(float (&x)[KTile<BITS>::NX], uint32_t codes, uint32_t srow0, uint32_t qrow,
                                               const float (*zq)[MAX_R4][KWARPS], float scale, float pscale, int gk_shift) {
  using TL = KTile<BITS>;
  constexpr bool ONE_GROUP = TL::ONE_GROUP;         // the columns are hi and lo of a head
  constexpr int UNITS = BITS == 4 ? 2 : 1;          // accumulator sets
  constexpr int NM = BITS >= 4 ? 2 : 4;             // M-tiles per set
  constexpr int SETS = WG ? 1 : UNITS;              // of scales
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tig = lane & 3;
  const uint32_t remainder = (g & 1) ? 0xFFFFFFFFu : 0u;
  // scale rows of this lane's B column
  uint32_t srow[SETS];
#pragma unroll
  for (int u = 0; u < SETS; ++u) srow[u] = srow0 + ((warp * TL::WTOK + 32 * (ONE_GROUP ? u : (g & 1))) >> gk_shift) * K_SROW + tig * 16;
  // ldmatrix row address of this lane for step 0
  uint32_t kb = codes, kb1 = 0;
  if constexpr (BITS == 8) {
    const int mi = lane >> 3, rr = lane & 7;        // matrices (octet, piece): (0,0), (0,1), (1,0), (1,1)
    kb += (8 * (mi >> 1) + rr) * 128 + (((2 * warp + (mi & 1)) ^ rr) << 4);
  } else if constexpr (BITS == 4) {
    kb += lane * 128 + (((2 * warp) ^ (lane & 7)) << 4);   // octets 0..3 of 32 channels; unit 1: the other piece of the pair
    kb1 = kb ^ 16u;
  } else if constexpr (BITS == 2) {
    kb += lane * 64 + ((warp ^ ((lane >> 1) & 3)) << 4);
  } else {
    kb += (2 * tig) * TL::PITCH + 8 * warp + 2 * (g & 3);  // block g & 3 of channel 2tig
  }
  float acc[UNITS][NM][4];
#pragma unroll
  for (int u = 0; u < UNITS; ++u)
#pragma unroll
    for (int i = 0; i < NM; ++i) acc[u][i][0] = acc[u][i][1] = acc[u][i][2] = acc[u][i][3] = 0.f;
  // Two 16-channel steps per iteration.  The operands of the next iteration are requested before this one's are used:
  // with four warps per scheduler the round trip to shared memory is not covered by other warps.
  uint32_t Rb[2][2][4];
  uint4 qb[2], sb4[2][SETS];
  auto fetch = [&](int p) {
    uint32_t(&R)[2][4] = Rb[p & 1];
    if constexpr (BITS == 8) {
      ldmatrix_x4_trans(R[0], kb + p * 4096);
      ldmatrix_x4_trans(R[1], kb + p * 4096 + 2048);
    } else if constexpr (BITS == 4) {
      ldmatrix_x4_trans(R[0], kb + p * 4096);
      ldmatrix_x4_trans(R[1], kb1 + p * 4096);
    } else if constexpr (BITS == 2) {
      ldmatrix_x4_trans(R[0], kb + p * 2048);
    } else {  // 16-bit pieces of channels 2tig, 2tig+1 (+8, +9; next step)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        R[0][i] = pack_lo16(lds16(kb + (32 * p + 8 * i) * TL::PITCH), lds16(kb + (32 * p + 8 * i + 1) * TL::PITCH));
    }
    qb[p & 1] = lds128(qrow + p * sizeof(KShared::q[0]));
#pragma unroll
    for (int u = 0; u < SETS; ++u) sb4[p & 1][u] = lds128(srow[u] + p * 64);
  };
  fetch(0);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    if (p < 3) fetch(p + 1);
    const uint32_t(&R)[2][4] = Rb[p & 1];
    const uint4 q4 = qb[p & 1];
    const uint32_t q[2][2] = {{q4.x, q4.y}, {q4.z, q4.w}};
    if constexpr (ONE_GROUP) {
      uint32_t qm[2][2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) qm[k][h] = (q[k][h] ^ 0x80008000u) & remainder;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        // even columns (qm = 0): hi = fp16(q*s); odd columns (qm = -q): the exact remainder q*s - hi
        uint32_t b[SETS][2];
#pragma unroll
        for (int u = 0; u < SETS; ++u) {
          const uint4 s4 = sb4[p & 1][u];
          const uint32_t s0 = k ? s4.z : s4.x, s1 = k ? s4.w : s4.y;
          b[u][0] = h2_fma(q[k][0], s0, h2_mul(qm[k][0], s0));
          b[u][1] = h2_fma(q[k][1], s1, h2_mul(qm[k][1], s1));
        }
        if constexpr (BITS == 8) {
          const uint32_t* r = R[k];
          mma16816(acc[0][0], r[0] & 0x00FF00FFu, r[1] & 0x00FF00FFu, r[2] & 0x00FF00FFu, r[3] & 0x00FF00FFu, b[0][0], b[0][1]);
          mma16816(acc[0][1], __byte_perm(r[0], 0u, 0x4341), __byte_perm(r[1], 0u, 0x4341), __byte_perm(r[2], 0u, 0x4341),
                   __byte_perm(r[3], 0u, 0x4341), b[0][0], b[0][1]);
        } else {
#pragma unroll
          for (int u = 0; u < UNITS; ++u) {
            const uint32_t ra = R[u][2 * k], rb = R[u][2 * k + 1], sa = ra >> 8, sb = rb >> 8;
#pragma unroll
            for (int i = 0; i < NM; ++i) {
              const uint32_t m = 0x000F000Fu << (4 * i);
              mma16816(acc[u][i], ra & m, sa & m, rb & m, sb & m, b[u < SETS ? u : 0][0], b[u < SETS ? u : 0][1]);
            }
          }
        }
      }
    } else {
      const uint4 s4 = sb4[p & 1][0];
      const uint32_t s[2][2] = {{s4.x, s4.y}, {s4.z, s4.w}};
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t h0 = h2_mul(q[k][0], s[k][0]), h1 = h2_mul(q[k][1], s[k][1]);
        const uint32_t l0 = h2_rem(q[k][0], s[k][0], h0), l1 = h2_rem(q[k][1], s[k][1], h1);
        uint32_t a[4][4];  // [register][M-tile]
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          const uint32_t lo = BITS == 2 ? R[0][2 * k + o] : R[0][2 * k + o] >> (4 * (g >> 2));
          const uint32_t hi = lo >> 8;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t m = BITS == 2 ? 0x00030003u << (2 * i) : 0x00010001u << i;
            a[2 * o][i] = lo & m;
            a[2 * o + 1][i] = hi & m;
          }
        }
        // the two MMAs into one accumulator are issued four apart (they depend on each other)
#pragma unroll
        for (int i = 0; i < 4; ++i) mma16816(acc[0][i], a[0][i], a[1][i], a[2][i], a[3][i], h0, h1);
#pragma unroll
        for (int i = 0; i < 4; ++i) mma16816(acc[0][i], a[0][i], a[1][i], a[2][i], a[3][i], l0, l1);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < UNITS; ++u) {
    const bool second = !ONE_GROUP && k_lane_unit<BITS>() == 1;
    const int gam = (warp * TL::WTOK + 32 * (BITS == 4 ? u : k_lane_unit<BITS>())) >> gk_shift;
    const float4 zp = *reinterpret_cast<const float4*>(zq[gam][tig]);
    const float z = ((zp.x + zp.y) + (zp.z + zp.w)) * scale;
#pragma unroll
    for (int i = 0; i < NM; ++i)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        constexpr int SH = BITS == 8 ? 0 : BITS;  // M-tile i holds the field at bit SH * i
        const float unscale = static_cast<float>(1 << 24) / static_cast<float>(1 << (SH * i));
        const float* a = &acc[u][i][2 * r];
        x[(u * NM + i) * 2 + r] = fmaf(ONE_GROUP ? a[0] + a[1] : (second ? a[1] : a[0]), pscale * unscale, z);
      }
  }
}

// Positions of the warp's tokens: pu[u] = position of stored token 32*u + lane of the warp (low word of the int64).
template <int BITS>
__device__ __forceinline__ void k_positions(const TierDev& T, uint32_t (&pu)[KTile<BITS>::HALVES], int t0) {
  const int t = t0 + (threadIdx.x >> 5) * KTile<BITS>::WTOK + (threadIdx.x & 31);
#pragma unroll
  for (int u = 0; u < KTile<BITS>::HALVES; ++u)
    pu[u] = t + 32 * u < T.n_k ? __ldg(reinterpret_cast<const uint32_t*>(T.k_idx + t + 32 * u)) : 0u;
}

// Any positions, any number of heads, masks: the lane's logits, as they count (-inf: none), in x.
template <int BITS>
__device__ __forceinline__ void k_store_any(const DecodeParams& P, const TierDev& T, const Where& w, float (&x)[KTile<BITS>::NX],
                                         const uint32_t (&pu)[KTile<BITS>::HALVES], int wt0) {
  using TL = KTile<BITS>;
  constexpr int NX = TL::NX, HALVES = TL::HALVES;
  const int tig = threadIdx.x & 3, lb = k_lane_base<BITS>();
  float* out = P.logits + static_cast<int64_t>(w.bvh) * P.L * P.r4;
  bool valid[HALVES];
#pragma unroll
  for (int u = 0; u < HALVES; ++u) valid[u] = wt0 + 32 * u < T.n_k;
  const bool on = tig < P.r4;
  const __half* mrow = P.mask ? P.mask + w.b * P.mask_bstride + (w.h0 + (on ? tig : 0)) * P.mask_hstride : nullptr;
#pragma unroll
  for (int j = 0; j < NX; ++j) {
    const int src = lb + k_step<BITS>(j);
    uint32_t pos = __shfl_sync(0xffffffffu, pu[BITS == 4 ? j >> 2 : 0], src);
    bool ok = on && valid[BITS == 4 ? j >> 2 : 0];
    if constexpr (BITS <= 2) {
      const uint32_t pos1 = __shfl_sync(0xffffffffu, pu[HALVES - 1], src);
      if (k_lane_unit<BITS>() == 1) {
        pos = pos1;
        ok = on && valid[HALVES - 1];
      }
    }
    ok = ok && HQKV_INDEX_OK(pos, P.L);
    if (ok) {
      if (mrow) x[j] += __half2float(mrow[pos]);
      out[logit_at(pos, tig, P.r4, P.L)] = x[j];
    } else {
      x[j] = -INFINITY;
    }
  }
}

// Store the lane's logits at their positions and add them to its running softmax statistics.  wt0 = the warp's first
// token in the tier.
template <int BITS>
__device__ __forceinline__ void k_emit(const DecodeParams& P, const TierDev& T, const Where& w, float (&x)[KTile<BITS>::NX],
                                       const uint32_t (&pu)[KTile<BITS>::HALVES], int wt0, float& m, float& l) {
  using TL = KTile<BITS>;
  constexpr int NX = TL::NX, HALVES = TL::HALVES;
  const int lane = threadIdx.x & 31, tig = lane & 3;
  const int lb = k_lane_base<BITS>();
  float* out = P.logits + static_cast<int64_t>(w.bvh) * P.L * P.r4 + 4 * tig;
  // whole 32-token units are valid or not (a tier holds a multiple of 32 tokens)
  bool valid[HALVES], dense = P.r4 >= 2 && P.mask == nullptr;
  uint32_t base[HALVES];
#pragma unroll
  for (int u = 0; u < HALVES; ++u) {
    valid[u] = wt0 + 32 * u < T.n_k;
    base[u] = __shfl_sync(0xffffffffu, pu[u], 0);
    dense = dense && (!valid[u] || (pu[u] == base[u] + lane && (base[u] & 3) == 0 && HQKV_INDEX_OK(pu[u], P.L)));
  }
  if (__all_sync(0xffffffffu, dense)) {
    const bool on = tig < P.r4;
    auto store = [&](auto heads) {
      constexpr int R = decltype(heads)::value;
      // N logits at consecutive positions from `token` of unit u on, x[j], x[j + 2], ...; two heads start on 8-byte boundaries
      auto run = [&](auto count, uint32_t unit, int token, int j, bool ok) {
        constexpr int N = decltype(count)::value;
        float* o = out + static_cast<int64_t>(unit + (token & ~3)) * R + (token & 3);
        if (!ok) {
#pragma unroll
          for (int i = 0; i < N; ++i) x[j + 2 * i] = -INFINITY;
        } else if constexpr (R == MAX_R4 && N == 4) {
          *reinterpret_cast<float4*>(o) = make_float4(x[j], x[j + 2], x[j + 4], x[j + 6]);
        } else {
#pragma unroll
          for (int i = 0; i < N; i += 2) *reinterpret_cast<float2*>(o + i) = make_float2(x[j + 2 * i], x[j + 2 * i + 2]);
        }
      };
      using Two = std::integral_constant<int, 2>;
      using Four = std::integral_constant<int, 4>;
      if constexpr (BITS == 8) {
        const bool ok = valid[0] && (R == MAX_R4 || on);
        run(Two(), base[0], lb, 0, ok);
        run(Two(), base[0], lb + 16, 1, ok);
      } else if constexpr (BITS == 4) {  // x[4u ...]: tokens 0, 2, 1, 3 of the lane's quad
#pragma unroll
        for (int u = 0; u < HALVES; ++u) {
          const bool ok = valid[u] && (R == MAX_R4 || on);
          float* o = out + static_cast<int64_t>(base[u] + lb) * R;
          if (!ok) {
#pragma unroll
            for (int j = 4 * u; j < 4 * u + 4; ++j) x[j] = -INFINITY;
          } else if constexpr (R == MAX_R4) {
            *reinterpret_cast<float4*>(o) = make_float4(x[4 * u], x[4 * u + 2], x[4 * u + 1], x[4 * u + 3]);
          } else {
            reinterpret_cast<float2*>(o)[0] = make_float2(x[4 * u], x[4 * u + 2]);
            reinterpret_cast<float2*>(o)[1] = make_float2(x[4 * u + 1], x[4 * u + 3]);
          }
        }
      } else {
        const bool second = k_lane_unit<BITS>() == 1;
        const bool ok = (second ? valid[HALVES - 1] : valid[0]) && (R == MAX_R4 || on);
        const uint32_t unit = second ? base[HALVES - 1] : base[0];
        run(Four(), unit, lb, 0, ok);
        run(Four(), unit, lb + (BITS == 2 ? 4 : 8), 1, ok);
      }
    };
    if (P.r4 == MAX_R4) store(std::integral_constant<int, MAX_R4>());
    else store(std::integral_constant<int, 2>());
  } else {
    k_store_any<BITS>(P, T, w, x, pu, wt0);
  }
  softmax_push<NX>(m, l, x);
}

// Tokens [t0, t1) of a quantised tier; m, l: the lane's running softmax pair (head tig).  `first`: nothing has run before
// in this CTA.
template <int BITS, bool WG>
__device__ __forceinline__ void k_run(const DecodeParams& P, const TierDev& T, KShared& sh, const Where& w, int t0, int t1,
                                      float& m, float& l, bool& first) {
  using TL = KTile<BITS>;
  constexpr int PER_BLOCK = K_BLOCK / TL::TOKENS;   // chunks per fetch of scales
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
  const int chunks = (t1 - t0 + TL::TOKENS - 1) / TL::TOKENS;
  const bool wide2 = BITS == 2 && (T.n_k & 63) == 0;
  const bool normal = BITS == 1 && T.normal != 0;   // Gaussian-codebook 1-bit tier: the code term carries the factor 2C
  const float pscale = normal ? P.scale * (2.f * HQKV_NORMAL1_CENTER) : P.scale;
  const uint32_t codes = smem_u32(sh.u.codes), srows = smem_u32(sh.s), qrow = smem_u32(&sh.q[0][lane]);
  KScales k;
  k.G = T.n_k >> P.gk_shift;
  k.row0 = (static_cast<int64_t>(w.bh) * D + 32 * warp) * k.G;
  k.raw = smem_u32(sh.v.raw[0][warp]);
  k.s_at = srows + 2 * k_order(tid);
  k.z_at = smem_u32(sh.z[warp]) + 2 * lane;
  k.z_row = smem_u32(sh.z[warp]) + ((lane & 7) + 8 * ((lane >> 3) & 1)) * K_ZROW + 16 * (lane >> 4);
  auto tokens = [&](int c) { return min(TL::TOKENS, t1 - t0 - c * TL::TOKENS); };
  auto groups = [&](int blk) { return (min(K_BLOCK, t1 - t0 - blk * K_BLOCK) + (1 << P.gk_shift) - 1) >> P.gk_shift; };
  auto first_group = [&](int blk) { return (t0 + blk * K_BLOCK) >> P.gk_shift; };
  if (!first) __syncthreads();  // every warp is done with the buffers
  k_scales_request(T, k, first_group(0), groups(0));
  cp_async_commit();
  const KCopy<BITS> copy = k_copy_init<BITS>(T, w.bh, t0, codes, wide2);
  k_codes_request<BITS>(copy, 0, tokens(0) * BITS / 8, wide2);
  cp_async_commit();
  if (chunks > 1) k_codes_request<BITS>(copy, 1, tokens(1) * BITS / 8, wide2);
  cp_async_commit();
  uint32_t pu[TL::HALVES];
  k_positions<BITS>(T, pu, t0);
  cp_async_wait<2>();
  __syncwarp();
  k_scales_transpose(k, first_group(0), groups(0));
  // Everything above reads only the cache.  From here on this grid reads q - the one input an earlier kernel of the
  // stream may still be writing - and writes the scratch that the previous decode call may still be using: wait for the
  // kernels before it.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  first = false;
  // every warp fetches the fragments of its own 32 channels, which it also needs for the zero term
  uint4 qz = make_uint4(0u, 0u, 0u, 0u);
  if ((g >> 1) < P.r4) {
    const uint32_t* qh = reinterpret_cast<const uint32_t*>(P.q + (static_cast<int64_t>(w.b) * P.nh_q + w.h0 + (g >> 1)) * D) +
                         16 * warp + tig;
    qz = make_uint4(qh[0], qh[4], qh[8], qh[12]);
  }
  sh.q[warp][lane] = qz;
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    if (c == 0) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();  // the codes of chunk c are there; every warp is done with chunk c - 1
    if (c > 0 && c + 1 < chunks) k_codes_request<BITS>(copy, c + 1, tokens(c + 1) * BITS / 8, wide2);
    cp_async_commit();
    if (c % PER_BLOCK == 0) {
      const int blk = c / PER_BLOCK;
      if (c > 0) k_scales_transpose(k, first_group(blk), groups(blk));
      __syncwarp();
      k_zero_term(k, qz, sh.zq, srows + g * K_SROW + warp * 64 + tig * 16, normal);
      __syncthreads();
      if (c + PER_BLOCK < chunks) k_scales_request(T, k, first_group(blk + 1), groups(blk + 1));
      cp_async_commit();
    }
    const int wt0 = t0 + c * TL::TOKENS + warp * TL::WTOK;
    if (wt0 < t1) {
      uint32_t at[TL::HALVES];
#pragma unroll
      for (int u = 0; u < TL::HALVES; ++u) at[u] = pu[u];
      if (c + 1 < chunks) k_positions<BITS>(T, pu, t0 + (c + 1) * TL::TOKENS);
      const int in_block = (c % PER_BLOCK) * TL::TOKENS;
      float x[TL::NX];
      const int g0 = in_block >> P.gk_shift;  // first group of the chunk within the block
      k_chunk_logits<BITS, WG>(x, codes + (c & 1) * K_CODES, srows + g0 * K_SROW, qrow, sh.zq + g0, P.scale, pscale, P.gk_shift);
      k_emit<BITS>(P, T, w, x, at, wt0, m, l);
    }
  }
}

// Write out a warp's logit tile [ntok][K_TROW] (already scaled) at the tokens' logical positions and
// add them to the running softmax pairs.  Element = (token, head) with the head
// fastest across lanes, so every lane owns ONE head for the whole call (r4 divides 32).
// (fp16 tier and residual window only; the quantised tiers write from registers.)
__device__ __forceinline__ void k_write_tile(const DecodeParams& P, const Where& w, float* tile, int ntok, const int64_t* idx,
                                             int64_t first_pos, float& m_out, float& l_out) {
  const int lane = threadIdx.x & 31;
  const int rep = P.r4, rshift = P.r4_shift;
  const int h = lane & (rep - 1);
  float* out = P.logits + static_cast<int64_t>(w.bvh) * P.L * rep;
  const __half* mrow = P.mask ? P.mask + w.b * P.mask_bstride + static_cast<int64_t>(w.h0 + h) * P.mask_hstride : nullptr;
  const int tpr = 32 >> rshift;  // tokens per round
  float m = -INFINITY, l = 0.f;
#pragma unroll 2
  for (int t = lane >> rshift; t < ntok; t += tpr) {
    const int64_t pos = idx ? idx[t] : first_pos + t;
    float x[1] = {-INFINITY};
    if (HQKV_INDEX_OK(pos, P.L)) {
      x[0] = tile[t * K_TROW + h];
      if (mrow) x[0] += __half2float(mrow[pos]);
      out[logit_at(pos, h, rep, P.L)] = x[0];
    }
    softmax_push<1>(m, l, x);
  }
  float mx = m;
  for (int off = rep; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  float sum = l * fast_exp2((m - (mx == -INFINITY ? 0.f : mx)) * LOG2E);  // every position masked out: 0, not NaN
  for (int off = rep; off < 32; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  // lane h now holds head h; lanes 0-3 take it into their pairs (head tig)
  if (lane < rep) softmax_merge(m_out, l_out, mx, sum);
}

// B fragment of q for the fp16 tier / residual: column n = g is head n; qh: that head's row at channel 2*tig (null: none)
__device__ __forceinline__ uint2 k_plain_q(const uint32_t* qh, int kt) {
  return qh ? make_uint2(qh[8 * kt], qh[8 * kt + 4]) : make_uint2(0u, 0u);
}

// fp16 tier, channel-major rows [D][n]: four tokens per 8-byte slot, no scales; B = q exactly.  64 tokens by the whole CTA,
// a warp for 32 of the channels: all of a warp's loads are in flight together (one warp for all channels went through
// eight dependent rounds of them); the partial logits meet in shared memory.
__device__ __forceinline__ void k_f16_block(const DecodeParams& P, const TierDev& T, KShared& sh, const Where& w, const uint32_t* qh,
                                            int t0, float& m, float& l) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tig = lane & 3;
  const int n = T.n_k;
  const int64_t nslot = n / K_SLOT;
  const uint2* base = reinterpret_cast<const uint2*>(T.k_data) + static_cast<int64_t>(w.bh) * D * nslot;
  int64_t sl[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) sl[r] = min(static_cast<int64_t>(t0 / K_SLOT + r * 8 + g), nslot - 1);
  float acc[K_SLOT][4];
#pragma unroll
  for (int i = 0; i < K_SLOT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int kt = 2 * warp + k;
    uint2 v[4][2];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int ch = 16 * kt + 8 * (e >> 1) + 2 * tig + (e & 1);
#pragma unroll
      for (int r = 0; r < 2; ++r) v[e][r] = ld_stream(base + ch * nslot + sl[r]);
    }
    const uint2 bq = k_plain_q(qh, kt);
    // token i of a slot: halfs (x.lo, x.hi, y.lo, y.hi); pair the same token of two channel rows
    uint32_t a[K_SLOT][4];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint2 va = v[2 * q][r], vb = v[2 * q + 1][r];
        a[0][q * 2 + r] = pack_lo16(va.x, vb.x);
        a[1][q * 2 + r] = pack_hi16(va.x, vb.x);
        a[2][q * 2 + r] = pack_lo16(va.y, vb.y);
        a[3][q * 2 + r] = pack_hi16(va.y, vb.y);
      }
#pragma unroll
    for (int i = 0; i < K_SLOT; ++i) mma16816(acc[i], a[i][0], a[i][1], a[i][2], a[i][3], bq.x, bq.y);
  }
  float* part = sh.u.tile[warp];
  if (tig < 2) {  // columns 0-3 are heads, 4-7 are empty
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int i = 0; i < K_SLOT; ++i) part[((r * 8 + g) * K_SLOT + i) * K_TROW + 2 * tig + e] = acc[i][r * 2 + e] * P.scale;
  }
  __syncthreads();
  // 16 tokens per warp: the sum goes into the first partial tile
  constexpr int MINE = K_SPAN / KWARPS * K_TROW;
  float* tile = sh.u.tile[0] + warp * MINE;
  for (int i = lane; i < MINE; i += 32) {
    float v = tile[i];
#pragma unroll
    for (int o = 1; o < KWARPS; ++o) v += sh.u.tile[o][warp * MINE + i];
    tile[i] = v;
  }
  __syncwarp();
  const int first = t0 + warp * (K_SPAN / KWARPS);
  k_write_tile(P, w, tile, min(K_SPAN / KWARPS, n - first), T.k_idx + first, 0, m, l);
  __syncthreads();
}

// fp16 residual window, token-major [r][D]: A fragments are read directly; one 16-token tile per warp.
__device__ __forceinline__ void k_residual_tile(const DecodeParams& P, const TierDev& T, KShared& sh, const Where& w, const uint32_t* qh, int tile_t0, float& m, float& l) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tig = lane & 3;
  const int n = T.n_k;
  const __half* base = reinterpret_cast<const __half*>(T.k_data) + static_cast<int64_t>(w.bh) * n * D;
  const int t[2] = {min(tile_t0 + g, n - 1), min(tile_t0 + g + 8, n - 1)};
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int kt = 0; kt < 8; ++kt) {
    uint32_t a[4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const __half* p = base + static_cast<int64_t>(t[r]) * D + 16 * kt + 2 * tig;
      a[r] = *reinterpret_cast<const uint32_t*>(p);
      a[2 + r] = *reinterpret_cast<const uint32_t*>(p + 8);
    }
    const uint2 bq = k_plain_q(qh, kt);
    mma16816(acc, a[0], a[1], a[2], a[3], bq.x, bq.y);
  }
  float* tile = sh.u.tile[warp];
  if (tig < 2) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) tile[(r * 8 + g) * K_TROW + 2 * tig + e] = acc[r * 2 + e] * P.scale;
  }
  __syncwarp();
  k_write_tile(P, w, tile, min(16, n - tile_t0), nullptr, static_cast<int64_t>(P.L) - n + tile_t0, m, l);
}

// ONE_TIER: no CTA has units of two tiers.  WG: K groups of 64 or 128, which hold all 64 tokens of a warp: at 4 bits one set of
// scales and B operands instead of two.  (At 2 and 1 bits one MMA with hi and lo in neighbouring columns would do, too: 8 x 16 k g 64
// 27.5 us instead of 28.3.  But then the logits of the same codes and scales depend on the size of the group, in their last bits.)
template <bool ONE_TIER, bool WG>
__global__ void __launch_bounds__(KTHREADS, K_MIN_CTAS) k_pass_kernel(const __grid_constant__ DecodeParams P) {
  extern __shared__ __align__(128) unsigned char k_smem[];
  KShared& sh = *reinterpret_cast<KShared*>(k_smem);
  const Where w = where(P);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;

  // Let the V pass of this call (launched with programmatic stream serialisation) start its own
  // prologue - V words, index lists, scale/zero tiles - as soon as SM resources free up; it waits for
  // this grid to finish (griddepcontrol.wait) before it touches the logits or the softmax pairs.
  asm volatile("griddepcontrol.launch_dependents;");
  float m = -INFINITY, l = 0.f;  // this lane's softmax pair: head tig
  bool first = true;
  auto plain = [&](int ti, int t0, int t1) {  // fp16 tier, residual window
    const TierDev& T = P.tier[ti];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!first) __syncthreads();
    first = false;
    const uint32_t* q =
        g < P.r4 ? reinterpret_cast<const uint32_t*>(P.q + (static_cast<int64_t>(w.b) * P.nh_q + w.h0 + g) * D) + tig : nullptr;
    if (ti == 0) {
      for (int t = t0; t < t1; t += K_SPAN) k_f16_block(P, T, sh, w, q, t, m, l);
    } else {
      for (int t = t0 + warp * 16; t < t1; t += KWARPS * 16) k_residual_tile(P, T, sh, w, q, t, m, l);
    }
  };
  int t0, t1;
  if constexpr (ONE_TIER) {
    const int ti = only_share<false>(P, t0, t1);
    if (ti == 1) k_run<8, WG>(P, P.tier[1], sh, w, t0, t1, m, l, first);
    else if (ti == 2) k_run<4, WG>(P, P.tier[2], sh, w, t0, t1, m, l, first);
    else if (ti == 3) k_run<2, WG>(P, P.tier[3], sh, w, t0, t1, m, l, first);
    else if (ti == 4) k_run<1, WG>(P, P.tier[4], sh, w, t0, t1, m, l, first);
    else plain(ti, t0, t1);
  } else {
    if (share_of<false>(P, 1, t0, t1)) k_run<8, WG>(P, P.tier[1], sh, w, t0, t1, m, l, first);
    if (share_of<false>(P, 2, t0, t1)) k_run<4, WG>(P, P.tier[2], sh, w, t0, t1, m, l, first);
    if (share_of<false>(P, 3, t0, t1)) k_run<2, WG>(P, P.tier[3], sh, w, t0, t1, m, l, first);
    if (share_of<false>(P, 4, t0, t1)) k_run<1, WG>(P, P.tier[4], sh, w, t0, t1, m, l, first);
    for (int ti = 0; ti <= HQKV_NUM_TIERS; ti += HQKV_NUM_TIERS)
      if (share_of<false>(P, ti, t0, t1)) plain(ti, t0, t1);
  }
  // the warp's (max, sum-exp) per head: the eight lanes with the same tig
  {
    float mx = m;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = l * fast_exp2((m - (mx == -INFINITY ? 0.f : mx)) * LOG2E);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane < MAX_R4) {
      sh.v.red.m[warp][tig] = mx;
      sh.v.red.l[warp][tig] = sum;
    }
  }

  // the output accumulators of these heads start from zero in every call (the V pass, which
  // adds into them, starts after this grid has finished); everything above has passed its
  // griddepcontrol.wait, so the previous call is done with them
  if (blockIdx.y == 0) {
    const int64_t out0 = (static_cast<int64_t>(w.b) * P.nh_q + w.h0) * D;
    for (int i = 2 * tid; i < P.r4 * D; i += 2 * KTHREADS) {
      *reinterpret_cast<double2*>(P.v_acc + out0 + i) = make_double2(0., 0.);
      if (P.v_lows) *reinterpret_cast<ulonglong2*>(P.v_lows + out0 + i) = make_ulonglong2(0ull, 0ull);
    }
  }
  // (max, sum) of this CTA per head from the warps' pairs
  __syncthreads();
  if (tid < P.r4) {
    float m = sh.v.red.m[0][tid], l = sh.v.red.l[0][tid];
#pragma unroll
    for (int i = 1; i < KWARPS; ++i) softmax_merge(m, l, sh.v.red.m[i][tid], sh.v.red.l[i][tid]);
    P.k_part[(static_cast<int64_t>(w.bvh) * P.r4 + tid) * P.nk_ctas + blockIdx.y] = make_float2(m, l);
  }
}

// ------------------------------------------------------------------------------------------------
// v_pass
// ------------------------------------------------------------------------------------------------
// V tier, token-major rows of 128 channels.  Every warp of a CTA walks TILES of 64 consecutive tokens of one tier on its own
// and keeps the output of all 128 channels x four heads in its accumulators from tile to tile, so nothing but the end of the
// kernel needs the other warps.  (Tiles of 32 where the work is small.)  The contraction runs over tokens, 16 per step.
// ldmatrix.trans over 8 token rows x 16 bytes hands lane (g, tig) the 16-bit block g (2 / 4 / 8 channels) of two K-neighbours in one register: an m16n8k16 A fragment.
// As in the K pass the codes enter the tensor pipe as fp16 subnormals (one AND per pair of codes) and the scale - here per
// token and channel group - is folded into the B operand: out[h][c] = sum_t (p_t * scale_t,G) * code_t,c + sum_t p_t * zero_t,G,
// with p*scale carried exactly as hi + lo in neighbouring columns (below 4 bits, where 16 bytes are 64 channels, the columns
// are two groups of 32 and hi and lo are two MMAs).
//
// What bounds the kernel is the number of instructions and of shared-memory wavefronts per token, so:
//  * A lane takes four consecutive tokens (a QUAD) of one head through the softmax: one 16-byte load of their logits, one
//    8-byte store of their probabilities, one position fetched per lane and compared with its neighbours'.
//  * The k-order of a step's tokens is that of its quads (k = 2i, 2i+1, 2i+8, 2i+9 are the tokens of quad i), so that a
//    lane's own probabilities are a column of the B operand, and those of the other step one exchange away: the operand is
//    formed in registers.  (Formed once and left in shared memory it took as many bytes there, both ways, as the codes.)
//  * The scales and zeros of a quad are transposed to [group][token] once per tile: pairs as the B operand (and the A
//    operand of the zero term) wants them.
//  * One loop serves all widths, with a copy of the MMA part per width: what a kernel executes has to come from L2 into every SM
//    that has not run it lately, and a CTA of one or two tiles runs little of it twice.
// us a launch, before (operand through shared memory, a copy of the loop per width, a last CTA that writes) and now: batch 1 of
// 32 k tokens 12.6 / 10.1, 8 x 16 k g 64 30.7 / 26.0, 4 x 128 k 69 / 57.6, 32 x 4 k g 128 31.8 / 28.2, 57 x 8 planes of 1.6 k in
// five tiers 71 / 55.  At 8 x 16 k a launch executes 11.1 M warp instructions (12.3 M before); issue slots 44 %, HBM 43 % used.
// Codes are streamed through ONE tile buffer: the copy of 32 tokens of the next tile is issued when this tile's have been
// consumed, so a whole tile's work lies between a request and its use.
// CTAs of eight warps (half as many outputs to add up, half as many softmax pairs to fold), or of four where those fill the SMs better.
constexpr int V_SM_WARPS = 16;             // warps per SM the V pass is compiled for (128 registers)
constexpr int V_TILE = 64;                 // tokens per tile of a warp at most

// importance row emitted by the V pass: staging limits (positions + per-head halfs live in the warps' buffers)
constexpr int HS_TOKENS = 512;   // tokens per round
constexpr int HS_HEADS = 32;     // query heads it is built for (beyond that a separate launch sums the heads)
struct VWarpShared {
  alignas(128) unsigned char codes[V_TILE * D];   // rows in k-order
  unsigned char raw[2][V_TILE * 8];               // scales, zeros as in memory: [token][group]
  unsigned char t[2][V_TILE * 8];                 // scales, zeros as [quad][group][token]; four groups: see v_swizzle
  float red[MAX_R4][D];                           // output of the tiers that are done
};
template <int NW>
struct VShared {
  VWarpShared w[NW];
  float gm[MAX_R4], ginv[MAX_R4];                 // max * log2(e) and 1 / sum of the query heads
  unsigned is_last;
  unsigned pad_[3];
};
// Four groups: a quad is two 16-byte pieces; those of every second step lie the other way round (bank conflicts).
__device__ __forceinline__ uint32_t v_swizzle(uint32_t byte) { return byte ^ ((byte >> 3) & 16u); }

// Where the probabilities come from: the softmax of the scratch logits of four query heads, of two or one, or the caller.
enum VMode { V_FOUR, V_FEWER, V_GIVEN };
constexpr uint32_t V_NONE = 0xFFFFFFFFu;

// A value that the compiler cannot work out again from thread and block indices: what a loop uses of them is computed once.
__device__ __forceinline__ uint32_t keep(uint32_t v) { return __shfl_sync(0xffffffffu, v, threadIdx.x & 31); }

// Logits (or given weights) of the lane's NP quads, tokens 0 .. 3 and 32 .. 35 below `left`; -inf (0) beyond.  at: positions as the
// warp has them, of token `head` of the lane's quads.  dense (the same for the warp): they are quad[j] and the next three, quads of the
// scratch.  Fewer query heads: the lanes of the others read the first ones'.  Given weights are those of `rows`, the head's from
// `row` on (V_NONE: no such head); whole: its quads start on 8-byte boundaries.
// What is not a quad goes four tokens at a time: eight at a time cost the usual path 7 of 311 us (16 layers of 32 k tokens) in registers.
// us a call at 8 x 16 k, before quads (four tokens' loads together) / quads, the rest one by one / now: one head 74 / 81 / 59, any
// positions 91 / 111 / 96, given weights 38 / 41 / 28, and 55 / 50 / 44 at any positions.  Consecutive positions that start between quads
// take 57 / 86 / 72: the K pass writes their logits four bytes at a time.
template <int MODE, int NP>
__device__ __forceinline__ void v_gather(const DecodeParams& P, const Where& w, int head, const __half* rows, uint32_t row, bool whole, bool dense,
                                         const uint32_t (&quad)[NP], const uint32_t (&at)[NP], int left, float (&x)[NP][4]) {
  const float* logits = P.logits + static_cast<int64_t>(w.bvh) * P.L * P.r4;
  const unsigned short* given = reinterpret_cast<const unsigned short*>(rows) + (row != V_NONE ? row : 0u);
  if (dense) {
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      if constexpr (MODE == V_FOUR) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(logits) + (quad[j] + static_cast<uint32_t>(head)));
        x[j][0] = v.x, x[j][1] = v.y, x[j][2] = v.z, x[j][3] = v.w;
      } else if (MODE == V_GIVEN) {
        uint2 v = make_uint2(0u, 0u);
        if (row != V_NONE) {
          const unsigned short* p = given + quad[j];
          if (whole) v = __ldcg(reinterpret_cast<const uint2*>(p));
          else v = make_uint2(pack_lo16(__ldcg(p), __ldcg(p + 1)), pack_lo16(__ldcg(p + 2), __ldcg(p + 3)));
        }
        const float2 a = __half22float2(u32_as_h2(v.x)), b = __half22float2(u32_as_h2(v.y));
        x[j][0] = a.x, x[j][1] = a.y, x[j][2] = b.x, x[j][3] = b.y;
      } else if (P.r4 == 2) {  // (rows of two heads start on 8-byte boundaries)
        const float2* q = reinterpret_cast<const float2*>(logits) + (quad[j] + 2u * static_cast<uint32_t>(head & 1));
        const float2 a = __ldcg(q), b = __ldcg(q + 1);
        x[j][0] = a.x, x[j][1] = a.y, x[j][2] = b.x, x[j][3] = b.y;
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[j][i] = __ldcg(logits + (quad[j] + i));
      }
    }
    return;
  }
  uint32_t mine = at[0];
#pragma unroll 1
  for (int j = 0; j < NP; ++j) {
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] = MODE == V_GIVEN ? 0.f : -INFINITY;
      const uint32_t pos = __shfl_sync(0xffffffffu, mine, 8 * i + (threadIdx.x & 7));
      if (32 * j + i < left && pos != V_NONE && HQKV_INDEX_OK(pos, P.L)) {
        if constexpr (MODE == V_GIVEN) {
          if (row != V_NONE) y[i] = __half2float(__ushort_as_half(__ldcg(given + pos)));
        } else {
          y[i] = __ldcg(logits + logit_at(pos, head & (P.r4 - 1), P.r4, P.L));
        }
      }
    }
    mine = at[NP - 1];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[0][i] = x[NP - 1][i], x[NP - 1][i] = y[i];
  }
}

// The probabilities n of the lane's quads (tokens 0 1, 2 3 of each), whose positions are idx[0 .. 3] and idx[32 .. 35], to the row that starts
// at `at` elements of rows.  whole: all rows' quads start on 8-byte boundaries.
template <int NP>
__device__ __forceinline__ void v_store_probs(__half* rows, uint32_t at, bool whole, bool dense, const uint32_t (&quad)[NP], const int64_t* idx,
                                              int left, int L, const uint32_t (&n)[NP][2]) {
  if (dense) {
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      __half* a = rows + (at + quad[j]);
      if (whole) {
        *reinterpret_cast<uint2*>(a) = make_uint2(n[j][0], n[j][1]);
      } else if ((reinterpret_cast<uintptr_t>(a) & 2u) == 0u) {
        reinterpret_cast<uint32_t*>(a)[0] = n[j][0];
        reinterpret_cast<uint32_t*>(a)[1] = n[j][1];
      } else {
        a[0] = __ushort_as_half(static_cast<unsigned short>(n[j][0]));
        *reinterpret_cast<uint32_t*>(a + 1) = pack_hi_lo(n[j][0], n[j][1]);
        a[3] = __ushort_as_half(static_cast<unsigned short>(n[j][1] >> 16));
      }
    }
    return;
  }
  uint32_t a = n[0][0], b = n[0][1];
#pragma unroll 1
  for (int j = 0; j < NP; ++j) {
    uint32_t pos[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) pos[i] = 32 * j + i < left ? __ldg(reinterpret_cast<const uint32_t*>(idx + 32 * j + i)) : V_NONE;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (pos[i] != V_NONE && (!HQKV_CHECKS_ENABLED || pos[i] < static_cast<uint32_t>(L)))
        rows[at + pos[i]] = __ushort_as_half(static_cast<unsigned short>((i < 2 ? a : b) >> 16 * (i & 1)));
    a = n[NP - 1][0], b = n[NP - 1][1];
  }
}

// -C * std, to 22 bits, as two halfs
__device__ __forceinline__ void v_normal_offset(uint32_t sd, uint32_t& hi, uint32_t& lo) {
  const float2 t = __half22float2(u32_as_h2(sd));
  const float x = -HQKV_NORMAL1_CENTER * t.x, y = -HQKV_NORMAL1_CENTER * t.y;
  const __half2 h = __floats2half2_rn(x, y);
  const float2 r = __half22float2(h);
  hi = h2_as_u32(h), lo = pack_f16x2(x - r.x, y - r.y);
}

// field f of a 16-bit block as the fp16 subnormal code * 2^(k-24), k = v_shift(f)
template <int BITS>
__host__ __device__ constexpr int v_shift(int f) { return BITS == 8 ? 0 : BITS * f; }

// A CTA's way through the tiles of a tier, and a lane's places in them.
struct VRun {
  const unsigned char *codes, *s, *z;   // the CTA's next tiles to request
  uint32_t src, dst;                    // the lane's first piece of a step's codes: offset from there, place in shared memory
  uint32_t lm;                          // its ldmatrix row of the first step (1 bit: its first 2-byte block)
};
// Copy tokens [32 j, 32 j + 32) of the next tile.  WHOLE: all of them; otherwise those of which the tier has `left`.
template <int BITS, bool WHOLE>
__device__ __forceinline__ void v_request_pair(const VRun& r, int j, int left) {
  constexpr int STEP = 256 * BITS, LP = BITS == 8 ? 3 : BITS == 4 ? 2 : BITS == 2 ? 1 : 0;   // bytes; log2 of the pieces of a row
  constexpr int N = BITS >= 4 ? STEP / 512 : 1;                                             // copies per lane and step
  const int k = (threadIdx.x & 31) >> LP;
  const int first = (k & 16) + ((k & 6) << 1) + ((k >> 2) & 2) + (k & 1);   // the token in place k
  // (one bit: a step is 16 pieces, so the two halves of the warp take a step each)
#pragma unroll
  for (int st = 0; st < (BITS == 1 ? 1 : 2); ++st)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      // rows 4 i (8 bits) or 8 i (4 bits) on in k-order: tokens 0, 8, 2, 10 or 0, 2 on
      constexpr int T8[4] = {0, 8, 2, 10};
      const int tok = 32 * j + 16 * st + (BITS == 8 ? T8[i] : 2 * i);
      const uint32_t at = (BITS == 8 ? r.dst ^ ((i & 1) * 64u) : r.dst) + (2 * j + st) * STEP + i * 512;
      if (WHOLE || tok + first < left) cp_async_16(at, r.codes + r.src + tok * 16 * BITS);
    }
}
template <bool WHOLE, int NP>
__device__ __forceinline__ void v_request_tile(int bits, const VRun& r, int left) {
#pragma unroll 1
  for (int j = 0; j < NP; ++j) {
    if (bits == 4) v_request_pair<4, WHOLE>(r, j, left);
    else if (bits == 2) v_request_pair<2, WHOLE>(r, j, left);
    else if (bits == 8) v_request_pair<8, WHOLE>(r, j, left);
    else if (bits == 1) v_request_pair<1, WHOLE>(r, j, left);
    cp_async_commit();
  }
}

// Tokens [32 j, 32 j + 32) of a tile into acc[M-tile] (channels x columns, see v_store_output): p[step][tokens 0 1, 2 3 of quad
// tig] of the lane's head; st: the lane's quad in the scales of the tile's first step; rem: all ones in the lanes of the lo columns.
template <int BITS, int GV>
__device__ __forceinline__ void v_pair_mma(float (&acc)[8][4], const uint32_t (&p)[2][2], uint32_t lm, uint32_t st, uint32_t rem) {
  constexpr int NG = D >> GV;
  constexpr bool PAIR = BITS <= 2 && GV == 5;   // neighbouring columns are two groups
  const int g = (threadIdx.x & 31) >> 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t row = lm + k * 256 * BITS, sq = st + k * (32 * NG);
    if constexpr (PAIR) {
      uint32_t R[4];
      if constexpr (BITS == 2) ldmatrix_x4_trans(R, row);   // (octet, piece): (0, 0), (1, 0), (0, 1), (1, 1)
#pragma unroll
      for (int c = 0; c < 2; ++c) {      // 64 channels
        // (the lane's group of the two: 8 bytes on)
        const uint2 s = lds64((k ? sq + ((c * 16) ^ 16) : sq + c * 16) + (rem & 8u));
        const uint32_t h0 = h2_mul(p[k][0], s.x), h1 = h2_mul(p[k][1], s.y), l0 = h2_rem(p[k][0], s.x, h0), l1 = h2_rem(p[k][1], s.y, h1);
        uint32_t lo0, lo1;
        if constexpr (BITS == 2) {
          lo0 = R[2 * c], lo1 = R[2 * c + 1];
        } else {
          const uint32_t tb = row + 8 * c;
          lo0 = pack_lo16(lds16(tb), lds16(tb + 16)) >> (4 * (g >> 2));
          lo1 = pack_lo16(lds16(tb + 128), lds16(tb + 144)) >> (4 * (g >> 2));
        }
        const uint32_t hi0 = lo0 >> 8, hi1 = lo1 >> 8;
        uint32_t a[4][4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const uint32_t m = (BITS == 2 ? 0x00030003u : 0x00010001u) << v_shift<BITS>(f);
          a[f][0] = lo0 & m, a[f][1] = hi0 & m, a[f][2] = lo1 & m, a[f][3] = hi1 & m;
        }
#pragma unroll
        for (int f = 0; f < 4; ++f) mma16816(acc[4 * c + f], a[f][0], a[f][1], a[f][2], a[f][3], h0, h1);
#pragma unroll
        for (int f = 0; f < 4; ++f) mma16816(acc[4 * c + f], a[f][0], a[f][1], a[f][2], a[f][3], l0, l1);
      }
    } else {
      uint32_t s[NG][2], b[NG][2];
      if constexpr (NG == 1) {
        const uint2 u = lds64(sq);
        s[0][0] = u.x, s[0][1] = u.y;
      } else {
#pragma unroll
        for (int i = 0; i < NG / 2; ++i) {
          const uint4 u = lds128(NG == 4 && k ? sq + ((i * 16) ^ 16) : sq + i * 16);
          s[2 * i][0] = u.x, s[2 * i][1] = u.y, s[2 * i + 1][0] = u.z, s[2 * i + 1][1] = u.w;
        }
      }
      // even columns: hi = fp16(p*s); odd columns (m = -p): the exact remainder p*s - hi
      const uint32_t m0 = (p[k][0] ^ 0x80008000u) & rem, m1 = (p[k][1] ^ 0x80008000u) & rem;
#pragma unroll
      for (int G = 0; G < NG; ++G) b[G][0] = h2_fma(p[k][0], s[G][0], h2_mul(m0, s[G][0])), b[G][1] = h2_fma(p[k][1], s[G][1], h2_mul(m1, s[G][1]));
      if constexpr (BITS >= 4) {
        uint32_t R[4];
#pragma unroll
        for (int cb = 0; cb < 4; ++cb) {   // 32 channels: two M-tiles
          const int G = cb >> (GV - 5);
          uint32_t a[2][4];
          if constexpr (BITS == 8) {       // (octet, piece): (0, 2cb), (0, 2cb + 1), (1, 2cb), (1, 2cb + 1)
            ldmatrix_x4_trans(R, row ^ (cb * 32u));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              a[0][i] = R[i] & 0x00FF00FFu;
              a[1][i] = __byte_perm(R[i], 0u, 0x4341);
            }
          } else {                         // (octet, piece): (0, cb), (1, cb), (0, cb + 1), (1, cb + 1)
            if ((cb & 1) == 0) ldmatrix_x4_trans(R, row ^ (cb * 16u));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint32_t r = R[2 * (cb & 1) + i], rs = r >> 8;
              a[0][2 * i] = r & 0x000F000Fu, a[1][2 * i] = r & 0x00F000F0u;
              a[0][2 * i + 1] = rs & 0x000F000Fu, a[1][2 * i + 1] = rs & 0x00F000F0u;
            }
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) mma16816(acc[2 * cb + i], a[i][0], a[i][1], a[i][2], a[i][3], b[G][0], b[G][1]);
        }
      } else {
        uint32_t R[4];
        if constexpr (BITS == 2) ldmatrix_x4_trans(R, row);
#pragma unroll
        for (int c = 0; c < 2; ++c) {      // 64 channels of one group
          const int G = NG == 2 ? c : 0;
          uint32_t lo0, lo1;
          if constexpr (BITS == 2) {
            lo0 = R[2 * c], lo1 = R[2 * c + 1];
          } else {
            const uint32_t tb = row + 8 * c;
            lo0 = pack_lo16(lds16(tb), lds16(tb + 16)) >> (4 * (g >> 2));
            lo1 = pack_lo16(lds16(tb + 128), lds16(tb + 144)) >> (4 * (g >> 2));
          }
          const uint32_t hi0 = lo0 >> 8, hi1 = lo1 >> 8;
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const uint32_t m = (BITS == 2 ? 0x00030003u : 0x00010001u) << v_shift<BITS>(f);
            mma16816(acc[4 * c + f], lo0 & m, hi0 & m, lo1 & m, hi1 & m, b[G][0], b[G][1]);
          }
        }
      }
    }
  }
}

// The MMA part of a tile: pairs of steps, each refilled with the next tile's tokens when it is done.
template <int BITS, int GV, int NP>
__device__ __forceinline__ void v_tile(float (&acc)[8][4], const uint32_t (&p)[NP][2], const VRun& r, uint32_t t_s, uint32_t rem, bool refill) {
  const bool odd = threadIdx.x & 4;
  uint32_t p0 = p[0][0], p1 = p[0][1];
#pragma unroll 1
  for (int j = 0; j < NP; ++j) {
    // own probabilities are those of step lane bit 2 (of the pair) of the lane's head; the other step's are four lanes away
    const uint32_t a = __shfl_xor_sync(0xffffffffu, p0, 4), b = __shfl_xor_sync(0xffffffffu, p1, 4);
    const uint32_t ps[2][2] = {{odd ? a : p0, odd ? b : p1}, {odd ? p0 : a, odd ? p1 : b}};
    cp_async_wait<NP>();
    __syncwarp();
    v_pair_mma<BITS, GV>(acc, ps, r.lm + j * 512 * BITS, t_s + j * (64 * (D >> GV)), rem);
    // The codes make room for the next tile's.  At 8, 4 and 2 bits ldmatrix has read them for the whole warp; at 1 bit every lane
    // reads for itself, and the MMAs between need not stay before the copies.
    if constexpr (BITS == 1) __syncwarp();
    if (refill) v_request_pair<BITS, true>(r, j, 0);
    cp_async_commit();
    p0 = p[NP - 1][0], p1 = p[NP - 1][1];
  }
}

// Accumulators and zero term (lane: channel rows g, head tig) added to red[head tig][channel].
//   8 / 4 bits: M-tile 2*cb + i: rows g / g+8 = channels 32cb + 2g + i / + 16 (8 bits), 32cb + 4g + i / + 2 (4 bits);
//               a head's neighbouring columns are hi and lo
//   2 bits:     M-tile 4c + f: 64c + 8g + f / + 4;   1 bit: 64c + 16(g&3) + 4(g>>2) + f / + 8; in groups of 32 the columns
//               are two groups, a row keeps its own
// zt: zero term of channel group g % groups, head tig.
template <int GV>
__device__ __forceinline__ void v_store_output(float (*red)[D], const float (&acc)[8][4], int bits, float gain, float zt) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const bool wide = bits >= 4, pair = GV == 5 && !wide;
  const int second = bits == 2 ? g >> 2 : (g & 3) >> 1;                   // which group of the 64 channels the lane's rows are in
  const int other = bits == 8 ? 16 : bits == 4 ? 2 : bits == 2 ? 4 : 8;   // from rows g to rows g + 8
  float* out = red[tig] + (bits == 8 ? 2 * g : bits == 4 ? 4 * g : bits == 2 ? 8 * g : 16 * (g & 3) + 4 * (g >> 2));
  const float base = static_cast<float>(1 << 24) * gain, step = bits == 8 ? 1.f : bits == 4 ? 0x1p-4f : bits == 2 ? 0x1p-2f : 0x1p-1f;
#pragma unroll
  for (int mt = 0; mt < 8; ++mt) {
    const int f = wide ? mt & 1 : mt & 3;
    const float unscale = base * (f == 0 ? 1.f : f == 1 ? step : f == 2 ? step * step : step * step * step);   // 2^24 / 2^v_shift(f)
    const int block = wide ? mt >> 1 : 2 * (mt >> 2) + second;   // 32 channels
    const float z = __shfl_sync(0xffffffffu, zt, 4 * (block >> (GV - 5)) + tig);
    float* o = out + (wide ? 32 * (mt >> 1) : 64 * (mt >> 2)) + f;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float* a = &acc[mt][2 * r];
      o[r ? other : 0] += fmaf(pair ? (second ? a[1] : a[0]) : a[0] + a[1], unscale, z);
    }
  }
}

// fp16 tier and residual window, token-major rows [n][D] halfs: one 16-token step per warp straight
// from global memory; B = p, column n = head n.  The result is added to red.  ps: 128 bytes of shared memory.
template <int MODE, int NW>
__device__ __forceinline__ void v_plain_tile(const DecodeParams& P, const TierDev& T, const VShared<NW>& sh, __half* ps, float (*red)[D], const Where& w,
                                             int t0, int ntok, bool is_res) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const uint2* base = reinterpret_cast<const uint2*>(T.v_data) + (static_cast<int64_t>(w.bh) * T.n_v + t0) * 32;
  uint2 v[4][2];   // tokens 2tig, +1, +8, +9 x four channels of two rows of pieces
  auto load = [&](int half) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int tl = min(2 * tig + (p & 1) + (p >> 1) * 8, ntok - 1);
#pragma unroll
      for (int s = 0; s < 2; ++s) v[p][s] = ld_stream(base + tl * 32 + (2 * half + s) * 8 + g);
    }
  };
  load(0);
  {
    const int t = lane & 15;
    uint32_t pos = 0xFFFFFFFFu;
    if (t < ntok) pos = is_res ? static_cast<uint32_t>(P.L - T.n_v + t0 + t) : __ldg(reinterpret_cast<const uint32_t*>(T.v_idx + t0 + t));
    if (pos != 0xFFFFFFFFu && !HQKV_INDEX_OK(pos, P.L)) pos = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int h = 2 * (lane >> 4) + i;
      const bool on = h < P.r4 && pos != 0xFFFFFFFFu;
      const int64_t at = (static_cast<int64_t>(w.b) * P.nh_q + w.h0 + h) * P.L + pos;
      __half e = __float2half_rn(0.f);
      if (on) {
        if constexpr (MODE == V_GIVEN) {
          e = __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(P.probs_in) + at));
        } else {
          const float x = __ldcg(P.logits + static_cast<int64_t>(w.bvh) * P.L * P.r4 + logit_at(pos, h, P.r4, P.L));
          const float f = fast_exp2(fmaf(x, LOG2E, -sh.gm[h]));
          e = __float2half_rn(f);
          P.weights[at] = __float2half_rn(f * sh.ginv[h]);
        }
      }
      ps[h * 16 + t] = e;
    }
  }
  __syncwarp();
  uint32_t b0 = 0u, b1 = 0u;
  if (g < MAX_R4) {
    b0 = *reinterpret_cast<const uint32_t*>(ps + g * 16 + 2 * tig);
    b1 = *reinterpret_cast<const uint32_t*>(ps + g * 16 + 2 * tig + 8);
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    if (half) load(1);
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // M-tile: half k of the lane's four channels
      uint32_t a[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // fragment register: row slot q & 1, token pair q >> 1
        const uint2 x0 = v[2 * (q >> 1)][q & 1], x1 = v[2 * (q >> 1) + 1][q & 1];
        const uint32_t u0 = k < 2 ? x0.x : x0.y, u1 = k < 2 ? x1.x : x1.y;
        a[q] = k & 1 ? pack_hi16(u0, u1) : pack_lo16(u0, u1);
      }
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      mma16816(acc, a[0], a[1], a[2], a[3], b0, b1);
      if (tig < 2) {  // rows g, g + 8: channels of the two rows of pieces; columns 2tig, 2tig+1 = heads (4-7: none)
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int e = 0; e < 2; ++e) red[2 * tig + e][4 * ((2 * half + s) * 8 + g) + k] += acc[s * 2 + e];
      }
    }
  }
  __syncwarp();
}

// Cross-GPU barrier of one call, run by up to `world` threads of one CTA: thread r tells peer r "my stores
// of call number n are done" by raising a counter in the peer's signal pad, then waits until peer r has
// told it the same.  The call number lives in device memory and is advanced here, so the launch can
// sit in a CUDA graph that is replayed.  Every wait is bounded: after max_spins polls the thread gives
// up, records which peer was missing in the status word and returns, so a rank that died cannot hang
// the others' GPUs (the step's gathered data is then incomplete; the host checks the status).
template <bool FENCE_FIRST>
__device__ __forceinline__ void peer_barrier_device(unsigned* const* pad, int rank, int world, unsigned* call_no,
                                                    int* status, long long max_spins, unsigned* shared_n) {
  const int r = threadIdx.x;
  if (r == 0) *shared_n = *call_no + 1u;
  __syncthreads();
  const unsigned n = *shared_n;
  if (r < world && r != rank) {
    if (FENCE_FIRST) __threadfence_system();  // this GPU's earlier peer stores first (the V pass has fenced them already)
    atomicAdd_system(pad[r] + rank, 1u);      // slot `rank` of peer r's pad counts my arrivals
    volatile unsigned* mine = pad[rank] + r;  // slot r of my pad counts peer r's arrivals
    long long spins = 0;
    while (static_cast<int>(*mine - n) < 0) {
      if (++spins > max_spins) {
        atomicExch(status, r + 1);  // gave up waiting for peer r
        break;
      }
      __nanosleep(20);
    }
    __threadfence_system();
  }
  __syncthreads();
  if (r == 0) *call_no = n;
}

static_assert(sizeof(VShared<4>::w) >= HS_TOKENS * 4 + HS_TOKENS * HS_HEADS * 2, "importance-row staging fits the tile buffers");
// Importance row of n tokens from token c0 of a tier on, run by the last CTA to finish their grid row (not inlined: its registers are its own).
template <int NW>
__device__ __noinline__ void head_sum_chunk(const DecodeParams& P, const TierDev& T, VShared<NW>& sh, int c0, int n, bool is_res) {
  constexpr int VTHREADS = NW * 32;
  const int tid = threadIdx.x;
  __threadfence();
  __syncthreads();  // the round before is done with the staging buffers
  // The warps' buffers are free by now: they stage the chunk's positions and, per token and head, the sum
  // over the batch rounded to fp16.  Loads first, all of them independent: an item is (token, eight heads),
  // four items - 32 gathers per batch entry - are in flight per thread; then one thread per token adds the
  // heads in head order.
  uint32_t* pos_s = reinterpret_cast<uint32_t*>(&sh);                        // [HS_TOKENS]
  __half* stage = reinterpret_cast<__half*>(pos_s + HS_TOKENS);              // [HS_TOKENS][HS_HEADS]
  for (int t = tid; t < n; t += VTHREADS)
    pos_s[t] = is_res ? static_cast<uint32_t>(P.L - T.n_v + c0 + t) : static_cast<uint32_t>(T.v_idx[c0 + t]);
  __syncthreads();
  constexpr int ITEMS = 4;
  const int nhq = P.nh_q, ngr = (nhq + 7) >> 3, items = n * ngr;
  const unsigned short* w = reinterpret_cast<const unsigned short*>(P.weights);
  for (int base = tid; base < items; base += ITEMS * VTHREADS) {
    float ob[ITEMS][8];
#pragma unroll
    for (int q = 0; q < ITEMS; ++q)
#pragma unroll
      for (int j = 0; j < 8; ++j) ob[q][j] = 0.f;
    for (int bb = 0; bb < P.B; ++bb) {
      unsigned short v[ITEMS][8];
#pragma unroll
      for (int q = 0; q < ITEMS; ++q) {
        const int item = base + q * VTHREADS;
        const int gq = item / n, t = item - gq * n;  // token fastest: neighbouring threads read neighbouring positions
        const bool live = item < items && HQKV_INDEX_OK(pos_s[t], P.L);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int h = 8 * gq + j;
          v[q][j] = (live && h < nhq) ? __ldcg(w + (static_cast<int64_t>(bb) * nhq + h) * P.L + pos_s[t])
                                      : static_cast<unsigned short>(0);
        }
      }
#pragma unroll
      for (int q = 0; q < ITEMS; ++q)
#pragma unroll
        for (int j = 0; j < 8; ++j) ob[q][j] = __fadd_rn(ob[q][j], __half2float(__ushort_as_half(v[q][j])));
    }
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
      const int item = base + q * VTHREADS;
      if (item >= items) continue;
      const int gq = item / n, t = item - gq * n;
#pragma unroll
      for (int j = 0; j < 8; ++j) stage[t * HS_HEADS + 8 * gq + j] = __float2half_rn(ob[q][j]);
    }
  }
  __syncthreads();
  for (int t = tid; t < n; t += VTHREADS) {
    if (!HQKV_INDEX_OK(pos_s[t], P.L)) continue;
    float over_heads = 0.f;
    for (int h = 0; h < nhq; ++h) over_heads = __fadd_rn(over_heads, __half2float(stage[t * HS_HEADS + h]));
    P.head_sum[pos_s[t]] = __float2half_rn(over_heads);
  }
}

// A plane's outputs without anybody reading them back.  An output has two 64-bit words, and every share adds its (not yet
// normalised) part to them as whole numbers: to the high word multiples of 2^-f, to the low word what that rounds off, in
// multiples of 2^-(f + 42), and a count to the bits above both.  The thread that finds both counts complete in what its own
// additions return has the whole sum; it normalises and writes it.  (Reductions, a fence, a counter and a last CTA that reads
// the sums are three round trips to L2 in a row, 2 us; this is one.)
//   Bits 0-51 the sum, 52-61 the count (up to V_MAX_SHARES = 512 shares), and of the high word 62 / 63 +inf / -inf, both NaN.
//   A value of V is below 2^25 (255 x 65504 + 65504) and a probability at most 1, so a plane of up to 2^b tokens sums up to
//   less than 2^(25 + b) in whatever order and combination of shares: with f = 25 - b that is 2^50 units.  The low word's shares
//   are at most 2^41 units each.
//   What the words round off is 2^-(68 - b) a share at most, 2^-42 of an output for 512 shares of 128 k tokens (the smallest
//   half is 2^-24, and its parts come as fp32 sums): the sum of fp32 parts, like the fp64 sum of the other form below, but the same
//   whatever the order.  One word with the fraction that is left beside the largest V (27 bits) rounded small outputs visibly.
// Whether high and low word become complete in the same thread's additions is for the memory system to say; mostly they do.
// Otherwise the thread with the high word marks the low one: either it finds it complete by then, or whoever completes it
// finds the mark and takes the high word.
// (Not direct - more shares, more than 4 M tokens, or peers that get the outputs too: fp64 sums, read by the last CTA.)
constexpr int V_MAX_SHARES = 512, V_MAX_BITS = 22, V_COUNT_AT = 52, V_LOW_BITS = 42;
constexpr unsigned long long V_MARK = 1ull << 63;
__device__ __forceinline__ int v_count(unsigned long long word) { return static_cast<int>((word + (1ull << (V_COUNT_AT - 1)) & ~(3ull << 62)) >> V_COUNT_AT); }  // (a negative sum borrows from the count)
__device__ __forceinline__ double v_part(unsigned long long word) {
  return static_cast<double>(static_cast<long long>(word << (64 - V_COUNT_AT)) >> (64 - V_COUNT_AT));
}
template <int NW, bool FOUR>
__device__ __forceinline__ void v_finish(const DecodeParams& P, const VShared<NW>& sh, int64_t out0) {
  constexpr int EACH = MAX_R4 * D / (NW * 32), STEP = MAX_R4 / EACH;   // outputs of a thread: heads h0, h0 + STEP, ...
  const int c = threadIdx.x & (D - 1), h0 = threadIdx.x / D;
  unsigned long long* high = reinterpret_cast<unsigned long long*>(P.v_acc) + out0 + c;
  unsigned long long* low = P.v_lows + out0 + c;
  unsigned long long a[EACH], b[EACH];
#pragma unroll
  for (int k = 0; k < EACH; ++k) {
    const int h = h0 + STEP * k;
    if (!FOUR && h >= P.r4) break;
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < NW; ++i) v += sh.w[i].red[h][c];
    a[k] = b[k] = 1ull << V_COUNT_AT;
    if (fabsf(v) < P.v_limit) {
      const float units = rintf(v * P.v_units);
      a[k] += static_cast<unsigned long long>(__float2ll_rn(units));
      b[k] += static_cast<unsigned long long>(__float2ll_rn(fmaf(v, P.v_units, -units) * static_cast<float>(1ull << V_LOW_BITS)));  // (the difference is exact)
    } else {
      atomicOr(high + h * D, v > 0.f ? 1ull << 62 : v < 0.f ? 1ull << 63 : 3ull << 62);   // (before the thread's own addition to the word)
    }
  }
#pragma unroll
  for (int k = 0; k < EACH; ++k) {
    const int h = h0 + STEP * k;
    if (!FOUR && h >= P.r4) break;
    b[k] += atomicAdd(low + h * D, b[k]);
    a[k] += atomicAdd(high + h * D, a[k]);
  }
#pragma unroll
  for (int k = 0; k < EACH; ++k) {
    const int h = h0 + STEP * k;
    if (!FOUR && h >= P.r4) break;
    const bool high_done = v_count(a[k]) == P.nv_ctas;
    bool low_done = v_count(b[k]) == P.nv_ctas;
    if (high_done && !low_done) {
      // (the missing additions were issued before those that the high word has: mostly another look is enough)
#pragma unroll 1
      for (int looks = 0; looks < 4 && !low_done; ++looks) {
        b[k] = *const_cast<volatile unsigned long long*>(low + h * D);
        low_done = v_count(b[k]) == P.nv_ctas;
      }
      if (!low_done) {
        __threadfence();   // (whoever finds the mark finds the high word complete)
        b[k] = atomicOr(low + h * D, V_MARK);
        low_done = v_count(b[k]) == P.nv_ctas;
      }
    } else if (!high_done && low_done) {
      low_done = (b[k] & V_MARK) != 0;
      if (low_done) {
        __threadfence();
        a[k] = atomicAdd(high + h * D, 0ull);
      }
    }
    if (!low_done) continue;
    const unsigned odd = static_cast<unsigned>(a[k] >> 62);
    double sum = (v_part(a[k]) + v_part(b[k]) * (1. / (1ull << V_LOW_BITS))) * P.v_unit;
    if (odd) sum = odd == 1u ? INFINITY : odd == 2u ? -INFINITY : __int_as_float(0x7FC00000);
    P.out[out0 + h * D + c] = __float2half_rn(static_cast<float>(sum) * sh.ginv[h]);
    high[h * D] = low[h * D] = 0ull;   // (nobody else comes: a V pass without a K pass before it starts from zero, too)
  }
}

// GV: log2 of the channel group.  NP: pairs of 16-token steps in a tile.  NW: warps.
template <int GV, int MODE, int NP, int NW>
__global__ void __launch_bounds__(NW * 32, V_SM_WARPS / NW) v_pass_kernel(const __grid_constant__ DecodeParams P) {
  constexpr int NG = D >> GV, VTHREADS = NW * 32;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  VShared<NW>& sh = *reinterpret_cast<VShared<NW>*>(smem_raw);
  const Where w = where(P);
  // (the warp's number in a form that the compiler knows to be the same in all lanes: what depends on it is uniform)
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), g = lane >> 2, tig = lane & 3;

  // The next kernel of the stream - the K pass of the next decode call, if it was launched with
  // programmatic stream serialisation - may start its cache-only prologue while this grid drains.
  asm volatile("griddepcontrol.launch_dependents;");
  VWarpShared& ws = sh.w[warp];
#pragma unroll
  for (int i = 0; i < MAX_R4; ++i) reinterpret_cast<float4*>(ws.red[i])[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  // The lane in the softmax: head lane / 8, quad lane % 8 of the eight of a pair of steps.
  constexpr int tile = 32 * NP, stride = NW * tile;   // tokens of a warp, of the CTA at a time
  const int head = lane >> 3, wtok = warp * tile + 4 * (lane & 7), mine = keep(wtok + head);   // first token of its first quad; whose position it fetches
  __half* rows = (MODE == V_GIVEN ? const_cast<__half*>(P.probs_in) : P.weights) + (static_cast<int64_t>(w.b) * P.nh_q + w.h0) * P.L;   // (given ones are read)
  const uint32_t row = head < P.r4 ? static_cast<uint32_t>(head) * static_cast<uint32_t>(P.L) : V_NONE;
  float mh = INFINITY, inv = 0.f;   // max * log2(e), 1 / sum; of a head that is not there: probability 0
  const bool whole = ((reinterpret_cast<uintptr_t>(rows) | (static_cast<uintptr_t>(P.L) << 1)) & 7u) == 0u;
  const uint32_t rem = keep((g & 1) ? 0xFFFFFFFFu : 0u);
  // Its places in shared memory: 8 bytes of scales as they come; the quad it transposes (lanes 16 - 31: of the zeros), from and
  // to; quad tig in the scales, and with channel group g % NG in the zeros, of the first step.
  const uint32_t raw = smem_u32(ws.raw);
  const uint32_t sdst = keep(raw + (NG == 4 ? v_swizzle(lane * 8) : lane * 8));
  const uint32_t from = keep(raw + (lane >> 4) * (V_TILE * 8) + (NG == 4 ? v_swizzle((lane & 15) * 32) : (lane & 15) * (8 * NG)));
  const uint32_t t_s = keep(smem_u32(ws.t) + tig * (8 * NG));
  const uint32_t t_z = keep(smem_u32(ws.t[1]) + tig * (8 * NG) + (g & (NG - 1)) * 8);
  constexpr uint32_t TO = sizeof(VWarpShared::raw);   // from raw to t

  int f16_0, f16_1, res_0, res_1;   // (looked up here, where there is time)
  const bool f16 = share_of<true>(P, 0, f16_0, f16_1), res = share_of<true>(P, HQKV_NUM_TIERS, res_0, res_1);
  // One round per quantised tier, and an empty one where a CTA has none.
  bool begun = false;
#pragma unroll 1
  for (int ti = 1; ti <= HQKV_NUM_TIERS; ++ti) {
    int t0 = 0, t1 = 0;
    if (ti < HQKV_NUM_TIERS ? !share_of<true>(P, ti, t0, t1) : begun) continue;
    const TierDev& T = P.tier[ti];
    const int bits = T.bits;
    const bool normal = T.normal != 0;
    int left = t1 - t0;   // tokens from the CTA's next tiles on; those of the warp start tile * warp further
    const int64_t tok0 = static_cast<int64_t>(w.bh) * T.n_v + t0;
    VRun r;
    {
      const int lp = bits == 8 ? 3 : bits == 4 ? 2 : bits == 2 ? 1 : 0;   // log2 of the pieces of a row
      // codes: the 16-byte pieces of a step are shared out in the order they lie in shared memory, rows in k-order, the piece
      // index XORed with row bits so that the eight rows of an ldmatrix spread over all banks
      const int k = lane >> lp, piece = lane & ((1 << lp) - 1);
      const int token = (k & 16) + ((k & 6) << 1) + ((k >> 2) & 2) + (k & 1);
      const uint32_t codes = smem_u32(ws.codes);
      r.src = keep(((warp * tile + token) << (lp + 4)) + piece * 16);
      r.dst = keep(codes + (k << (lp + 4)) + ((piece ^ ((k >> (3 - lp)) & ((1 << lp) - 1))) << 4));
      // ldmatrix: matrices (octet, piece) (0, 0), (0, 1), (1, 0), (1, 1) at 8 bits, else (0, 0), (1, 0), (0, 1), (1, 1)
      const int octet = bits == 8 ? lane >> 4 : (lane >> 3) & 1, c = bits == 8 ? (lane >> 3) & 1 : lane >> 4, kk = 8 * octet + (lane & 7);
      r.lm = keep(bits == 1 ? codes + 2 * tig * 16 + 2 * (g & 3)
                            : codes + (kk << (lp + 4)) + ((c ^ ((kk >> (3 - lp)) & ((1 << lp) - 1))) << 4));
      r.codes = static_cast<const unsigned char*>(T.v_data) + (tok0 << (lp + 4));
      r.s = reinterpret_cast<const unsigned char*>(T.v_scale) + tok0 * (NG * 2);
      r.z = reinterpret_cast<const unsigned char*>(T.v_zero) + tok0 * (NG * 2);
    }
    const int64_t* idx = T.v_idx + t0;   // positions of the tiles
    // (what lies beyond the tier is filled with zeros)
    auto request_scales = [&](int left) {
#pragma unroll
      for (int o = 0; o < V_TILE * NG * 2; o += 256) {
        const int mine = o + lane * 8;
        if (mine < tile * (NG * 2)) {
          const int at = warp * (tile * (NG * 2)) + mine, valid = max(0, min(8, left * (NG * 2) - at));
          const uint32_t from = valid ? at : 0;
          cp_async_8_fill(sdst + o, r.s + from, valid);
          cp_async_8_fill(sdst + V_TILE * 8 + o, r.z + from, valid);
        }
      }
    };
    // position of token `head` of the lane's quads (low word), of the tile after the next
    uint32_t at[NP], quad[NP];
    bool dense = false;
    auto positions = [&](const int64_t* idx, int left) {
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        // (Beyond the tier, whose last 32 tokens are all there wherever it holds a multiple of 32: those once more.  Their
        // probabilities are stored once more, too, and count with scales and zeros of 0.)
        int t = mine + 32 * j;
        if (t >= left && left >= 32) t = left - 32 + (t & 31);
        at[j] = t < left ? __ldg(reinterpret_cast<const uint32_t*>(idx + t)) : V_NONE;
      }
    };
    float x[NP][4];
    // Requested for the tiles that have `left` tokens from the first on: the logits (positions in at), the positions of the ones after them.
    auto gather = [&](int left) {
      bool ok = true;
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        quad[j] = __shfl_sync(0xffffffffu, at[j], lane & 7);
        ok = ok && at[j] == quad[j] + head && (quad[j] & 3u) == 0u && quad[j] < (static_cast<uint32_t>(P.L) & ~3u);
      }
      dense = __all_sync(0xffffffffu, ok);
      v_gather<MODE, NP>(P, w, head, rows, row, whole, dense, quad, at, min(left - wtok, tile), x);
      positions(idx + stride, left - stride);
    };
    __syncwarp();   // (the buffers may have served another tier)
    if (left > 0) {
      request_scales(left);
      cp_async_commit();
      if (left >= stride) v_request_tile<true, NP>(bits, r, 0);
      else v_request_tile<false, NP>(bits, r, left - warp * tile);
      positions(idx, left);
    }
    const bool waited = begun;
    begun = true;
    // (what reads only the cache has been requested before the K pass is known to be complete)
    if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (left > 0) gather(left);
    if (!waited && MODE != V_GIVEN) {
      // global (max, sum) of the heads from the K pass's pairs: warp = head, up to four pairs per lane in flight
      if (warp < P.r4) {
        const float2* pairs = P.k_part + (static_cast<int64_t>(w.bvh) * P.r4 + warp) * P.nk_ctas;
        float m = -INFINITY, l = 0.f;
#pragma unroll 1
        for (int c0 = lane; c0 < P.nk_ctas; c0 += 4 * 32) {
          float2 v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = c0 + 32 * j < P.nk_ctas ? __ldcg(pairs + c0 + 32 * j) : make_float2(-INFINITY, 0.f);
          const float mx = fmaxf(fmaxf(fmaxf(v[0].x, v[1].x), fmaxf(v[2].x, v[3].x)), m);
          const float ref = mx == -INFINITY ? 0.f : mx;   // every position masked out: 0, not NaN
          l *= fast_exp2((m - ref) * LOG2E);
#pragma unroll
          for (int j = 0; j < 4; ++j) l += v[j].y * fast_exp2((v[j].x - ref) * LOG2E);
          m = mx;
        }
        float mx = m;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, k));
        float sum = l * fast_exp2((m - (mx == -INFINITY ? 0.f : mx)) * LOG2E);
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
        if (lane == 0) {
          sh.gm[warp] = mx * LOG2E;
          sh.ginv[warp] = 1.f / sum;
        }
      }
      __syncthreads();
      if (head < P.r4) mh = sh.gm[head], inv = sh.ginv[head];
    }
    if (left <= 0) continue;
    float acc[8][4], za[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 1
    for (; left > 0; left -= stride) {
      const int next = left - stride;
      r.codes += stride * 16 * bits;
      r.s += stride * NG * 2;
      r.z += stride * NG * 2;
      cp_async_wait<NP>();   // scales and zeros (the codes of the tile may still be on their way)
      __syncwarp();
      // [token][group] -> [group][token] of a quad
      if constexpr (NG == 4) {
        const uint4 u = lds128(from), v = lds128(from ^ 16u);
        sts128(from + TO, pack_lo16(u.x, u.z), pack_lo16(v.x, v.z), pack_hi16(u.x, u.z), pack_hi16(v.x, v.z));
        sts128((from ^ 16u) + TO, pack_lo16(u.y, u.w), pack_lo16(v.y, v.w), pack_hi16(u.y, u.w), pack_hi16(v.y, v.w));
      } else if constexpr (NG == 2) {
        const uint4 u = lds128(from);
        sts128(from + TO, pack_lo16(u.x, u.y), pack_lo16(u.z, u.w), pack_hi16(u.x, u.y), pack_hi16(u.z, u.w));
      } else {
        const uint2 u = lds64(from);
        sts64(from + TO, u.x, u.y);
      }
      __syncwarp();
      if (next > 0) request_scales(next);
      cp_async_commit();
      uint32_t p[NP][2], n[NP][2];
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        if constexpr (MODE == V_GIVEN) {
          p[j][0] = pack_f16x2(x[j][0], x[j][1]), p[j][1] = pack_f16x2(x[j][2], x[j][3]);
        } else {
          float e[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) e[i] = fast_exp2(fmaf(x[j][i], LOG2E, -mh));  // exp2(-inf) = 0 beyond the tier
          p[j][0] = pack_f16x2(e[0], e[1]), p[j][1] = pack_f16x2(e[2], e[3]);
          n[j][0] = pack_f16x2(e[0] * inv, e[1] * inv), n[j][1] = pack_f16x2(e[2] * inv, e[3] * inv);
        }
        // Zero term.  Rows g of A are the channel groups of the even step's quads, rows g + 8 of the odd one's; B is the lane's own
        // probabilities: of the columns, head * 2 + (lane's step & 1), a lane keeps head tig of the step that the row is of:
        // acc[0] and acc[3].
        const uint32_t zq = t_z + j * (64 * NG);
        const uint32_t zo = (NG == 4 ? zq ^ 16u : zq) + 32 * NG;
        const uint2 ze = lds64(zq), zp = lds64(zo);
        mma16816(za, ze.x, zp.x, ze.y, zp.y, p[j][0], p[j][1]);
        if (normal) {  // value = std * C * (2 code - 1) + mean: the code-free term is sum_t p (mean - C std)
          const uint2 se = lds64(zq - V_TILE * 8), so = lds64(zo - V_TILE * 8);
          const uint32_t sd[4] = {se.x, so.x, se.y, so.y};
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v_normal_offset(sd[i], hi[i], lo[i]);
          mma16816(za, hi[0], hi[1], hi[2], hi[3], p[j][0], p[j][1]);
          mma16816(za, lo[0], lo[1], lo[2], lo[3], p[j][0], p[j][1]);
        }
      }
      if (MODE == V_FOUR || (MODE == V_FEWER && row != V_NONE)) v_store_probs<NP>(rows, row, whole, dense, quad, idx + wtok, min(left - wtok, tile), P.L, n);
      idx += stride;
      if (next > 0) gather(next);
      const bool refill = next >= stride;
      if (bits == 4) v_tile<4, GV, NP>(acc, p, r, t_s, rem, refill);
      else if (bits == 2) v_tile<2, GV, NP>(acc, p, r, t_s, rem, refill);
      else if (bits == 8) v_tile<8, GV, NP>(acc, p, r, t_s, rem, refill);
      else v_tile<1, GV, NP>(acc, p, r, t_s, rem, refill);
      if (next > 0 && !refill) {   // the tier ends within the next tiles
        __syncwarp();
        v_request_tile<false, NP>(bits, r, next - warp * tile);
      }
    }
    cp_async_wait<0>();
    __syncwarp();
    v_store_output<GV>(ws.red, acc, bits, normal ? 2.f * HQKV_NORMAL1_CENTER : 1.f, za[0] + za[3]);
  }
  __syncwarp();
  // ---- fp16 tier, residual window
#pragma unroll 1
  for (int ti = 0; ti <= HQKV_NUM_TIERS; ti += HQKV_NUM_TIERS) {
    if (!(ti ? res : f16)) continue;
    const int t0 = ti ? res_0 : f16_0, t1 = ti ? res_1 : f16_1;
    for (int t = t0 + 16 * warp; t < t1; t += 16 * NW)
      v_plain_tile<MODE>(P, P.tier[ti], sh, reinterpret_cast<__half*>(ws.raw), ws.red, w, t, min(16, t1 - t), ti != 0);
  }
  __syncthreads();
  // ---- the output of this CTA (warps added in index order) joins those of its plane
  const int64_t out0 = (static_cast<int64_t>(w.b) * P.nh_q + w.h0) * D;
  // (Weights given by the caller may add up to anything.)  fp64 reductions: their sum depends on the order of the fp32
  // partials only below 2^-53.
  double* accum = P.v_acc + out0;
  if (MODE != V_GIVEN && P.direct) {
    v_finish<NW, MODE == V_FOUR>(P, sh, out0);
  } else {
    for (int k = tid; k < P.r4 * D; k += VTHREADS) {
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < NW; ++i) v += sh.w[i].red[k >> 7][k & (D - 1)];
      atomicAdd(accum + k, static_cast<double>(v));
    }
  }
  // ---- not direct: the last CTA of this (batch, virtual kv head) normalises and writes the output
  if (tid == 0) sh.is_last = 0u;
  if (!P.direct) {
    __syncthreads();
    if (tid == 0) {
      __threadfence();  // the CTA's adds, which the barrier has ordered before this thread's fence
      const unsigned prev = atomicAdd(&P.counters[w.bvh], 1u);
      sh.is_last = (prev == static_cast<unsigned>(P.nv_ctas) - 1u) ? 1u : 0u;
      if (sh.is_last) P.counters[w.bvh] = 0u;  // ready for the next call
    }
    __syncthreads();
  } else if (!P.head_sum) {
    return;
  }
  if (!P.direct && sh.is_last) {
    __threadfence();
    for (int i = tid * 2; i < P.r4 * D; i += VTHREADS * 2) {
      const double2 v = __ldcg(reinterpret_cast<const double2*>(accum + i));
      *reinterpret_cast<double2*>(accum + i) = make_double2(0., 0.);   // (as in v_finish)
      const float inv = MODE == V_GIVEN ? 1.f : sh.ginv[i >> 7];
      const __half2 o = __floats2half2_rn(static_cast<float>(v.x) * inv, static_cast<float>(v.y) * inv);
      const int64_t at = (static_cast<int64_t>(w.b) * P.nh_q + w.h0) * D + i;
      *reinterpret_cast<__half2*>(P.out + at) = o;
      // kv-head sharding: the same rows go straight into every peer's copy of the gathered output
      // (plain stores over NVLink; the callers' cross-GPU barrier makes them visible before use)
      if (P.peer_flagged) {
        // value and call number travel in ONE 8-byte store: the receiver needs no fence and no signal
        const uint2 e = make_uint2(h2_as_u32(o), P.peer_state[0] + 1u);
        for (int p = 0; p < P.n_peers; ++p) reinterpret_cast<uint2*>(P.peer_out[p])[at >> 1] = e;
      } else {
        for (int p = 0; p < P.n_peers; ++p) *reinterpret_cast<__half2*>(P.peer_out[p] + at) = o;
      }
    }
    if (P.world > 1) {
      // the CTA that finishes the last (batch, kv head) of this GPU runs the cross-GPU barrier: when this
      // kernel completes, every rank's rows are in this GPU's gathered buffer
      __threadfence_system();
      __syncthreads();
      if (tid == 0) {
        const unsigned done = atomicAdd(P.peer_state + 2, 1u);
        sh.is_last = (done == gridDim.x * gridDim.z - 1u) ? 1u : 0u;
        if (sh.is_last) P.peer_state[2] = 0u;
      }
      __syncthreads();
      if (sh.is_last) {
        __threadfence();
        // every CTA fenced its peer stores system-wide before it counted itself in, and this CTA saw the
        // full count: the signal may go out at once
        peer_barrier_device<false>(P.pad, P.rank, P.world, P.peer_state, reinterpret_cast<int*>(P.peer_state + 1),
                                   P.max_spins, &sh.pad_[0]);
      }
    }
  }
  // ---- importance row: sum of the probabilities over batch, then over heads, for the tokens of this share.
  //      The CTAs of all (batch, kv head) pairs with the same share wrote these tokens' probabilities; the
  //      last of them to arrive adds them in fixed order with the roundings of attn_weights.sum(0).sum(0) on fp16
  //      tensors (fp32 accumulation, one fp16 rounding per sum; model/public_func.py:253-254 of the reference).
  if (P.head_sum) {
    __threadfence();  // this CTA's probabilities
    __syncthreads();
    if (tid == 0) {
      const unsigned prev = atomicAdd(&P.hs_count[blockIdx.y], 1u);
      sh.is_last = (prev == gridDim.x * gridDim.z - 1u) ? 1u : 0u;
      if (sh.is_last) P.hs_count[blockIdx.y] = 0u;  // ready for the next call
    }
    __syncthreads();
    if (sh.is_last) {
      int t0, t1;
      for (int ti = 0; ti <= HQKV_NUM_TIERS; ++ti)
        if (share_of<true>(P, ti, t0, t1))
          for (int c0 = t0; c0 < t1; c0 += HS_TOKENS) head_sum_chunk(P, P.tier[ti], sh, c0, min(HS_TOKENS, t1 - c0), ti == HQKV_NUM_TIERS);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
// Both passes ask for the same amount of shared memory: their CTAs follow each other on an SM, and with two sizes the
// gaps that one kind leaves do not fit the other (four of one kind, then only three of the other, half the SMs a wave
// behind: 77 against 60 us per layer at batch 8).
constexpr size_t PASS_SMEM = sizeof(KShared) > sizeof(VShared<4>) ? sizeof(KShared) : sizeof(VShared<4>);
static_assert(4 * (PASS_SMEM + 1024) <= 228 * 1024, "four CTAs per SM");
constexpr size_t PASS_SMEM_8 = 2 * PASS_SMEM + 1024;   // a CTA of eight warps takes the place of two
static_assert(sizeof(VShared<8>) <= PASS_SMEM_8, "two CTAs of eight warps per SM");

static int ilog2(int v) {
  int s = 0;
  while ((1 << s) < v) ++s;
  return s;
}

struct Layout {
  size_t acc_off, logits_off, kpart_off, lows_off, total;   // (scratch that ends before the low words is taken, too)
};

// How the CTAs of a plane share its units.  Whatever it walks, a CTA pays about a unit for its prologue and the softmax pairs,
// and one more in the V pass for the output (16 x 8 planes of 33 units: V 30 us with four CTAs each, 0.9 of a wave, 33 with nine,
// 1.95; 20 x 8 planes: 33.8 with three, 34.8 with seven), and runs about as fast beside three others on its SM as beside one (its chain of loads
// bounds it): up to one wave the number of CTAs that are on the GPU does not count, only how long each is.  Beyond, the time
// lies between the load of the SMs and that of whole waves (the last wave starts as the first CTAs end).  13 x 16 planes of
// 15 units: 53 us with two CTAs each (0.7 of a wave), 50 with four; 30 x 8 planes of 15 units: 50 with two (0.8), 55 with
// three (1.2).
// Where one or two units per CTA make a wave, a second tier would double a CTA's latency: there a CTA keeps to one tier
// (two units at 8 bits).
//
// warps: 4 (K pass), 4 or 8 (V pass).  Returns what the longest of the waves takes in units of cost, 0 for CTAs of one tier.
static double divide(DecodeParams& P, int64_t planes, bool v, int warps) {
  const int slots = 148 * 16 / warps;
  int total = 0, unit = 0;  // cost of a plane; of a unit of most widths
  auto tokens = [&](const TierDev& t) { return v ? t.n_v : t.n_k; };
  auto set_units = [&](int pairs) {
    total = 0;
    for (TierDev& t : P.tier) {
      TierDev::Units& u = t.unit[v];
      u.tokens = !v || t.bits == 16 ? unit_tokens(t.bits) : 32 * warps * pairs;
      u.cost = !v || t.bits == 16 ? unit_cost(t.bits) : t.bits == 8 ? 6 * pairs : 4 * pairs;
      u.per_cost = 0xFFFFFFFFu / u.cost + 1u;
      u.cost0 = total;
      total += static_cast<int>(ceil_div(tokens(t), u.tokens)) * u.cost;
    }
    unit = P.tier[2].unit[v].cost;
  };
  // CTAs of one tier each, of at most this cost (at least a unit each)
  auto one_tier = [&](int budget, bool set) {
    int n = 0;
    for (TierDev& t : P.tier) {
      TierDev::Units& u = t.unit[v];
      if (set) u.cta0 = n;
      n += static_cast<int>(ceil_div(tokens(t), u.tokens * (budget < u.cost ? 1 : budget / u.cost)));
    }
    return n;
  };
  auto take = [&](int ctas, int per, int more) {
    (v ? P.nv_ctas : P.nk_ctas) = ctas;
    (v ? P.v_per : P.k_per) = per;
    (v ? P.v_more : P.k_more) = more;
  };
  if (v) {
    P.v_warps = warps;
    set_units(P.v_pairs = 1);
    if (warps == 8 && total > 0 && one_tier(unit, false) * planes <= slots) {
      take(one_tier(unit, true), unit, -1);
      return 0.;
    }
    P.v_pairs = 2;
  }
  set_units(2);
  if (total == 0) {
    take(0, 0, 0);
    return 0.;
  }
  // the smallest cost with which the planes' CTAs of one tier fit one wave (with more cost there are never more of them)
  if (one_tier(2 * unit, false) * planes <= slots) {
    int budget = v ? unit : 2 * unit_cost(8);
    while (one_tier(budget, false) * planes > slots) ++budget;
    take(one_tier(budget, true), budget, -1);
    return 0.;
  }
  // Up to one wave more CTAs only make it shorter: the search begins there, and ends where whole waves without a gap would take
  // longer than the best so far: the same number as of a search through all, in (host us for the three divisions of a call, before
  // and now) 1.7 / 0.6 at 8 planes of 32 k tokens, 4.7 / 0.3 at 8 of 130 k, 1.1 / 0.35 at 256 of 4 k.
  const double fixed = v ? 2 * unit : unit, per_wave = static_cast<double>(planes) / slots;
  const int64_t most = max(int64_t{1}, min(min(int64_t{1023}, static_cast<int64_t>(total / (2 * unit))), (4 * slots - 1) / planes + 1));
  int ctas = 0;
  double best = 0.;
  for (int n = static_cast<int>(max(int64_t{1}, min(most, slots / planes))); n <= most; ++n) {
    if (ctas && (total + fixed * n) * per_wave > best * (1. + 1e-9)) break;
    const double waves = static_cast<double>(n * planes) / slots;
    const double cost = (static_cast<double>(total) / n + fixed) * (waves <= 1. ? 1. : 0.5 * (waves + ceil(waves)));
    if (!ctas || cost < best) best = cost, ctas = n;
  }
  take(ctas, total / ctas, total % ctas);
  return best;
}

// sides: 1 = only the K side of the descriptor is looked at, 2 = only the V side, 3 = both
static int build_params(const hqkv_cache_desc_t* c, DecodeParams& P, Layout& lay, int sides = 3) {
  HQKV_REQUIRE(c != nullptr, "decode: null cache descriptor");
  HQKV_REQUIRE(c->B > 0 && c->H > 0 && c->nh_q > 0, "decode: B, H and nh_q must be positive");
  HQKV_REQUIRE(c->D == D, "decode: head dim must be 128 (got %d)", c->D);
  HQKV_REQUIRE(c->nh_q % c->H == 0 && c->nh_q / c->H <= MAX_REP,
               "decode: nh_q (%d) must be a multiple of H (%d) with at most %d query heads per kv head", c->nh_q,
               c->H, MAX_REP);
  HQKV_REQUIRE(valid_group(c->group_k) && valid_group(c->group_v), "decode: group sizes must be 32, 64 or 128");
  HQKV_REQUIRE(static_cast<int64_t>(c->B) * c->H <= 1024, "decode: B*H must not exceed 1024");
  HQKV_REQUIRE(c->n_new >= 0, "decode: negative residual length");
  memset(&P, 0, sizeof(P));
  P.B = c->B;
  P.H = c->H;
  P.nh_q = c->nh_q;
  const int rep = c->nh_q / c->H;
  HQKV_REQUIRE((rep & (rep - 1)) == 0, "decode: nh_q / H must be 1, 2, 4 or 8 (got %d)", rep);
  P.halves = rep > MAX_R4 ? 2 : 1;
  P.r4 = rep / P.halves;
  P.r4_shift = ilog2(P.r4);
  P.gk_shift = ilog2(c->group_k);
  P.gv_shift = ilog2(c->group_v);
  P.scale = c->softmax_scale;
  static const int expect_bits[HQKV_NUM_TIERS] = {16, 8, 4, 2, 1};
  int64_t nk_total = 0, nv_total = 0;
  for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
    const hqkv_tier_t& s = c->tier[t];
    TierDev& d = P.tier[t];
    HQKV_REQUIRE(s.n_k >= 0 && s.n_v >= 0, "decode: negative tier size");
    d.bits = expect_bits[t];
    d.n_k = (sides & 1) ? s.n_k : 0;
    d.n_v = (sides & 2) ? s.n_v : 0;
    if (d.n_k > 0 || d.n_v > 0) {
      HQKV_REQUIRE(s.bits == expect_bits[t], "decode: tier %d must hold %d-bit data (got %d)", t, expect_bits[t], s.bits);
      HQKV_REQUIRE(s.codec == HQKV_CODEC_UNIFORM || (s.codec == HQKV_CODEC_NORMAL && s.bits == 1),
                   "decode: tier %d: codec %d is not valid at %d bits (the Gaussian codebook is built for the 1-bit tier)", t,
                   s.codec, s.bits);
      d.normal = s.codec == HQKV_CODEC_NORMAL ? 1 : 0;
    }
    if (d.n_k > 0) {
      HQKV_REQUIRE(s.k_data && s.k_idx && aligned(s.k_idx, 8), "decode: tier %d K pointers are null or the index list is misaligned", t);
      if (s.bits < 16) {
        HQKV_REQUIRE(s.k_scale && s.k_zero && aligned(s.k_scale, 16) && aligned(s.k_zero, 16),
                     "decode: tier %d K scale/zero pointers are null or not 16-byte aligned", t);
        HQKV_REQUIRE(s.n_k % c->group_k == 0, "decode: tier %d K holds %d tokens, not a multiple of the K group %d", t,
                     s.n_k, c->group_k);
        HQKV_REQUIRE(aligned(s.k_data, 16), "decode: tier %d K codes must be 16-byte aligned", t);
      } else {
        HQKV_REQUIRE(s.n_k % 8 == 0 && aligned(s.k_data, 16),
                     "decode: the fp16 K tier needs a token count that is a multiple of 8 and 16-byte alignment");
      }
    }
    if (d.n_v > 0) {
      HQKV_REQUIRE(s.v_data && s.v_idx && aligned(s.v_idx, 8), "decode: tier %d V pointers are null or the index list is misaligned", t);
      if (s.bits < 16)
        HQKV_REQUIRE(s.v_scale && s.v_zero && aligned(s.v_scale, 8) && aligned(s.v_zero, 8),
                     "decode: tier %d V scale/zero pointers are null or not 8-byte aligned", t);
      HQKV_REQUIRE(aligned(s.v_data, 16), "decode: tier %d V data must be 16-byte aligned", t);
    }
    d.k_data = s.k_data;
    d.k_scale = static_cast<const __half*>(s.k_scale);
    d.k_zero = static_cast<const __half*>(s.k_zero);
    d.k_idx = s.k_idx;
    d.v_data = s.v_data;
    d.v_scale = static_cast<const __half*>(s.v_scale);
    d.v_zero = static_cast<const __half*>(s.v_zero);
    d.v_idx = s.v_idx;
    HQKV_REQUIRE(static_cast<int64_t>(s.n_k) * D * d.bits / 8 < (1ll << 31), "decode: tier %d K plane of one head exceeds 2 GiB", t);
    nk_total += d.n_k;
    nv_total += d.n_v;
  }
  if (sides == 3)
    HQKV_REQUIRE(nk_total == nv_total, "decode: K side holds %lld quantised tokens, V side %lld", (long long)nk_total,
                 (long long)nv_total);
  TierDev& r = P.tier[HQKV_NUM_TIERS];
  r.bits = 16;
  r.n_k = r.n_v = c->n_new;
  if (c->n_new > 0) {
    if (sides & 1) HQKV_REQUIRE(c->new_k && aligned(c->new_k, 16), "decode: residual K is null or not 16-byte aligned");
    if (sides & 2) HQKV_REQUIRE(c->new_v && aligned(c->new_v, 16), "decode: residual V is null or not 16-byte aligned");
  }
  r.k_data = c->new_k;
  r.v_data = c->new_v;
  const int64_t L = ((sides & 1) ? nk_total : nv_total) + c->n_new;
  HQKV_REQUIRE(L > 0, "decode: the cache is empty");
  HQKV_REQUIRE(L < (1ll << 30), "decode: cache too long");
  P.L = static_cast<int>(L);
  const int64_t planes = static_cast<int64_t>(c->B) * c->H * P.halves;
  divide(P, planes, false, KWARPS);
  // V pass: eight warps where one wave or as good a last wave comes of it.  (Batch 4 of 128 k tokens: 123 us a layer with eight
  // and 127 with four; batch 8 of 16 k, where four CTAs of eight warps per plane fill 86 % of the places: 57 and 55.)
  if (const double eight = divide(P, planes, true, 8)) {
    const DecodeParams with_eight = P;
    if (1.04 * divide(P, planes, true, 4) >= eight) P = with_eight;
  }
  lay.acc_off = HQKV_WS_HEADER_BYTES;
  lay.logits_off = (lay.acc_off + static_cast<size_t>(c->B) * c->nh_q * D * sizeof(double) + 255) & ~static_cast<size_t>(255);
  size_t off = lay.logits_off + static_cast<size_t>(c->B) * c->nh_q * L * sizeof(float);
  off = (off + 255) & ~static_cast<size_t>(255);
  lay.kpart_off = off;
  off += static_cast<size_t>(c->B) * c->nh_q * P.nk_ctas * sizeof(float2);
  lay.lows_off = (off + 255) & ~static_cast<size_t>(255);
  lay.total = lay.lows_off + ((static_cast<size_t>(c->B) * c->nh_q * D * sizeof(unsigned long long) + 255) & ~static_cast<size_t>(255));
  return HQKV_OK;
}

}  // namespace hqkv

using namespace hqkv;

extern "C" size_t hqkv_decode_workspace_bytes(const hqkv_cache_desc_t* cache_host) {
  DecodeParams P;
  Layout lay;
  if (build_params(cache_host, P, lay) != HQKV_OK) return 0;
  return lay.total;
}

extern "C" size_t hqkv_decode_workspace_zero_bytes(const hqkv_cache_desc_t* cache_host) {
  DecodeParams P;
  Layout lay;
  if (build_params(cache_host, P, lay) != HQKV_OK) return 0;
  return HQKV_WS_HEADER_BYTES;
}

namespace hqkv {
struct PeerArgs {
  void* const* out = nullptr;   // where this rank's block starts in each peer's gathered buffer
  int n_peers = 0;
  bool flagged = false;         // peers take flagged 8-byte entries
  void* const* pads = nullptr;  // signal pads of all ranks (own one included); null: no barrier
  int rank = 0, world = 0;
  void* state = nullptr;
  long long max_spins = 0;
};
static int decode_launch(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights, void* attn_output,
                         void* workspace, size_t workspace_bytes, int phases, const PeerArgs& peers, void* stream,
                         const void* probs_in = nullptr, const void* mask = nullptr, long long mask_bstride = 0,
                         long long mask_hstride = 0, void* head_sum = nullptr);
// the V pass emits the importance row itself up to these sizes (a CTA reads B*nh_q probabilities per token)
constexpr int HEAD_SUM_MAX_ROWS = 64;
constexpr int HEAD_SUM_MAX_CHUNKS = (HQKV_WS_HEADER_BYTES - 4096) / 4;
}

extern "C" int hqkv_decode_attention_phases(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights,
                                            void* attn_output, void* workspace, size_t workspace_bytes, int phases,
                                            void* stream) {
  return decode_launch(cache_host, q, attn_weights, attn_output, workspace, workspace_bytes, phases, hqkv::PeerArgs(), stream);
}

extern "C" int hqkv_decode_attention_gather(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights,
                                            void* attn_output, void* workspace, size_t workspace_bytes,
                                            void* const* peer_outputs_host, int n_peers, void* const* peer_pads_host,
                                            int rank, int world, void* state, long long max_spins, void* stream) {
  HQKV_REQUIRE(n_peers >= 0 && n_peers <= HQKV_MAX_PEERS, "decode_gather: at most %d peers (got %d)", HQKV_MAX_PEERS, n_peers);
  HQKV_REQUIRE(n_peers == 0 || peer_outputs_host, "decode_gather: null peer list");
  for (int p = 0; p < n_peers; ++p)
    HQKV_REQUIRE(peer_outputs_host[p] && aligned(peer_outputs_host[p], 4), "decode_gather: peer output %d is null or misaligned", p);
  hqkv::PeerArgs pa;
  pa.out = peer_outputs_host;
  pa.n_peers = n_peers;
  if (peer_pads_host) {
    HQKV_REQUIRE(world >= 2 && world <= HQKV_MAX_PEERS + 1 && rank >= 0 && rank < world, "decode_gather: bad rank/world");
    HQKV_REQUIRE(state && aligned(state, 4) && max_spins > 0, "decode_gather: null state or non-positive spin limit");
    for (int r = 0; r < world; ++r)
      HQKV_REQUIRE(peer_pads_host[r] && aligned(peer_pads_host[r], 4), "decode_gather: pad %d is null or misaligned", r);
    pa.pads = peer_pads_host;
    pa.rank = rank;
    pa.world = world;
    pa.state = state;
    pa.max_spins = max_spins;
  }
  return decode_launch(cache_host, q, attn_weights, attn_output, workspace, workspace_bytes, 3, pa, stream);
}

using PassKernel = void (*)(const DecodeParams);
static constexpr PassKernel k_kernels[4] = {k_pass_kernel<false, false>, k_pass_kernel<true, false>, k_pass_kernel<false, true>,
                                            k_pass_kernel<true, true>};  // [groups of more than 32][one tier per CTA]
template <int MODE, int NP, int NW>
static constexpr PassKernel v_kernels_of[3] = {v_pass_kernel<5, MODE, NP, NW>, v_pass_kernel<6, MODE, NP, NW>, v_pass_kernel<7, MODE, NP, NW>};
static constexpr const PassKernel* v_kernels[3][2][2] = {  // [VMode][8, 4 warps][pairs of steps - 1][log2 of the channel group - 5]
    {{v_kernels_of<V_FOUR, 1, 8>, v_kernels_of<V_FOUR, 2, 8>}, {nullptr, v_kernels_of<V_FOUR, 2, 4>}},
    {{v_kernels_of<V_FEWER, 1, 8>, v_kernels_of<V_FEWER, 2, 8>}, {nullptr, v_kernels_of<V_FEWER, 2, 4>}},
    {{v_kernels_of<V_GIVEN, 1, 8>, v_kernels_of<V_GIVEN, 2, 8>}, {nullptr, v_kernels_of<V_GIVEN, 2, 4>}}};

static int hqkv::decode_launch(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights, void* attn_output,
                               void* workspace, size_t workspace_bytes, int phases, const PeerArgs& peers, void* stream,
                               const void* probs_in, const void* mask, long long mask_bstride, long long mask_hstride,
                               void* head_sum) {
  HQKV_REQUIRE(phases >= 1 && phases <= 3, "decode: phases must be 1 (K pass), 2 (V pass) or 3 (both)");
  DecodeParams P;
  Layout lay;
  // a K-only call whose logits are the result, and a V-only call on given weights, look at one side only
  const int sides = probs_in ? 2 : ((phases == 1 && !attn_output) ? 1 : 3);
  int rc = build_params(cache_host, P, lay, sides);
  if (rc) return rc;
  P.n_peers = peers.n_peers;
  P.peer_flagged = peers.flagged ? 1 : 0;
  if (peers.flagged) P.peer_state = static_cast<unsigned*>(peers.state);
  for (int p = 0; p < peers.n_peers; ++p) P.peer_out[p] = static_cast<__half*>(peers.out[p]);
  if (peers.pads) {
    P.rank = peers.rank;
    P.world = peers.world;
    for (int r = 0; r < peers.world; ++r) P.pad[r] = static_cast<unsigned*>(peers.pads[r]);
    P.peer_state = static_cast<unsigned*>(peers.state);
    P.max_spins = peers.max_spins;
  }
  HQKV_REQUIRE(workspace, "decode: null pointer");
  if (phases & 1) HQKV_REQUIRE(q && aligned(q, 4), "decode: q is null or not 4-byte aligned");
  if (phases & 2) HQKV_REQUIRE(attn_output && (attn_weights || probs_in), "decode: null pointer");
  HQKV_REQUIRE(!probs_in || phases == 2, "decode: given weights go with the V pass alone");
  P.probs_in = static_cast<const __half*>(probs_in);
  HQKV_REQUIRE(!mask || (aligned(mask, 2) && mask_bstride >= 0 && mask_hstride >= 0), "decode: misaligned mask or negative stride");
  P.mask = static_cast<const __half*>(mask);
  P.mask_bstride = mask_bstride;
  P.mask_hstride = mask_hstride;
  HQKV_REQUIRE(aligned(workspace, 256), "decode: workspace must be 256-byte aligned");
  if (workspace_bytes < lay.lows_off)
    return fail(HQKV_E_WORKSPACE, "decode: workspace holds %zu bytes, %zu needed", workspace_bytes, lay.lows_off);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  P.q = static_cast<const __half*>(q);
  P.weights = static_cast<__half*>(attn_weights);
  P.out = static_cast<__half*>(attn_output);
  P.counters = reinterpret_cast<unsigned*>(ws);
  P.hs_count = reinterpret_cast<unsigned*>(ws + 4096);
  P.head_sum = static_cast<__half*>(head_sum);
  P.logits = reinterpret_cast<float*>(ws + lay.logits_off);
  P.k_part = reinterpret_cast<float2*>(ws + lay.kpart_off);
  P.v_acc = reinterpret_cast<double*>(ws + lay.acc_off);
  if (workspace_bytes >= lay.total) P.v_lows = reinterpret_cast<unsigned long long*>(ws + lay.lows_off);
  const int bits = ilog2(P.L);
  P.direct = !probs_in && peers.n_peers == 0 && !peers.pads && P.v_lows && P.nv_ctas <= V_MAX_SHARES && bits <= V_MAX_BITS;
  P.v_limit = ldexpf(1.f, 25 + bits);
  P.v_units = ldexpf(1.f, 25 - bits);
  P.v_unit = ldexpf(1.f, bits - 25);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned VH = static_cast<unsigned>(P.H * P.halves);
  HQKV_REQUIRE(P.nk_ctas <= 65535 && P.nv_ctas <= 65535, "decode: too many chunks");
  {
    // opt in to >48 KB of dynamic shared memory once per device
    static bool attr_set[64] = {};
    int dev = 0;
    HQKV_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
      // all of them with the same (largest) share of the L1 for shared memory: CTAs of kernels that ask for different
      // shares cannot be on an SM together
      auto opt_in = [](PassKernel f, size_t bytes) {
        HQKV_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
        HQKV_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        return 0;
      };
      for (PassKernel f : k_kernels)
        if (int rc = opt_in(f, PASS_SMEM)) return rc;
      for (const auto& mode : v_kernels)
        for (int four = 0; four < 2; ++four)
          for (const PassKernel* groups : mode[four])
            for (int g = 0; groups && g < 3; ++g)
              if (int rc = opt_in(groups[g], four ? PASS_SMEM : PASS_SMEM_8)) return rc;
      if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
  }
  // Both launches use programmatic stream serialisation: a grid may place its CTAs while the kernel before it
  // drains (if that kernel allows it - both of these do), and everything it does before its
  // griddepcontrol.wait reads only the cache tiers.
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  if ((phases & 1) && P.nk_ctas > 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(VH, P.nk_ctas, P.B);
    cfg.blockDim = dim3(KTHREADS);
    cfg.dynamicSmemBytes = PASS_SMEM;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    HQKV_CUDA(cudaLaunchKernelEx(&cfg, k_kernels[2 * (P.gk_shift > 5) + (P.k_more < 0)], P));
  }
  if ((phases & 2) && P.nv_ctas > 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(VH, P.nv_ctas, P.B);
    cfg.blockDim = dim3(32 * P.v_warps);
    cfg.dynamicSmemBytes = P.v_warps == 4 ? PASS_SMEM : PASS_SMEM_8;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    HQKV_CUDA(cudaLaunchKernelEx(&cfg, v_kernels[P.probs_in ? V_GIVEN : P.r4 == MAX_R4 ? V_FOUR : V_FEWER][P.v_warps == 4][P.v_pairs - 1][P.gv_shift - 5], P));
  }
  return HQKV_OK;
}

extern "C" int hqkv_decode_attention(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights,
                                     void* attn_output, void* workspace, size_t workspace_bytes, void* stream) {
  return hqkv_decode_attention_phases(cache_host, q, attn_weights, attn_output, workspace, workspace_bytes, 3, stream);
}

extern "C" int hqkv_decode_attention_masked(const hqkv_cache_desc_t* cache_host, const void* q, const void* mask,
                                            int64_t mask_b_stride, int64_t mask_h_stride, void* attn_weights,
                                            void* attn_output, void* workspace, size_t workspace_bytes, void* stream) {
  HQKV_REQUIRE(mask != nullptr, "decode_masked: null mask");
  return decode_launch(cache_host, q, attn_weights, attn_output, workspace, workspace_bytes, 3, hqkv::PeerArgs(), stream,
                       nullptr, mask, mask_b_stride, mask_h_stride);
}

extern "C" int hqkv_decode_attention_headsum(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights,
                                             void* attn_output, void* head_sum_row, void* workspace,
                                             size_t workspace_bytes, void* stream) {
  HQKV_REQUIRE(head_sum_row && aligned(head_sum_row, 2), "decode_headsum: null or misaligned row");
  DecodeParams P;
  Layout lay;
  int rc = build_params(cache_host, P, lay);
  if (rc) return rc;
  const bool fused = P.B * P.nh_q <= HEAD_SUM_MAX_ROWS && P.nh_q <= HS_HEADS && P.nv_ctas <= HEAD_SUM_MAX_CHUNKS;
  rc = decode_launch(cache_host, q, attn_weights, attn_output, workspace, workspace_bytes, 3, hqkv::PeerArgs(), stream,
                     nullptr, nullptr, 0, 0, fused ? head_sum_row : nullptr);
  if (rc || fused) return rc;
  // larger batches: one more launch over the probabilities just written
  return hqkv_head_sum(attn_weights, P.B, P.nh_q, P.L, P.L, head_sum_row, stream);
}

// ------------------------------------------------------------------------------------------------
// The two passes as operators of their own: raw logits of every tier, and the product of given weights with V
// ------------------------------------------------------------------------------------------------
namespace hqkv {
// fp32 logits of the scratch -> fp16 rows [plane][head][L]
__global__ void __launch_bounds__(256) logits_out_kernel(const float* logits, __half* out, int64_t planes, int64_t L, int heads) {
  const int64_t n = planes * L, stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int64_t plane = i / L, pos = i - plane * L;
    for (int h = 0; h < heads; ++h)
      out[(plane * heads + h) * L + pos] = __float2half_rn(__ldcg(logits + plane * L * heads + logit_at(pos, h, heads, static_cast<int>(L))));
  }
}
}  // namespace hqkv

extern "C" int hqkv_decode_logits(const hqkv_cache_desc_t* cache_host, const void* q, void* logits_f16, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  HQKV_REQUIRE(logits_f16 && aligned(logits_f16, 2), "decode_logits: null or misaligned output");
  int rc = decode_launch(cache_host, q, nullptr, nullptr, workspace, workspace_bytes, 1, hqkv::PeerArgs(), stream);
  if (rc) return rc;
  DecodeParams P;
  Layout lay;
  rc = build_params(cache_host, P, lay, 1);
  if (rc) return rc;
  const int64_t planes = static_cast<int64_t>(P.B) * P.H * P.halves, n = planes * P.L;
  const int blocks = static_cast<int>(n / 512 > 592 ? 592 : (n / 512 > 0 ? n / 512 : 1));
  hqkv::logits_out_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float*>(static_cast<unsigned char*>(workspace) + lay.logits_off),
      static_cast<__half*>(logits_f16), planes, P.L, P.r4);
  HQKV_LAUNCH_CHECK("decode_logits");
  return HQKV_OK;
}

extern "C" int hqkv_decode_weighted_sum(const hqkv_cache_desc_t* cache_host, const void* weights_f16, void* out,
                                        void* workspace, size_t workspace_bytes, void* stream) {
  HQKV_REQUIRE(weights_f16 && aligned(weights_f16, 2), "decode_weighted_sum: null or misaligned weights");
  {
    // no K pass runs in this call, so nobody clears the output accumulators: a stream-ordered memset does
    DecodeParams P;
    Layout lay;
    int rc = build_params(cache_host, P, lay, 2);
    if (rc) return rc;
    HQKV_REQUIRE(workspace && workspace_bytes >= lay.lows_off, "decode_weighted_sum: workspace too small");
    HQKV_CUDA(cudaMemsetAsync(static_cast<unsigned char*>(workspace) + lay.acc_off, 0, lay.logits_off - lay.acc_off,
                              static_cast<cudaStream_t>(stream)));
  }
  return decode_launch(cache_host, nullptr, nullptr, out, workspace, workspace_bytes, 2, hqkv::PeerArgs(), stream, weights_f16);
}

namespace hqkv {
unsigned decode_check_failures(bool reset) {
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
}  // namespace hqkv

extern "C" int hqkv_checks_enabled(void) { return HQKV_CHECKS_ENABLED; }

extern "C" int hqkv_check_failures(int reset, unsigned* count_host) {
  HQKV_REQUIRE(count_host != nullptr, "check_failures: null pointer");
  HQKV_CUDA(cudaDeviceSynchronize());
  *count_host = hqkv::decode_check_failures(reset != 0) + hqkv::policy_check_failures(reset != 0);
  return HQKV_OK;
}

// ------------------------------------------------------------------------------------------------
// Decode attention for callers that may not allocate device memory
// ------------------------------------------------------------------------------------------------
// Some hosts of this library cannot obtain scratch at call time: a serving loop that has handed all
// of the GPU's memory to its own pool, a latency-critical loop whose rules forbid allocation after
// start-up (cudaMalloc may synchronise the device, and may fail late), or a binding whose language
// runtime owns no device allocator.  For them the scratch of the two decode kernels lives in this
// fixed array, which every GPU that loads the library holds until the process exits.
//
// g_static_scratch names the array in DEVICE code.  In host code the same identifier is only a
// stand-in for the symbol, not a device address, so the host asks the runtime for the address once
// per device (cudaGetSymbolAddress with that device current) and passes the pointer it gets.
static __device__ __align__(256) unsigned char g_static_scratch[HQKV_STATIC_SCRATCH_BYTES];

namespace hqkv {
static void* g_static_scratch_ptr[64] = {};  // device address of the array, per device ordinal

static int static_scratch_address(void** out) {
  int dev = 0;
  HQKV_CUDA(cudaGetDevice(&dev));
  HQKV_REQUIRE(dev >= 0 && dev < 64, "decode_static: device ordinal %d out of range", dev);
  void* p = __atomic_load_n(&g_static_scratch_ptr[dev], __ATOMIC_ACQUIRE);
  if (!p) {
    HQKV_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
    HQKV_REQUIRE(p != nullptr, "decode_static: the scratch symbol has no address on device %d", dev);
    __atomic_store_n(&g_static_scratch_ptr[dev], p, __ATOMIC_RELEASE);  // every thread would store the same address
  }
  *out = p;
  return HQKV_OK;
}
}  // namespace hqkv

extern "C" size_t hqkv_decode_static_scratch_bytes(void) { return HQKV_STATIC_SCRATCH_BYTES; }

extern "C" int hqkv_decode_attention_static(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights,
                                            void* attn_output, void* stream) {
  DecodeParams P;
  Layout lay;
  const size_t need = build_params(cache_host, P, lay) == HQKV_OK ? lay.lows_off : 0;
  if (need == 0)  // invalid descriptor: let the regular path produce the precise message
    return hqkv_decode_attention(cache_host, q, attn_weights, attn_output, nullptr, 0, stream);
  if (need > HQKV_STATIC_SCRATCH_BYTES)
    return fail(HQKV_E_WORKSPACE,
                "decode_static: this cache needs %zu bytes of scratch, the built-in array holds %zu "
                "(HQKV_STATIC_SCRATCH_BYTES); use hqkv_decode_attention with caller-provided scratch",
                need, static_cast<size_t>(HQKV_STATIC_SCRATCH_BYTES));
  void* scratch = nullptr;
  int rc = static_scratch_address(&scratch);
  if (rc) return rc;
  // The array keeps whatever the previous call left.  Only the arrival counters have to start at
  // zero; a finished call leaves them zero, an aborted one might not, so they are cleared every time
  // (a stream-ordered memset, not an allocation).
  HQKV_CUDA(cudaMemsetAsync(scratch, 0, HQKV_WS_HEADER_BYTES, static_cast<cudaStream_t>(stream)));
  return hqkv_decode_attention(cache_host, q, attn_weights, attn_output, scratch, HQKV_STATIC_SCRATCH_BYTES, stream);
}

// ------------------------------------------------------------------------------------------------
// Cross-GPU barrier for the kv-head-sharded decode (one process per GPU)
// ------------------------------------------------------------------------------------------------
// After hqkv_decode_attention_gather every rank has written its heads' output rows into every peer's
// gathered buffer.  This kernel, launched by every rank on the same stream right after, (1) tells every
// peer "my stores of call number n are done" by raising a counter in the peer's signal pad, and (2)
// waits until every peer has told it the same.  The call number lives in device memory and is advanced
// by the kernel itself, so the launch can sit in a CUDA graph that is replayed.  Every wait is bounded:
// after max_spins polls the kernel gives up, records which peer was missing in *status and returns, so
// a rank that died cannot hang the others' GPUs (the data of that step is then incomplete and the host
// must check *status before it trusts it).
namespace hqkv {
struct PeerPads {
  unsigned* pad[HQKV_MAX_PEERS + 1];  // the ranks' signal pads, own one included
};

__global__ void peer_barrier_kernel(const __grid_constant__ PeerPads pads, int rank, int world, unsigned* call_no,
                                    int* status, long long max_spins) {
  __shared__ unsigned n;
  peer_barrier_device<true>(pads.pad, rank, world, call_no, status, max_spins, &n);
}
}  // namespace hqkv

extern "C" int hqkv_peer_barrier(void* const* peer_pads_host, int rank, int world, void* state, long long max_spins,
                                 void* stream) {
  HQKV_REQUIRE(world >= 1 && world <= HQKV_MAX_PEERS + 1 && rank >= 0 && rank < world, "peer_barrier: bad rank/world");
  HQKV_REQUIRE(peer_pads_host && state && aligned(state, 8) && max_spins > 0,
               "peer_barrier: null or misaligned pointer, or non-positive spin limit");
  hqkv::PeerPads pads = {};
  for (int r = 0; r < world; ++r) {
    HQKV_REQUIRE(peer_pads_host[r] && aligned(peer_pads_host[r], 4), "peer_barrier: pad %d is null or misaligned", r);
    pads.pad[r] = static_cast<unsigned*>(peer_pads_host[r]);
  }
  // state (8 bytes of this GPU's memory, zero before the first call): call number, status
  unsigned* st = static_cast<unsigned*>(state);
  hqkv::peer_barrier_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(pads, rank, world, st,
                                                                             reinterpret_cast<int*>(st + 1), max_spins);
  HQKV_LAUNCH_CHECK("peer_barrier");
  return HQKV_OK;
}

// ------------------------------------------------------------------------------------------------
// Flagged exchange: the low-latency form of the kv-head-sharded gather
// ------------------------------------------------------------------------------------------------
// hqkv_decode_attention_gather_flagged makes the V pass store every pair of output values together with
// the call number as ONE 8-byte word into the peers' receive buffers: a word whose flag equals the
// call number is complete, so no fence, no signal and no round trip is needed - the exchange costs
// one NVLink store latency.  hqkv_peer_unpack, enqueued by every rank right after, polls its own
// receive buffer (bounded), strips the flags into the plain gathered buffer [world][entries] of fp16
// pairs and advances the call number (device memory: the pair of launches replays from a CUDA graph).
// A receive buffer must not be reused before the peers have unpacked it: callers rotate at least two.
namespace hqkv {
__global__ void __launch_bounds__(256) peer_unpack_kernel(const uint2* recv, uint32_t* plain, int rank, int world,
                                                          int entries, unsigned* state, long long max_spins) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // this GPU's own decode call has finished
  const unsigned n = state[0] + 1u;
  // Four words per thread are requested together, so that a pass over words that have already arrived costs one
  // round trip, not one per word; a word that is still old is polled on its own.
  const int total = world * entries;
  for (int base = threadIdx.x; base < total; base += 4 * 256) {
    uint2 e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = base + j * 256;
      e[j] = make_uint2(0u, n);
      if (i < total && i / entries != rank)  // own rows were written in place by the decode kernel
        asm volatile("ld.volatile.global.v2.u32 {%0,%1}, [%2];" : "=r"(e[j].x), "=r"(e[j].y) : "l"(recv + i));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = base + j * 256;
      if (i >= total || i / entries == rank) continue;
      long long spins = 0;
      while (e[j].y != n) {
        if (++spins > max_spins) {
          atomicExch(reinterpret_cast<int*>(state + 1), i / entries + 1);  // gave up waiting for that rank
          break;
        }
        __nanosleep(20);
        asm volatile("ld.volatile.global.v2.u32 {%0,%1}, [%2];" : "=r"(e[j].x), "=r"(e[j].y) : "l"(recv + i));
      }
      plain[i] = e[j].x;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) state[0] = n;
}
}  // namespace hqkv

extern "C" int hqkv_decode_attention_gather_flagged(const hqkv_cache_desc_t* cache_host, const void* q, void* attn_weights,
                                                    void* attn_output, void* workspace, size_t workspace_bytes,
                                                    void* const* peer_recv_host, int n_peers, void* state, void* stream) {
  HQKV_REQUIRE(n_peers >= 1 && n_peers <= HQKV_MAX_PEERS, "decode_gather_flagged: 1..%d peers (got %d)", HQKV_MAX_PEERS, n_peers);
  HQKV_REQUIRE(peer_recv_host && state && aligned(state, 4), "decode_gather_flagged: null pointer");
  for (int p = 0; p < n_peers; ++p)
    HQKV_REQUIRE(peer_recv_host[p] && aligned(peer_recv_host[p], 8), "decode_gather_flagged: peer buffer %d is null or misaligned", p);
  hqkv::PeerArgs pa;
  pa.out = peer_recv_host;
  pa.n_peers = n_peers;
  pa.flagged = true;
  pa.state = state;
  return decode_launch(cache_host, q, attn_weights, attn_output, workspace, workspace_bytes, 3, pa, stream);
}

extern "C" int hqkv_peer_unpack(const void* recv, void* gathered, int rank, int world, int entries_per_rank, void* state,
                                long long max_spins, void* stream) {
  HQKV_REQUIRE(world >= 2 && world <= HQKV_MAX_PEERS + 1 && rank >= 0 && rank < world, "peer_unpack: bad rank/world");
  HQKV_REQUIRE(recv && gathered && state && aligned(recv, 8) && aligned(gathered, 4) && aligned(state, 4),
               "peer_unpack: null or misaligned pointer");
  HQKV_REQUIRE(entries_per_rank > 0 && max_spins > 0, "peer_unpack: sizes and the spin limit must be positive");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(256);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // polls may start while the decode call drains
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HQKV_CUDA(cudaLaunchKernelEx(&cfg, hqkv::peer_unpack_kernel, static_cast<const uint2*>(recv),
                               static_cast<uint32_t*>(gathered), rank, world, entries_per_rank,
                               static_cast<unsigned*>(state), max_spins));
  return HQKV_OK;
}
