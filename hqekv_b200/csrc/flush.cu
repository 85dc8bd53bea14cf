// Phase 2 of the flush (sm_100a): the destination tiers of one side from the plan - kept blocks are copied, arrivals are
// dequantised if they were quantised and re-quantised at the destination width.  One launch per side builds all tiers,
// their index lists and the part of the residual window that stays.
//
// HBM-bound copying and quantising: what matters is that loads are wide, coalesced and many at a time.
#include <string.h>

#include <type_traits>

#include "common.cuh"

namespace hqkv {

constexpr int D = 128;
constexpr int BUILD_THREADS = 256;

struct BuildDst {
  const int32_t* plan;  // [n] source of every token, see hqkv_flush_plan
  const int64_t* ids;   // [n] its id, copied to ids_out (null: not wanted)
  int64_t* ids_out;
  int64_t n;
  void* data;
  __half* scale;
  __half* zero;
  int tile0;            // first tile of this destination in the grid
};
struct BuildArgs {
  const void* data[HQKV_NUM_TIERS];
  const __half* scale[HQKV_NUM_TIERS];
  const __half* zero[HQKV_NUM_TIERS];
  int32_t n[HQKV_NUM_TIERS];
  const __half* residual;
  int64_t res_b_stride, res_h_stride;
  int wide;             // the residual's rows may be read, and what stays of it stored, 16 bytes at a time
  int tiers_wide;       // picks WIDE, see below (read by the host)
  int H, gshift;
  int normal_low;       // the 1-bit destination is written in the Gaussian-codebook codec
  BuildDst dst[HQKV_NUM_TIERS];
  int tiles;            // of all destinations; one more column of the grid copies the rest of the residual window
  const __half* rest;   // its first row of (batch 0, head 0), strides as the residual's
  __half* rest_out;
  int64_t rest_n;       // halfs per (batch, head)
};

// WIDE: sources and outputs lie where the widest accesses want them - codes on 16-byte boundaries, scales and zeros on 8-byte
// ones - and K tiers hold whole runs of 32 tokens.  Else everything goes by the tensors' own types (views into larger
// buffers may start anywhere): the same kernels, with words and halfs in the place of the wide pieces.
template <bool WIDE>
__device__ __forceinline__ uint2 load_words(const uint32_t* p) {
  return WIDE ? *reinterpret_cast<const uint2*>(p) : make_uint2(p[0], p[1]);
}

__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ uint32_t lo16(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410); }
__device__ __forceinline__ uint32_t hi16(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

// Two codes (bits [0,10) and [16,26)) -> half(half(code * scale) + zero), one rounding per step: 1024 + code is exact in fp16
__device__ __forceinline__ __half2 dequant2(uint32_t codes, __half2 scale, __half2 zero) {
  const __half2 c = __hsub2(as_h2(codes | 0x64006400u), as_h2(0x64006400u));
  return __hadd2_rn(__hmul2_rn(c, scale), zero);
}
// The minimum is the group's zero point: a zero has to have the sign of its first occurrence, and a NaN is treated as the
// element-by-element comparison treats it; both are rare and left to that comparison.
__device__ __forceinline__ bool doubtful(__half lo, __half hi) {
  return (__half_as_ushort(lo) & 0x7FFFu) == 0 || __hisnan(lo) || __hisnan(hi);
}
// the tail of the residual window: a copy
__device__ __forceinline__ void copy_rest(const BuildArgs& A, int bh) {
  const int b = bh / A.H, h = bh - b * A.H;
  const __half* src = A.rest + b * A.res_b_stride + h * A.res_h_stride;
  __half* dst = A.rest_out + bh * A.rest_n;
  if (A.wide) {
    for (int64_t i = threadIdx.x; i < A.rest_n / 8; i += BUILD_THREADS)
      reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
  } else {
    for (int64_t i = threadIdx.x; i < A.rest_n; i += BUILD_THREADS) dst[i] = src[i];
  }
}

// ------------------------------------------------------------------------------------------------
// K side: channel-major tiers, groups of tokens per channel
// ------------------------------------------------------------------------------------------------
// CTA = tile of one destination tier and (batch, head): 128 channel rows x 128 bytes of codes at 16 / 8 / 4 bits, 64 / 32
// bytes at 2 / 1 bits.  The tokens of a destination group come from one source and are consecutive there (tiers are
// filled and emptied in whole groups).  Kept groups are copied with eight lanes per row: runs of 128 bytes, four rows in
// flight per thread, where a thread per channel copied a word at a time, a row apart from its neighbour's.  An arrival is a
// thread per pair of channels and 32 tokens, all 32 in registers; its words and scales meet in shared memory and are
// stored in the same runs.  32 tokens into 24 k: 36 us (126 with a launch per tier and a thread per channel), into 8 x 16 k:
// 51 us (302; what it copies takes 28 at the copy rate); a prefill of 32 k tokens: 30 us (174).  What bounds a small flush is
// latency: the chain plan - source - store of a tile, and the few tiles with arrivals, which are started first for that
// reason (issue slots 23 % used, warps wait for memory).  A prefill, all arrivals: instructions (41 %) and their fetch.
// 64 registers a thread, for four CTAs per SM, are less than an arrival wants: the kernel spills 666 bytes and reads 626 back
// (-Xptxas -v), a codebook group 732 and 388.  Local loads and stores are 2 % of the instructions of that prefill, and
// 8 % of the 32 tokens into 24 k, where groups arrive in the codebook tier.
template <int BITS>
struct KBuild {
  static constexpr int TOKENS = BITS == 16 ? 64 : BITS == 8 ? 128 : 256;
  static constexpr int SUBS = TOKENS / 32;                                  // 32-token sub-blocks
  static constexpr int PIECE = BITS >= 4 ? 16 : 4 * BITS;                   // bytes per lane: eight pieces per row
  static constexpr int WPS = BITS;                                          // words per sub-block and row
  static __device__ __forceinline__ int sub_of(int piece) { return BITS == 16 ? piece >> 2 : BITS == 8 ? piece >> 1 : piece; }
};
constexpr int KB_MAX_SUBS = 8;
struct KBuildShared {
  uint32_t words[D * 33];  // [channel][words of the tile], one word of padding
  __half s[D * KB_MAX_SUBS], z[D * KB_MAX_SUBS];    // [channel][group of the tile]
  __half lo[D * KB_MAX_SUBS], hi[D * KB_MAX_SUBS];  // [channel][sub-block], groups of several sub-blocks
  int src[KB_MAX_SUBS], pos[KB_MAX_SUBS];
};

// 32 values of channels ch, ch + 1 from source tier `src` at pos: v[t] = (ch, ch + 1) of token pos + t
template <bool WIDE>
__device__ __forceinline__ void k_load32(const BuildArgs& A, int src, int64_t pos, int bh, int ch, __half2 (&v)[32]) {
  if (src < 0) {
    const int b = bh / A.H, h = bh - b * A.H;
    const __half* p = A.residual + b * A.res_b_stride + h * A.res_h_stride + pos * D + ch;
    if (A.wide) {
#pragma unroll
      for (int t = 0; t < 32; ++t) v[t] = *reinterpret_cast<const __half2*>(p + t * D);
    } else {
#pragma unroll
      for (int t = 0; t < 32; ++t) v[t] = __halves2half2(p[t * D], p[t * D + 1]);
    }
    return;
  }
  const int64_t row = static_cast<int64_t>(bh) * D + ch, n = A.n[src];
  if (src == 0) {
    const __half *p = reinterpret_cast<const __half*>(A.data[0]) + row * n + pos, *q = p + n;
    const int last = WIDE ? 31 : static_cast<int>(min(n - 1 - pos, static_cast<int64_t>(31)));
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const int i = WIDE ? t : min(t, last);
      v[t] = __halves2half2(p[i], q[i]);
    }
    return;
  }
  const int64_t G = n >> A.gshift, gi = row * G + (pos >> A.gshift);
  const __half2 sc = __halves2half2(A.scale[src][gi], A.scale[src][gi + G]), ze = __halves2half2(A.zero[src][gi], A.zero[src][gi + G]);
  if (src == 1) {
    const uint32_t *p = reinterpret_cast<const uint32_t*>(reinterpret_cast<const unsigned char*>(A.data[1]) + row * n + pos);
    const uint32_t *q = reinterpret_cast<const uint32_t*>(reinterpret_cast<const unsigned char*>(p) + n);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint2 a = load_words<WIDE>(p + 2 * w), b = load_words<WIDE>(q + 2 * w);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t x = k ? a.y : a.x, y = k ? b.y : b.x;
#pragma unroll
        for (int i = 0; i < 4; ++i) v[8 * w + 4 * k + i] = dequant2(((x >> (8 * i)) & 0xFFu) | (((y >> (8 * i)) & 0xFFu) << 16), sc, ze);
      }
    }
  } else if (src == 2) {
    const uint32_t *p = reinterpret_cast<const uint32_t*>(reinterpret_cast<const unsigned char*>(A.data[2]) + row * (n / 2) + pos / 2);
    const uint32_t *q = reinterpret_cast<const uint32_t*>(reinterpret_cast<const unsigned char*>(p) + n / 2);
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const uint2 a = load_words<WIDE>(p + 2 * w), b = load_words<WIDE>(q + 2 * w);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t x = k ? a.y : a.x, y = k ? b.y : b.x;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[16 * w + 8 * k + i] = dequant2(((x >> (4 * i)) & 0xFu) | (((y >> (4 * i)) & 0xFu) << 16), sc, ze);
      }
    }
  } else {
    const int bits = src == 3 ? 2 : 1;  // (nothing moves out of the 1-bit tier; read like the others all the same)
    const uint32_t *p = reinterpret_cast<const uint32_t*>(A.data[src]) + (row * n + pos) * bits / 32, *q = p + n * bits / 32;
    const uint64_t x = p[0] | (bits == 2 ? static_cast<uint64_t>(p[1]) << 32 : 0), y = q[0] | (bits == 2 ? static_cast<uint64_t>(q[1]) << 32 : 0);
    const uint32_t m = (1u << bits) - 1u;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      v[i] = dequant2((static_cast<uint32_t>(x >> (i * bits)) & m) | ((static_cast<uint32_t>(y >> (i * bits)) & m) << 16), sc, ze);
  }
}

// minimum and maximum of 32 values per channel of the pair
__device__ __forceinline__ void k_min_max(const __half2 (&v)[32], __half2& lo, __half2& hi) {
  lo = hi = v[0];
#pragma unroll
  for (int t = 1; t < 32; ++t) {
    lo = __hmin2_nan(lo, v[t]);
    hi = __hmax2_nan(hi, v[t]);
  }
  if (doubtful(__low2half(lo), __low2half(hi)) || doubtful(__high2half(lo), __high2half(hi))) {
    __half l0 = __low2half(v[0]), h0 = l0, l1 = __high2half(v[0]), h1 = l1;
#pragma unroll
    for (int t = 1; t < 32; ++t) {
      l0 = h_min(l0, __low2half(v[t]));
      h0 = h_max(h0, __low2half(v[t]));
      l1 = h_min(l1, __high2half(v[t]));
      h1 = h_max(h1, __high2half(v[t]));
    }
    lo = __halves2half2(l0, l1);
    hi = __halves2half2(h0, h1);
  }
}

// fp64 statistics of a group of the codebook tier in token order, channels ch and ch + 1: mean, std
template <bool WIDE>
__device__ __noinline__ void k_normal_stats(const BuildArgs& A, const KBuildShared& sh, int run0, int bh, int ch, __half2& mean, __half2& sd) {
  const int group = 1 << A.gshift;
  const double share = static_cast<double>(1.f / static_cast<float>(group));  // (exact: a power of two)
  double s0 = 0.0, s1 = 0.0, q0 = 0.0, q1 = 0.0;
  __half2 v[32];
  for (int i = 0; i < group; i += 32) {
    k_load32<WIDE>(A, sh.src[run0 + i / 32], sh.pos[run0 + i / 32], bh, ch, v);
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      s0 += static_cast<double>(__low2float(v[t]));
      s1 += static_cast<double>(__high2float(v[t]));
    }
  }
  const double m0 = s0 * share, m1 = s1 * share;
  for (int i = 0; i < group; i += 32) {
    if (group > 32) k_load32<WIDE>(A, sh.src[run0 + i / 32], sh.pos[run0 + i / 32], bh, ch, v);
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const double a = static_cast<double>(__low2float(v[t])) - m0, b = static_cast<double>(__high2float(v[t])) - m1;
      q0 += a * a;
      q1 += b * b;
    }
  }
  mean = __halves2half2(__double2half(m0), __double2half(m1));
  sd = __halves2half2(normal1_sd(q0, group), normal1_sd(q1, group));
}

// One arrival group of the codebook tier, channels ch and ch + 1.
template <bool WIDE>
__device__ __noinline__ void k_normal_group(const BuildArgs& A, KBuildShared& sh, int bh, int g, int ch) {
  const int per = 1 << (A.gshift - 5), s0 = g * per, group = 1 << A.gshift;
  __half2 v[32];
  float s[2][2] = {}, c[2][2] = {}, ss[2][4] = {};
  for (int i = 0; i < per; ++i) {
    k_load32<WIDE>(A, sh.src[s0 + i], sh.pos[s0 + i], bh, ch, v);
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      add_compensated(s[0][t & 1], c[0][t & 1], __low2float(v[t]));
      add_compensated(s[1][t & 1], c[1][t & 1], __high2float(v[t]));
    }
  }
  float m[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    c[k][0] += c[k][1];
    add_compensated(s[k][0], c[k][0], s[k][1]);
    m[k] = (s[k][0] + c[k][0]) * (1.f / static_cast<float>(group));
  }
  for (int i = 0; i < per; ++i) {
    if (per > 1) k_load32<WIDE>(A, sh.src[s0 + i], sh.pos[s0 + i], bh, ch, v);
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const float a = __low2float(v[t]) - m[0], b = __high2float(v[t]) - m[1];
      ss[0][t & 3] = fmaf(a, a, ss[0][t & 3]);
      ss[1][t & 3] = fmaf(b, b, ss[1][t & 3]);
    }
  }
  __half mean[2], sd[2];
  bool sure = true;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    sure &= normal1_fast(s[k][0], c[k][0], (ss[k][0] + ss[k][1]) + (ss[k][2] + ss[k][3]), group, mean[k], sd[k]);
  __half2 mean2 = __halves2half2(mean[0], mean[1]), sd2 = __halves2half2(sd[0], sd[1]);
  if (!sure) k_normal_stats<WIDE>(A, sh, s0, bh, ch, mean2, sd2);
  const __half2 bound = __halves2half2(normal1_bound(__low2half(sd2)), normal1_bound(__high2half(sd2)));
  for (int i = 0; i < per; ++i) {
    if (per > 1) k_load32<WIDE>(A, sh.src[s0 + i], sh.pos[s0 + i], bh, ch, v);
    uint32_t a = 0, b = 0;
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const uint32_t k = normal1_code2(v[t], mean2, bound);
      a |= (k & 1u) << t;
      b |= (k >> 16) << t;
    }
    sh.words[ch * 33 + s0 + i] = a;
    sh.words[(ch + 1) * 33 + s0 + i] = b;
  }
  sh.s[ch * KB_MAX_SUBS + g] = __low2half(sd2);
  sh.z[ch * KB_MAX_SUBS + g] = __low2half(mean2);
  sh.s[(ch + 1) * KB_MAX_SUBS + g] = __high2half(sd2);
  sh.z[(ch + 1) * KB_MAX_SUBS + g] = __high2half(mean2);
}

template <int PIECE>
struct PieceType;
template <>
struct PieceType<16> {
  using type = uint4;
};
template <>
struct PieceType<8> {
  using type = uint2;
};
template <>
struct PieceType<4> {
  using type = uint32_t;
};

// a piece of a row of codes (fp16 values at 16 bits, of which the tier has `left` from here on)
template <int BITS, bool WIDE, typename Piece>
__device__ __forceinline__ Piece load_piece(const unsigned char* p, int64_t left) {
  if constexpr (WIDE) return *reinterpret_cast<const Piece*>(p);
  Piece v;
  uint32_t* u = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
  for (int i = 0; i < static_cast<int>(sizeof(Piece) / 4); ++i) {
    if constexpr (BITS == 16) {
      const __half* h = reinterpret_cast<const __half*>(p);
      u[i] = as_u32(__halves2half2(h[min(static_cast<int64_t>(2 * i), left - 1)], h[min(static_cast<int64_t>(2 * i + 1), left - 1)]));
    } else {
      u[i] = reinterpret_cast<const uint32_t*>(p)[i];
    }
  }
  return v;
}
template <int BITS, bool WIDE, typename Piece>
__device__ __forceinline__ void store_piece(unsigned char* p, const Piece& v) {
  if constexpr (WIDE) {
    *reinterpret_cast<Piece*>(p) = v;
    return;
  }
  const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
  for (int i = 0; i < static_cast<int>(sizeof(Piece) / 4); ++i) {
    if constexpr (BITS == 16) {
      __half* h = reinterpret_cast<__half*>(p) + 2 * i;
      h[0] = __low2half(as_h2(u[i]));
      h[1] = __high2half(as_h2(u[i]));
    } else {
      reinterpret_cast<uint32_t*>(p)[i] = u[i];
    }
  }
}

template <int BITS, bool WIDE>
__device__ __forceinline__ void k_build_tile(const BuildArgs& A, KBuildShared& sh, int t, int tile, int bh) {
  using KB = KBuild<BITS>;
  using Piece = typename PieceType<KB::PIECE>::type;
  const BuildDst& dst = A.dst[t];
  const int tid = threadIdx.x;
  const int64_t j0 = static_cast<int64_t>(tile) * KB::TOKENS;
  const int nsub = static_cast<int>((dst.n - j0) / 32 < KB::SUBS ? (dst.n - j0) / 32 : KB::SUBS);
  if (tid < nsub) {
    const int32_t enc = dst.plan[j0 + 32 * tid];
    const int src = (enc >> 28) - 1;
    sh.src[tid] = src;
    // Runs of 32 start on multiples of 32.  The positions of ids that split blocks do not; there is no right result for them,
    // but no access may leave its boundary or its tier for them either (an fp16 tier that does not hold whole runs: see the
    // loads without WIDE).
    sh.pos[tid] = enc & (WIDE || src > 0 ? 0x0FFFFFE0 : 0x0FFFFFFF);
  }
  if (bh == 0 && dst.ids_out)
    for (int i = tid; i < 32 * nsub; i += BUILD_THREADS) dst.ids_out[j0 + i] = dst.ids[j0 + i];
  __syncthreads();
  const int piece = tid & 7, r0 = tid >> 3, sub = KB::sub_of(piece);
  const bool mine = sub < nsub, kept = mine && sh.src[sub] == t;
  // Scales of kept groups, requested together with their codes: a thread has one group of the tile and every `rstep`-th row.
  constexpr int SPT = 4;                                                 // scales per thread at most
  const int gs = (BITS == 8 ? 7 : 8) - A.gshift;                         // log2(groups per tile)
  const int sg = tid & ((1 << gs) - 1), srow = tid >> gs, rstep = BUILD_THREADS >> gs, sfirst = sg << (A.gshift - 5);
  const bool scaled = BITS < 16 && sfirst < nsub, scale_kept = scaled && sh.src[sfirst] == t;
  __half ks[SPT], kz[SPT];
  if (scale_kept) {
    const int64_t Gs = static_cast<int64_t>(A.n[t]) >> A.gshift, from = (static_cast<int64_t>(bh) * D + srow) * Gs + (sh.pos[sfirst] >> A.gshift);
    const __half *ps = A.scale[t] + from, *pz = A.zero[t] + from;
    const int64_t step = rstep * Gs;
#pragma unroll
    for (int k = 0; k < SPT; ++k)
      if (srow + k * rstep < D) {
        ks[k] = ps[k * step];
        kz[k] = pz[k * step];
      }
  }
  const int64_t out_row = dst.n * BITS / 8;
  unsigned char* out = reinterpret_cast<unsigned char*>(dst.data) + (static_cast<int64_t>(bh) * D + r0) * out_row + j0 * BITS / 8 + piece * KB::PIECE;
  if (kept) {
    const int64_t in_row = static_cast<int64_t>(A.n[t]) * BITS / 8;
    const unsigned char* in = reinterpret_cast<const unsigned char*>(A.data[t]) + static_cast<int64_t>(bh) * D * in_row +
                              static_cast<int64_t>(sh.pos[sub]) * BITS / 8 + (piece * KB::PIECE - sub * 4 * BITS);
    in += r0 * in_row;
    Piece v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = load_piece<BITS, WIDE, Piece>(in + 32 * i * in_row, A.n[t] - sh.pos[sub] - (piece * KB::PIECE / 2 - sub * 32));
#pragma unroll
    for (int i = 0; i < 4; ++i) store_piece<BITS, WIDE>(out + 32 * i * out_row, v[i]);
  }
  bool arrivals = false;
#pragma unroll
  for (int i = 0; i < KB::SUBS; ++i) arrivals |= i < nsub && sh.src[i] != t;
  const int ch = 2 * (tid & 63), set = tid >> 6;  // channel pair; four sub-blocks (groups) at a time
  if (arrivals) {
    uint32_t *w0 = sh.words + ch * 33, *w1 = w0 + 33;
    if constexpr (BITS == 16) {
      for (int i = set; i < nsub; i += 4) {
        if (sh.src[i] == t) continue;
        __half2 v[32];
        k_load32<WIDE>(A, sh.src[i], sh.pos[i], bh, ch, v);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          w0[16 * i + k] = lo16(as_u32(v[2 * k]), as_u32(v[2 * k + 1]));
          w1[16 * i + k] = hi16(as_u32(v[2 * k]), as_u32(v[2 * k + 1]));
        }
      }
    } else if (BITS == 1 && A.normal_low) {
      for (int g = set; g < (nsub << 5) >> A.gshift; g += 4)
        if (sh.src[g << (A.gshift - 5)] != t) k_normal_group<WIDE>(A, sh, bh, g, ch);
    } else {
      constexpr float levels = static_cast<float>((1 << BITS) - 1);
      auto finish = [&](const __half2(&v)[32], __half2 lo, __half2 hi, int i, int g) {
        const __half s0 = quant_scale(__low2half(lo), __low2half(hi), levels), s1 = quant_scale(__high2half(lo), __high2half(hi), levels);
        uint32_t a[BITS], b[BITS];
        quant_cols32<BITS, true>(v, quant_pair(__low2half(lo), s0, __high2half(lo), s1), a, b);
#pragma unroll
        for (int w = 0; w < BITS; ++w) {
          w0[i * KB::WPS + w] = a[w];
          w1[i * KB::WPS + w] = b[w];
        }
        sh.s[ch * KB_MAX_SUBS + g] = s0;
        sh.z[ch * KB_MAX_SUBS + g] = __low2half(lo);
        sh.s[(ch + 1) * KB_MAX_SUBS + g] = s1;
        sh.z[(ch + 1) * KB_MAX_SUBS + g] = __high2half(lo);
      };
      if (A.gshift == 5) {
        for (int i = set; i < nsub; i += 4) {
          if (sh.src[i] == t) continue;
          __half2 v[32], lo, hi;
          k_load32<WIDE>(A, sh.src[i], sh.pos[i], bh, ch, v);
          k_min_max(v, lo, hi);
          finish(v, lo, hi, i, i);
        }
      } else {  // groups of two or four sub-blocks: their minima meet in shared memory, the values are read once more
        for (int i = set; i < nsub; i += 4) {
          if (sh.src[i] == t) continue;
          __half2 v[32], lo, hi;
          k_load32<WIDE>(A, sh.src[i], sh.pos[i], bh, ch, v);
          k_min_max(v, lo, hi);
          sh.lo[ch * KB_MAX_SUBS + i] = __low2half(lo);
          sh.lo[(ch + 1) * KB_MAX_SUBS + i] = __high2half(lo);
          sh.hi[ch * KB_MAX_SUBS + i] = __low2half(hi);
          sh.hi[(ch + 1) * KB_MAX_SUBS + i] = __high2half(hi);
        }
        __syncthreads();
        const int per = 1 << (A.gshift - 5);
        for (int i = set; i < nsub; i += 4) {
          if (sh.src[i] == t) continue;
          const int s0 = i & ~(per - 1);
          __half l[2], h[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            l[c] = sh.lo[(ch + c) * KB_MAX_SUBS + s0];
            h[c] = sh.hi[(ch + c) * KB_MAX_SUBS + s0];
            for (int k = 1; k < per; ++k) {
              l[c] = h_min(l[c], sh.lo[(ch + c) * KB_MAX_SUBS + s0 + k]);
              h[c] = h_max(h[c], sh.hi[(ch + c) * KB_MAX_SUBS + s0 + k]);
            }
          }
          __half2 v[32];
          k_load32<WIDE>(A, sh.src[i], sh.pos[i], bh, ch, v);
          finish(v, __halves2half2(l[0], l[1]), __halves2half2(h[0], h[1]), i, i >> (A.gshift - 5));
        }
      }
    }
    __syncthreads();
    if (mine && !kept) {
      constexpr int W = KB::PIECE / 4;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t* w = sh.words + (r0 + 32 * i) * 33 + piece * W;
        Piece v;
        uint32_t* u = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
        for (int k = 0; k < W; ++k) u[k] = w[k];
        store_piece<BITS, WIDE>(out + 32 * i * out_row, v);
      }
    }
  }
  if constexpr (BITS < 16) {
    if (scaled) {
      const int64_t Gd = dst.n >> A.gshift, at = (static_cast<int64_t>(bh) * D + srow) * Gd + (j0 >> A.gshift) + sg, step = rstep * Gd;
#pragma unroll
      for (int k = 0; k < SPT; ++k) {
        const int r = srow + k * rstep;
        if (r >= D) break;
        dst.scale[at + k * step] = scale_kept ? ks[k] : sh.s[r * KB_MAX_SUBS + sg];
        dst.zero[at + k * step] = scale_kept ? kz[k] : sh.z[r * KB_MAX_SUBS + sg];
      }
    }
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(BUILD_THREADS, 4) flush_build_k_kernel(const __grid_constant__ BuildArgs A) {
  __shared__ KBuildShared sh;
  // From the back: arrivals, which take longer than copies, are at the end of a tier's list, and the lowest tier's longest.
  const int x = A.tiles - 1 - static_cast<int>(blockIdx.x), bh = blockIdx.y;
  if (x < 0) {
    copy_rest(A, bh);
    return;
  }
  if (x >= A.dst[4].tile0) k_build_tile<1, WIDE>(A, sh, 4, x - A.dst[4].tile0, bh);
  else if (x >= A.dst[3].tile0) k_build_tile<2, WIDE>(A, sh, 3, x - A.dst[3].tile0, bh);
  else if (x >= A.dst[2].tile0) k_build_tile<4, WIDE>(A, sh, 2, x - A.dst[2].tile0, bh);
  else if (x >= A.dst[1].tile0) k_build_tile<8, WIDE>(A, sh, 1, x - A.dst[1].tile0, bh);
  else k_build_tile<16, WIDE>(A, sh, 0, x, bh);
}

// ------------------------------------------------------------------------------------------------
// V side: token-major tiers, groups of channels per token
// ------------------------------------------------------------------------------------------------
// A warp takes 32 consecutive destination tokens of a (batch, head).  Blocks of tokens move together, so they are nearly always
// consecutive in one source (one vote): kept ones are then a contiguous copy, 16 bytes per lane, and arrivals are eight
// tokens per step, 32 channels per lane: a group's scale and reciprocal are one lane's.  (With eight channels per lane four
// lanes repeated them, and those instructions were most of the kernel.)  Any other run of tokens goes one by one.
// A prefill of 32 k tokens takes 20 us and is bound by instructions (63 % of the issue slots), 32 tokens into 24 k take 18 us and
// are bound by latency.  64 registers a thread: 1160 bytes spilled, 2324 read back (-Xptxas -v), most of it on ways that few
// warps take: 0.6 and 1.4 % of the instructions of the two are local loads and stores.
__device__ __forceinline__ __half v_get(const void* p, int bits, int c) {  // code c of a packed row
  const uint32_t w = reinterpret_cast<const uint32_t*>(p)[c * bits / 32];
  return __uint2half_rn((w >> ((c * bits) & 31)) & ((1u << bits) - 1u));
}

// fp64 statistics of a group of the codebook tier: sums of four channels, then pairwise over the group
__device__ __forceinline__ void v_normal_stats(const __half2 (&v)[16], int gshift, __half& mean, __half& sd) {
  const int lanes = 1 << (gshift - 5), group = 1 << gshift;
  auto over_group = [&](auto value) {
    double part[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      part[q] = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) part[q] += value(i & 1 ? __high2float(v[2 * q + (i >> 1)]) : __low2float(v[2 * q + (i >> 1)]));
    }
    double sum = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
    for (int off = 1; off < lanes; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    return sum;
  };
  const double mean64 = over_group([](float x) { return static_cast<double>(x); }) * static_cast<double>(1.f / static_cast<float>(group));
  const double ss = over_group([&](float x) {
    const double d = static_cast<double>(x) - mean64;
    return d * d;
  });
  mean = __double2half(mean64);
  sd = normal1_sd(ss, group);
}

// 32 values per lane quantised in groups of 2^(gshift - 5) adjacent lanes; codes -> words, the group's scale and zero (std
// and mean) -> sc, lo.  The whole warp takes part.
template <int BITS>
__device__ __forceinline__ void v_quantise32(const __half2 (&v)[16], int gshift, bool normal, uint32_t (&words)[BITS], __half& sc, __half& lo) {
  const int lanes = 1 << (gshift - 5), lane = threadIdx.x & 31, first = lane & ~(lanes - 1);
  if (BITS == 1 && normal) {
    const int group = 1 << gshift;
    float s[2] = {0.f, 0.f}, c[2] = {0.f, 0.f}, ss[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      add_compensated(s[0], c[0], __low2float(v[i]));
      add_compensated(s[1], c[1], __high2float(v[i]));
    }
    c[0] += c[1];
    add_compensated(s[0], c[0], s[1]);
    for (int off = 1; off < lanes; off <<= 1) {
      const float other = __shfl_xor_sync(0xffffffffu, s[0], off);
      c[0] += __shfl_xor_sync(0xffffffffu, c[0], off);
      add_compensated(s[0], c[0], other);
    }
    const float m = __shfl_sync(0xffffffffu, (s[0] + c[0]) * (1.f / static_cast<float>(group)), first);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float a = __low2float(v[i]) - m, b = __high2float(v[i]) - m;
      ss[(2 * i) & 3] = fmaf(a, a, ss[(2 * i) & 3]);
      ss[(2 * i + 1) & 3] = fmaf(b, b, ss[(2 * i + 1) & 3]);
    }
    float sq = (ss[0] + ss[1]) + (ss[2] + ss[3]);
    for (int off = 1; off < lanes; off <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
    const bool sure = normal1_fast(s[0], c[0], sq, group, lo, sc);
    if (__any_sync(0xffffffffu, !sure)) v_normal_stats(v, gshift, lo, sc);
    lo = __shfl_sync(0xffffffffu, lo, first);  // one lane's result for the group
    sc = __shfl_sync(0xffffffffu, sc, first);
    const __half2 mean2 = __half2half2(lo), bound = __half2half2(normal1_bound(sc));
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t k = normal1_code2(v[i], mean2, bound);
      w |= ((k | (k >> 15)) & 3u) << (2 * i);
    }
    words[0] = w;
    return;
  }
  constexpr float levels = static_cast<float>((1 << BITS) - 1);
  __half2 lo2 = v[0], hi2 = v[0];
#pragma unroll
  for (int i = 1; i < 16; ++i) {
    lo2 = __hmin2_nan(lo2, v[i]);
    hi2 = __hmax2_nan(hi2, v[i]);
  }
  // minimum and negated maximum together
  __half2 m = __halves2half2(__hmin_nan(__low2half(lo2), __high2half(lo2)), __hneg(__hmax_nan(__low2half(hi2), __high2half(hi2))));
  for (int off = 1; off < lanes; off <<= 1) m = __hmin2_nan(m, __shfl_xor_sync(0xffffffffu, m, off));
  lo = __low2half(m);
  __half hi = __hneg(__high2half(m));
  if (__any_sync(0xffffffffu, doubtful(lo, hi))) {  // element by element, the first lane of a group decides
    __half l = __low2half(v[0]), h = l;
#pragma unroll
    for (int i = 1; i < 32; ++i) {
      const __half x = i & 1 ? __high2half(v[i >> 1]) : __low2half(v[i >> 1]);
      l = h_min(l, x);
      h = h_max(h, x);
    }
    for (int off = 1; off < lanes; off <<= 1) {
      l = h_min(l, __shfl_xor_sync(0xffffffffu, l, off));
      h = h_max(h, __shfl_xor_sync(0xffffffffu, h, off));
    }
    lo = __shfl_sync(0xffffffffu, l, first);
    hi = __shfl_sync(0xffffffffu, h, first);
  }
  sc = quant_scale(lo, hi, levels);
  quant_row32<BITS, true>(v, quant_pair(lo, sc), words);
}
// Store a lane's quarter q of token `tok` (32 channels, 4 * BITS bytes) and, from the first lane of a group, its scale and
// zero.  live: the lane has a token.
template <int BITS, bool WIDE>
__device__ __forceinline__ void v_store32(const BuildArgs& A, const BuildDst& dst, int64_t tok, int q, const __half2 (&v)[16], bool live) {
  uint32_t* row = reinterpret_cast<uint32_t*>(dst.data) + tok * (4 * BITS) + q * BITS;
  if constexpr (BITS == 16) {
    if (live && !WIDE) {
      __half* out = static_cast<__half*>(dst.data) + tok * D + 32 * q;
#pragma unroll
      for (int i = 0; i < 16; ++i) out[2 * i] = __low2half(v[i]), out[2 * i + 1] = __high2half(v[i]);
    } else if (live) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        reinterpret_cast<uint4*>(row)[i] = make_uint4(as_u32(v[4 * i]), as_u32(v[4 * i + 1]), as_u32(v[4 * i + 2]), as_u32(v[4 * i + 3]));
    }
  } else {
    __half sc, lo;
    uint32_t w[BITS];
    v_quantise32<BITS>(v, A.gshift, A.normal_low != 0, w, sc, lo);
    if (!live) return;
    if constexpr (!WIDE) {
#pragma unroll
      for (int i = 0; i < BITS; ++i) row[i] = w[i];
    } else if constexpr (BITS == 8) {
      reinterpret_cast<uint4*>(row)[0] = make_uint4(w[0], w[1], w[2], w[3]);
      reinterpret_cast<uint4*>(row)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    } else if constexpr (BITS == 4) {
      *reinterpret_cast<uint4*>(row) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if constexpr (BITS == 2) {
      *reinterpret_cast<uint2*>(row) = make_uint2(w[0], w[1]);
    } else {
      *row = w[0];
    }
    if ((q & ((1 << (A.gshift - 5)) - 1)) == 0) {
      const int64_t at = tok * (D >> A.gshift) + (q >> (A.gshift - 5));
      dst.scale[at] = sc;
      dst.zero[at] = lo;
    }
  }
}

// Quarter q of a token's row of a source tier with SB bits (row at `row`, tok = its number over the (batch, head) planes).
template <int SB>
struct VUnit {
  uint32_t raw[SB];
  __half sc, ze;
};
template <int SB>
__device__ __forceinline__ void v_unit_load(const BuildArgs& A, VUnit<SB>& u, const unsigned char* row, int src, int64_t tok, int q) {
  const unsigned char* p = row + q * (4 * SB);
  if constexpr (SB >= 4) {
#pragma unroll
    for (int i = 0; i < SB / 4; ++i) {
      const uint4 x = reinterpret_cast<const uint4*>(p)[i];
      u.raw[4 * i] = x.x, u.raw[4 * i + 1] = x.y, u.raw[4 * i + 2] = x.z, u.raw[4 * i + 3] = x.w;
    }
  } else {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    u.raw[0] = x.x, u.raw[1] = x.y;
  }
  if constexpr (SB < 16) {
    const int64_t at = tok * (D >> A.gshift) + (q >> (A.gshift - 5));
    u.sc = A.scale[src][at];
    u.ze = A.zero[src][at];
  }
}
template <int SB>
__device__ __forceinline__ void v_unit_values(const VUnit<SB>& u, __half2 (&v)[16]) {
  if constexpr (SB == 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = as_h2(u.raw[i]);
  } else {
    const __half2 sc = __half2half2(u.sc), ze = __half2half2(u.ze);
    constexpr int PAIRS = 16 / SB;  // per word
    constexpr uint32_t M = (1u << SB) - 1u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t w = u.raw[i / PAIRS] >> ((i % PAIRS) * 2 * SB);
      v[i] = dequant2((w & M) | (((w >> SB) & M) << 16), sc, ze);
    }
  }
}
// 32 consecutive tokens that arrive from one source: rows at `rows`, 16 * SB bytes apart, tok = number of the first
template <int BITS, int SB>
__device__ __forceinline__ void v_arrive(const BuildArgs& A, const BuildDst& dst, const unsigned char* rows, int src, int64_t tok, int64_t out_tok) {
  const int lane = threadIdx.x & 31, q = lane & 3, row = lane >> 2;
  VUnit<SB> u;
  v_unit_load<SB>(A, u, rows + row * (16 * SB), src, tok + row, q);
#pragma unroll 1
  for (int s = 0; s < 32; s += 8) {
    __half2 v[16];
    v_unit_values<SB>(u, v);
    if (s + 8 < 32) v_unit_load<SB>(A, u, rows + (s + 8 + row) * (16 * SB), src, tok + s + 8 + row, q);
    v_store32<BITS, true>(A, dst, out_tok + s + row, q, v, true);
  }
}

// One token from any source, by the first four lanes of the warp.
template <int BITS, bool WIDE>
__device__ __noinline__ void v_one_token(const BuildArgs& A, int t, int32_t enc, int64_t j, int bh) {
  const BuildDst& dst = A.dst[t];
  const int lane = threadIdx.x & 31, q = lane & 3, ng = D >> A.gshift;
  const int src = (enc >> 28) - 1;
  const int64_t pos = enc & 0x0FFFFFFF, out_tok = static_cast<int64_t>(bh) * dst.n + j;
  if (src == t) {  // kept: copy the row verbatim
    const int64_t tok = static_cast<int64_t>(bh) * A.n[t] + pos;
    using Item = typename std::conditional<BITS == 16 && !WIDE, __half, uint32_t>::type;
    constexpr int N = 16 * BITS / sizeof(Item);  // per row
    for (int w = lane; w < N; w += 32) static_cast<Item*>(dst.data)[out_tok * N + w] = static_cast<const Item*>(A.data[t])[tok * N + w];
    if (BITS < 16 && lane < ng) {
      dst.scale[out_tok * ng + lane] = A.scale[t][tok * ng + lane];
      dst.zero[out_tok * ng + lane] = A.zero[t][tok * ng + lane];
    }
    return;
  }
  __half2 v[16];
  if (src < 0 || src == 0) {
    const int b = bh / A.H, h = bh - b * A.H;
    const __half* p = src < 0 ? A.residual + b * A.res_b_stride + h * A.res_h_stride + pos * D
                              : reinterpret_cast<const __half*>(A.data[0]) + (static_cast<int64_t>(bh) * A.n[0] + pos) * D;
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __halves2half2(p[32 * q + 2 * i], p[32 * q + 2 * i + 1]);
  } else {
    const int sb = 16 >> src;
    const int64_t tok = static_cast<int64_t>(bh) * A.n[src] + pos, at = tok * ng + (q >> (A.gshift - 5));
    const __half sc = A.scale[src][at], ze = A.zero[src][at];
    const uint32_t* w = reinterpret_cast<const uint32_t*>(A.data[src]) + tok * (4 * sb);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      v[i] = __halves2half2(h_add(h_mul(v_get(w, sb, 32 * q + 2 * i), sc), ze), h_add(h_mul(v_get(w, sb, 32 * q + 2 * i + 1), sc), ze));
  }
  v_store32<BITS, WIDE>(A, dst, out_tok, q, v, lane < 4);
}

template <int BITS, bool WIDE>
__device__ __forceinline__ void v_build_run(const BuildArgs& A, int t, int64_t run, int bh) {
  const BuildDst& dst = A.dst[t];
  const int lane = threadIdx.x & 31;
  const int64_t j0 = run * 32;
  const int ntok = static_cast<int>(dst.n - j0 < 32 ? dst.n - j0 : 32);
  int32_t enc = 0;
  if (lane < ntok) {
    enc = dst.plan[j0 + lane];
    if (bh == 0 && dst.ids_out) dst.ids_out[j0 + lane] = dst.ids[j0 + lane];
  }
  const int32_t enc0 = __shfl_sync(0xffffffffu, enc, 0);
  if (!WIDE || ntok < 32 || !__all_sync(0xffffffffu, enc == enc0 + lane) || !A.wide) {
    for (int i = 0; i < ntok; ++i) v_one_token<BITS, WIDE>(A, t, __shfl_sync(0xffffffffu, enc, i), j0 + i, bh);
    return;
  }
  const int src = (enc0 >> 28) - 1;
  const int64_t pos = enc0 & 0x0FFFFFFF, out_tok = static_cast<int64_t>(bh) * dst.n + j0;
  if (src == t) {
    const int64_t tok = static_cast<int64_t>(bh) * A.n[t] + pos;
    const uint4* in = reinterpret_cast<const uint4*>(A.data[t]) + tok * BITS + lane;
    uint4* out = reinterpret_cast<uint4*>(dst.data) + out_tok * BITS + lane;
    constexpr int N = BITS < 8 ? BITS : 8;
#pragma unroll
    for (int k = 0; k < BITS; k += N) {
      uint4 v[N];
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = in[(k + i) * 32];
#pragma unroll
      for (int i = 0; i < N; ++i) out[(k + i) * 32] = v[i];
    }
    if constexpr (BITS < 16) {  // 32 tokens x 1, 2 or 4 groups: 2, 4 or 8 bytes per lane
      const int ng = D >> A.gshift;
      const __half *s = A.scale[t] + tok * ng, *z = A.zero[t] + tok * ng;
      __half *so = dst.scale + out_tok * ng, *zo = dst.zero + out_tok * ng;
      if (ng == 4) {
        reinterpret_cast<uint2*>(so)[lane] = reinterpret_cast<const uint2*>(s)[lane];
        reinterpret_cast<uint2*>(zo)[lane] = reinterpret_cast<const uint2*>(z)[lane];
      } else if (ng == 2) {
        reinterpret_cast<uint32_t*>(so)[lane] = reinterpret_cast<const uint32_t*>(s)[lane];
        reinterpret_cast<uint32_t*>(zo)[lane] = reinterpret_cast<const uint32_t*>(z)[lane];
      } else {
        so[lane] = s[lane];
        zo[lane] = z[lane];
      }
    }
    return;
  }
  if (src < 0) {
    const int b = bh / A.H, h = bh - b * A.H;
    v_arrive<BITS, 16>(A, dst, reinterpret_cast<const unsigned char*>(A.residual + b * A.res_b_stride + h * A.res_h_stride + pos * D), src,
                       0, out_tok);
    return;
  }
  const int64_t tok = static_cast<int64_t>(bh) * A.n[src] + pos;
  const int sb = 16 >> src;
  const unsigned char* rows = reinterpret_cast<const unsigned char*>(A.data[src]) + tok * (16 * sb);
  if (sb == 16) v_arrive<BITS, 16>(A, dst, rows, src, tok, out_tok);
  else if (BITS < 8 && sb == 8) v_arrive<BITS, 8>(A, dst, rows, src, tok, out_tok);
  else if (BITS < 4 && sb == 4) v_arrive<BITS, 4>(A, dst, rows, src, tok, out_tok);
  else if (BITS < 2 && sb == 2) v_arrive<BITS, 2>(A, dst, rows, src, tok, out_tok);
  else
    for (int i = 0; i < 32; ++i) v_one_token<BITS, WIDE>(A, t, enc0 + i, j0 + i, bh);  // (not to wider tiers; all the same)
}

constexpr int VB_WARPS = BUILD_THREADS / 32;
template <bool WIDE>
__global__ void __launch_bounds__(BUILD_THREADS, 4) flush_build_v_kernel(const __grid_constant__ BuildArgs A) {
  const int x = A.tiles - 1 - static_cast<int>(blockIdx.x), bh = blockIdx.y;  // from the back, as above
  if (x < 0) {
    copy_rest(A, bh);
    return;
  }
  const int t = x >= A.dst[4].tile0 ? 4 : x >= A.dst[3].tile0 ? 3 : x >= A.dst[2].tile0 ? 2 : x >= A.dst[1].tile0 ? 1 : 0;
  const int64_t run = static_cast<int64_t>(x - A.dst[t].tile0) * VB_WARPS + (threadIdx.x >> 5);
  if (run * 32 >= A.dst[t].n) return;
  if (t == 4) v_build_run<1, WIDE>(A, 4, run, bh);
  else if (t == 3) v_build_run<2, WIDE>(A, 3, run, bh);
  else if (t == 2) v_build_run<4, WIDE>(A, 2, run, bh);
  else if (t == 1) v_build_run<8, WIDE>(A, 1, run, bh);
  else v_build_run<16, WIDE>(A, 0, run, bh);
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
static int fill_build_args(BuildArgs& A, bool v_side, const hqkv_flush_src_t* src, int B, int H, int Dd, int group, const char* who) {
  HQKV_REQUIRE(src != nullptr, "%s: null source descriptor", who);
  HQKV_REQUIRE(Dd == D, "%s: head dim must be 128", who);
  HQKV_REQUIRE(B > 0 && H > 0 && static_cast<int64_t>(B) * H <= 65535, "%s: bad B/H", who);
  HQKV_REQUIRE(valid_group(group), "%s: group must be 32, 64 or 128", who);
  HQKV_REQUIRE(src->low_codec == HQKV_CODEC_UNIFORM || src->low_codec == HQKV_CODEC_NORMAL, "%s: unknown low_codec %d",
               who, src->low_codec);
  memset(&A, 0, sizeof(A));
  A.tiers_wide = 1;
  A.wide = aligned(src->residual, 16) && src->residual_b_stride % 8 == 0 && src->residual_h_stride % 8 == 0;
  for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
    A.data[t] = src->data[t];
    A.scale[t] = static_cast<const __half*>(src->scale[t]);
    A.zero[t] = static_cast<const __half*>(src->zero[t]);
    A.n[t] = src->n[t];
    if (src->n[t] <= 0) continue;
    // (a K tier's scales are those of whole groups; the fp16 tier has none, and may hold any number of tokens)
    HQKV_REQUIRE(v_side || t == 0 || src->n[t] % group == 0, "%s: tier %d holds %d tokens, not a multiple of the group %d", who, t,
                 src->n[t], group);
    A.tiers_wide &= aligned(src->data[t], 16) && aligned(src->scale[t], 8) && aligned(src->zero[t], 8) && (v_side || src->n[t] % 32 == 0);
  }
  A.residual = static_cast<const __half*>(src->residual);
  A.res_b_stride = src->residual_b_stride;
  A.res_h_stride = src->residual_h_stride;
  A.H = H;
  A.normal_low = src->low_codec == HQKV_CODEC_NORMAL ? 1 : 0;
  while ((32 << (A.gshift)) < group) ++A.gshift;
  A.gshift += 5;
  return HQKV_OK;
}
static int add_dst(BuildArgs& A, bool v_side, int t, int group, const int32_t* plan, int64_t n, void* data, void* scale, void* zero,
                   const char* who) {
  HQKV_REQUIRE(n >= 0, "%s: negative n_dst", who);
  if (n > 0) {
    HQKV_REQUIRE(plan && data, "%s: null pointer", who);
    HQKV_REQUIRE(t == 0 || (scale && zero), "%s: null scale/zero output", who);
    HQKV_REQUIRE(v_side || n % group == 0, "%s: n_dst (%lld) is not a multiple of the group %d", who, (long long)n, group);
  }
  A.tiers_wide &= n == 0 || (aligned(data, 16) && aligned(scale, 8) && aligned(zero, 8));
  BuildDst& d = A.dst[t];
  d.plan = plan;
  d.n = n;
  d.data = data;
  d.scale = static_cast<__half*>(scale);
  d.zero = static_cast<__half*>(zero);
  return HQKV_OK;
}
static int launch_build(BuildArgs& A, bool v_side, int B, int H, const char* who, void* stream) {
  static constexpr int k_tokens[HQKV_NUM_TIERS] = {KBuild<16>::TOKENS, KBuild<8>::TOKENS, KBuild<4>::TOKENS, KBuild<2>::TOKENS, KBuild<1>::TOKENS};
  int64_t tiles = 0;
  for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
    A.dst[t].tile0 = static_cast<int>(tiles);
    tiles += ceil_div(A.dst[t].n, v_side ? 32 * VB_WARPS : k_tokens[t]);
  }
  A.tiles = static_cast<int>(tiles);
  const dim3 grid(static_cast<unsigned>(tiles + (A.rest_n > 0 ? 1 : 0)), B * H);
  if (grid.x == 0) return HQKV_OK;
  const auto kernel = v_side ? (A.tiers_wide ? flush_build_v_kernel<true> : flush_build_v_kernel<false>)
                             : (A.tiers_wide ? flush_build_k_kernel<true> : flush_build_k_kernel<false>);
  kernel<<<grid, BUILD_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(A);
  HQKV_LAUNCH_CHECK(who);
  return HQKV_OK;
}
static int build_one(bool v_side, const hqkv_flush_src_t* src_host, int B, int H, int Dd, int group, int dst_tier,
                     const int32_t* plan_src_row, int64_t n_dst, void* out_data, void* out_scale, void* out_zero, const char* who,
                     void* stream) {
  BuildArgs A;
  int rc = fill_build_args(A, v_side, src_host, B, H, Dd, group, who);
  if (rc) return rc;
  HQKV_REQUIRE(dst_tier >= 0 && dst_tier < HQKV_NUM_TIERS, "%s: dst_tier out of range", who);
  rc = add_dst(A, v_side, dst_tier, group, plan_src_row, n_dst, out_data, out_scale, out_zero, who);
  return rc ? rc : launch_build(A, v_side, B, H, who, stream);
}

}  // namespace hqkv

using namespace hqkv;

extern "C" int hqkv_flush_build_k(const hqkv_flush_src_t* src_host, int B, int H, int Dd, int group, int dst_tier,
                                  const int32_t* plan_src_row, int64_t n_dst, void* out_data, void* out_scale,
                                  void* out_zero, void* stream) {
  return build_one(false, src_host, B, H, Dd, group, dst_tier, plan_src_row, n_dst, out_data, out_scale, out_zero, "flush_build_k", stream);
}
extern "C" int hqkv_flush_build_v(const hqkv_flush_src_t* src_host, int B, int H, int Dd, int group, int dst_tier,
                                  const int32_t* plan_src_row, int64_t n_dst, void* out_data, void* out_scale,
                                  void* out_zero, void* stream) {
  return build_one(true, src_host, B, H, Dd, group, dst_tier, plan_src_row, n_dst, out_data, out_scale, out_zero, "flush_build_v", stream);
}

extern "C" int hqkv_flush_build(int v_side, const hqkv_flush_src_t* src_host, int B, int H, int Dd, int group,
                                const int32_t* plan_src, const int64_t* plan_ids, int64_t total, const int32_t* counts_host,
                                void* const* out_data_host, void* const* out_scale_host, void* const* out_zero_host,
                                int64_t* const* out_ids_host, int64_t compress, int64_t rest, void* rest_out, void* stream) {
  HQKV_REQUIRE(plan_src && plan_ids && counts_host && out_data_host && out_scale_host && out_zero_host && out_ids_host,
               "flush_build: null pointer");
  HQKV_REQUIRE(rest >= 0 && (rest == 0 || rest_out), "flush_build: bad residual output");
  BuildArgs A;
  int rc = fill_build_args(A, v_side != 0, src_host, B, H, Dd, group, "flush_build");
  if (rc) return rc;
  for (int t = 0; t < HQKV_NUM_TIERS; ++t) {
    HQKV_REQUIRE(counts_host[t] >= 0 && counts_host[t] <= total, "flush_build: bad count of tier %d", t);
    rc = add_dst(A, v_side != 0, t, group, plan_src + t * total, counts_host[t], out_data_host[t], out_scale_host[t], out_zero_host[t],
                 "flush_build");
    if (rc) return rc;
    HQKV_REQUIRE(counts_host[t] == 0 || out_ids_host[t], "flush_build: null id output");
    A.dst[t].ids = plan_ids + t * total;
    A.dst[t].ids_out = out_ids_host[t];
  }
  A.rest = A.residual + compress * D;
  A.rest_out = static_cast<__half*>(rest_out);
  A.rest_n = rest * D;
  A.wide &= aligned(rest_out, 16);
  return launch_build(A, v_side != 0, B, H, "flush_build", stream);
}
