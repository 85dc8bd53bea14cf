// Group quantise + bit-pack, unpack + dequantise (sm_100a).
//
// HBM-bound elementwise work: every element is read once and every packed word written once.
// Algorithmic bytes per element: 2 in, bits/8 + 4/group out.
#include <stdarg.h>
#include <stdio.h>

#include "common.cuh"

namespace hqkv {

// ------------------------------------------------------------------------------------------------
// error plumbing shared by all translation units
// ------------------------------------------------------------------------------------------------
static thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int check_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return 0;
  return fail(HQKV_E_CUDA, "%s failed: %s", what, cudaGetErrorString(e));
}

// ------------------------------------------------------------------------------------------------
// Row path: groups are contiguous in memory (t_stride == 1).  One thread owns 32 consecutive elements, GROUP/32 adjacent
// lanes own one group: what is done once per group (two divisions) is shared by 32 elements, and a thread's words are
// one store.  Bound by HBM at large sizes: 131072 x 8 rows of 128 at 4 bits in 50 us (352 MB; 106 us with a lane per 8
// elements, six instructions per quotient pair and a shuffle reduction per group, which the issue slots bounded).
// ------------------------------------------------------------------------------------------------
template <int BYTES>  // BYTES consecutive bytes, 16 at a time or, where the address allows it, 32
__device__ __forceinline__ void load_run(void* dst, const void* src, bool by32) {
  uint32_t* d = static_cast<uint32_t*>(dst);
  const char* p = static_cast<const char*>(src);
  if (by32) {
#pragma unroll
    for (int i = 0; i < BYTES / 32; ++i)
      asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(d[8 * i]), "=r"(d[8 * i + 1]), "=r"(d[8 * i + 2]), "=r"(d[8 * i + 3]), "=r"(d[8 * i + 4]),
                     "=r"(d[8 * i + 5]), "=r"(d[8 * i + 6]), "=r"(d[8 * i + 7])
                   : "l"(p + 32 * i));
  } else {
#pragma unroll
    for (int i = 0; i < BYTES / 16; ++i) {
      const uint4 v = *reinterpret_cast<const uint4*>(p + 16 * i);
      d[4 * i] = v.x, d[4 * i + 1] = v.y, d[4 * i + 2] = v.z, d[4 * i + 3] = v.w;
    }
  }
}

template <int BITS, int GROUP>
__global__ void __launch_bounds__(256) quantize_rows_kernel(const __half* __restrict__ x, int64_t n_units, int64_t T,
                                                            int64_t inner, int64_t outer_stride, int64_t inner_stride,
                                                            int align, bool vec_out, uint32_t* __restrict__ code,
                                                            __half* __restrict__ scale, __half* __restrict__ mn_out) {
  constexpr int LPG = GROUP / 32;  // lanes per group
  const float levels = static_cast<float>((1 << BITS) - 1);
  const int64_t unit = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t u = unit < n_units ? unit : n_units - 1;  // every lane takes part in the shuffles
  const __half* src = x + u * 32;
  if (inner_stride != T || outer_stride != inner * T) {  // rows that do not follow one another
    const int64_t units_per_row = T / 32, row = u / units_per_row;
    src = x + (row / inner) * outer_stride + (row % inner) * inner_stride + (u - row * units_per_row) * 32;
  }
  __half2 v[16];
  if (align >= 16) {
    load_run<64>(v, src, align >= 32);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __halves2half2(src[2 * i], src[2 * i + 1]);
  }
  // min / max of the group on half2 pairs (NaN propagates, as in torch.min / torch.max)
  __half2 lo2 = v[0], hi2 = v[0];
#pragma unroll
  for (int i = 1; i < 16; ++i) {
    lo2 = __hmin2_nan(lo2, v[i]);
    hi2 = __hmax2_nan(hi2, v[i]);
  }
#pragma unroll
  for (int off = 1; off < LPG; off <<= 1) {
    lo2 = __hmin2_nan(lo2, __shfl_xor_sync(0xffffffffu, lo2, off));
    hi2 = __hmax2_nan(hi2, __shfl_xor_sync(0xffffffffu, hi2, off));
  }
  const __half lo = __low2half(__hmin2_nan(lo2, __lowhigh2highlow(lo2))), hi = __low2half(__hmax2_nan(hi2, __lowhigh2highlow(hi2)));
  const __half sc = quant_scale(lo, hi, levels);
  uint32_t word[BITS];
  quant_row32<BITS, false>(v, quant_pair(lo, sc), word);
  if (unit >= n_units) return;
  uint32_t* dst = code + u * BITS;
  if (vec_out) {
    if constexpr (BITS >= 4) {
#pragma unroll
      for (int i = 0; i < BITS / 4; ++i)
        reinterpret_cast<uint4*>(dst)[i] = make_uint4(word[4 * i], word[4 * i + 1], word[4 * i + 2], word[4 * i + 3]);
    } else if constexpr (BITS == 2) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(word[0], word[1]);
    } else {
      *dst = word[0];
    }
  } else {
#pragma unroll
    for (int i = 0; i < BITS; ++i) dst[i] = word[i];
  }
  if (u % LPG == 0) {
    scale[u / LPG] = sc;
    mn_out[u / LPG] = lo;
  }
}

// ------------------------------------------------------------------------------------------------
// Column path (K): source is token-major [outer, T, inner] and is quantised as [outer*inner, T] with
// groups of GROUP tokens per channel — the transposed view, never materialised.  One thread owns
// one channel; a warp reads 64 contiguous bytes per token.  Two passes over the group (the second
// hits L1/L2): min/max, then codes.
// ------------------------------------------------------------------------------------------------
template <int BITS>
__global__ void __launch_bounds__(128) quantize_cols_kernel(const __half* __restrict__ x, int64_t inner, int64_t T,
                                                            int64_t outer_stride, int64_t t_stride, int group,
                                                            uint32_t* __restrict__ code, __half* __restrict__ scale,
                                                            __half* __restrict__ mn_out) {
  constexpr int FPI = 32 / BITS;
  const float levels = static_cast<float>((1 << BITS) - 1);
  const int64_t d = static_cast<int64_t>(blockIdx.y) * blockDim.x + threadIdx.x;
  if (d >= inner) return;
  const int64_t o = blockIdx.z;
  const int64_t gi = blockIdx.x;  // group index along T
  const __half* src = x + o * outer_stride + d + gi * group * t_stride;
  __half lo = src[0], hi = src[0];
  for (int t = 1; t < group; ++t) {
    const __half v = src[t * t_stride];
    lo = h_min(lo, v);
    hi = h_max(hi, v);
  }
  const __half sc = quant_scale(lo, hi, levels);
  const QuantGroup qg = quant_group(lo, sc, levels);
  const int64_t row = o * inner + d;
  const int64_t W = T / FPI;
  uint32_t* dst = code + row * W + gi * (group / FPI);
  for (int w = 0; w < group / FPI; ++w) {
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < FPI; ++i) word |= quant_code_fast(src[(w * FPI + i) * t_stride], qg) << (i * BITS);
    dst[w] = word;
  }
  const int64_t G = T / group;
  scale[row * G + gi] = sc;
  mn_out[row * G + gi] = lo;
}

// The usual case of an even, 4-byte aligned channel count: a tile of 128 tokens x 128 channels per CTA, 32 tokens of two
// adjacent channels per thread, kept in registers (one pass over the source, 128 contiguous bytes per token and warp).
// Groups of 64 and 128 tokens exchange their minima and maxima through shared memory.  The words and the scale / zero
// halfs of the tile meet in shared memory too, and each channel's run (16 x BITS bytes of codes, up to 8 of scales or minima)
// is stored by consecutive threads, at addresses that advance by constants.  Four small CTAs per SM rather than fewer large
// ones: a CTA loads, computes and stores in turn, and only other CTAs fill the gaps.  Issue slots are what it runs short of
// (68 % used with 833 instructions per warp and tile), so rows of TS = 128 elements, a cache's, have their token offsets in
// the load instructions (TS = 0: computed for any distance), the output loops carry no divisions and 64-bit products, and a
// quotient is one multiplication.  131072 x 8 heads at 8 / 4 / 2 / 1 bits: 66 / 60 / 58 / 60 us (80 / 74 / 74 / 74 before;
// HBM allows 64 / 53 / 48 / 46); 32768 x 8 at 4 bits 18.7 (23.4).  Loads of the next tile by cp.async in a persistent CTA
// took 89 us at 4 bits: the loads were not what it waited for.  64 registers a thread, nothing spilled.
constexpr int QT_SUBS = 4;       // runs of 32 tokens per tile
constexpr int QT_CH = 128;       // channels per tile
template <int BITS, int TS>
__global__ void __launch_bounds__(256, 4) quantize_cols_tile_kernel(const __half* __restrict__ x, int64_t inner, int64_t T,
                                                                    int64_t outer_stride, int64_t t_stride, int gshift,
                                                                    int vec_out, uint32_t* __restrict__ code,
                                                                    __half* __restrict__ scale, __half* __restrict__ mn_out) {
  // words of a staged channel row: 16-byte steps, and the rows of neighbouring lanes (every other channel: even channels
  // are staged before odd ones) start in different banks
  constexpr int ROW = QT_SUBS * BITS + 4;
  __shared__ __align__(16) uint32_t s_words[QT_CH * ROW];
  __shared__ __half2 s_lo[256], s_hi[256];
  __shared__ __align__(4) __half s_group[2][QT_SUBS][QT_CH];  // scales and minima: [group of the tile][channel]
  const float levels = static_cast<float>((1 << BITS) - 1);
  const int tid = threadIdx.x, cp = tid & 63, sub = tid >> 6, gs = gshift - 5;  // 2^gs runs per group
  const int64_t subs = T / 32, first = static_cast<int64_t>(blockIdx.x) * QT_SUBS;
  const int nsub = static_cast<int>(subs - first < QT_SUBS ? subs - first : QT_SUBS);
  const int64_t d0 = static_cast<int64_t>(blockIdx.y) * QT_CH;
  const int nch = static_cast<int>(inner - d0 < QT_CH ? inner - d0 : QT_CH);  // even: the host checks inner % 2 == 0
  const int64_t o = blockIdx.z;
  const int ch = 2 * cp;
  const bool live = ch < nch && sub < nsub;
  __half2 v[32], lo, hi;
  if (live) {
    const __half* src = x + o * outer_stride + d0 + ch + (first + sub) * 32 * t_stride;
#pragma unroll
    for (int t = 0; t < 32; ++t) v[t] = *reinterpret_cast<const __half2*>(src + t * (TS ? TS : t_stride));
    lo = hi = v[0];
#pragma unroll
    for (int t = 1; t < 32; ++t) {
      lo = __hmin2_nan(lo, v[t]);
      hi = __hmax2_nan(hi, v[t]);
    }
  }
  if (gs > 0) {
    if (live) {
      s_lo[tid] = lo;
      s_hi[tid] = hi;
    }
    __syncthreads();
    if (live) {
      for (int k = 1; k < (1 << gs); ++k) {  // a group's runs are all in the tile: T is a multiple of the group
        lo = __hmin2_nan(lo, s_lo[(sub ^ k) * 64 + cp]);
        hi = __hmax2_nan(hi, s_hi[(sub ^ k) * 64 + cp]);
      }
    }
  }
  if (live) {
    const __half sc0 = quant_scale(__low2half(lo), __low2half(hi), levels);
    const __half sc1 = quant_scale(__high2half(lo), __high2half(hi), levels);
    uint32_t w0[BITS], w1[BITS];
    quant_cols32<BITS, false>(v, quant_pair(__low2half(lo), sc0, __high2half(lo), sc1), w0, w1);
    uint32_t *r0 = s_words + cp * ROW + sub * BITS, *r1 = r0 + 64 * ROW;
    if constexpr (BITS >= 4) {
#pragma unroll
      for (int i = 0; i < BITS / 4; ++i) {
        reinterpret_cast<uint4*>(r0)[i] = make_uint4(w0[4 * i], w0[4 * i + 1], w0[4 * i + 2], w0[4 * i + 3]);
        reinterpret_cast<uint4*>(r1)[i] = make_uint4(w1[4 * i], w1[4 * i + 1], w1[4 * i + 2], w1[4 * i + 3]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < BITS; ++i) {
        r0[i] = w0[i];
        r1[i] = w1[i];
      }
    }
    if ((sub & ((1 << gs) - 1)) == 0) {
      *reinterpret_cast<__half2*>(&s_group[0][sub >> gs][ch]) = __halves2half2(sc0, sc1);
      *reinterpret_cast<__half2*>(&s_group[1][sub >> gs][ch]) = lo;
    }
  }
  __syncthreads();
  const int64_t row0 = o * inner + d0, W = subs * BITS, G = subs >> gs, g_first = first >> gs;
  auto staged = [&](int r) { return s_words + ((r & 1) * 64 + (r >> 1)) * ROW; };
  const int per = 2 - gs;  // log2(groups per tile)
  if ((vec_out & 1) && nsub == QT_SUBS) {
    // BITS lanes store a channel's codes, and a step takes 256 / BITS channels: addresses by constant steps
    const int r = tid / BITS, w = tid % BITS;
    uint4* dst = reinterpret_cast<uint4*>(code + (row0 + r) * W + first * BITS) + w;
    const uint4* src = reinterpret_cast<const uint4*>(staged(r)) + w;
#pragma unroll
    for (int k = 0; k < (BITS + 1) / 2; ++k)
      if (r + k * (256 / BITS) < nch) dst[k * (64 / BITS) * W] = src[k * (128 / BITS) * (ROW / 4)];
  } else {
    for (int i = tid; i < nch * QT_SUBS * BITS; i += 256) {
      const int r = i / (QT_SUBS * BITS), w = i % (QT_SUBS * BITS);
      if (w < nsub * BITS) code[(row0 + r) * W + first * BITS + w] = staged(r)[w];
    }
  }
  if ((vec_out & 2) && nsub == QT_SUBS) {
    // a thread stores a channel's scales or its minima
    const int c = tid & (QT_CH - 1), which = tid >> 7;
    if (c < nch) {
      __half* to = (which ? mn_out : scale) + (row0 + c) * G + g_first;
      const unsigned short* from = reinterpret_cast<const unsigned short*>(&s_group[which][0][c]);
      if (per == 2) *reinterpret_cast<uint2*>(to) = make_uint2(from[0] | from[QT_CH] << 16, from[2 * QT_CH] | from[3 * QT_CH] << 16);
      else if (per == 1) *reinterpret_cast<uint32_t*>(to) = from[0] | from[QT_CH] << 16;
      else *reinterpret_cast<unsigned short*>(to) = from[0];
    }
  } else {
    for (int i = tid; i < nch << per; i += 256) {
      const int r = i >> per, g = i & ((1 << per) - 1);
      if (g << gs >= nsub) continue;
      scale[(row0 + r) * G + g_first + g] = s_group[0][g][r];
      mn_out[(row0 + r) * G + g_first + g] = s_group[1][g][r];
    }
  }
}

template <int BITS>
static void launch_quant_cols(dim3 tiles, const __half* x, int64_t inner, int64_t T, int64_t outer_stride, int64_t t_stride, int gshift,
                              int vec_out, uint32_t* code, __half* scale, __half* mn, cudaStream_t st) {
  auto* f = t_stride == QT_CH ? quantize_cols_tile_kernel<BITS, QT_CH> : quantize_cols_tile_kernel<BITS, 0>;
  f<<<tiles, 256, 0, st>>>(x, inner, T, outer_stride, t_stride, gshift, vec_out, code, scale, mn);
}

// ------------------------------------------------------------------------------------------------
// unpack + two-rounding dequantise.  A thread writes 16 consecutive fp16 values (one 32-byte store where the address allows
// it: whole sectors, a warp's store is contiguous), DQ_UNITS times, all loads before the first store; pairs of
// elements in fp16 arithmetic, whose one rounding equals the two of "widen, operate, narrow".  Bound by HBM: 131072 x 8 rows
// of 128 at 4 bits in 52 us (80 with 8 values per thread, one load in flight, a 64-bit division and fp32 arithmetic).
// ------------------------------------------------------------------------------------------------
constexpr int DQ_UNITS = 2;
template <int BITS>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint32_t* __restrict__ code,
                                                         const __half* __restrict__ scale,
                                                         const __half* __restrict__ mn, int64_t n_units, int gshift,
                                                         bool vec_in, bool by32, __half* __restrict__ out) {
  constexpr int WORDS = BITS >= 2 ? BITS / 2 : 1;  // words of 16 codes (1 bit: half a word)
  const int64_t u0 = static_cast<int64_t>(blockIdx.x) * (256 * DQ_UNITS) + threadIdx.x;
  uint32_t w[DQ_UNITS][WORDS];
  __half sc[DQ_UNITS], z[DQ_UNITS];
#pragma unroll
  for (int k = 0; k < DQ_UNITS; ++k) {
    const int64_t u = u0 + 256 * k;
    if (u >= n_units) break;
    const uint32_t* src = code + u * BITS / 2;
    if (WORDS > 1 && vec_in) {
      if constexpr (WORDS == 4) {
        const uint4 c = *reinterpret_cast<const uint4*>(src);
        w[k][0] = c.x, w[k][1] = c.y, w[k][2] = c.z, w[k][3] = c.w;
      } else if constexpr (WORDS == 2) {
        const uint2 c = *reinterpret_cast<const uint2*>(src);
        w[k][0] = c.x, w[k][1] = c.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < WORDS; ++i) w[k][i] = src[i];
      if (BITS == 1) w[k][0] >>= 16 * (u & 1);
    }
    const int64_t g = (u * 16) >> gshift;
    sc[k] = scale[g];
    z[k] = mn[g];
  }
#pragma unroll
  for (int k = 0; k < DQ_UNITS; ++k) {
    const int64_t u = u0 + 256 * k;
    if (u >= n_units) break;
    const __half2 s2 = __half2half2(sc[k]), z2 = __half2half2(z[k]);
    auto value = [&](uint32_t c) {  // codes in bits [0, 10) and [16, 26) over a biased exponent
      const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&c), __float2half2_rn(1024.f));
      const __half2 r = __hadd2_rn(__hmul2_rn(h, s2), z2);
      return *reinterpret_cast<const uint32_t*>(&r);
    };
    uint32_t v[8];
    if constexpr (BITS == 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = value(__byte_perm(w[k][i / 2], 0x64646464u, i % 2 ? 0x4342 : 0x4140));
    } else {
      // codes i and i + HALF meet in a pair, and are put beside their neighbours at the end
      constexpr int HALF = 16 / BITS, PER = BITS == 4 ? 8 : 16;  // codes in half a word (of 2 and 4 bits) and per run
      const uint32_t m = ((1u << BITS) - 1) * 0x00010001u;
#pragma unroll
      for (int r = 0; r < 16 / PER; ++r) {
        constexpr int H = BITS == 1 ? 8 : HALF;
        const uint32_t x = BITS == 1 ? (w[k][0] & 0xFFu) | (w[k][0] & 0xFF00u) << 8 : w[k][r];
        uint32_t p[H];
#pragma unroll
        for (int i = 0; i < H; ++i) p[i] = value(((x >> (i * BITS)) & m) | 0x64006400u);
#pragma unroll
        for (int i = 0; i < H / 2; ++i) {
          v[r * PER / 2 + i] = __byte_perm(p[2 * i], p[2 * i + 1], 0x5410);
          v[r * PER / 2 + H / 2 + i] = __byte_perm(p[2 * i], p[2 * i + 1], 0x7632);
        }
      }
    }
    __half* dst = out + u * 16;
    if (by32) {
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                   "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                   : "memory");
    } else {
      reinterpret_cast<uint4*>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
      reinterpret_cast<uint4*>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
  }
}

template <int BITS>
__global__ void __launch_bounds__(256) pack_kernel(const int32_t* __restrict__ codes, int64_t n_words,
                                                   uint32_t* __restrict__ words) {
  constexpr int FPI = 32 / BITS;
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= n_words) return;
  uint32_t word = 0;
#pragma unroll
  for (int i = 0; i < FPI; ++i) word |= static_cast<uint32_t>(codes[w * FPI + i]) << (i * BITS);
  words[w] = word;
}

template <int BITS>
__global__ void __launch_bounds__(256) unpack_kernel(const uint32_t* __restrict__ words, int64_t n_words,
                                                     __half* __restrict__ out) {
  constexpr int FPI = 32 / BITS;
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= n_words) return;
  const uint32_t word = words[w];
#pragma unroll
  for (int i = 0; i < FPI; ++i) out[w * FPI + i] = __uint2half_rn((word >> (i * BITS)) & ((1u << BITS) - 1));
}

static int log2_group(int group) { return group == 32 ? 5 : group == 64 ? 6 : 7; }

template <int BITS>
static void launch_quant_rows(const __half* x, int64_t rows, int64_t T, int64_t inner, int64_t os, int64_t is, int group,
                              uint32_t* code, __half* scale, __half* mn, cudaStream_t st) {
  const int64_t units = rows * (T / 32);
  const unsigned blocks = static_cast<unsigned>(ceil_div(units, 256));
  int align = 2;
  if (aligned(x, 16) && os % 8 == 0 && is % 8 == 0) align = aligned(x, 32) && os % 16 == 0 && is % 16 == 0 ? 32 : 16;
  const bool vec_out = aligned(code, 16);
  switch (group) {
    case 32: quantize_rows_kernel<BITS, 32><<<blocks, 256, 0, st>>>(x, units, T, inner, os, is, align, vec_out, code, scale, mn); break;
    case 64: quantize_rows_kernel<BITS, 64><<<blocks, 256, 0, st>>>(x, units, T, inner, os, is, align, vec_out, code, scale, mn); break;
    default: quantize_rows_kernel<BITS, 128><<<blocks, 256, 0, st>>>(x, units, T, inner, os, is, align, vec_out, code, scale, mn); break;
  }
}

// ------------------------------------------------------------------------------------------------
// Gaussian-codebook codec at 1 bit (the low tier of 'high_uniform_group_low_normal_group')
// ------------------------------------------------------------------------------------------------
// One thread per group, two passes over its `group` elements.  std and mean are the unbiased
// torch.std_mean of the group computed in fp64 (the sum of fp16 values is exact there) and rounded ONCE
// to fp16, which is what torch returns for fp16 input; then (x - mean) / std in fp16 with a rounding after
// each step, code = 1 where the quotient is > 0 (decision bounds [0, inf]; NaN gives 0).
__global__ void __launch_bounds__(128) normal1_quantize_kernel(const __half* __restrict__ x, int64_t rows, int64_t T,
                                                               int64_t inner, int64_t outer_stride, int64_t inner_stride,
                                                               int64_t t_stride, int group, uint32_t* __restrict__ code,
                                                               __half* __restrict__ std_out, __half* __restrict__ mean_out) {
  const int64_t G = T / group;
  const int64_t gid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (gid >= rows * G) return;
  const int64_t row = gid / G, gi = gid - row * G;
  const __half* src = x + (row / inner) * outer_stride + (row % inner) * inner_stride + gi * group * t_stride;
  double sum = 0.0;
  for (int t = 0; t < group; ++t) sum += static_cast<double>(__half2float(src[t * t_stride]));
  const double mean64 = sum / group;
  double ss = 0.0;
  for (int t = 0; t < group; ++t) {
    const double d = static_cast<double>(__half2float(src[t * t_stride])) - mean64;
    ss += d * d;
  }
  const __half mean = __double2half(mean64);
  const __half sd = normal1_sd(ss, group), bound = normal1_bound(sd);
  uint32_t* dst = code + (row * T + gi * group) / 32;
  for (int w = 0; w < group / 32; ++w) {
    uint32_t word = 0;
    for (int i = 0; i < 32; ++i) {
      word |= normal1_code(src[(w * 32 + i) * t_stride], mean, bound) << i;
    }
    dst[w] = word;
  }
  std_out[gid] = sd;
  mean_out[gid] = mean;
}

// x = half(half(center[code] * std) + mean), center = +-fp16(0.67448974); one thread per packed word
__global__ void __launch_bounds__(256) normal1_dequantize_kernel(const uint32_t* __restrict__ code,
                                                                 const __half* __restrict__ sd,
                                                                 const __half* __restrict__ mean, int64_t n_words,
                                                                 int group, __half* __restrict__ out) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= n_words) return;
  const uint32_t word = code[w];
  const int64_t gi = (w * 32) / group;
  const __half s = sd[gi], m = mean[gi];
  const __half cpos = __float2half_rn(HQKV_NORMAL1_CENTER), cneg = __float2half_rn(-HQKV_NORMAL1_CENTER);
  __half* dst = out + w * 32;
  for (int i = 0; i < 32; ++i) dst[i] = h_add(h_mul((word >> i) & 1u ? cpos : cneg, s), m);
}

}  // namespace hqkv

using namespace hqkv;

extern "C" const char* hqkv_last_error(void) { return g_err; }
extern "C" int hqkv_version(void) { return 100; }
#ifndef HQKV_BUILD_ID
#define HQKV_BUILD_ID "unstamped"
#endif
// the marker lets a build script read the stamp out of the file without loading the library
static const char g_build_stamp[] = "HQKV_BUILD_ID=" HQKV_BUILD_ID;
extern "C" const char* hqkv_build_id(void) { return g_build_stamp + 14; }

extern "C" int hqkv_quantize_pack(const void* x, int64_t rows, int64_t T, int64_t inner, int64_t outer_stride,
                                  int64_t inner_stride, int64_t t_stride, int group, int bits, void* code,
                                  void* scale, void* mn, void* stream) {
  HQKV_REQUIRE(bits == 8 || bits == 4 || bits == 2 || bits == 1, "quantize_pack: bits must be 8, 4, 2 or 1 (got %d)", bits);
  HQKV_REQUIRE(valid_group(group), "quantize_pack: group must be 32, 64 or 128 (got %d)", group);
  HQKV_REQUIRE(rows >= 0 && T >= 0 && inner > 0, "quantize_pack: negative size");
  HQKV_REQUIRE(T % group == 0, "quantize_pack: T (%lld) is not a multiple of the group size %d", (long long)T, group);
  HQKV_REQUIRE(rows % inner == 0, "quantize_pack: rows (%lld) is not a multiple of inner (%lld)", (long long)rows,
               (long long)inner);
  if (rows == 0 || T == 0) return HQKV_OK;
  HQKV_REQUIRE(x && code && scale && mn, "quantize_pack: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* xs = static_cast<const __half*>(x);
  uint32_t* c = static_cast<uint32_t*>(code);
  __half* s = static_cast<__half*>(scale);
  __half* m = static_cast<__half*>(mn);
  if (t_stride == 1) {
    switch (bits) {
      case 8: launch_quant_rows<8>(xs, rows, T, inner, outer_stride, inner_stride, group, c, s, m, st); break;
      case 4: launch_quant_rows<4>(xs, rows, T, inner, outer_stride, inner_stride, group, c, s, m, st); break;
      case 2: launch_quant_rows<2>(xs, rows, T, inner, outer_stride, inner_stride, group, c, s, m, st); break;
      default: launch_quant_rows<1>(xs, rows, T, inner, outer_stride, inner_stride, group, c, s, m, st); break;
    }
  } else if (inner_stride == 1) {
    const int64_t outer = rows / inner;
    HQKV_REQUIRE(outer <= 65535 && ceil_div(inner, 128) <= 65535, "quantize_pack: too many rows for the column path");
    dim3 grid(static_cast<unsigned>(T / group), static_cast<unsigned>(ceil_div(inner, 128)),
              static_cast<unsigned>(outer));
    if (inner % 2 == 0 && aligned(x, 4) && outer_stride % 2 == 0 && t_stride % 2 == 0) {
      const dim3 tiles(static_cast<unsigned>(ceil_div(T, 32 * QT_SUBS)), grid.y, grid.z);
      // codes in pieces of 16 bytes; a tile's scales or minima of a channel (up to 8 bytes) in one
      const int vec_out = (aligned(code, 16) && T / 32 * bits % 4 == 0 ? 1 : 0) |
                          (T % (32 * QT_SUBS) == 0 && aligned(s, 8) && aligned(m, 8) ? 2 : 0);
      const int gshift = log2_group(group);
      switch (bits) {
        case 8: launch_quant_cols<8>(tiles, xs, inner, T, outer_stride, t_stride, gshift, vec_out, c, s, m, st); break;
        case 4: launch_quant_cols<4>(tiles, xs, inner, T, outer_stride, t_stride, gshift, vec_out, c, s, m, st); break;
        case 2: launch_quant_cols<2>(tiles, xs, inner, T, outer_stride, t_stride, gshift, vec_out, c, s, m, st); break;
        default: launch_quant_cols<1>(tiles, xs, inner, T, outer_stride, t_stride, gshift, vec_out, c, s, m, st); break;
      }
    } else
    switch (bits) {
      case 8: quantize_cols_kernel<8><<<grid, 128, 0, st>>>(xs, inner, T, outer_stride, t_stride, group, c, s, m); break;
      case 4: quantize_cols_kernel<4><<<grid, 128, 0, st>>>(xs, inner, T, outer_stride, t_stride, group, c, s, m); break;
      case 2: quantize_cols_kernel<2><<<grid, 128, 0, st>>>(xs, inner, T, outer_stride, t_stride, group, c, s, m); break;
      default: quantize_cols_kernel<1><<<grid, 128, 0, st>>>(xs, inner, T, outer_stride, t_stride, group, c, s, m); break;
    }
  } else {
    return fail(HQKV_E_INVALID, "quantize_pack: unsupported strides (need t_stride == 1 or inner_stride == 1)");
  }
  HQKV_LAUNCH_CHECK("quantize_pack");
  return HQKV_OK;
}

extern "C" int hqkv_dequantize_unpack(const void* code, const void* scale, const void* mn, int64_t rows, int64_t T,
                                      int group, int bits, void* out, void* stream) {
  HQKV_REQUIRE(bits == 8 || bits == 4 || bits == 2 || bits == 1, "dequantize_unpack: bits must be 8, 4, 2 or 1");
  HQKV_REQUIRE(valid_group(group), "dequantize_unpack: group must be 32, 64 or 128");
  HQKV_REQUIRE(rows >= 0 && T >= 0 && T % group == 0, "dequantize_unpack: T is not a multiple of the group size");
  if (rows == 0 || T == 0) return HQKV_OK;
  HQKV_REQUIRE(code && scale && mn && out, "dequantize_unpack: null pointer");
  HQKV_REQUIRE(aligned(out, 16), "dequantize_unpack: output must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t units = rows * T / 16;
  const unsigned blocks = static_cast<unsigned>(ceil_div(units, 256 * DQ_UNITS));
  const bool vec_in = aligned(code, 16), by32 = aligned(out, 32);
  const int gshift = log2_group(group);
  const uint32_t* c = static_cast<const uint32_t*>(code);
  const __half* s = static_cast<const __half*>(scale);
  const __half* m = static_cast<const __half*>(mn);
  __half* o = static_cast<__half*>(out);
  switch (bits) {
    case 8: dequantize_kernel<8><<<blocks, 256, 0, st>>>(c, s, m, units, gshift, vec_in, by32, o); break;
    case 4: dequantize_kernel<4><<<blocks, 256, 0, st>>>(c, s, m, units, gshift, vec_in, by32, o); break;
    case 2: dequantize_kernel<2><<<blocks, 256, 0, st>>>(c, s, m, units, gshift, vec_in, by32, o); break;
    default: dequantize_kernel<1><<<blocks, 256, 0, st>>>(c, s, m, units, gshift, vec_in, by32, o); break;
  }
  HQKV_LAUNCH_CHECK("dequantize_unpack");
  return HQKV_OK;
}

extern "C" int hqkv_pack(const void* codes_i32, int64_t rows, int64_t T, int bits, void* words, void* stream) {
  HQKV_REQUIRE(bits == 8 || bits == 4 || bits == 2 || bits == 1, "pack: bits must be 8, 4, 2 or 1");
  HQKV_REQUIRE(rows >= 0 && T >= 0 && T % (32 / bits) == 0, "pack: T is not a multiple of 32/bits");
  const int64_t n_words = rows * T / (32 / bits);
  if (n_words == 0) return HQKV_OK;
  HQKV_REQUIRE(codes_i32 && words, "pack: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned blocks = static_cast<unsigned>(ceil_div(n_words, 256));
  const int32_t* c = static_cast<const int32_t*>(codes_i32);
  uint32_t* w = static_cast<uint32_t*>(words);
  switch (bits) {
    case 8: pack_kernel<8><<<blocks, 256, 0, st>>>(c, n_words, w); break;
    case 4: pack_kernel<4><<<blocks, 256, 0, st>>>(c, n_words, w); break;
    case 2: pack_kernel<2><<<blocks, 256, 0, st>>>(c, n_words, w); break;
    default: pack_kernel<1><<<blocks, 256, 0, st>>>(c, n_words, w); break;
  }
  HQKV_LAUNCH_CHECK("pack");
  return HQKV_OK;
}

extern "C" int hqkv_unpack(const void* words, int64_t rows, int64_t W, int bits, void* out_f16, void* stream) {
  HQKV_REQUIRE(bits == 8 || bits == 4 || bits == 2 || bits == 1, "unpack: bits must be 8, 4, 2 or 1");
  HQKV_REQUIRE(rows >= 0 && W >= 0, "unpack: negative size");
  const int64_t n_words = rows * W;
  if (n_words == 0) return HQKV_OK;
  HQKV_REQUIRE(words && out_f16, "unpack: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned blocks = static_cast<unsigned>(ceil_div(n_words, 256));
  const uint32_t* w = static_cast<const uint32_t*>(words);
  __half* o = static_cast<__half*>(out_f16);
  switch (bits) {
    case 8: unpack_kernel<8><<<blocks, 256, 0, st>>>(w, n_words, o); break;
    case 4: unpack_kernel<4><<<blocks, 256, 0, st>>>(w, n_words, o); break;
    case 2: unpack_kernel<2><<<blocks, 256, 0, st>>>(w, n_words, o); break;
    default: unpack_kernel<1><<<blocks, 256, 0, st>>>(w, n_words, o); break;
  }
  HQKV_LAUNCH_CHECK("unpack");
  return HQKV_OK;
}

extern "C" int hqkv_normal1_quantize_pack(const void* x, int64_t rows, int64_t T, int64_t inner, int64_t outer_stride,
                                          int64_t inner_stride, int64_t t_stride, int group, void* code, void* std_out,
                                          void* mean_out, void* stream) {
  HQKV_REQUIRE(valid_group(group), "normal1_quantize_pack: group size must be 32, 64 or 128 (got %d)", group);
  HQKV_REQUIRE(rows >= 0 && T >= 0 && inner > 0, "normal1_quantize_pack: negative size");
  HQKV_REQUIRE(T % group == 0, "normal1_quantize_pack: T (%lld) is not a multiple of the group size %d", (long long)T, group);
  HQKV_REQUIRE(rows % inner == 0, "normal1_quantize_pack: rows is not a multiple of inner");
  if (rows == 0 || T == 0) return HQKV_OK;
  HQKV_REQUIRE(x && code && std_out && mean_out, "normal1_quantize_pack: null pointer");
  const int64_t groups = rows * (T / group);
  normal1_quantize_kernel<<<static_cast<unsigned>(ceil_div(groups, 128)), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __half*>(x), rows, T, inner, outer_stride, inner_stride, t_stride, group,
      static_cast<uint32_t*>(code), static_cast<__half*>(std_out), static_cast<__half*>(mean_out));
  HQKV_LAUNCH_CHECK("normal1_quantize_pack");
  return HQKV_OK;
}

extern "C" int hqkv_normal1_dequantize_unpack(const void* code, const void* std_in, const void* mean_in, int64_t rows,
                                              int64_t T, int group, void* out, void* stream) {
  HQKV_REQUIRE(valid_group(group), "normal1_dequantize_unpack: group size must be 32, 64 or 128 (got %d)", group);
  HQKV_REQUIRE(rows >= 0 && T >= 0 && T % group == 0, "normal1_dequantize_unpack: bad sizes");
  if (rows == 0 || T == 0) return HQKV_OK;
  HQKV_REQUIRE(code && std_in && mean_in && out, "normal1_dequantize_unpack: null pointer");
  const int64_t n_words = rows * T / 32;
  normal1_dequantize_kernel<<<static_cast<unsigned>(ceil_div(n_words, 256)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint32_t*>(code), static_cast<const __half*>(std_in), static_cast<const __half*>(mean_in),
      n_words, group, static_cast<__half*>(out));
  HQKV_LAUNCH_CHECK("normal1_dequantize_unpack");
  return HQKV_OK;
}
