// Shared host/device helpers of libhqkv (sm_100a).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "hqkv.h"

namespace hqkv {

// ---- host-side error reporting ---------------------------------------------------------------
int fail(int code, const char* fmt, ...);  // records the message for hqkv_last_error(), returns code
int check_cuda(cudaError_t e, const char* what);

#define HQKV_REQUIRE(cond, ...)                                \
  do {                                                         \
    if (!(cond)) return ::hqkv::fail(HQKV_E_INVALID, __VA_ARGS__); \
  } while (0)

#define HQKV_CUDA(call)                                        \
  do {                                                         \
    int rc_ = ::hqkv::check_cuda((call), #call);               \
    if (rc_) return rc_;                                       \
  } while (0)

#define HQKV_LAUNCH_CHECK(name) HQKV_CUDA((cudaGetLastError()))

// ---- bounds-check build (-DHQKV_CHECKS) --------------------------------------------------------
// Every index that comes out of a caller-supplied list (logical positions of the decode, token ids of the
// flush plan) is range-checked before it addresses memory; a violation is counted in a device counter of
// the translation unit and the access is skipped - no trap.  hqkv_check_failures() reports the sum.  The
// regular build compiles the checks away.  (The stand-in for compute-sanitizer's memcheck on small cases.)
#ifdef HQKV_CHECKS
#define HQKV_CHECKS_ENABLED 1
#define HQKV_DEFINE_CHECK_COUNTER static __device__ unsigned int g_check_failures = 0u;
#define HQKV_INDEX_OK(idx, bound) \
  ((static_cast<unsigned long long>(idx) < static_cast<unsigned long long>(bound)) ? true : (atomicAdd(&g_check_failures, 1u), false))
#else
#define HQKV_CHECKS_ENABLED 0
#define HQKV_DEFINE_CHECK_COUNTER
#define HQKV_INDEX_OK(idx, bound) true
#endif
unsigned decode_check_failures(bool reset);  // decode.cu
unsigned policy_check_failures(bool reset);  // policy.cu

static inline bool valid_group(int g) { return g == 32 || g == 64 || g == 128; }
static inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }
static inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// ---- fp16 arithmetic with one rounding per operation -----------------------------------------
// "One torch op on fp16 tensors": widen to fp32, operate, round to nearest-even fp16.  The
// intrinsics with explicit rounding keep the compiler from contracting separate operations
// into an FMA, which would drop an intermediate rounding.
__device__ __forceinline__ __half h_sub(__half a, __half b) {
  return __float2half_rn(__fsub_rn(__half2float(a), __half2float(b)));
}
__device__ __forceinline__ __half h_divf(__half a, float b) {
  return __float2half_rn(__fdiv_rn(__half2float(a), b));
}
__device__ __forceinline__ __half h_mul(__half a, __half b) {
  return __float2half_rn(__fmul_rn(__half2float(a), __half2float(b)));
}
__device__ __forceinline__ __half h_add(__half a, __half b) {
  return __float2half_rn(__fadd_rn(__half2float(a), __half2float(b)));
}

// Code of one element: clamp(half(half(x - mn) / scale), 0, levels) rounded half-to-even; a NaN quotient (constant
// group: scale == 0) gives code 0, as the float->int conversion on the GPU does for the reference.
// For many elements of one group: x - mn with the native fp16 subtract (one rounding
// of the exact difference equals the two roundings of "widen, subtract, narrow": fp32 carries 2*11 + 2
// bits).  The quotient by Markstein's sequence: r = RN(1/scale) once per group, q0 = RN(d*r),
// e = d - q0*scale (exact in one FMA), q1 = RN(q0 + e*r) is the correctly rounded fp32 quotient (the
// scale has an 11-bit significand, never the all-ones fp32 significand the theorem excludes), so
// half(q1) is the fp16 quotient; three FP32 instructions per element instead of a full IEEE divide.
// A NaN or infinite intermediate (scale 0 or inf) ends as code 0.
struct QuantGroup {
  __half mn;
  float scale, rcp, levels;
};
__device__ __forceinline__ QuantGroup quant_group(__half mn, __half scale, float levels) {
  QuantGroup g;
  g.mn = mn;
  g.scale = __half2float(scale);
  g.rcp = __frcp_rn(g.scale);
  g.levels = levels;
  return g;
}
__device__ __forceinline__ float quant_quotient(float d, const QuantGroup& g) {
  const float q0 = __fmul_rn(d, g.rcp);
  const float e = __fmaf_rn(-q0, g.scale, d);
  return __fmaf_rn(e, g.rcp, q0);
}
__device__ __forceinline__ uint32_t quant_code_fast(__half x, const QuantGroup& g) {
  float u = __half2float(__float2half_rn(quant_quotient(__half2float(__hsub(x, g.mn)), g)));
  u = fminf(fmaxf(u, 0.f), g.levels);  // fmaxf(NaN, 0) == 0
  return static_cast<uint32_t>(__float2int_rn(u));
}
// Codes of 32 values at a time.  Only half(d / scale) is wanted, and half(RN(d * RN(1 / scale))) is that for every pair of
// 11-bit significands and every exponent between a quotient of 1/8 and one of 256, ties included (all 12 million of them:
// tests/test_quantise_quotient.py); smaller ones have code 0 and larger ones the largest code either way.  One instruction
// for a pair of elements (f32x2); a group whose scale is 0, inf or NaN has all codes 0, by one mask for its words instead of a
// test per element.  Pairs are gathered into bytes and the bytes into words, four elements at a time.  NAN_IN: a NaN element may be in a
// group whose scale is a number (where minimum and maximum are taken element by element); its code is 0.
struct QuantPair {  // low half of a pair in one group, high half in another or the same
  __half2 mn;
  float2 rcp;
  uint32_t keep0, keep1;  // 0 where all codes of the group are 0
};
__device__ __forceinline__ QuantPair quant_pair(__half mn0, __half sc0, __half mn1, __half sc1) {
  QuantPair g;
  g.mn = __halves2half2(mn0, mn1);
  const float s0 = __half2float(sc0), s1 = __half2float(sc1);
  g.rcp = make_float2(__frcp_rn(s0), __frcp_rn(s1));
  g.keep0 = s0 > 0.f && s0 < __int_as_float(0x7F800000) ? 0xFFFFFFFFu : 0u;
  g.keep1 = s1 > 0.f && s1 < __int_as_float(0x7F800000) ? 0xFFFFFFFFu : 0u;
  return g;
}
__device__ __forceinline__ QuantPair quant_pair(__half mn, __half sc) { return quant_pair(mn, sc, mn, sc); }
// the codes of a pair in bytes 0 and 2 (bytes 1 and 3 are not 0)
template <int BITS, bool NAN_IN>
__device__ __forceinline__ uint32_t quant_pair_bytes(__half2 x, const QuantPair& g) {
  const float2 d = __half22float2(__hsub2(x, g.mn));
  float2 q;
  asm("{\n.reg .b64 d, r, q;\nmov.b64 d, {%2, %3};\nmov.b64 r, {%4, %5};\nmul.rn.f32x2 q, d, r;\nmov.b64 {%0, %1}, q;\n}"
      : "=f"(q.x), "=f"(q.y)
      : "f"(d.x), "f"(d.y), "f"(g.rcp.x), "f"(g.rcp.y));
  __half2 u = __floats2half2_rn(q.x, q.y);
  if (NAN_IN) u = __hmax2(u, __float2half2_rn(0.f));  // max(NaN, 0) == 0
  u = __hmin2(u, __float2half2_rn(static_cast<float>((1 << BITS) - 1)));
  u = __hadd2(u, __float2half2_rn(1024.f));  // 1024 + rint(u): fp16 has unit spacing there, ties to even
  return *reinterpret_cast<uint32_t*>(&u);
}
// BITS words from 32 codes in 8 registers of 4 bytes
template <int BITS>
__device__ __forceinline__ void pack_bytes(const uint32_t* q, uint32_t keep, uint32_t* word) {
#pragma unroll
  for (int w = 0; w < BITS; ++w) {
    if constexpr (BITS == 8) {
      word[w] = q[w] & keep;
    } else if constexpr (BITS == 4) {
      const uint32_t a = q[2 * w] | q[2 * w] >> 4, b = q[2 * w + 1] | q[2 * w + 1] >> 4;
      word[w] = __byte_perm(a, b, 0x6420) & keep;
    } else {
      uint32_t b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        b[i] = BITS == 2 ? __dp4a(q[4 * w + i], 0x40100401u, 0u)
                         : __dp4a(q[2 * i + 1], 0x80402010u, __dp4a(q[2 * i], 0x08040201u, 0u));
      word[w] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410) & keep;
    }
  }
}
// 32 values of one group, in order: BITS words
template <int BITS, bool NAN_IN>
__device__ __forceinline__ void quant_row32(const __half2 (&v)[16], const QuantPair& g, uint32_t* word) {
  uint32_t q[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] = __byte_perm(quant_pair_bytes<BITS, NAN_IN>(v[2 * i], g), quant_pair_bytes<BITS, NAN_IN>(v[2 * i + 1], g), 0x6420);
  pack_bytes<BITS>(q, g.keep0, word);
}
// 32 pairs, low halves of one group and high halves of another: BITS words of each
template <int BITS, bool NAN_IN>
__device__ __forceinline__ void quant_cols32(const __half2 (&v)[32], const QuantPair& g, uint32_t* word0, uint32_t* word1) {
  uint32_t q0[8], q1[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t a = __byte_perm(quant_pair_bytes<BITS, NAN_IN>(v[4 * i], g), quant_pair_bytes<BITS, NAN_IN>(v[4 * i + 1], g), 0x6240);
    const uint32_t b = __byte_perm(quant_pair_bytes<BITS, NAN_IN>(v[4 * i + 2], g), quant_pair_bytes<BITS, NAN_IN>(v[4 * i + 3], g), 0x6240);
    q0[i] = __byte_perm(a, b, 0x5410);
    q1[i] = __byte_perm(a, b, 0x7632);
  }
  pack_bytes<BITS>(q0, g.keep0, word0);
  pack_bytes<BITS>(q1, g.keep1, word1);
}

// scale = half(half(mx - mn) / levels)
__device__ __forceinline__ __half quant_scale(__half mn, __half mx, float levels) {
  return h_divf(h_sub(mx, mn), levels);
}

// Gaussian-codebook codec at 1 bit.  std and mean of a group are torch.std_mean (unbiased) of its fp16
// values: computed in fp64 (the sum of up to 128 fp16 values is exact there) and rounded once to fp16.
__device__ __forceinline__ __half normal1_sd(double sum_sq_dev, int group) {
  return __double2half(sqrt(sum_sq_dev / (group - 1)));
}
// The same from fp32 sums, which decide the fp16 rounding of nearly every group (conversions to fp64, its divide and its
// square root take longer than everything else about a group): s + c = sum of the values, compensated; ss = sum of
// squared deviations from it, in four or more partial sums.  False where a bound on their error - 2^-22 of the mean, unless
// the values cancel to less than 2^-13 of their spread, and (group / 8 + 6) * 2^-25 of the deviation, which is 2^-21.6 for 32 -
// straddles a rounding boundary: one group in some 500.
__device__ __forceinline__ bool normal1_fast(float s, float c, float ss, int group, __half& mean, __half& sd) {
  const float m = (s + c) * (1.f / static_cast<float>(group));  // the group is a power of two
  const float d = __fsqrt_rn(__fdividef(ss, static_cast<float>(group - 1))), off = d * (static_cast<float>(group) * 0x1p-27f + 0x1p-22f);
  mean = __float2half_rn(m * (1.f - 0x1p-22f));
  sd = __float2half_rn(d - off);
  return __half_as_ushort(mean) == __half_as_ushort(__float2half_rn(m * (1.f + 0x1p-22f))) &&
         __half_as_ushort(sd) == __half_as_ushort(__float2half_rn(d + off)) && fabsf(m) >= d * 0x1p-13f && d > 1e-6f &&
         d < 6e4f && fabsf(m) < 6e4f;
}
// x added to s + c, the rounding error of the addition kept in c (Knuth's TwoSum)
__device__ __forceinline__ void add_compensated(float& s, float& c, float x) {
  const float t = __fadd_rn(s, x), back = __fsub_rn(t, s);
  c += __fadd_rn(__fsub_rn(s, __fsub_rn(t, back)), __fsub_rn(x, back));
  s = t;
}
// code = 1 where half(half(x - mean) / std) > 0 (decision bounds [0, inf]; a NaN quotient gives 0).  The quotient of two
// halfs rounds to zero up to 2^-25, so that is half(x - mean) > std * 2^-25, rounded down to a half (0 below std = 2).
__device__ __forceinline__ __half normal1_bound(__half sd) { return __float2half_rd(__half2float(sd) * 0x1p-25f); }
__device__ __forceinline__ uint32_t normal1_code(__half x, __half mean, __half bound) { return __hgt(h_sub(x, mean), bound) ? 1u : 0u; }
// two elements: codes in bits 0 and 16
__device__ __forceinline__ uint32_t normal1_code2(__half2 x, __half2 mean, __half2 bound) {
  return __hgt2_mask(__hsub2(x, mean), bound) & 0x00010001u;
}
#define HQKV_NORMAL1_CENTER 0.67448974f

__device__ __forceinline__ __half h_min(__half a, __half b) { return __half2float(b) < __half2float(a) ? b : a; }
__device__ __forceinline__ __half h_max(__half a, __half b) { return __half2float(b) > __half2float(a) ? b : a; }

}  // namespace hqkv
