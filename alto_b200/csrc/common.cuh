// Device-side arithmetic shared by the quantizer kernels: scale derivation, E2M1 / FP8
// encode and decode, exact division, packed-scale addressing.
//
// Every function restates arithmetic of the reference so that codes and scales are
// bit-identical to it; the citation next to each function names the reference lines.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include "../../include/altob200.h"

namespace altob200 {

// ---------------------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------------------
#define ALTOB200_CUDA_CHECK(expr)                 \
  do {                                            \
    cudaError_t _e = (expr);                      \
    if (_e != cudaSuccess) return ALTOB200_ECUDA; \
  } while (0)

static inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Programmatic dependent launch: a kernel launched through launch_after() may be scheduled while the
// kernel before it in the stream is still draining (its launch latency and the start-up of its CTAs
// then overlap that tail); it must call grid_dependency_wait() before it touches global memory, which
// blocks until the earlier kernel has completed and its writes are visible.  Launched any other way,
// the wait is a no-op.  ALTOB200_PDL=0 in the environment launches everything the plain way.
static inline bool pdl_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("ALTOB200_PDL");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v != 0;
}
template <class... KArgs, class... Args>
static inline cudaError_t launch_after(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                       Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------------------------------
// bit casts
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t f2u(float f) { return __float_as_uint(f); }
__device__ __forceinline__ float u2f(uint32_t u) { return __uint_as_float(u); }

// bf16 pair (little endian: element 0 in the low half) -> two floats, exact.
__device__ __forceinline__ float bf16lo_to_f32(uint32_t w) { return u2f(w << 16); }
// max(m, |a|, |b|), NaN if any is one
__device__ __forceinline__ float absmax3_nan(float m, float a, float b) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float bf16hi_to_f32(uint32_t w) { return u2f(w & 0xFFFF0000u); }

// float -> bf16 bits, round to nearest even (what Tensor.to(torch.bfloat16) does).
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float f) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f));
}

// ---------------------------------------------------------------------------------------
// packed scale layout (tiles of 128 rows x 4 scale columns, 512 bytes each)
// ---------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ int64_t packed_scale_offset(int64_t r, int64_t c,
                                                                int64_t ncol_tiles) {
  const int64_t tile = (r >> 7) * ncol_tiles + (c >> 2);
  return tile * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4 + (c & 3);
}

// ---------------------------------------------------------------------------------------
// E8M0 scale from a block amax, computed on the BITS of the amax in the input dtype.
//   alto/kernels/fp4/mxfp4/mxfp_quantization.py:79-95  (mbits=1, target_max_pow2=2)
//   alto/kernels/mxfp8/mxfp8_quantization.py:70-78      (e4m3: 3/8, e5m2: 2/15)
// `amax_bits` is the non-negative amax as bf16 bits (IS_BF16) or fp32 bits.
// ---------------------------------------------------------------------------------------
template <bool IS_BF16>
__device__ __forceinline__ uint32_t e8m0_from_amax_bits(uint32_t amax_bits, int mbits,
                                                        int target_max_pow2) {
  int e;
  if (IS_BF16) {
    // int16 arithmetic in the reference: wrap to 16 bits, arithmetic shift.
    const int32_t v = (int32_t)(int16_t)(((amax_bits + (1u << (7 - mbits - 1))) & 0xFF80u));
    e = (v >> 7) - target_max_pow2;
  } else {
    const int32_t v = (int32_t)((amax_bits + (1u << (23 - mbits - 1))) & 0xFF800000u);
    e = (v >> 23) - target_max_pow2;
  }
  e = e < 1 ? 1 : e;
  return (uint32_t)e & 0xFFu;  // .to(uint8)
}

// ---------------------------------------------------------------------------------------
// float -> E4M3 (float8_e4m3fn) round-to-nearest-even for inputs already clamped to
// [2^-6, 448] (all normal in E4M3), returned both as the byte and as the fp32 value.
//   alto/kernels/fp4/nvfp4/nvfp_quantization.py:278-282
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float round_to_e4m3_grid(float x, uint32_t* code) {
  uint32_t b = f2u(x);
  b += 0x7FFFFu + ((b >> 20) & 1u);  // RNE on the 20 dropped mantissa bits
  b &= 0xFFF00000u;
  // E4M3 bias 7: exponent field = e32 - 127 + 7
  const uint32_t e8 = (b >> 23) - 120u;
  *code = (e8 << 3) | ((b >> 20) & 7u);
  return u2f(b);
}

// NVFP4 block scales (inner on the E4M3 grid, quant = inner * outer).
//   alto/kernels/fp4/nvfp4/nvfp_quantization.py:255-289
// `raw` = amax / outer / 6 (or amax / 6), correctly rounded.
__device__ __forceinline__ void nvfp4_block_scale_from_raw(float raw, bool use_outer, float outer,
                                                           float* inner, float* quant, uint32_t* code) {
  raw = fminf(fmaxf(raw, 0.015625f), 448.0f);
  const float in = round_to_e4m3_grid(raw, code);
  *inner = in;
  *quant = use_outer ? __fmul_rn(in, outer) : in;
}
__device__ __forceinline__ void nvfp4_block_scale(float amax, bool use_outer, float outer,
                                                  float* inner, float* quant, uint32_t* code) {
  if (amax != amax) amax = 0.0f;  // NaN amax -> 0
  const float raw = use_outer ? __fdiv_rn(__fdiv_rn(amax, outer), 6.0f) : __fdiv_rn(amax, 6.0f);
  nvfp4_block_scale_from_raw(raw, use_outer, outer, inner, quant, code);
}

// ---------------------------------------------------------------------------------------
// Factor of a macro block (two-level scaling) from its maximum, and from its stored code:
//   alto/kernels/fp4/mxfp4/macro_block_scaling.py:70-85
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float macro_factor_from_amax(float amax, uint32_t* code) {
  amax = fmaxf(amax, 1e-12f);
  const uint32_t bits = f2u(__fdiv_rn(6.0f, amax)) & 0x007F8000u;
  *code = bits >> 15;
  return u2f(bits + (127u << 23));
}
__device__ __forceinline__ float macro_factor_from_code(uint32_t code) { return u2f((code << 15) + (127u << 23)); }

// ---------------------------------------------------------------------------------------
// Exact fp32 division x / q.
//
// For a bf16-valued numerator the sequence  y = x*r; e = fma(-y, q, x); y' = fma(e, r, y)
// with r = RN(1/q) returns the correctly rounded quotient (checked exhaustively over all
// 2^7 numerator and 2^23 denominator mantissas); it needs q and the quotient to stay away
// from the subnormal range, which callers guarantee by testing q once per block
// (`div_fast_ok`).  Written with e negated - e = fma(y, q, -x), y' = fma(-r, e, y), the same roundings -
// it also keeps the sign of a zero x (y is that zero, and an exact e is +0, so -r * e is -0), as IEEE
// division does (the reference ORs that sign into the code, triton_fp4_ops.py:40-41,90-92).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ bool div_fast_ok(float q) {
  const uint32_t e = (f2u(q) >> 23) & 0xFFu;
  return e >= 67u && e <= 187u;  // 2^-60 <= q < 2^61
}
__device__ __forceinline__ float div_bf16_num(float x, float q, float r) {
  const float y = __fmul_rn(x, r);
  const float e = __fmaf_rn(y, q, -x);
  return __fmaf_rn(-r, e, y);
}

// The same for an fp32 numerator, whose first product can be more than an ulp off: one correction makes it
// faithful, and correcting a faithful quotient with r = RN(1/q) rounds it correctly (Markstein's theorem).  It needs
// the quotient to stay finite (callers bound it per block); a residual that underflows belongs to a quotient below
// 2^-34, which every encoder treats alike.
__device__ __forceinline__ float div_f32_num(float x, float q, float r) {
  float y = __fmul_rn(x, r);
  y = __fmaf_rn(-r, __fmaf_rn(y, q, -x), y);
  return __fmaf_rn(-r, __fmaf_rn(y, q, -x), y);
}

// x / 6 for a normal x whose quotient and residual stay normal (callers keep |x| in [2^-91, 2^120) or
// zero): y = x * r, e = fma(-y, 6, x), y' = fma(e, r, y) with r = RN(1/6) is the correctly rounded
// quotient for every one of the 2^23 mantissas of x (checked exhaustively in integer arithmetic).
__device__ __forceinline__ float div_by_6(float x) {
  const float r = 0.16666667163372040f;
  const float y = __fmul_rn(x, r);
  const float e = __fmaf_rn(-y, 6.0f, x);
  return __fmaf_rn(e, r, y);
}

// ---------------------------------------------------------------------------------------
// E2M1 encode, round to nearest even, saturating:
//   alto/kernels/fp4/fp4_common/triton_fp4_ops.py:26-93 with USE_SR=False.
// Two floats -> one byte of E2M1 codes (v0 in the low nibble) with the hardware converter, which
// computes what the reference's bit arithmetic computes for every finite input: round to nearest
// even on the E2M1 grid including its subnormal 0.5, saturation to 6, sign of zero kept (checked
// against the oracle on the golden vectors and on random data in the GPU tests).
// ---------------------------------------------------------------------------------------
// Eight floats -> four bytes, element 0 in the lowest nibble: the converters write into the bytes of one
// register, nothing is shifted or merged.
__device__ __forceinline__ uint32_t e2m1x8_rtn_hw(const float* v) {
  uint32_t r;
  asm("{\n\t.reg .b8 t0, t1, t2, t3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t3, %8, %7;\n\t"
      "mov.b32 %0, {t0, t1, t2, t3};\n\t}"
      : "=r"(r)
      : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  return r;
}

// ---------------------------------------------------------------------------------------
// E2M1 encode with stochastic rounding from 32 random bits.  Restatement of
//   alto/kernels/fp4/fp4_common/triton_fp4_ops.py:26-93 with USE_SR=True.
// ---------------------------------------------------------------------------------------
// The reference rounds the normal range [1, 6) by adding 22 random bits below the kept mantissa bit and
// truncating; in the E2M1-subnormal range [0, 1), with 2a = k + frac, it compares the random word with
// uint32(a * fp32(2^33 - 2)) for a < 0.5 and with uint32((2a - 1) * fp32(2^32 - 1)) otherwise; both
// constants round to powers of two in fp32, so both thresholds are trunc(frac * 2^32) and the code is
// k + [rnd <= threshold].
//
// The general form (any v; the quantizers use it for blocks that hold an infinity or a NaN, or whose scale
// rules out the reciprocal division).  `v` is the scaled value up to the sign of a zero; the sign bit of the
// code is taken from `sign_bits` (the bits of the unscaled element: scales are positive).
// With a = min(|v|, 6):
//   normal range   code = (bits(a) + (rnd & (2^22 - 1)) - (126 << 23)) >> 22: the carry out of the low
//                  22 mantissa bits rounds up, and 6.0 itself maps to 7, so saturation needs no
//                  separate test;
//   a < 1          with T = trunc(a * 2^33) = k * 2^32 + threshold (k = [a >= 0.5]),
//                  code = T.hi + [T.lo >= rnd].
// A NaN saturates to 7 (the reference's code for a NaN element is an accident of its payload).
__device__ __forceinline__ uint32_t e2m1_sr_code(float v, uint32_t sign_bits, uint32_t rnd) {
  const float a = fminf(fabsf(v), 6.0f);
  const uint32_t ab = f2u(a);
  const uint32_t cn = (ab + (rnd & 0x3FFFFFu) - (126u << 23)) >> 22;
  const uint64_t t = __float2ull_rz(__fmul_rn(a, 8589934592.0f));
  const uint32_t cd = (uint32_t)(t >> 32) + ((uint32_t)t >= rnd ? 1u : 0u);
  return ((sign_bits >> 31) << 3) | (a < 1.0f ? cd : cn);
}

// The same for finite v whose zeros carry their sign, as the VALUE of the code (which the hardware converter
// then packs with its neighbours), without selects, shifts or integer conversions of v - the quantizers are
// bound by the integer pipe, whose compares, selects, shifts and permutes take two cycles a warp and its
// 64-bit float conversion eight:
//   a < 1    [rnd <= threshold] is a >= rnd * 2^-33 (plus 0.5 when k = 1), and since a and a - 0.5 are fp32
//            numbers, rnd may first be rounded UP to fp32.  With t = RZ(a - u), u = RU(rnd) * 2^-33, whose
//            rounding towards zero never moves it across 0 or 0.5, the value is (floor(2t) + 1) / 2: the
//            round-down multiply-add with 1.5 * 2^23 is floor(2t), and saturating the rest at 1 makes it 1 for
//            every a >= 1 (u <= 0.5, so t >= 0.5 there);
//   a >= 1   (bits(v) + 22 random bits) with the low bits cut is the rounded value; what it exceeds 1 by is
//            added (saturated at 8, which the converter saturates to 6); below 1 there is no excess.
// Bit for bit the code of e2m1_sr_code.
__device__ __forceinline__ float e2m1_sr_value(float v, uint32_t rnd) {
  const float u = __uint2float_ru(rnd);
  const float t = __fmaf_rz(u, -1.16415321826934814453125e-10f, fabsf(v));
  const float g = __fmaf_rd(t, 2.0f, 12582912.0f);
  float below, above;
  asm("fma.rn.sat.f32 %0, %1, 0f3F000000, %2;" : "=f"(below) : "f"(g), "f"(-6291455.5f));
  const uint32_t n = (f2u(v) + (rnd & 0x3FFFFFu)) & 0x7FC00000u;
  asm("fma.rn.sat.f32 %0, %1, 0f3E000000, 0fBE000000;" : "=f"(above) : "f"(u2f(n)));
  const float w = __fmaf_rn(above, 8.0f, below);
  return u2f(f2u(w) | (f2u(v) & 0x80000000u));
}

// E2M1 decode (alto/kernels/fp4/fp4_common/triton_fp4_ops.py:100-132).
// The two codes of a byte (low nibble first) -> two floats with the hardware converter; exact, sign of zero kept.
__device__ __forceinline__ float2 e2m1x2_decode(uint32_t byte) {
  uint32_t h2;
  asm("{ .reg .b8 lo, hi; mov.b16 {lo, hi}, %1; cvt.rn.f16x2.e2m1x2 %0, lo; }" : "=r"(h2) : "h"((uint16_t)byte));
  const __half2 h = *reinterpret_cast<const __half2*>(&h2);
  return __half22float2(h);
}

// ---------------------------------------------------------------------------------------
// FP8 encode: saturating round-to-nearest-even (the emulation clamps to +-max and then
// casts, tests/unittest/mxfp8/utils.py:126-132; the Triton cast saturates natively,
// alto/kernels/mxfp8/mxfp8_quantization.py:263-281).  v0 goes to the low byte.
// ---------------------------------------------------------------------------------------
template <bool E5M2>
__device__ __forceinline__ uint32_t fp8x2_rtn_hw(float v0, float v1) {
  uint16_t r;
  if (E5M2) {
    asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(r) : "f"(v1), "f"(v0));
  } else {
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(v1), "f"(v0));
  }
  return (uint32_t)r;
}

// Two FP8 bytes (low byte first) -> two floats; exact (both formats embed in fp16).
template <bool E5M2>
__device__ __forceinline__ float2 fp8x2_decode(uint32_t c) {
  uint32_t h2;
  const uint16_t c16 = (uint16_t)c;
  if (E5M2) {
    asm("cvt.rn.f16x2.e5m2x2 %0, %1;" : "=r"(h2) : "h"(c16));
  } else {
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(c16));
  }
  const __half2 h = *reinterpret_cast<const __half2*>(&h2);
  return __half22float2(h);
}

// ---------------------------------------------------------------------------------------
// Philox-4x32-10 with the counter/key convention of triton.language.randint4x(seed, offset):
// counter = (offset_lo, offset_hi, 0, 0), key = (seed_lo, seed_hi); each of the ten rounds is
//   c0' = hi(B * c2) ^ c1 ^ k0,  c2' = hi(A * c0) ^ c3 ^ k1,  c1' = lo(B * c2),  c3' = lo(A * c0)
// with A = 0xD2511F53, B = 0xCD9E8D57 and the key advanced by (0x9E3779B9, 0xBB67AE85) per round.
// The ten round keys are precomputed on the host (they depend on the seed only), so that each round
// is two wide multiplies and two three-input XORs.
// ---------------------------------------------------------------------------------------
struct PhiloxKeys {
  uint32_t k[20];  // k[2i], k[2i+1]: key of round i
};
static inline void philox_make_keys(uint64_t seed, PhiloxKeys* pk) {
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int i = 0; i < 10; ++i) {
    pk->k[2 * i] = k0;
    pk->k[2 * i + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}
__device__ __forceinline__ void philox4x32_10_keys(uint32_t c0, uint32_t c1, const PhiloxKeys& pk, uint32_t out[4]) {
  const uint32_t A = 0xD2511F53u, B = 0xCD9E8D57u;
  uint32_t c2 = 0u, c3 = 0u;
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    const uint64_t pb = (uint64_t)B * c2, pa = (uint64_t)A * c0;
    c0 = (uint32_t)(pb >> 32) ^ c1 ^ pk.k[2 * i];
    c2 = (uint32_t)(pa >> 32) ^ c3 ^ pk.k[2 * i + 1];
    c1 = (uint32_t)pb;
    c3 = (uint32_t)pa;
  }
  out[0] = c0;
  out[1] = c1;
  out[2] = c2;
  out[3] = c3;
}

}  // namespace altob200
