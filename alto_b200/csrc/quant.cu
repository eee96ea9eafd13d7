// Bandwidth kernels of the low-precision linear path: block quantizers (row-wise,
// column-wise with the optional randomised Hadamard transform, 2D with dual packing),
// tensor amax, dequantizers and the standalone Hadamard transform.
//
// Work layout (every global access is a full 32-byte sector or better, and every thread keeps one
// quantisation block or a fixed part of it in registers; the counters show all of these kernels
// bound by instruction issue rather than by HBM):
//   row-wise  : a warp task is 4 rows x 512 contiguous elements, a lane 16 elements of each row
//               (two 128-bit loads per row for bf16, all issued first).  NVFP4 blocks (16) live in
//               one lane, MX blocks (32) in a lane pair.
//   col-wise  : a CTA owns a 128-row x 64-column tile; a lane owns two adjacent columns of one
//               block of rows, so the Hadamard butterfly and the block amax need no shuffles.
//               Codes are transposed through shared memory so that every output row receives 64
//               (FP4) or 128 (FP8) contiguous bytes.
//   2D        : a warp owns 64 rows x 64 columns (FP8: 32 x 128), a thread 16 rows x 8 columns in
//               registers; block maxima by shuffles, the second packing by an in-register
//               transpose; no shared memory.
#include <type_traits>

#include <atomic>

#include "common.cuh"

namespace altob200 {

// ---------------------------------------------------------------------------------------
// format traits
// ---------------------------------------------------------------------------------------
template <int FMT>
struct Fmt;
template <>
struct Fmt<ALTOB200_FMT_NVFP4> {
  static constexpr int B = 16;
  static constexpr bool FP4 = true, MX = false, E5M2 = false;
  static constexpr int MBITS = 0, TMAX = 0;
};
template <>
struct Fmt<ALTOB200_FMT_MXFP4> {
  static constexpr int B = 32;
  static constexpr bool FP4 = true, MX = true, E5M2 = false;
  static constexpr int MBITS = 1, TMAX = 2;
};
template <>
struct Fmt<ALTOB200_FMT_MXFP8_E4M3> {
  static constexpr int B = 32;
  static constexpr bool FP4 = false, MX = true, E5M2 = false;
  static constexpr int MBITS = 3, TMAX = 8;
};
template <>
struct Fmt<ALTOB200_FMT_MXFP8_E5M2> {
  static constexpr int B = 32;
  static constexpr bool FP4 = false, MX = true, E5M2 = true;
  static constexpr int MBITS = 2, TMAX = 15;
};

// Scale of one quantisation block, in the forms the element loop needs.
struct BlockScale {
  float q;        // divisor applied to the elements
  float r;        // reciprocal used by the fast paths
  bool fast;      // fast path valid
  uint32_t byte;  // stored scale byte (E8M0 exponent or E4M3 code)
  float plain;    // NVFP4: inner scale as fp32 (plain layout)
};

// The tensor-wide outer scale of NVFP4 in the forms the block-scale arithmetic needs (per thread, once).
struct OuterScale {
  bool use;    // an outer scale is applied
  float v;     // its value (1 when unused)
  float r;     // RN(1 / v)
  bool fast;   // v allows the reciprocal form of amax / v
};
__device__ __forceinline__ OuterScale make_outer_scale(bool use, const float* p) {
  OuterScale o;
  o.use = use;
  o.v = use ? __ldg(p) : 1.0f;
  o.r = __frcp_rn(o.v);
  o.fast = div_fast_ok(o.v);
  return o;
}

// amax_abs_bits: max over the block of (bits & 0x7FFF..) in the input dtype's bit width
// (bf16 bits or fp32 bits); integer max propagates NaN like torch.amax does.
template <int FMT, bool IN_BF16>
__device__ __forceinline__ BlockScale make_block_scale(uint32_t amax_abs_bits, const OuterScale& os) {
  using F = Fmt<FMT>;
  BlockScale s;
  if (F::MX) {
    const uint32_t e = e8m0_from_amax_bits<IN_BF16>(amax_abs_bits, F::MBITS, F::TMAX);
    s.byte = e;
    s.q = u2f(e << 23);
    s.fast = e <= 253u;
    s.r = u2f((254u - e) << 23);
    s.plain = 0.0f;
  } else {
    const float amax = IN_BF16 ? u2f(amax_abs_bits << 16) : u2f(amax_abs_bits);
    // bf16 amax of 0 or in [2^-30, 2^60): amax / outer / 6 by reciprocals with one correction step each
    // (exact, see div_bf16_num and div_by_6); everything else divides
    const uint32_t e8 = amax_abs_bits >> 7;
    if (IN_BF16 && (amax_abs_bits == 0u || (e8 >= 97u && e8 < 187u)) && (!os.use || os.fast)) {
      const float t = os.use ? div_bf16_num(amax, os.v, os.r) : amax;
      nvfp4_block_scale_from_raw(div_by_6(t), os.use, os.v, &s.plain, &s.q, &s.byte);
    } else {
      nvfp4_block_scale(amax, os.use, os.v, &s.plain, &s.q, &s.byte);
    }
    s.r = __frcp_rn(s.q);
    s.fast = div_fast_ok(s.q) && (IN_BF16 || __fmul_rn(amax, s.r) < 1.2676506e30f);
  }
  return s;
}

// ---------------------------------------------------------------------------------------
// Options of the MXFP4 quantizer (alto/kernels/fp4/mxfp4/mxfp_quantization.py:29-95, 321-322;
// arithmetic as in the reference's emulation, tests/unittest/mxfp4/utils.py:320-358, which works
// in the input dtype: with bf16 inputs every intermediate is rounded to bf16).
//   clip 1 (static) : elements are multiplied by 3/4 before encoding; the scale is unchanged
//   clip 2 (dynamic): the scale is taken from 2.92247856/6 * std(block) + 1e-8 instead of the amax,
//                     with target exponent 0 instead of 2
//   uos             : scale = ceil(log2(amax / 7.25)) + 127 (128 for an all-zero block)
// ---------------------------------------------------------------------------------------
struct MxOpts {
  int clip;
  int uos;
};

template <bool IN_BF16>
__device__ __forceinline__ float round_in(float v) {
  return IN_BF16 ? u2f(f32_to_bf16_bits(v) << 16) : v;
}

// E8M0 byte of an MX block from its statistics.  `amax_abs_bits` as in make_block_scale; `sum` and
// `sumsq` (of the squares rounded to the input dtype) over the n elements are used by clip 2 only.
template <int FMT, bool IN_BF16>
__device__ __forceinline__ BlockScale make_block_scale_opts(uint32_t amax_abs_bits, float sum, float sumsq, int n,
                                                            MxOpts o) {
  using F = Fmt<FMT>;
  float max_abs = IN_BF16 ? u2f(amax_abs_bits << 16) : u2f(amax_abs_bits);
  int tmax = F::TMAX;
  if (o.clip == 2) {
    const float inv_n = 1.0f / (float)n;
    const float mean_sq = round_in<IN_BF16>(__fmul_rn(sumsq, inv_n));
    const float mean = round_in<IN_BF16>(__fmul_rn(sum, inv_n));
    const float var = round_in<IN_BF16>(__fsub_rn(mean_sq, round_in<IN_BF16>(__fmul_rn(mean, mean))));
    const float sd = round_in<IN_BF16>(__fsqrt_rn(var));
    max_abs = round_in<IN_BF16>(__fadd_rn(round_in<IN_BF16>(__fmul_rn(sd, (float)(2.92247856 / 6.0))), 1e-8f));
    tmax = 0;
  }
  uint32_t e;
  if (o.uos) {
    const float r = round_in<IN_BF16>(__fdiv_rn(max_abs, 7.25f));
    float s = ceilf(round_in<IN_BF16>(log2f(r)));
    if (max_abs == 0.0f) s = 1.0f;
    s += 127.0f;
    // NaN compares false everywhere and converts to 0, which the clamp turns into 1
    e = s < 1.0f ? 1u : (s > 255.0f ? 255u : (uint32_t)s);
    if (!(s == s)) e = 1u;
  } else {
    const uint32_t bits = IN_BF16 ? (f2u(max_abs) >> 16) : f2u(max_abs);
    e = e8m0_from_amax_bits<IN_BF16>(bits, F::MBITS, tmax);
  }
  BlockScale s;
  s.byte = e;
  s.q = u2f(e << 23);
  s.fast = e <= 253u;
  s.r = u2f((254u - e) << 23);
  s.plain = 0.0f;
  return s;
}

// One element divided by its block scale.  FAST is decided once per warp (every lane's block scale
// allows the reciprocal forms), so that the element loops carry no per-element branch; the other
// variant divides.  Both give the correctly rounded quotient.
template <int FMT, bool IN_BF16, bool FAST>
__device__ __forceinline__ float scale_elem(float x, const BlockScale& s) {
  if (!FAST) return __fdiv_rn(x, s.q);
  if (Fmt<FMT>::MX) return __fmul_rn(x, s.r);
  return IN_BF16 ? div_bf16_num(x, s.q, s.r) : div_f32_num(x, s.q, s.r);
}

// acc | (x << sh) for disjoint bits, as one integer multiply-add.
__device__ __forceinline__ uint32_t merge_shifted(uint32_t x, int sh, uint32_t acc) {
  uint32_t r;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(x), "r"(1u << sh), "r"(acc));
  return r;
}

// Eight elements of one block scaled and quantised into four FP4 bytes (element 0 in the lowest nibble).
// SR words: r0[j] for element 2j, r1[j] for element 2j + 1; FAST also means that the elements are finite.
template <int FMT, bool IN_BF16, int ROUND, bool FAST>
__device__ __forceinline__ uint32_t fp4_octet(const float* x, const BlockScale& s, const uint32_t* r0, const uint32_t* r1) {
  float q[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) q[j] = scale_elem<FMT, IN_BF16, FAST>(x[j], s);
  if (ROUND == ALTOB200_ROUND_RTN) return e2m1x8_rtn_hw(q);
  if (FAST) {
#pragma unroll
    for (int j = 0; j < 8; ++j) q[j] = e2m1_sr_value(q[j], (j & 1) ? r1[j >> 1] : r0[j >> 1]);
    return e2m1x8_rtn_hw(q);
  }
  uint32_t word = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    word = merge_shifted(e2m1_sr_code(q[j], f2u(x[j]), (j & 1) ? r1[j >> 1] : r0[j >> 1]), 4 * j, word);
  return word;
}

// Two values that are bf16 numbers as one word.
__device__ __forceinline__ uint32_t pack_bf16_bits(float lo, float hi) { return __byte_perm(f2u(lo), f2u(hi), 0x7632); }

// The random words of eight elements in the forms that e2m1_sr_value takes from a word: -RU(word) * 2^-33 and the
// low 22 bits.  Elements that share words (rows a table's period apart) share these.
struct SrOctet {
  float nu[8];
  uint32_t m[8];
};
__device__ __forceinline__ SrOctet sr_octet(const uint4& even, const uint4& odd) {
  const uint32_t w[8] = {even.x, odd.x, even.y, odd.y, even.z, odd.z, even.w, odd.w};
  SrOctet o;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    o.nu[j] = __fmul_rn(__uint2float_ru(w[j]), -1.16415321826934814453125e-10f);
    o.m[j] = w[j] & 0x3FFFFFu;
  }
  return o;
}

// fp4_octet<FAST> with such words: the steps of e2m1_sr_value, two elements to an instruction where there is one, and
// the sign from the element itself.
template <int FMT, bool IN_BF16>
__device__ __forceinline__ uint32_t fp4_octet_sr(const float* x, const BlockScale& s, const SrOctet& o) {
  float c[8];
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    float2 v = make_float2(x[j], x[j + 1]);
    const float2 r = make_float2(s.r, s.r);
    if (Fmt<FMT>::MX) {
      v = __fmul2_rn(v, r);
    } else if (IN_BF16) {   // div_bf16_num up to the sign of a zero
      const float2 y = __fmul2_rn(v, r), nq = make_float2(-s.q, -s.q);
      v = __ffma2_rn(__ffma2_rn(y, nq, v), r, y);
    } else {
      v = make_float2(div_f32_num(v.x, s.q, s.r), div_f32_num(v.y, s.q, s.r));
    }
    const float2 t = make_float2(__fadd_rz(fabsf(v.x), o.nu[j]), __fadd_rz(fabsf(v.y), o.nu[j + 1]));
    const float2 g = __ffma2_rd(t, make_float2(2.0f, 2.0f), make_float2(12582912.0f, 12582912.0f));
    float2 below, above;
    asm("fma.rn.sat.f32 %0, %1, 0f3F000000, %2;" : "=f"(below.x) : "f"(g.x), "f"(-6291455.5f));
    asm("fma.rn.sat.f32 %0, %1, 0f3F000000, %2;" : "=f"(below.y) : "f"(g.y), "f"(-6291455.5f));
    const uint32_t n0 = (f2u(v.x) + o.m[j]) & 0x7FC00000u, n1 = (f2u(v.y) + o.m[j + 1]) & 0x7FC00000u;
    asm("fma.rn.sat.f32 %0, %1, 0f3E000000, 0fBE000000;" : "=f"(above.x) : "f"(u2f(n0)));
    asm("fma.rn.sat.f32 %0, %1, 0f3E000000, 0fBE000000;" : "=f"(above.y) : "f"(u2f(n1)));
    const float2 w = __ffma2_rn(above, make_float2(8.0f, 8.0f), below);
    c[j] = u2f(f2u(w.x) | (f2u(x[j]) & 0x80000000u));
    c[j + 1] = u2f(f2u(w.y) | (f2u(x[j + 1]) & 0x80000000u));
  }
  return e2m1x8_rtn_hw(c);
}

// Whether a block may take the reciprocal forms: with stochastic rounding only without infinities and NaNs.
template <bool IN_BF16, int ROUND>
__device__ __forceinline__ bool block_fast(const BlockScale& s, uint32_t amax_abs_bits) {
  return s.fast && (ROUND == ALTOB200_ROUND_RTN || amax_abs_bits < (IN_BF16 ? 0x7F80u : 0x7F800000u));
}

// Runs body(std::true_type) when every lane of the warp may use the reciprocal forms, else
// body(std::false_type); must be reached by the whole warp.
template <class Body>
__device__ __forceinline__ void with_uniform_fast(bool lane_fast, Body body) {
  if (__all_sync(0xFFFFFFFFu, lane_fast)) body(std::true_type{});
  else body(std::false_type{});
}

// Quotient and remainder with a 32-bit divide whenever the operands fit (a 64-bit divide costs
// several dozen instructions per task).
__device__ __forceinline__ void divmod_fast(int64_t t, int64_t d, int64_t* q, int64_t* r) {
  if ((((uint64_t)t | (uint64_t)d) >> 32) == 0) {
    const uint32_t qq = (uint32_t)t / (uint32_t)d;
    *q = qq;
    *r = (uint32_t)t - qq * (uint32_t)d;
  } else {
    *q = t / d;
    *r = t - *q * d;
  }
}

__device__ __forceinline__ uint32_t absmax_bf16x2(uint32_t acc, uint32_t w) {
  return __vmaxu2(acc, w & 0x7FFF7FFFu);
}
// maximum over two words at once (one three-input instruction)
__device__ __forceinline__ uint32_t absmax2_bf16x2(uint32_t acc, uint32_t w0, uint32_t w1) {
  return __vimax3_u16x2(acc, w0 & 0x7FFF7FFFu, w1 & 0x7FFF7FFFu);
}
__device__ __forceinline__ uint32_t fold_bf16x2(uint32_t acc) {
  const uint32_t lo = acc & 0xFFFFu, hi = acc >> 16;
  return lo > hi ? lo : hi;
}

__device__ __forceinline__ uint32_t warp_max_u32(uint32_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint32_t t = __shfl_xor_sync(0xFFFFFFFFu, v, o);
    v = t > v ? t : v;
  }
  return v;
}

// =======================================================================================
// Row-wise quantizer
// =======================================================================================
struct RowwiseArgs {
  const void* x;
  int64_t rows, cols, ld;
  uint8_t* codes;
  void* scale_plain;
  uint8_t* scale_packed;
  int64_t ncol_tiles;  // ceil(cols / B / 4)
  const float* outer;
  const uint32_t* rand_bits;
  // rand_bits as a periodic tile [2][tile_rows][tile_pairs] (0 = full planes [2][rows][cols/2])
  int64_t tile_rows, tile_pairs;
  uint64_t philox_seed, philox_offset;
  PhiloxKeys pk;
  MxOpts mx;
  uint8_t* macro_codes;  // MACRO: [rows, ceil(cols / 128)] factor codes, written
};

// A warp task is 4 consecutive rows x 512 contiguous columns (a lane: 16 columns of each row).  The
// loads of all four rows are issued before the first is consumed (128 bytes per lane in flight), and
// the index arithmetic of a task (row and chunk, pointers, position in the periodic random table) is
// paid once per 64 elements of a lane.
// Three resident blocks of 256 threads per SM (at most 85 registers per thread): other block sizes and counts
// measured within 3 %.
//
// SHARED, words from a table: the four rows are a period of the table apart, so that they meet the same words, which are
// loaded and converted once, behind the scales of all four rows.  Bound by the instructions of the rounding (26 an element
// with macro factors, 20 without, the scheduler 64 % busy).  Four blocks of 128 threads (128 registers) keep bf16 rows
// free of spills; five, or three of 256, spill and are slower than words loaded by row.  8192 x 14336 from bf16, words by
// row -> shared: MXFP4 119 -> 106 us, with macro factors 141 -> 133, NVFP4 125 -> 113; fp32 141 -> 131 and 178 -> 147.
constexpr int ROW_R = 4;

// Words by row (full planes, or few rows: `rowwise_shares_words`) are loaded in front of a row's scale arithmetic, which
// hides them.  Asked for behind it, in the registers of SHARED, 8192 x 14336 from bf16 took MXFP4 172 us for 150, with
// macro factors 193 for 156, NVFP4 180 for 151.
constexpr int rowwise_threads(bool shared) { return shared ? 128 : 256; }

// Groups of rows that tasks take, rows `step` apart: neighbours, or a period of the random table (SHARED).
__host__ __device__ __forceinline__ int64_t rowwise_row_groups(int64_t rows, int64_t step) {
  return (rows + ROW_R * step - 1) / (ROW_R * step) * step;
}

// MACRO (MXFP4 from bf16): the two-level recipe's scaling runs in front of the quantisation; a macro block of
// 128 columns is eight neighbouring lanes.
template <int FMT, bool IN_BF16, int ROUND, bool MACRO, bool SHARED>
__global__ void __launch_bounds__(rowwise_threads(SHARED), SHARED ? 4 : 3) quantize_rowwise_kernel(RowwiseArgs a) {
  grid_dependency_wait();
  using F = Fmt<FMT>;
  static_assert(!MACRO || (FMT == ALTOB200_FMT_MXFP4 && IN_BF16), "macro blocks");
  const int64_t macro_chunks = (a.cols + 127) >> 7;
  constexpr int LPB = F::B / 16;  // lanes per block
  constexpr int ESZ = IN_BF16 ? 2 : 4;
  constexpr int NV = IN_BF16 ? 2 : 4;  // 16-byte vectors per lane and row
  const int lane = threadIdx.x & 31;
  const int64_t chunks_per_row = (a.cols + 511) >> 9;
  static_assert(!SHARED || ROUND == ALTOB200_ROUND_SR_BITS, "words from a table");
  const int64_t step = SHARED ? a.tile_rows : 1;
  const int64_t n_tasks = rowwise_row_groups(a.rows, step) * chunks_per_row;
  const int64_t warp0 = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t n_warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const OuterScale os = make_outer_scale((!F::MX) && a.outer != nullptr, a.outer);
  const int64_t half_cols = a.cols >> 1;
  const int64_t nkb = a.cols / F::B;
  const bool tiled = a.tile_rows != 0;
  const uint32_t t_rows = (uint32_t)a.tile_rows, t_pairs = (uint32_t)a.tile_pairs;

  for (int64_t task = warp0; task < n_tasks; task += n_warps) {
    int64_t rg, chunk;
    divmod_fast(task, chunks_per_row, &rg, &chunk);
    int64_t row0 = rg * ROW_R;
    if (SHARED) {
      int64_t period, first;
      divmod_fast(rg, step, &period, &first);
      row0 = period * (ROW_R * step) + first;
    }
    const int64_t col = (chunk << 9) + lane * 16;
    const bool col_ok = col < a.cols;
    const uint8_t* src = reinterpret_cast<const uint8_t*>(a.x) + (row0 * a.ld + col) * ESZ;
    const int64_t pitch = a.ld * ESZ * step;
    // rows of the task that exist, and the place of their codes, from a count and a pitch where registers are left for them
    constexpr bool COUNTED = SHARED || (IN_BF16 && ROUND == ALTOB200_ROUND_RTN);
    constexpr int EPB = F::FP4 ? 2 : 1;   // elements per byte of codes
    int n_ok = 0;
#pragma unroll
    for (int i = 0; COUNTED && i < ROW_R; ++i) n_ok += row0 + i * step < a.rows ? 1 : 0;
    uint8_t* const dst0 = a.codes + (row0 * a.cols + col) / EPB;
    const int64_t dst_pitch = step * (a.cols / EPB);
    const auto row_ok = [&](int i) { return COUNTED ? i < n_ok : row0 + i * step < a.rows; };
    const auto dst = [&](int i) { return COUNTED ? dst0 + i * dst_pitch : a.codes + ((row0 + i * step) * a.cols + col) / EPB; };

    // ---- all loads of the task ----
    uint4 raw[ROW_R][NV];
#pragma unroll
    for (int i = 0; i < ROW_R; ++i) {
      const bool ok = col_ok && row_ok(i);
#pragma unroll
      for (int q = 0; q < NV; ++q)
        raw[i][q] = ok ? __ldg(reinterpret_cast<const uint4*>(src + i * pitch) + q) : make_uint4(0u, 0u, 0u, 0u);
    }
    // position of the task in the periodic random table (32-bit: the host refuses larger extents)
    uint32_t rr0 = 0, pp = 0;
    if (ROUND == ALTOB200_ROUND_SR_BITS && !SHARED && tiled) {
      rr0 = (uint32_t)row0 % t_rows;
      pp = (uint32_t)(col >> 1) % t_pairs;
    }
    const int64_t kb = (chunk << 9) / F::B + lane / LPB;  // scale column of this lane
    const bool holder = col_ok && (lane % LPB == 0);
    static_assert(ROW_R == 4, "the packed scales are transposed four rows at a time");
    uint32_t scale_bytes = 0;   // byte i: scale of row i

    BlockScale scales[SHARED ? ROW_R : 1];
    bool all_fast = true;
#pragma unroll
    for (int i = 0; i < ROW_R; ++i) {
      const int64_t row = row0 + i * step;
      if (SHARED && !row_ok(i)) break;   // the whole warp
      const bool active = col_ok && row_ok(i);
      uint32_t r0[8], r1[8];
      if (ROUND == ALTOB200_ROUND_SR_BITS && !SHARED) {
        // random words first: their loads overlap the scale arithmetic below.  Full planes [2][rows][cols/2], or a
        // [2][tile_rows][tile_pairs] table repeated over the matrix (the 8 pairs of a lane never straddle a tile:
        // tile_pairs is a multiple of 8)
        uint32_t rr = rr0 + (uint32_t)i;
        while (tiled && rr >= t_rows) rr -= t_rows;
        const int64_t off = tiled ? (int64_t)(rr * t_pairs + pp) : row * half_cols + (col >> 1);
        const int64_t plane = tiled ? (int64_t)(t_rows * t_pairs) : a.rows * half_cols;
        uint4 a0 = make_uint4(0u, 0u, 0u, 0u), a1 = a0, b0 = a0, b1 = a0;
        if (active) {
          const uint4* p0 = reinterpret_cast<const uint4*>(a.rand_bits + off);
          const uint4* p1 = reinterpret_cast<const uint4*>(a.rand_bits + plane + off);
          a0 = __ldg(p0); a1 = __ldg(p0 + 1); b0 = __ldg(p1); b1 = __ldg(p1 + 1);
        }
        r0[0] = a0.x; r0[1] = a0.y; r0[2] = a0.z; r0[3] = a0.w;
        r0[4] = a1.x; r0[5] = a1.y; r0[6] = a1.z; r0[7] = a1.w;
        r1[0] = b0.x; r1[1] = b0.y; r1[2] = b0.z; r1[3] = b0.w;
        r1[4] = b1.x; r1[5] = b1.y; r1[6] = b1.z; r1[7] = b1.w;
      } else if (ROUND == ALTOB200_ROUND_SR_PHILOX) {
        // one Philox call feeds two element pairs: call index = pair index / 2
        const uint64_t q0 = a.philox_offset + (uint64_t)((row * half_cols + (col >> 1)) >> 1);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[4];
          const uint64_t ctr = q0 + c;
          philox4x32_10_keys((uint32_t)ctr, (uint32_t)(ctr >> 32), a.pk, o);
          r0[2 * c] = o[0]; r1[2 * c] = o[1]; r0[2 * c + 1] = o[2]; r1[2 * c + 1] = o[3];
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) r0[j] = r1[j] = 0;
      }

      // ---- unpack, block maximum ----
      float v[16];
      uint32_t amax_bits = 0;
      if (IN_BF16) {
        const uint32_t w[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w,
                               raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
        uint32_t acc = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (j & 1) acc = absmax2_bf16x2(acc, w[j - 1], w[j]);
          v[2 * j] = bf16lo_to_f32(w[j]);
          v[2 * j + 1] = bf16hi_to_f32(w[j]);
        }
        amax_bits = fold_bf16x2(acc);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          v[4 * q] = u2f(raw[i][q % NV].x); v[4 * q + 1] = u2f(raw[i][q % NV].y);
          v[4 * q + 2] = u2f(raw[i][q % NV].z); v[4 * q + 3] = u2f(raw[i][q % NV].w);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t b = f2u(v[j]) & 0x7FFFFFFFu;
          amax_bits = b > amax_bits ? b : amax_bits;
        }
      }
      if (MACRO) {
        // factor of the row's 128 columns (NaNs do not take part in the maximum, csrc/macro_scale.cu), then
        // y = bf16(x * factor); rounding is monotone, so the lane's maximum is scaled instead of searched again
        float m = u2f(amax_bits << 16);
        if (__any_sync(0xFFFFFFFFu, amax_bits > 0x7F80u)) {
          m = 0.0f;
#pragma unroll
          for (int j = 0; j < 16; ++j) m = fmaxf(m, fabsf(v[j]));
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
        uint32_t code;
        const float f = macro_factor_from_amax(m, &code);
        if (active && (lane & 7) == 0) a.macro_codes[row * macro_chunks + (col >> 7)] = (uint8_t)code;
        amax_bits = f32_to_bf16_bits(__fmul_rn(u2f(amax_bits << 16), f)) & 0x7FFFu;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const __nv_bfloat162 p2 = __floats2bfloat162_rn(__fmul_rn(v[j], f), __fmul_rn(v[j + 1], f));
          const uint32_t w = *reinterpret_cast<const uint32_t*>(&p2);
          v[j] = bf16lo_to_f32(w);
          v[j + 1] = bf16hi_to_f32(w);
        }
      }
      if (LPB == 2) {
        const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, amax_bits, 1);
        amax_bits = o > amax_bits ? o : amax_bits;
      }
      BlockScale s;
      if (F::MX && (a.mx.clip | a.mx.uos)) {
        float sum = 0.0f, sumsq = 0.0f;
        if (a.mx.clip == 2) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            sum = __fadd_rn(sum, v[j]);
            sumsq = __fadd_rn(sumsq, round_in<IN_BF16>(__fmul_rn(v[j], v[j])));
          }
          if (LPB == 2) {
            sum = __fadd_rn(sum, __shfl_xor_sync(0xFFFFFFFFu, sum, 1));
            sumsq = __fadd_rn(sumsq, __shfl_xor_sync(0xFFFFFFFFu, sumsq, 1));
          }
        }
        s = make_block_scale_opts<FMT, IN_BF16>(amax_bits, sum, sumsq, F::B, a.mx);
        if (a.mx.clip == 1) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = round_in<IN_BF16>(__fmul_rn(v[j], 0.75f));
        }
      } else {
        s = make_block_scale<FMT, IN_BF16>(amax_bits, os);
      }

      // ---- encode and store ----
      if constexpr (SHARED) {   // behind the loop; what clip and factors made of the elements goes back into their words
        scales[i] = s;
        all_fast = all_fast && block_fast<IN_BF16, ROUND>(s, amax_bits);
        if (MACRO || (F::MX && a.mx.clip == 1)) {
          if (IN_BF16) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
              raw[i][q] = make_uint4(pack_bf16_bits(v[8 * q], v[8 * q + 1]), pack_bf16_bits(v[8 * q + 2], v[8 * q + 3]),
                                     pack_bf16_bits(v[8 * q + 4], v[8 * q + 5]), pack_bf16_bits(v[8 * q + 6], v[8 * q + 7]));
          } else {
#pragma unroll
            for (int q = 0; q < NV; ++q)
              raw[i][q] = make_uint4(f2u(v[(4 * q) & 15]), f2u(v[(4 * q + 1) & 15]), f2u(v[(4 * q + 2) & 15]), f2u(v[(4 * q + 3) & 15]));
          }
        }
      } else
      with_uniform_fast(block_fast<IN_BF16, ROUND>(s, amax_bits), [&](auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        if (F::FP4) {
          const uint32_t lo = fp4_octet<FMT, IN_BF16, ROUND, FAST>(v, s, r0, r1);
          const uint32_t hi = fp4_octet<FMT, IN_BF16, ROUND, FAST>(v + 8, s, r0 + 4, r1 + 4);
          if (active) *reinterpret_cast<uint2*>(dst(i)) = make_uint2(lo, hi);
        } else {
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float q[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) q[c] = scale_elem<FMT, IN_BF16, FAST>(v[4 * j + c], s);
            o[j] = fp8x2_rtn_hw<F::E5M2>(q[0], q[1]) | (fp8x2_rtn_hw<F::E5M2>(q[2], q[3]) << 16);
          }
          if (active) *reinterpret_cast<uint4*>(dst(i)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      });

      // ---- scales ----
      if (a.scale_plain != nullptr && holder && row_ok(i)) {
        if (F::MX) reinterpret_cast<uint8_t*>(a.scale_plain)[row * nkb + kb] = (uint8_t)s.byte;
        else reinterpret_cast<float*>(a.scale_plain)[row * nkb + kb] = s.plain;
      }
      scale_bytes = merge_shifted((holder && row_ok(i)) ? s.byte : 0u, 8 * i, scale_bytes);
    }
    if constexpr (SHARED) {
      const uint32_t* const at = a.rand_bits + (int64_t)(((uint32_t)row0 % t_rows) * t_pairs + (uint32_t)(col >> 1) % t_pairs);
      with_uniform_fast(all_fast, [&](auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        uint32_t first[ROW_R];
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          uint4 even = make_uint4(0u, 0u, 0u, 0u), odd = even;
          if (col_ok) {
            even = __ldg(reinterpret_cast<const uint4*>(at) + o);
            odd = __ldg(reinterpret_cast<const uint4*>(at + (int64_t)(t_rows * t_pairs)) + o);
          }
          SrOctet words;
          if (FAST) words = sr_octet(even, odd);
#pragma unroll
          for (int i = 0; i < ROW_R; ++i) {
            if (!row_ok(i)) break;
            float v[8];
            if (IN_BF16) {
              const uint32_t w[4] = {raw[i][o].x, raw[i][o].y, raw[i][o].z, raw[i][o].w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                v[2 * j] = bf16lo_to_f32(w[j]);
                v[2 * j + 1] = bf16hi_to_f32(w[j]);
              }
            } else {
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const uint4 w = raw[i][(2 * o + q) % NV];
                v[4 * q] = u2f(w.x); v[4 * q + 1] = u2f(w.y); v[4 * q + 2] = u2f(w.z); v[4 * q + 3] = u2f(w.w);
              }
            }
            uint32_t code;
            if constexpr (FAST) {
              code = fp4_octet_sr<FMT, IN_BF16>(v, scales[i], words);
            } else {
              const uint32_t r0[4] = {even.x, even.y, even.z, even.w}, r1[4] = {odd.x, odd.y, odd.z, odd.w};
              code = fp4_octet<FMT, IN_BF16, ROUND, false>(v, scales[i], r0, r1);
            }
            if (o == 0) first[i] = code;
            else if (col_ok) *reinterpret_cast<uint2*>(dst(i)) = make_uint2(first[i], code);
          }
        }
      });
    }
    // ---- packed scales: four lanes hold four rows of four scale columns each; a 4 x 4 byte transpose in two
    // exchanges leaves each of them one row's word (a word is four scale columns of one row) ----
    if (a.scale_packed != nullptr) {
      const int h = (lane / LPB) & 3;
      uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, scale_bytes, 2 * LPB);
      scale_bytes = __byte_perm(scale_bytes, o, (h & 2) ? 0x3276 : 0x5410);
      o = __shfl_xor_sync(0xFFFFFFFFu, scale_bytes, LPB);
      scale_bytes = __byte_perm(scale_bytes, o, (h & 1) ? 0x3715 : 0x6240);
      const int64_t kb4 = kb - h;
      const int64_t row = row0 + h * step;
      if (lane % LPB == 0 && kb4 < a.ncol_tiles * 4 && row_ok(h))
        *reinterpret_cast<uint32_t*>(a.scale_packed + packed_scale_offset(row, kb4, a.ncol_tiles)) = scale_bytes;
    }
  }
}

// =======================================================================================
// Hadamard helpers (n = 16, Sylvester ordering, in registers)
// =======================================================================================
struct RhtParams {
  int n;           // 0 or 16
  int8_t pinv[16]; // slot k reads row pinv[k] of the block
  float sign[16];  // sign applied to slot k after the butterfly
  int64_t row_off[16];  // byte offset of row pinv[k] from the first row of a 16-row group (column passes)
  float qsign[16];      // sign[k] / sqrt(16): the factor applied to slot k
  uint32_t psel[4], pmask[4];  // output word w of four positions: byte selectors within each half of the slots, half mask
};

__device__ __forceinline__ void hadamard16(float* z) {
#pragma unroll
  for (int h = 1; h < 16; h <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if ((i & h) == 0) {
        const float a = z[i], b = z[i + h];
        z[i] = __fadd_rn(a, b);
        z[i + h] = __fsub_rn(a, b);
      }
    }
  }
}

// The same butterfly on the two columns of a lane at once, as packed fp32 operations (one instruction
// per pair of sums): a - b is fma(b, -1, a), which rounds once like the subtraction.
__device__ __forceinline__ void hadamard16_pair(float* za, float* zb) {
  float2 z[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) z[i] = make_float2(za[i], zb[i]);
  const float2 neg = make_float2(-1.0f, -1.0f);
#pragma unroll
  for (int h = 1; h < 16; h <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if ((i & h) == 0) {
        const float2 a = z[i], b = z[i + h];
        z[i] = __fadd2_rn(a, b);
        z[i + h] = __ffma2_rn(b, neg, a);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    za[i] = z[i].x;
    zb[i] = z[i].y;
  }
}

// =======================================================================================
// Column-wise quantizer (axis 0) with optional Hadamard transform
// =======================================================================================
struct ColwiseArgs {
  const void* x;
  int64_t rows, cols, ld;
  uint8_t* codes;       // [cols, rows/2] or [cols, rows]
  void* scale_plain;    // [cols, rows/B]
  uint8_t* scale_packed;
  int64_t ncol_tiles;   // ceil(rows / B / 4)
  const float* outer;
  const uint32_t* rand_bits;  // [2][cols][rows/2], or a periodic tile [2][tile_rows][tile_pairs]
  int64_t tile_rows, tile_pairs;
  bool rand_vec;              // the words of 16 rows can be read in 16-byte vectors
  uint64_t philox_seed, philox_offset;
  PhiloxKeys pk;
  RhtParams rht;
  MxOpts mx;
  uint8_t* macro_codes;  // MACRO: [cols, ceil(rows / 128)] factor codes, written
  const float* dense;    // DENSE: the 32 x 32 matrix
  float dense_scale;     // DENSE: 1 / sqrt(32)
};

// A warp's 32 rows x 64 columns times the 32 x 32 matrix of +-1, as bf16 words of a lane's two columns by row.  The
// matrix is not of Sylvester type, so there is no butterfly: mma.sync on a tile in shared memory, as in
// csrc/rht_dense.cu and with its roundings.  Here it spares that kernel's pass over memory.  Bound by issue slots
// behind the loads, which is why all of them are asked for before anything else (176 us without).  With macro blocks:
// 69 632 x 2880 RTN 167 + 110 us (transform, then quantizer) -> 165 us, 5760 columns with random words 329 + 366 -> 508.
constexpr int DENSE_PITCH = 64 * 2 + 16;   // bytes per tile row: rows 16 bytes apart modulo 128
__device__ __forceinline__ void dense32_words(const uint8_t* src, int64_t pitch, int n_cols, bool rows_ok, const float* w,
                                              float scale, uint8_t* tile, int lane, uint32_t* words) {
  uint4 raw[8];
  {
    const bool ok = rows_ok && (lane & 7) * 8 < n_cols;
    const uint8_t* p = src + (lane >> 3) * pitch + (lane & 7) * 16;
#pragma unroll
    for (int i = 0; i < 8; ++i, p += 4 * pitch) raw[i] = ok ? __ldg(reinterpret_cast<const uint4*>(p)) : make_uint4(0u, 0u, 0u, 0u);
  }
  uint32_t fa[2][2][4];   // A fragments of the matrix (16 x 16 tiles)
  {
    const int r = lane >> 2, c2 = 2 * (lane & 3);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int kt = 0; kt < 2; ++kt)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = __ldg(reinterpret_cast<const float2*>(w + (mt * 16 + r + 8 * (q & 1)) * 32 + kt * 16 + c2 + 8 * (q >> 1)));
          const __nv_bfloat162 p2 = __floats2bfloat162_rn(f.x, f.y);
          fa[mt][kt][q] = *reinterpret_cast<const uint32_t*>(&p2);
        }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(tile + (i * 4 + (lane >> 3)) * DENSE_PITCH + (lane & 7) * 16) = raw[i];
  __syncwarp();
  const uint32_t tile_s = (uint32_t)__cvta_generic_to_shared(tile);
#pragma unroll
  for (int t = 0; t < 8; ++t) {                // 8 columns
    uint32_t b[4];                             // rows 0-15, 16-31
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(tile_s + (uint32_t)lane * DENSE_PITCH + t * 16)
                 : "memory");
    float acc[2][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.0f;
#pragma unroll
      for (int kt = 0; kt < 2; ++kt)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(acc[mt][0]), "+f"(acc[mt][1]), "+f"(acc[mt][2]), "+f"(acc[mt][3])
                     : "r"(fa[mt][kt][0]), "r"(fa[mt][kt][1]), "r"(fa[mt][kt][2]), "r"(fa[mt][kt][3]),
                       "r"(b[2 * kt]), "r"(b[2 * kt + 1]));
    }
    __syncwarp();   // every lane's fragment of these columns has been read
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // the fused +0 turns the product of a -0 sum into +0, as the matmul's accumulation from zero does
        const float2 y = __ffma2_rn(make_float2(acc[mt][2 * h], acc[mt][2 * h + 1]), make_float2(scale, scale), make_float2(0.0f, 0.0f));
        const __nv_bfloat162 p2 = __floats2bfloat162_rn(y.x, y.y);
        *reinterpret_cast<uint32_t*>(tile + (mt * 16 + (lane >> 2) + 8 * h) * DENSE_PITCH + t * 16 + (lane & 3) * 4) =
            *reinterpret_cast<const uint32_t*>(&p2);
      }
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 32; ++k) words[k] = *reinterpret_cast<const uint32_t*>(tile + k * DENSE_PITCH + lane * 4);
}

// Threads per CTA = rows per CTA tile.  128 rather than 256: more, smaller CTAs per SM, so that the start-up
// loads and the barrier of one overlap the arithmetic of the others.
constexpr int COL_NT = 128;
constexpr int COL_TN = 64;   // columns per CTA tile

// What bounds the kernel is the integer pipe, so codes are never handled one by one: the converter packs the
// codes of a lane's two columns into one byte, four slots into one word; the output permutation of the
// Hadamard transform moves those bytes (three instructions for four positions of both columns), and the two
// columns are separated eight codes at a time.  The random words of stochastic rounding belong to output
// positions: with ROUND_SR_SLOTS the table is laid out by slot (altob200_philox_slots), so that the codes can
// be made in slot order and neighbouring lanes read neighbouring words.
// MACRO (MXFP4 from bf16): the two-level recipe's scaling runs in front of the quantisation - a CTA tile is one
// macro block of 128 rows per column, so its maxima only have to cross the four warps.
// DENSE (MXFP4 from bf16, no RHT): the dense transform of 32 rows runs in front of all that.
template <int FMT, bool IN_BF16, int ROUND, bool RHT, bool MACRO, bool DENSE = false>
// (fp32 blocks of 32 with words by position are held to the 128 registers of four CTAs an SM: 63 -> 58 us for
// 8192 x 4096; drawn in the kernel, only behind the transform, 24.0 -> 22.6 us for 4096 x 2880 (without it 5.2 -> 5.4
// for 512 x 4096); 0 leaves the others to the compiler)
__global__ void __launch_bounds__(COL_NT, !IN_BF16 && Fmt<FMT>::B == 32 &&
                                  (ROUND == ALTOB200_ROUND_SR_BITS || (ROUND == ALTOB200_ROUND_SR_PHILOX && RHT)) ? 4 : 0)
quantize_colwise_kernel(ColwiseArgs a) {
  grid_dependency_wait();
  using F = Fmt<FMT>;
  constexpr int B = F::B;
  constexpr int NT = COL_NT;   // threads per CTA
  constexpr int WARPS = NT / 32;
  constexpr int COL_TM = NT;               // rows per CTA tile
  constexpr int NBLK = COL_TM / B;          // row blocks per tile (8 or 4)
  constexpr int ITERS = NBLK / WARPS;       // per warp
  constexpr int ROW_BYTES = F::FP4 ? COL_TM / 2 : COL_TM;  // bytes per output row per tile
  constexpr int BLK_BYTES = F::FP4 ? B / 2 : B;            // bytes per block per column
  static_assert(!MACRO || (FMT == ALTOB200_FMT_MXFP4 && IN_BF16 && COL_TM == 128 && ITERS == 1), "macro blocks");
  static_assert(!DENSE || (IN_BF16 && B == 32 && ITERS == 1 && !RHT && COL_TN == 64), "a warp's rows are a block of the transform");
  __shared__ __align__(16) uint8_t s_dense[DENSE ? WARPS : 1][DENSE ? 32 * DENSE_PITCH : 16];
  // codes staged as [block][column][BLK_BYTES]; scales as [column][NBLK]
  __shared__ __align__(16) uint8_t s_codes[COL_TN * ROW_BYTES];
  __shared__ __align__(16) uint8_t s_sf[COL_TN * NBLK];
  __shared__ float s_sf_plain[Fmt<FMT>::MX ? 1 : COL_TN * NBLK];
  // words that come in position order: the values of a thread's two columns are moved there from slot order
  constexpr bool TO_POS = RHT && (ROUND == ALTOB200_ROUND_SR_PHILOX || ROUND == ALTOB200_ROUND_SR_BITS);
  using Pair = typename std::conditional<IN_BF16, uint32_t, float2>::type;
  __shared__ Pair s_pos[TO_POS ? 16 : 1][NT];
  __shared__ uint32_t s_macro[MACRO ? WARPS : 1][32];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t m0 = (int64_t)blockIdx.y * COL_TM;
  const int64_t n0 = (int64_t)blockIdx.x * COL_TN;
  const int64_t c = n0 + 2 * lane;  // first of this lane's two columns
  const bool col_ok = c < a.cols;   // cols is even, so c+1 is valid too
  const OuterScale os = make_outer_scale((!F::MX) && a.outer != nullptr, a.outer);
  const int64_t half_rows = a.rows >> 1;
  // rows of the periodic random table for this lane's two columns (rows of the axis-last view)
  // (32-bit arithmetic: with a periodic table the host refuses extents of 2^32 and more; a 64-bit
  // modulo is ~70 instructions, several per thread of a CTA that handles 64 elements per thread)
  const uint32_t tile_row0 = a.tile_rows != 0 ? (uint32_t)c % (uint32_t)a.tile_rows : 0u;
  const uint32_t tile_row1 = a.tile_rows != 0 ? (tile_row0 + 1u == (uint32_t)a.tile_rows ? 0u : tile_row0 + 1u) : 0u;

  // bf16: the words of every iteration are requested before the first is used (slot k <- row pinv[k]
  // when the transform is on; the identity otherwise), so the second block's loads fly under the
  // first block's arithmetic
  constexpr int ESZ = IN_BF16 ? 2 : 4;
  const int64_t half_blk = 16 * a.ld * ESZ;  // second 16-row group of a 32-row block
  uint32_t pre[IN_BF16 ? ITERS : 1][IN_BF16 ? B : 1];
  if constexpr (DENSE) {
    const int64_t mb = m0 + (int64_t)warp * B;
    const int64_t n_cols = a.cols - n0;
    dense32_words(reinterpret_cast<const uint8_t*>(a.x) + (mb * a.ld + n0) * ESZ, a.ld * ESZ,
                  (int)(n_cols < COL_TN ? n_cols : COL_TN), mb < a.rows, a.dense, a.dense_scale, s_dense[warp], lane, pre[0]);
  } else if (IN_BF16) {
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
      const int64_t mb = m0 + (int64_t)(warp + WARPS * it) * B;
      const bool ok = col_ok && mb < a.rows;
      const uint8_t* base = reinterpret_cast<const uint8_t*>(a.x) + (mb * a.ld + c) * ESZ;
#pragma unroll
      for (int k = 0; k < B; ++k)
        pre[it % (IN_BF16 ? ITERS : 1)][k % (IN_BF16 ? B : 1)] =
            ok ? __ldg(reinterpret_cast<const uint32_t*>(base + a.rht.row_off[k & 15] + (k >= 16 ? half_blk : 0))) : 0u;
    }
  }

#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int blk = warp + WARPS * it;
    const int64_t mb = m0 + (int64_t)blk * B;
    const bool ok = col_ok && mb < a.rows;  // rows % B == 0
    // bf16: both columns of a slot travel as one packed pair (pw); fp32: as two floats (v0, v1)
    uint32_t pw[IN_BF16 ? B : 1];
    float v0[IN_BF16 ? 16 : B], v1[IN_BF16 ? 16 : B];
    uint32_t am0 = 0, am1 = 0;   // block maxima of |x|, bits of the input type
    if (IN_BF16) {
      uint32_t acc = 0;
#pragma unroll
      for (int g = 0; g < B; g += 16) {
        uint32_t* w = pw + (IN_BF16 ? g : 0);
#pragma unroll
        for (int k = 0; k < 16; ++k) w[k % (IN_BF16 ? 16 : 1)] = pre[it % (IN_BF16 ? ITERS : 1)][(g + k) % (IN_BF16 ? B : 1)];
        if (RHT) {
          // y = (H z) / sqrt(16), rounded to bf16: one conversion per pair
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            v0[k] = bf16lo_to_f32(w[k % (IN_BF16 ? 16 : 1)]);
            v1[k] = bf16hi_to_f32(w[k % (IN_BF16 ? 16 : 1)]);
          }
          hadamard16_pair(v0, v1);
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            // the fused +0 turns a -0 product into the +0 that a dot product yields
            const float sg = a.rht.qsign[k];
            const float2 sc = __ffma2_rn(make_float2(v0[k], v1[k]), make_float2(sg, sg), make_float2(0.0f, 0.0f));
            const __nv_bfloat162 p2 = __floats2bfloat162_rn(sc.x, sc.y);
            w[k % (IN_BF16 ? 16 : 1)] = *reinterpret_cast<const uint32_t*>(&p2);
          }
        }
#pragma unroll
        for (int k = 0; k < 16; k += 2)
          acc = absmax2_bf16x2(acc, w[k % (IN_BF16 ? 16 : 1)], w[(k + 1) % (IN_BF16 ? 16 : 1)]);
      }
      if (MACRO) {
        // factor of the column's 128 rows (csrc/macro_scale.cu), then y = bf16(x * factor); rounding is
        // monotone, so the block maximum is scaled instead of searched again
        s_macro[MACRO ? warp : 0][lane] = acc;
        __syncthreads();
        uint32_t m = s_macro[0][lane];
#pragma unroll
        for (int w = 1; w < (MACRO ? WARPS : 1); ++w) m = __vmaxu2(m, s_macro[w][lane]);
        uint32_t code0, code1;
        const float f0 = macro_factor_from_amax(bf16lo_to_f32(m), &code0);
        const float f1 = macro_factor_from_amax(bf16hi_to_f32(m), &code1);
        if (warp == 0 && col_ok) {
          uint8_t* dst = a.macro_codes + c * gridDim.y + blockIdx.y;
          dst[0] = (uint8_t)code0;
          dst[gridDim.y] = (uint8_t)code1;
        }
        auto scaled = [&](uint32_t w) {
          const __nv_bfloat162 p2 = __floats2bfloat162_rn(__fmul_rn(bf16lo_to_f32(w), f0), __fmul_rn(bf16hi_to_f32(w), f1));
          return *reinterpret_cast<const uint32_t*>(&p2);
        };
        acc = scaled(acc) & 0x7FFF7FFFu;
#pragma unroll
        for (int k = 0; k < B; ++k) pw[k % (IN_BF16 ? B : 1)] = scaled(pw[k % (IN_BF16 ? B : 1)]);
      }
      am0 = acc & 0xFFFFu;
      am1 = acc >> 16;
    } else {
      const uint8_t* base = reinterpret_cast<const uint8_t*>(a.x) + (mb * a.ld + c) * ESZ;
#pragma unroll
      for (int k = 0; k < B; ++k) {
        float2 f = make_float2(0.f, 0.f);
        if (ok) f = __ldg(reinterpret_cast<const float2*>(base + a.rht.row_off[k & 15] + (k >= 16 ? half_blk : 0)));
        v0[k % (IN_BF16 ? 16 : B)] = f.x;
        v1[k % (IN_BF16 ? 16 : B)] = f.y;
      }
      if (RHT) {
#pragma unroll
        for (int g = 0; g < (IN_BF16 ? 16 : B); g += 16) hadamard16_pair(v0 + g, v1 + g);
#pragma unroll
        for (int k = 0; k < (IN_BF16 ? 16 : B); ++k) {
          const float sg = a.rht.qsign[k & 15];
          v0[k] = __fmaf_rn(v0[k], sg, 0.0f);
          v1[k] = __fmaf_rn(v1[k], sg, 0.0f);
        }
      }
#pragma unroll
      for (int k = 0; k < (IN_BF16 ? 16 : B); ++k) {
        const uint32_t b0 = f2u(v0[k]) & 0x7FFFFFFFu, b1 = f2u(v1[k]) & 0x7FFFFFFFu;
        am0 = b0 > am0 ? b0 : am0;
        am1 = b1 > am1 ? b1 : am1;
      }
    }
    // static clip (MXFP4): bf16 elements are clipped where they are read, fp32 ones in place (the test in the
    // element loop cost every fp32 launch 4 to 6 %, FP8 too; in place costs bf16 16 registers, 2 % of a large tensor)
    const bool clip = F::FP4 && F::MX && IN_BF16 && a.mx.clip == 1;
    // the two elements of slot k
    auto slot = [&](int k) -> float2 {
      float2 x = IN_BF16 ? make_float2(bf16lo_to_f32(pw[k % (IN_BF16 ? B : 1)]), bf16hi_to_f32(pw[k % (IN_BF16 ? B : 1)]))
                         : make_float2(v0[k % (IN_BF16 ? 16 : B)], v1[k % (IN_BF16 ? 16 : B)]);
      if (clip) x = make_float2(round_in<IN_BF16>(__fmul_rn(x.x, 0.75f)), round_in<IN_BF16>(__fmul_rn(x.y, 0.75f)));
      return x;
    };
    // slot order -> position order through a private column of shared memory (moving the words instead, behind
    // their loads, takes 20 % longer)
    auto to_positions = [&]() {
#pragma unroll
      for (int g = 0; g < B; g += 16) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          Pair& dst = s_pos[TO_POS ? a.rht.pinv[k] : 0][threadIdx.x];
          if constexpr (IN_BF16) dst = pw[g + k];
          else dst = make_float2(v0[g + k], v1[g + k]);
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const Pair src = s_pos[TO_POS ? k : 0][threadIdx.x];
          if constexpr (IN_BF16) pw[g + k] = src;
          else { v0[g + k] = src.x; v1[g + k] = src.y; }
        }
      }
    };
    // (the statistics of the dynamic clip are summed in slot order)
    if (TO_POS && !F::MX) to_positions();
    BlockScale s0, s1;
    if (F::MX && (a.mx.clip | a.mx.uos)) {
      float sum0 = 0.0f, sq0 = 0.0f, sum1 = 0.0f, sq1 = 0.0f;
      if (a.mx.clip == 2) {
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const float2 x = slot(k);
          sum0 = __fadd_rn(sum0, x.x);
          sq0 = __fadd_rn(sq0, round_in<IN_BF16>(__fmul_rn(x.x, x.x)));
          sum1 = __fadd_rn(sum1, x.y);
          sq1 = __fadd_rn(sq1, round_in<IN_BF16>(__fmul_rn(x.y, x.y)));
        }
      }
      s0 = make_block_scale_opts<FMT, IN_BF16>(am0, sum0, sq0, B, a.mx);
      s1 = make_block_scale_opts<FMT, IN_BF16>(am1, sum1, sq1, B, a.mx);
      if (F::FP4 && !IN_BF16 && a.mx.clip == 1) {
#pragma unroll
        for (int k = 0; k < (IN_BF16 ? 16 : B); ++k) {
          v0[k] = __fmul_rn(v0[k], 0.75f);
          v1[k] = __fmul_rn(v1[k], 0.75f);
        }
      }
    } else {
      s0 = make_block_scale<FMT, IN_BF16>(am0, os);
      s1 = make_block_scale<FMT, IN_BF16>(am1, os);
    }
    const bool fast = block_fast<IN_BF16, ROUND>(s0, am0) && block_fast<IN_BF16, ROUND>(s1, am1);
    if (TO_POS && F::MX) to_positions();

    // ---- quantise in slot order (position order after the move) ----
    if (F::FP4) {
#pragma unroll
      for (int h = 0; h < B / 16; ++h) {
        // random words in the order of the values: r[k] for columns c and c + 1
        uint2 r[ROUND == ALTOB200_ROUND_RTN ? 1 : 16];
        if (ROUND == ALTOB200_ROUND_SR_SLOTS) {
          // [64 positions, slot order within groups of 16][64 columns]
          const uint2* t = reinterpret_cast<const uint2*>(a.rand_bits + ((uint32_t)(mb + 16 * h) & 63u) * 64u + tile_row0);
#pragma unroll
          for (int k = 0; k < 16; ++k) r[k % (ROUND == ALTOB200_ROUND_RTN ? 1 : 16)] = __ldg(t + 32 * k);
        } else if (ROUND == ALTOB200_ROUND_SR_BITS) {
          // by position: the 8 pairs of these 16 rows are 8 words of either plane, consecutive and 32-byte aligned
          // unless the caller's table says otherwise (rand_vec).  NVFP4 bf16 8192 x 4096 with the transform, periodic
          // table / full planes: 62 / 61 us; with one 4-byte load (and one modulo) a word 144 / 166
          const bool tiled = a.tile_rows != 0;
          const int64_t idx = (mb + 16 * h) >> 1;
          const int64_t pitch = tiled ? a.tile_pairs : half_rows;
          const int64_t plane = (tiled ? a.tile_rows : a.cols) * pitch;
          const uint32_t* t0 = a.rand_bits + (tiled ? (int64_t)tile_row0 : c) * pitch;
          const uint32_t* t1 = a.rand_bits + (tiled ? (int64_t)tile_row1 : c + 1) * pitch;
          if (!ok) {
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i % (ROUND == ALTOB200_ROUND_RTN ? 1 : 16)] = make_uint2(0u, 0u);
          } else if (a.rand_vec) {
            const int64_t p = tiled ? (int64_t)((uint32_t)idx % (uint32_t)a.tile_pairs) : idx;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
              for (int odd = 0; odd < 2; ++odd) {
                const uint4 w0 = __ldg(reinterpret_cast<const uint4*>(t0 + odd * plane + p) + q);
                const uint4 w1 = __ldg(reinterpret_cast<const uint4*>(t1 + odd * plane + p) + q);
                const uint32_t u0[4] = {w0.x, w0.y, w0.z, w0.w}, u1[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  r[(8 * q + 2 * j + odd) % (ROUND == ALTOB200_ROUND_RTN ? 1 : 16)] = make_uint2(u0[j], u1[j]);
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int64_t pair = idx + (i >> 1);
              const int64_t p = (i & 1) * plane + (tiled ? (int64_t)((uint32_t)pair % (uint32_t)a.tile_pairs) : pair);
              r[i % (ROUND == ALTOB200_ROUND_RTN ? 1 : 16)] = make_uint2(__ldg(t0 + p), __ldg(t1 + p));
            }
          }
        } else if (ROUND == ALTOB200_ROUND_SR_PHILOX) {
          const uint64_t p0 = (uint64_t)(c * half_rows + ((mb + 16 * h) >> 1));        // pair index, column c
          const uint64_t p1 = (uint64_t)((c + 1) * half_rows + ((mb + 16 * h) >> 1));  // column c + 1
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t o0[4], o1[4];
            uint64_t ctr = a.philox_offset + (p0 >> 1) + i;
            philox4x32_10_keys((uint32_t)ctr, (uint32_t)(ctr >> 32), a.pk, o0);
            ctr = a.philox_offset + (p1 >> 1) + i;
            philox4x32_10_keys((uint32_t)ctr, (uint32_t)(ctr >> 32), a.pk, o1);
#pragma unroll
            for (int q = 0; q < 4; ++q) r[(4 * i + q) % (ROUND == ALTOB200_ROUND_RTN ? 1 : 16)] = make_uint2(o0[q], o1[q]);
          }
        }
        // byte k % 4 of word k / 4: code of slot k, column c in the low nibble and c + 1 in the high one
        uint32_t by_slot[4];
        with_uniform_fast(fast, [&](auto fast_tag) {
          constexpr bool FAST = decltype(fast_tag)::value;
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            float q[8], sgn[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 x = slot(16 * h + 4 * w + j);
              q[2 * j] = scale_elem<FMT, IN_BF16, FAST>(x.x, s0);
              q[2 * j + 1] = scale_elem<FMT, IN_BF16, FAST>(x.y, s1);
              sgn[2 * j] = x.x;
              sgn[2 * j + 1] = x.y;
            }
            if (ROUND == ALTOB200_ROUND_RTN) {
              by_slot[w] = e2m1x8_rtn_hw(q);
            } else if (FAST) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint2 rw = r[(4 * w + j) % (ROUND == ALTOB200_ROUND_RTN ? 1 : 16)];
                q[2 * j] = e2m1_sr_value(q[2 * j], rw.x);
                q[2 * j + 1] = e2m1_sr_value(q[2 * j + 1], rw.y);
              }
              by_slot[w] = e2m1x8_rtn_hw(q);
            } else {
              by_slot[w] = 0u;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint2 rw = r[(4 * w + j) % (ROUND == ALTOB200_ROUND_RTN ? 1 : 16)];
                by_slot[w] = merge_shifted(e2m1_sr_code(q[2 * j], f2u(sgn[2 * j]), rw.x), 8 * j, by_slot[w]);
                by_slot[w] = merge_shifted(e2m1_sr_code(q[2 * j + 1], f2u(sgn[2 * j + 1]), rw.y), 8 * j + 4, by_slot[w]);
              }
            }
          }
        });
        uint32_t u0[4], u1[4];   // bytes 0 and 2: two positions of column c / c + 1
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t o = by_slot[w];
          if (RHT && !TO_POS) {   // output position i takes slot perm[i]
            const uint32_t lo = __byte_perm(by_slot[0], by_slot[1], a.rht.psel[w]);
            const uint32_t hi = __byte_perm(by_slot[2], by_slot[3], a.rht.psel[w]);
            o = (lo & ~a.rht.pmask[w]) | (hi & a.rht.pmask[w]);
          }
          const uint32_t o4 = o >> 4, o8 = o >> 8;
          u0[w] = (o & 0x0F0F0F0Fu) | (o4 & 0xF0F0F0F0u);
          u1[w] = (o4 & 0x0F0F0F0Fu) | (o8 & 0xF0F0F0F0u);
        }
        uint8_t* d = s_codes + ((size_t)blk * COL_TN + 2 * lane) * BLK_BYTES + 8 * h;
        *reinterpret_cast<uint2*>(d) = make_uint2(__byte_perm(u0[0], u0[1], 0x6420), __byte_perm(u0[2], u0[3], 0x6420));
        *reinterpret_cast<uint2*>(d + BLK_BYTES) = make_uint2(__byte_perm(u1[0], u1[1], 0x6420), __byte_perm(u1[2], u1[3], 0x6420));
      }
    } else {
      // FP8: one byte per element, no transform (the reference asserts that MXFP8 runs
      // without Hadamard, alto/kernels/dispatch/tensor.py:448-454)
      uint8_t* d = s_codes + ((size_t)blk * COL_TN + 2 * lane) * BLK_BYTES;
      with_uniform_fast(s0.fast && s1.fast, [&](auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
#pragma unroll
        for (int k = 0; k < B; k += 4) {
          float q0[4], q1[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 x = slot(k + j);
            q0[j] = scale_elem<FMT, IN_BF16, FAST>(x.x, s0);
            q1[j] = scale_elem<FMT, IN_BF16, FAST>(x.y, s1);
          }
          *reinterpret_cast<uint32_t*>(d + k) = fp8x2_rtn_hw<F::E5M2>(q0[0], q0[1]) |
                                                (fp8x2_rtn_hw<F::E5M2>(q0[2], q0[3]) << 16);
          *reinterpret_cast<uint32_t*>(d + BLK_BYTES + k) =
              fp8x2_rtn_hw<F::E5M2>(q1[0], q1[1]) | (fp8x2_rtn_hw<F::E5M2>(q1[2], q1[3]) << 16);
        }
      });
    }
    s_sf[(2 * lane) * NBLK + blk] = ok ? (uint8_t)s0.byte : 0;
    s_sf[(2 * lane + 1) * NBLK + blk] = ok ? (uint8_t)s1.byte : 0;
    if (!F::MX) {
      s_sf_plain[(2 * lane) * NBLK + blk] = s0.plain;
      s_sf_plain[(2 * lane + 1) * NBLK + blk] = s1.plain;
    }
  }
  __syncthreads();

  // ---- write codes: output row n gets ROW_BYTES contiguous bytes, 16 bytes per thread ----
  constexpr int CHUNKS = ROW_BYTES / 16;  // 8 (FP4) or 16 (FP8) per output row
  for (int t = threadIdx.x; t < COL_TN * CHUNKS; t += NT) {
    const int n = t / CHUNKS, ch = t - n * CHUNKS;
    const int64_t col = n0 + n;
    const int64_t mrow = m0 + (int64_t)ch * (F::FP4 ? 32 : 16);  // first row covered by this chunk
    if (col >= a.cols || mrow >= a.rows) continue;
    // a 16-byte chunk covers 32 rows (FP4) or 16 rows (FP8)
    uint4 o;
    if (BLK_BYTES >= 16) {
      const int blk = (ch * 16) / BLK_BYTES, off = (ch * 16) % BLK_BYTES;
      o = *reinterpret_cast<const uint4*>(s_codes + ((size_t)blk * COL_TN + n) * BLK_BYTES + off);
    } else {  // BLK_BYTES == 8: two blocks per chunk
      const uint2 lo = *reinterpret_cast<const uint2*>(s_codes + ((size_t)(2 * ch) * COL_TN + n) * 8);
      const uint2 hi = *reinterpret_cast<const uint2*>(s_codes + ((size_t)(2 * ch + 1) * COL_TN + n) * 8);
      o = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
    uint8_t* dst = a.codes + col * (F::FP4 ? half_rows : a.rows) + (F::FP4 ? (m0 >> 1) : m0) + ch * 16;
    const int64_t rows_left = a.rows - mrow;
    if (rows_left >= (F::FP4 ? 32 : 16)) {
      *reinterpret_cast<uint4*>(dst) = o;
    } else {  // ragged tail: rows_left is a multiple of B = 16 here (NVFP4 only)
      *reinterpret_cast<uint2*>(dst) = make_uint2(o.x, o.y);
    }
  }
  // ---- write scales ----
  const int64_t nkb = a.rows / B;
  if (a.scale_plain != nullptr) {
    for (int t = threadIdx.x; t < COL_TN * NBLK; t += NT) {
      const int n = t / NBLK, b = t - n * NBLK;
      const int64_t col = n0 + n, kb = m0 / B + b;
      if (col < a.cols && kb < nkb) {
        if (F::MX) reinterpret_cast<uint8_t*>(a.scale_plain)[col * nkb + kb] = s_sf[n * NBLK + b];
        else reinterpret_cast<float*>(a.scale_plain)[col * nkb + kb] = s_sf_plain[n * NBLK + b];
      }
    }
  }
  if (a.scale_packed != nullptr) {
    for (int t = threadIdx.x; t < COL_TN * (NBLK / 4); t += NT) {
      const int n = t / (NBLK / 4), qd = t - n * (NBLK / 4);
      const int64_t col = n0 + n, kb = m0 / B + qd * 4;
      if (col < a.cols && kb < a.ncol_tiles * 4) {
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (kb + j < nkb) word |= (uint32_t)s_sf[n * NBLK + qd * 4 + j] << (8 * j);
        *reinterpret_cast<uint32_t*>(a.scale_packed + packed_scale_offset(col, kb, a.ncol_tiles)) = word;
      }
    }
  }
}

// =======================================================================================
// 2D block quantizer with dual packing
// =======================================================================================
struct Quant2dArgs {
  const void* w;
  int64_t rows, cols, ld;
  uint8_t* codes_k;   // [rows, cols/2] or [rows, cols]
  uint8_t* codes_t;   // [cols, rows/2] or [cols, rows]
  void* scale_plain;  // [rows/B, cols/B]
  uint8_t* packed_k;  // rows=rows, ncols=cols/B
  uint8_t* packed_t;  // rows=cols, ncols=rows/B
  int64_t nct_k, nct_t;
  const float* outer;
  MxOpts mx;          // clip 0/1/2 and uos
  // stochastic rounding (FP4): words by (row, pair of columns) as in the row-wise quantizer: full planes
  // [2][rows][cols/2], or a periodic table [2][tile_rows][tile_pairs]
  const uint32_t* rand_bits;
  int64_t tile_rows, tile_pairs;
  // batch of equally shaped matrices: input stride in elements, outputs stacked contiguously; the
  // rows of the stochastic-rounding view are the rows of all matrices, one after the other
  int64_t batch, batch_stride, packed_k_bytes, packed_t_bytes;
  uint8_t* macro_codes;  // MACRO: [batch, ceil(rows / 128), ceil(cols / 128)] factor codes, written
};

// 4 x 4 byte transpose: out[b] = (in[0].byte b, in[1].byte b, in[2].byte b, in[3].byte b)
__device__ __forceinline__ void transpose4x4_bytes(const uint32_t* in, uint32_t* out) {
  const uint32_t t0 = __byte_perm(in[0], in[1], 0x5140);  // a0 b0 a1 b1
  const uint32_t t1 = __byte_perm(in[2], in[3], 0x5140);  // c0 d0 c1 d1
  const uint32_t t2 = __byte_perm(in[0], in[1], 0x7362);  // a2 b2 a3 b3
  const uint32_t t3 = __byte_perm(in[2], in[3], 0x7362);  // c2 d2 c3 d3
  out[0] = __byte_perm(t0, t1, 0x5410);
  out[1] = __byte_perm(t0, t1, 0x7632);
  out[2] = __byte_perm(t2, t3, 0x5410);
  out[3] = __byte_perm(t2, t3, 0x7632);
}

// A thread owns 16 rows x 8 columns, kept in registers from the load to both stores; a warp owns LC x LR
// threads, whole blocks either way, so block maxima need shuffles only and the kernel uses no shared memory.
// The K packing is written row by row (4 or 8 bytes per row per lane, 32 or 128 contiguous bytes per row
// per warp); for the transposed packing the thread's 16 x 8 codes are
// transposed in registers (nibble merge of row pairs, then 4 x 4 byte transposes) and every column
// receives 8 (FP4) or 16 (FP8) contiguous bytes per lane, 32 contiguous bytes per warp and column (MXFP4 with
// warps of 32 x 128, 16 bytes a column, half sectors: 78 us for 8192 x 14336 against 56).
// MACRO (MXFP4 from bf16): the two-level recipe's scaling of 128 x 128 tiles runs in front of the quantisation;
// a tile is the four warps of a CTA, whose maxima meet in shared memory.
// CTAs of 128 threads, five of them an SM (four with the words of stochastic rounding): with 256 threads and 105
// registers two were resident and waited for their slowest warp.  8192 x 14336: NVFP4 73 -> 60 us, fp32
// (x 4096) 46 -> 39; two-level MXFP4, with the warp tile above, 90 -> 67.
constexpr int WARPS_2D = 4;
template <int FMT, bool IN_BF16, int ROUND, bool BATCHED, bool MACRO>
__global__ void __launch_bounds__(WARPS_2D * 32, ROUND == ALTOB200_ROUND_RTN ? 5 : 4) quantize_2d_kernel(Quant2dArgs a) {
  grid_dependency_wait();
  using F = Fmt<FMT>;
  constexpr int B = F::B;
  constexpr int LC = F::FP4 ? 8 : 16;  // lanes across columns, 8 columns each
  constexpr int LR = 32 / LC;          // 16-row groups per warp
  constexpr int TR = 16 * LR, TC = 8 * LC;  // warp tile: 64 x 64 (FP4) or 32 x 128: 32-byte sectors in both packings
  constexpr int ESZ = IN_BF16 ? 2 : 4;
  const int lane = threadIdx.x & 31;
  static_assert(!MACRO || (FMT == ALTOB200_FMT_MXFP4 && IN_BF16 && TR == 64 && TC == 64), "macro tiles");
  // MACRO: the four warps of a CTA take one macro tile, 2 x 2; tiles_r x tiles_c counts macro tiles then
  constexpr int PER = MACRO ? 2 : 1;   // warp tiles per counted tile in either direction
  const int64_t tiles_c = (a.cols + TC * PER - 1) / (TC * PER), tiles_r = (a.rows + TR * PER - 1) / (TR * PER);
  const int64_t warp_all = (int64_t)blockIdx.x * WARPS_2D + (threadIdx.x >> 5);
  // from the end, where the pass before (the maximum of the tensor) left what L2 holds
  const int64_t tile_all = tiles_c * tiles_r * a.batch - 1 - (MACRO ? warp_all >> 2 : warp_all);
  // (whole warps leave, with MACRO whole CTAs)
  if (tile_all < 0) return;
  // matrix `bi` of the batch: its outputs follow those of matrix bi - 1, so the batch index enters the
  // addresses as extra rows (bi * rows for the K packing, bi * cols for the transposed one)
  // (BATCHED is a template parameter so that the single-matrix kernel carries none of this arithmetic)
  int64_t bi = 0, tile = tile_all;
  if (BATCHED) divmod_fast(tile_all, tiles_c * tiles_r, &bi, &tile);
  const int64_t rows_before = BATCHED ? bi * a.rows : 0, cols_before = BATCHED ? bi * a.cols : 0;
  int64_t tr, tc;
  divmod_fast(tile, tiles_c, &tr, &tc);
  const int64_t macro_tile = (bi * tiles_r + tr) * tiles_c + tc;
  if (MACRO) {
    tr = tr * 2 + ((threadIdx.x >> 6) & 1);
    tc = tc * 2 + ((threadIdx.x >> 5) & 1);
  }
  const int lc = lane % LC, lr = lane / LC;
  const int64_t row0 = tr * TR + lr * 16, col0 = tc * TC + lc * 8;
  const bool ok = row0 < a.rows && col0 < a.cols;  // rows % B == 0 and cols % B == 0
  const OuterScale os = make_outer_scale((!F::MX) && a.outer != nullptr, a.outer);
  const uint8_t* src = reinterpret_cast<const uint8_t*>(a.w) + (bi * a.batch_stride + row0 * a.ld + col0) * ESZ;
  const int64_t pitch = a.ld * ESZ;

  // ---- load and block maximum ----
  uint4 raw[IN_BF16 ? 16 : 1];  // bf16: the 16 x 8 elements stay in registers; fp32: rows are read again
  uint32_t amax_bits = 0;
  // the dynamic clip (MX formats) takes the block's sum and sum of squares instead of its maximum
  const bool stats = F::MX && a.mx.clip == 2;
  float sum = 0.0f, sumsq = 0.0f;
  if (IN_BF16) {
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      raw[i] = ok ? __ldg(reinterpret_cast<const uint4*>(src + i * pitch)) : make_uint4(0u, 0u, 0u, 0u);
      acc = absmax2_bf16x2(absmax2_bf16x2(acc, raw[i].x, raw[i].y), raw[i].z, raw[i].w);
    }
    amax_bits = fold_bf16x2(acc);
    if (MACRO) {
      __shared__ uint32_t s_macro[WARPS_2D];
      const uint32_t wm = warp_max_u32(amax_bits);
      const int warp = threadIdx.x >> 5;
      if (lane == 0) s_macro[warp] = wm;
      __syncthreads();
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < WARPS_2D; ++i) m = s_macro[i] > m ? s_macro[i] : m;
      uint32_t code;
      const float f = macro_factor_from_amax(u2f(m << 16), &code);
      if (threadIdx.x == 0) a.macro_codes[macro_tile] = (uint8_t)code;
      // y = bf16(x * factor); rounding is monotone, so the maximum is scaled instead of searched again
      auto scaled = [&](uint32_t w) {
        const __nv_bfloat162 p2 = __floats2bfloat162_rn(__fmul_rn(bf16lo_to_f32(w), f), __fmul_rn(bf16hi_to_f32(w), f));
        return *reinterpret_cast<const uint32_t*>(&p2);
      };
#pragma unroll
      for (int i = 0; i < 16; ++i)
        raw[i % (IN_BF16 ? 16 : 1)] = make_uint4(scaled(raw[i % (IN_BF16 ? 16 : 1)].x), scaled(raw[i % (IN_BF16 ? 16 : 1)].y),
                                                 scaled(raw[i % (IN_BF16 ? 16 : 1)].z), scaled(raw[i % (IN_BF16 ? 16 : 1)].w));
      amax_bits = scaled(amax_bits) & 0x7FFFu;
    }
    if (stats) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float lo = bf16lo_to_f32(w[j]), hi = bf16hi_to_f32(w[j]);
          sum = __fadd_rn(__fadd_rn(sum, lo), hi);
          sumsq = __fadd_rn(__fadd_rn(sumsq, round_in<true>(__fmul_rn(lo, lo))), round_in<true>(__fmul_rn(hi, hi)));
        }
      }
    }
  } else if (ok) {
#pragma unroll 4
    for (int i = 0; i < 16; ++i) {
      const uint4 p = __ldg(reinterpret_cast<const uint4*>(src + i * pitch));
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(src + i * pitch) + 1);
      const uint32_t ws[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t b = ws[j] & 0x7FFFFFFFu;
        amax_bits = b > amax_bits ? b : amax_bits;
        if (stats) {
          sum = __fadd_rn(sum, u2f(ws[j]));
          sumsq = __fadd_rn(sumsq, __fmul_rn(u2f(ws[j]), u2f(ws[j])));
        }
      }
    }
  }
  // lanes of one block: B / 8 neighbours along the columns, B / 16 row groups
#pragma unroll
  for (int o = 1; o < B / 8; o <<= 1) {
    const uint32_t t = __shfl_xor_sync(0xFFFFFFFFu, amax_bits, o);
    amax_bits = t > amax_bits ? t : amax_bits;
    if (stats) {   // uniform: a launch argument
      sum = __fadd_rn(sum, __shfl_xor_sync(0xFFFFFFFFu, sum, o));
      sumsq = __fadd_rn(sumsq, __shfl_xor_sync(0xFFFFFFFFu, sumsq, o));
    }
  }
  if (B == 32) {
    const uint32_t t = __shfl_xor_sync(0xFFFFFFFFu, amax_bits, LC);
    amax_bits = t > amax_bits ? t : amax_bits;
    if (stats) {
      sum = __fadd_rn(sum, __shfl_xor_sync(0xFFFFFFFFu, sum, LC));
      sumsq = __fadd_rn(sumsq, __shfl_xor_sync(0xFFFFFFFFu, sumsq, LC));
    }
  }
  const BlockScale s = (F::MX && (a.mx.clip | a.mx.uos))
                           ? make_block_scale_opts<FMT, IN_BF16>(amax_bits, sum, sumsq, B * B, a.mx)
                           : make_block_scale<FMT, IN_BF16>(amax_bits, os);
  const bool clip = F::MX && a.mx.clip == 1;

  // ---- encode row by row, K packing ----
  uint32_t kw[F::FP4 ? 16 : 32];  // FP4: one word per row (8 codes); FP8: two words per row (8 bytes)
  with_uniform_fast(block_fast<IN_BF16, ROUND>(s, amax_bits), [&](auto fast_tag) {
    constexpr bool FAST = decltype(fast_tag)::value;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float v[8];
      if (IN_BF16) {
        const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[2 * j] = bf16lo_to_f32(w[j]);
          v[2 * j + 1] = bf16hi_to_f32(w[j]);
        }
      } else {
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
        if (ok) {
          p = __ldg(reinterpret_cast<const float4*>(src + i * pitch));
          q = __ldg(reinterpret_cast<const float4*>(src + i * pitch) + 1);
        }
        v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
        v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
      }
      if (clip) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = round_in<IN_BF16>(__fmul_rn(v[j], 0.75f));
      }
      if (F::FP4 && ROUND == ALTOB200_ROUND_SR_BITS) {
        // the lane's 4 column pairs are 4 consecutive, 16-byte aligned words of each plane
        const bool tiled = a.tile_rows != 0;
        const int64_t row = rows_before + row0 + i;  // row of the flattened view over the batch
        // (a 64-bit modulo only where the flattened row index needs it: it costs ~70 instructions)
        const int64_t rr = !tiled ? row
                           : ((uint64_t)row >> 32) == 0 ? (int64_t)((uint32_t)row % (uint32_t)a.tile_rows)
                                                        : (int64_t)((uint64_t)row % (uint64_t)a.tile_rows);
        const int64_t pp = tiled ? (int64_t)((uint32_t)(col0 >> 1) % (uint32_t)a.tile_pairs) : (col0 >> 1);
        const int64_t pitch = tiled ? a.tile_pairs : (a.cols >> 1);
        const int64_t plane = tiled ? a.tile_rows * a.tile_pairs : a.batch * a.rows * (a.cols >> 1);
        uint4 re = make_uint4(0u, 0u, 0u, 0u), ro = re;
        if (ok) {
          re = __ldg(reinterpret_cast<const uint4*>(a.rand_bits + rr * pitch + pp));
          ro = __ldg(reinterpret_cast<const uint4*>(a.rand_bits + plane + rr * pitch + pp));
        }
        const uint32_t e4[4] = {re.x, re.y, re.z, re.w}, o4[4] = {ro.x, ro.y, ro.z, ro.w};
        kw[i] = fp4_octet<FMT, IN_BF16, ROUND, FAST>(v, s, e4, o4);
        if (ok) *reinterpret_cast<uint32_t*>(a.codes_k + (rows_before + row0 + i) * (a.cols >> 1) + (col0 >> 1)) = kw[i];
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = scale_elem<FMT, IN_BF16, FAST>(v[j], s);
        if (F::FP4) {
          kw[i] = e2m1x8_rtn_hw(v);
          if (ok) *reinterpret_cast<uint32_t*>(a.codes_k + (rows_before + row0 + i) * (a.cols >> 1) + (col0 >> 1)) = kw[i];
        } else {
          kw[2 * i] = fp8x2_rtn_hw<F::E5M2>(v[0], v[1]) | (fp8x2_rtn_hw<F::E5M2>(v[2], v[3]) << 16);
          kw[2 * i + 1] = fp8x2_rtn_hw<F::E5M2>(v[4], v[5]) | (fp8x2_rtn_hw<F::E5M2>(v[6], v[7]) << 16);
          if (ok)
            *reinterpret_cast<uint2*>(a.codes_k + (rows_before + row0 + i) * a.cols + col0) = make_uint2(kw[2 * i], kw[2 * i + 1]);
        }
      }
    }
  });

  // ---- transposed packing: column col0 + c, rows row0 .. row0 + 15 along the packed axis ----
  if (a.codes_t != nullptr) {
    if (F::FP4) {
      // byte j of ev[..] / od[..]: rows 2j (low nibble) and 2j + 1 of an even / odd column
      uint32_t ev[8], od[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t lo = kw[2 * j], hi = kw[2 * j + 1];
        ev[j] = (lo & 0x0F0F0F0Fu) | ((hi << 4) & 0xF0F0F0F0u);  // byte b: column 2b
        od[j] = ((lo >> 4) & 0x0F0F0F0Fu) | (hi & 0xF0F0F0F0u);  // byte b: column 2b + 1
      }
      uint32_t e0[4], e1[4], o0[4], o1[4];
      transpose4x4_bytes(ev, e0);      // e0[b]: bytes 0..3 of column 2b
      transpose4x4_bytes(ev + 4, e1);  // e1[b]: bytes 4..7
      transpose4x4_bytes(od, o0);
      transpose4x4_bytes(od + 4, o1);
      if (ok) {
        uint8_t* dst = a.codes_t + (cols_before + col0) * (a.rows >> 1) + (row0 >> 1);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          *reinterpret_cast<uint2*>(dst + (2 * b) * (a.rows >> 1)) = make_uint2(e0[b], e1[b]);
          *reinterpret_cast<uint2*>(dst + (2 * b + 1) * (a.rows >> 1)) = make_uint2(o0[b], o1[b]);
        }
      }
    } else {
      // kw[2 i + h]: row i, bytes = columns 4h .. 4h + 3
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t t[4][4];  // t[g][b]: rows 4g .. 4g + 3 of column 4h + b
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint32_t in[4] = {kw[2 * (4 * g) + h], kw[2 * (4 * g + 1) + h], kw[2 * (4 * g + 2) + h],
                                  kw[2 * (4 * g + 3) + h]};
          transpose4x4_bytes(in, t[g]);
        }
        if (ok) {
#pragma unroll
          for (int b = 0; b < 4; ++b)
            *reinterpret_cast<uint4*>(a.codes_t + (cols_before + col0 + 4 * h + b) * a.rows + row0) =
                make_uint4(t[0][b], t[1][b], t[2][b], t[3][b]);
        }
      }
    }
  }

  // ---- scales ----
  const bool col_ok = col0 < a.cols, row_ok = row0 < a.rows;
  if (a.scale_plain != nullptr && ok && (lc % (B / 8)) == 0 && (lr % (B / 16)) == 0) {
    const int64_t idx = ((rows_before + row0) / B) * (a.cols / B) + col0 / B;
    if (F::MX) reinterpret_cast<uint8_t*>(a.scale_plain)[idx] = (uint8_t)s.byte;
    else reinterpret_cast<float*>(a.scale_plain)[idx] = s.plain;
  }
  const uint32_t my_byte = ok ? s.byte : 0u;  // blocks outside the matrix contribute zero bytes
  constexpr int BC = TC / B, BR = TR / B;   // the warp's blocks: 4 x 4 (NVFP4), 2 x 2 (MXFP4), 4 columns x 1 row (FP8)
  if (a.packed_k != nullptr) {
    // per row the scale bytes of the warp's BC block columns: a word, or half of one; the rows of a group
    // are shared out over its LC lanes
    uint32_t word = 0;
#pragma unroll
    for (int j = 0; j < BC; ++j) word |= __shfl_sync(0xFFFFFFFFu, my_byte, lr * LC + j * (B / 8)) << (8 * j);
    const int64_t kb = tc * BC;
    if (row_ok && (BC == 4 || kb < a.nct_k * 4)) {
#pragma unroll
      for (int i = 0; i < 16 / LC; ++i) {
        const int64_t row = row0 + lc * (16 / LC) + i;
        uint8_t* dst = a.packed_k + bi * a.packed_k_bytes + packed_scale_offset(row, kb, a.nct_k);
        if (BC == 4) *reinterpret_cast<uint32_t*>(dst) = word;
        else *reinterpret_cast<uint16_t*>(dst) = (uint16_t)word;
      }
    }
  }
  if (a.packed_t != nullptr) {
    // rows of this layout are the matrix columns, scale columns the row blocks
    if (BR > 1) {
      // the BR row blocks are the bytes of one word or half-word; the 8 columns of a lane are shared out over
      // the 4 row groups
      uint32_t word = 0;
#pragma unroll
      for (int j = 0; j < BR; ++j) word |= __shfl_sync(0xFFFFFFFFu, my_byte, j * (B / 16) * LC + lc) << (8 * j);
      const int64_t kb = tr * BR;
      if (col_ok && (BR == 4 || kb < a.nct_t * 4)) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint8_t* dst = a.packed_t + bi * a.packed_t_bytes + packed_scale_offset(col0 + 2 * lr + e, kb, a.nct_t);
          if (BR == 4) *reinterpret_cast<uint32_t*>(dst) = word;
          else *reinterpret_cast<uint16_t*>(dst) = (uint16_t)word;
        }
      }
    } else {
      // one row block, one byte per column
      if (ok) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          a.packed_t[bi * a.packed_t_bytes + packed_scale_offset(col0 + 4 * lr + e, tr, a.nct_t)] = (uint8_t)s.byte;
      }
    }
  }
}

// =======================================================================================
// Tensor amax (plain and Hadamard-transformed) with the outer-scale finalisation
// =======================================================================================
struct AmaxArgs {
  const void* x;
  int32_t steps;         // loads of a thread in a row, up to LOADS
  int64_t rows, cols, ld;
  uint32_t* amax_bits;   // [2], written by the last block
  float* outer_scale;    // [2] or NULL
  uint32_t* counter;     // scratch [4]: ticket counter, running maxima; zero on entry, zero on exit
  RhtParams rht;
};

// outer = max(nan_to_num(amax) / (448 * 6), 1e-30)
//   alto/kernels/fp4/nvfp4/nvfp_quantization.py:484-487
__device__ __forceinline__ float outer_from_amax_bits(uint32_t bits) {
  float amax = u2f(bits);
  if (bits > 0x7F800000u) amax = 0.0f;               // NaN -> 0
  if (bits == 0x7F800000u) amax = 3.4028234663852886e38f;  // nan_to_num(+inf) -> float max
  return fmaxf(__fdiv_rn(amax, 2688.0f), 1.0e-30f);
}

// LOADS: 16-byte loads of a thread in flight (without RHT).  Eight of them, neighbours of a block, from nine for each
// thread of the grid on: 117 MB of bf16 24.0 us, 268 MB 54.9, where four a grid's width apart took 26.7 and 58.3.  Below
// that four, which leaves room for eight blocks on an SM: 4 MB 5.2 us, 6.9 with eight; 36.4 MB (7.5 a thread) 9.4 and
// 10.6, 38.9 MB 10.3 and 11.0 (43.7 MB, nine: 11.2 with eight, 11.8 with those four).  Just above a multiple of the grid a part of the blocks has
// nothing to do, which costs nothing: 4.86 MB, one load a thread and a little, 5.0 us in half of the blocks, 5.8 spread out.
template <bool IN_BF16, bool RHT, int LOADS = 1>
__global__ void __launch_bounds__(256) amax_kernel(AmaxArgs a) {
  grid_dependency_wait();
  __shared__ uint32_t s_red[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t am_plain = 0, am_rht = 0;
  if (!RHT) {
    // flat pass, 16 bytes per thread per step; rows are contiguous when ld == cols
    const int64_t vec = IN_BF16 ? 8 : 4;
    const int64_t vec_per_row = a.cols / vec;
    const int64_t total = a.rows * vec_per_row;
    const bool dense = a.ld == a.cols;  // contiguous rows: no index arithmetic per load
    auto load = [&](int64_t i) -> uint4 {
      int64_t off = i * vec;
      if (!dense) {
        int64_t row, cv;
        divmod_fast(i, vec_per_row, &row, &cv);
        off = row * a.ld + cv * vec;
      }
      return __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(a.x) + off * (IN_BF16 ? 2 : 4)));
    };
    // the loads are issued before any of them is consumed: the pass is a pure stream and needs bytes in flight,
    // not arithmetic
    constexpr int U = LOADS;
    const int64_t chunk = a.steps * 256;
    for (int64_t b = blockIdx.x * chunk + threadIdx.x; b < total; b += gridDim.x * chunk) {
      uint4 wv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = b + u * 256;
        wv[u] = u < a.steps && i < total ? load(i) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
      const uint4 w = wv[u];
      if (IN_BF16) {
        const uint32_t acc = absmax2_bf16x2(absmax2_bf16x2(0, w.x, w.y), w.z, w.w);
        const uint32_t m = fold_bf16x2(acc) << 16;
        am_plain = m > am_plain ? m : am_plain;
      } else {
        const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t b = ws[j] & 0x7FFFFFFFu;
          am_plain = b > am_plain ? b : am_plain;
        }
      }
      }
    }
  } else {
    // column pass: 16-row groups x 2 columns per lane, as in the column-wise quantizer.  Rounding to
    // the input dtype and the factor 1/4 are monotone in the magnitude, so the maximum is taken over
    // the raw butterfly outputs and scaled and rounded once per thread.
    const int64_t groups = a.rows >> 4;
    const int64_t col_tiles = (a.cols + 63) >> 6;
    const int64_t n_tasks = groups * col_tiles;
    const int64_t warp0 = (int64_t)blockIdx.x * 8 + warp, n_warps = (int64_t)gridDim.x * 8;
    uint32_t plain16 = 0;
    float raw_rht = 0.0f;
    for (int64_t task = warp0; task < n_tasks; task += n_warps) {
      int64_t g, ct;
      divmod_fast(task, col_tiles, &g, &ct);
      const int64_t c = (ct << 6) + 2 * lane;
      if (c >= a.cols) continue;
      const uint8_t* base = reinterpret_cast<const uint8_t*>(a.x) + ((g << 4) * a.ld + c) * (IN_BF16 ? 2 : 4);
      float v0[16], v1[16];
      uint32_t before = 0;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        if (IN_BF16) {
          const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(base + a.rht.row_off[k]));
          if (k & 1) plain16 = absmax2_bf16x2(plain16, before, w);
          before = w;
          v0[k] = bf16lo_to_f32(w);
          v1[k] = bf16hi_to_f32(w);
        } else {
          const float2 f = __ldg(reinterpret_cast<const float2*>(base + a.rht.row_off[k]));
          const uint32_t b0 = f2u(f.x) & 0x7FFFFFFFu, b1 = f2u(f.y) & 0x7FFFFFFFu;
          am_plain = b0 > am_plain ? b0 : am_plain;
          am_plain = b1 > am_plain ? b1 : am_plain;
          v0[k] = f.x;
          v1[k] = f.y;
        }
      }
      hadamard16_pair(v0, v1);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        // one three-input instruction for both columns; a NaN wins, as in torch.amax
        raw_rht = absmax3_nan(raw_rht, v0[k], v1[k]);
      }
    }
    if (IN_BF16) am_plain = fold_bf16x2(plain16) << 16;
    // the row signs of the transform do not change magnitudes
    const float y = __fmul_rn(raw_rht, 0.25f);
    am_rht = IN_BF16 ? ((f32_to_bf16_bits(y) & 0x7FFFu) << 16) : (f2u(y) & 0x7FFFFFFFu);
  }
  am_plain = warp_max_u32(am_plain);
  am_rht = warp_max_u32(am_rht);
  if (lane == 0) {
    s_red[0][warp] = am_plain;
    s_red[1][warp] = am_rht;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t p = 0, h = 0;
    for (int i = 0; i < 8; ++i) {
      p = s_red[0][i] > p ? s_red[0][i] : p;
      h = s_red[1][i] > h ? s_red[1][i] : h;
    }
    // the running maxima live in the scratch words behind the counter, so that the result buffer needs
    // no clearing launch in front of the kernel; the last block moves them out and leaves the scratch zero
    atomicMax(a.counter + 1, p);
    if (RHT) atomicMax(a.counter + 2, h);
    __threadfence();
    const uint32_t ticket = atomicAdd(a.counter, 1u);
    if (ticket == gridDim.x - 1) {
      __threadfence();
      const uint32_t fp = atomicExch(a.counter + 1, 0u), fh = RHT ? atomicExch(a.counter + 2, 0u) : 0u;
      a.amax_bits[0] = fp;
      a.amax_bits[1] = fh;
      if (a.outer_scale != nullptr) {
        a.outer_scale[0] = outer_from_amax_bits(fp);
        if (RHT) a.outer_scale[1] = outer_from_amax_bits(fh);
      }
      *a.counter = 0u;
    }
  }
}

// =======================================================================================
// Tensor amax without any caller- or library-allocated scratch
// =======================================================================================
// Partial maxima (one word per block) and the completion counter live in this file-scope array.
// Every GPU that loads the library holds these bytes until the process exits.
constexpr int NOALLOC_MAX_BLOCKS = 8192;
constexpr int NOALLOC_VEC_PER_THREAD = 16;  // 16-byte vectors per thread -> 64 KiB of input per block
struct NoallocScratch {
  uint32_t counter;
  uint32_t pad[63];
  uint32_t partial[NOALLOC_MAX_BLOCKS];
};
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoallocScratch)];

struct AmaxNoallocArgs {
  const void* x;
  int64_t rows, cols, ld;
  uint32_t* amax_bits;   // [1]
  float* outer_scale;    // [1] or NULL
  NoallocScratch* scratch;
};

template <bool IN_BF16>
__global__ void __launch_bounds__(256) amax_noalloc_kernel(AmaxNoallocArgs a) {
  __shared__ uint32_t s_red[8];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t vec = IN_BF16 ? 8 : 4;
  const int64_t vec_per_row = a.cols / vec;
  const int64_t total = a.rows * vec_per_row;
  const bool dense = a.ld == a.cols;
  uint32_t am = 0;
  const int64_t base = (int64_t)blockIdx.x * (256 * NOALLOC_VEC_PER_THREAD) + threadIdx.x;
#pragma unroll 4
  for (int j = 0; j < NOALLOC_VEC_PER_THREAD; ++j) {
    const int64_t i = base + (int64_t)j * 256;
    if (i >= total) break;
    int64_t off = i * vec;
    if (!dense) {
      int64_t row, cv;
      divmod_fast(i, vec_per_row, &row, &cv);
      off = row * a.ld + cv * vec;
    }
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(
        reinterpret_cast<const uint8_t*>(a.x) + off * (IN_BF16 ? 2 : 4)));
    if (IN_BF16) {
      uint32_t acc = absmax_bf16x2(0, w.x);
      acc = absmax_bf16x2(acc, w.y);
      acc = absmax_bf16x2(acc, w.z);
      acc = absmax_bf16x2(acc, w.w);
      const uint32_t m = fold_bf16x2(acc) << 16;
      am = m > am ? m : am;
    } else {
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t b = ws[q] & 0x7FFFFFFFu;
        am = b > am ? b : am;
      }
    }
  }
  am = warp_max_u32(am);
  if (lane == 0) s_red[warp] = am;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t m = 0;
    for (int i = 0; i < 8; ++i) m = s_red[i] > m ? s_red[i] : m;
    a.scratch->partial[blockIdx.x] = m;
    __threadfence();
    s_last = atomicAdd(&a.scratch->counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (s_last) {  // the last block to finish folds every block's partial maximum
    __threadfence();
    uint32_t m = 0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) {
      const uint32_t p = *reinterpret_cast<volatile uint32_t*>(&a.scratch->partial[i]);
      m = p > m ? p : m;
    }
    m = warp_max_u32(m);
    __syncthreads();
    if (lane == 0) s_red[warp] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t f = 0;
      for (int i = 0; i < 8; ++i) f = s_red[i] > f ? s_red[i] : f;
      a.amax_bits[0] = f;
      if (a.outer_scale != nullptr) a.outer_scale[0] = outer_from_amax_bits(f);
      a.scratch->counter = 0u;  // ready for the next call
    }
  }
}

// =======================================================================================
// Dequantizer (row-major codes, plain scales)
// =======================================================================================
struct DequantArgs {
  const uint8_t* codes;
  const void* scales;
  const float* outer;
  int64_t rows, cols, ld_out;
  void* out;
  int is_2d;
  int static_clip;  // MXFP4: decoded values are multiplied by 4/3 in the output dtype before scaling
};

// A pure stream (a write of the output, 1/8 to 1/2 of that read): a thread makes 16-byte vectors of the output,
// neighbouring threads neighbouring vectors, several of them in flight where there are more vectors than threads.
// (16 elements per thread, which wrote each 32-byte sector in two instructions, and decoding E2M1 with compares took
// 75 us for 14336 x 4096 fp32; 60 us now.)  FP8 -> bf16 has the most arithmetic per vector: 14336 x 4096 takes 32 us
// with two in flight, 42 with four, 38 with 16 elements per thread.
template <int FMT, bool OUT_BF16>
__global__ void __launch_bounds__(256) dequantize_kernel(DequantArgs a) {
  grid_dependency_wait();
  using F = Fmt<FMT>;
  constexpr int V = OUT_BF16 ? 8 : 4;                     // elements per vector; a block is a whole number of them
  constexpr int CODE_BYTES = F::FP4 ? V / 2 : V;
  constexpr int U = OUT_BF16 && !F::FP4 ? 2 : 4;          // vectors in flight
  const int64_t vecs_per_row = a.cols / V;
  const int64_t total = a.rows * vecs_per_row;
  const float outer = (!F::MX && a.outer != nullptr) ? __ldg(a.outer) : 1.0f;
  const bool use_outer = (!F::MX && a.outer != nullptr);
  const int64_t nsc = a.cols / F::B;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < total; i0 += U * stride) {
    uint2 code[U];
    float scale[U];
    int64_t dst[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride;
      code[u] = make_uint2(0u, 0u);
      scale[u] = 0.0f;
      dst[u] = -1;
      if (i < total) {
        // rows of codes and of 1-D scales follow each other without gaps: only 2-D scales and an output with a
        // pitch of its own need the row
        int64_t row = 0, vec = i;
        if (a.is_2d || a.ld_out != a.cols) divmod_fast(i, vecs_per_row, &row, &vec);
        dst[u] = a.ld_out == a.cols ? i * V : row * a.ld_out + vec * V;
        const uint8_t* c = a.codes + i * CODE_BYTES;
        if (CODE_BYTES == 2) code[u].x = __ldg(reinterpret_cast<const uint16_t*>(c));
        else if (CODE_BYTES == 4) code[u].x = __ldg(reinterpret_cast<const uint32_t*>(c));
        else code[u] = __ldg(reinterpret_cast<const uint2*>(c));
        const int64_t si = a.is_2d ? row / F::B * nsc + vec * V / F::B : i * V / F::B;
        if (F::MX) scale[u] = u2f((uint32_t)__ldg(reinterpret_cast<const uint8_t*>(a.scales) + si) << 23);
        else scale[u] = __ldg(reinterpret_cast<const float*>(a.scales) + si);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (dst[u] < 0) break;
      const float s = use_outer ? __fmul_rn(scale[u], outer) : scale[u];
      float v[V];
#pragma unroll
      for (int j = 0; j < V; j += 2) {
        float2 f;
        if (F::FP4) {
          f = e2m1x2_decode((code[u].x >> (4 * j)) & 0xFFu);
          // tests/unittest/mxfp4/utils.py:381-384: cast, times 4/3 in the output dtype, then the scale
          if (a.static_clip) f = make_float2(round_in<OUT_BF16>(__fmul_rn(f.x, (float)(4.0 / 3.0))),
                                             round_in<OUT_BF16>(__fmul_rn(f.y, (float)(4.0 / 3.0))));
        } else {
          f = fp8x2_decode<F::E5M2>(((j < 4 ? code[u].x : code[u].y) >> (8 * (j & 3))) & 0xFFFFu);
        }
        v[j] = __fmul_rn(f.x, s);
        v[j + 1] = __fmul_rn(f.y, s);
      }
      if (OUT_BF16) {
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __nv_bfloat162 p2 = __floats2bfloat162_rn(v[(2 * j) % V], v[(2 * j + 1) % V]);
          o[j] = *reinterpret_cast<const uint32_t*>(&p2);
        }
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + dst[u]) = make_uint4(o[0], o[1], o[2], o[3]);
      } else {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + dst[u]) = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
  }
}

// =======================================================================================
// Standalone randomised Hadamard transform (n = 16)
// =======================================================================================
struct RhtArgs {
  const void* x;
  void* y;
  int64_t rows, cols, ld, ld_y;
  RhtParams rht;
};

template <bool IN_BF16>
__global__ void __launch_bounds__(256) rht_kernel(RhtArgs a) {
  grid_dependency_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t groups = a.rows >> 4;
  const int64_t col_tiles = (a.cols + 63) >> 6;
  const int64_t n_tasks = groups * col_tiles;
  const int64_t warp0 = (int64_t)blockIdx.x * 8 + warp, n_warps = (int64_t)gridDim.x * 8;
  for (int64_t task = warp0; task < n_tasks; task += n_warps) {
    int64_t g, ct;
    divmod_fast(task, col_tiles, &g, &ct);
    const int64_t c = (ct << 6) + 2 * lane;
    if (c >= a.cols) continue;
    float v0[16], v1[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int src = a.rht.pinv[k];
      float f0, f1;
      if (IN_BF16) {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(
            reinterpret_cast<const __nv_bfloat16*>(a.x) + ((g << 4) + src) * a.ld + c));
        f0 = bf16lo_to_f32(w);
        f1 = bf16hi_to_f32(w);
      } else {
        const float2 f = __ldg(reinterpret_cast<const float2*>(
            reinterpret_cast<const float*>(a.x) + ((g << 4) + src) * a.ld + c));
        f0 = f.x;
        f1 = f.y;
      }
      v0[k] = f0;
      v1[k] = f1;
    }
    hadamard16(v0);
    hadamard16(v1);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      // slot k is output row pinv[k] of the group (y[i] = sign[perm[i]] * u[perm[i]])
      const int64_t orow = (g << 4) + a.rht.pinv[k];
      const float sg = 0.25f * a.rht.sign[k];
      const float y0 = __fadd_rn(__fmul_rn(v0[k], sg), 0.0f), y1 = __fadd_rn(__fmul_rn(v1[k], sg), 0.0f);
      if (IN_BF16) {
        *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(a.y) + orow * a.ld_y + c) =
            f32_to_bf16_bits(y0) | (f32_to_bf16_bits(y1) << 16);
      } else {
        *reinterpret_cast<float2*>(reinterpret_cast<float*>(a.y) + orow * a.ld_y + c) = make_float2(y0, y1);
      }
    }
  }
}

// =======================================================================================
// host side
// =======================================================================================
static int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 148;
  }
  return n;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

static int fill_rht(RhtParams* r, int n, const int32_t* perm, const int32_t* sign) {
  r->n = n;
  if (n == 0) {
    for (int i = 0; i < 16; ++i) {
      r->pinv[i] = (int8_t)i; r->sign[i] = 1.0f;
      r->qsign[i] = 0.25f;
    }
    return ALTOB200_OK;
  }
  if (n != 16) return ALTOB200_EUNSUPPORTED;
  if (perm == nullptr || sign == nullptr) return ALTOB200_EINVAL_SHAPE;
  bool seen[16] = {false};
  for (int i = 0; i < 16; ++i) {
    if (perm[i] < 0 || perm[i] > 15 || seen[perm[i]]) return ALTOB200_EINVAL_SHAPE;
    if (sign[i] != 1 && sign[i] != -1) return ALTOB200_EINVAL_SHAPE;
    seen[perm[i]] = true;
  }
  // W[i][j] = sign[perm[i]] * H[perm[i]][perm[j]]:  z[k] = x[pinv[k]],  y[i] = sign[perm[i]] * (H z)[perm[i]]
  for (int i = 0; i < 16; ++i) {
    r->pinv[perm[i]] = (int8_t)i;
    r->sign[i] = (float)sign[i];
  }
  for (int k = 0; k < 16; ++k) {
    r->qsign[k] = 0.25f * r->sign[k];
    if ((k & 3) == 0) r->psel[k >> 2] = r->pmask[k >> 2] = 0u;
    r->psel[k >> 2] |= (uint32_t)(perm[k] & 7) << (4 * (k & 3));
    r->pmask[k >> 2] |= (perm[k] & 8) != 0 ? 0xFFu << (8 * (k & 3)) : 0u;
  }
  return ALTOB200_OK;
}

// Byte offsets of the rows that feed butterfly slots 0..15, for a matrix with leading dimension `ld`.
static void fill_rht_row_offsets(RhtParams* r, int64_t ld, int esz) {
  for (int k = 0; k < 16; ++k) r->row_off[k] = (int64_t)r->pinv[k] * ld * esz;
}

// Whether the rows of a task are taken a period of the table apart.  There are up to four times as many tasks then where
// rows are few, each with fewer loads in flight: faster while one wave of warps holds them (64 x 14336 6.4 -> 5.0 us) and
// with three rows or more in a task (192 x 65536 17.4 -> 16.2, 512 x 65536 33.5 -> 31.9), not below (64 x 131072
// 13.2 -> 17.7; 320 x 131072, five rows in eight places, 46.9 -> 49.7; NVFP4 from bf16).  fp32 rows are twice as long and
// the body with words by row spills: from three rows in two tasks on (96 x 65536 15.1 -> 14.3, 64 x 131072 18.8 -> 20.4).
static bool rowwise_shares_words(const RowwiseArgs& a, bool in_bf16) {
  if (a.tile_rows == 0 || a.tile_rows >= (1ll << 32)) return false;
  const int64_t groups = rowwise_row_groups(a.rows, a.tile_rows);
  return groups * ((a.cols + 511) >> 9) <= (int64_t)sm_count() * 16 || 2 * a.rows >= (in_bf16 ? 6 : 3) * groups;
}

template <int FMT, bool IN_BF16, int ROUND, bool SHARED>
static void launch_rowwise_kernel(const RowwiseArgs& a, cudaStream_t st) {
  const int64_t tasks = rowwise_row_groups(a.rows, SHARED ? a.tile_rows : 1) * ((a.cols + 511) >> 9);
  constexpr int NT = rowwise_threads(SHARED);
  int64_t blocks = ceil_div(tasks, NT / 32);
  const int64_t cap = (int64_t)sm_count() * (2048 / NT);
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  constexpr bool CAN_MACRO = FMT == ALTOB200_FMT_MXFP4 && IN_BF16 && ROUND != ALTOB200_ROUND_SR_PHILOX;
  if (CAN_MACRO && a.macro_codes != nullptr)
    (void)launch_after(quantize_rowwise_kernel<FMT, IN_BF16, ROUND, CAN_MACRO, SHARED>, dim3((unsigned)blocks), dim3(NT), 0, st, a);
  else
    (void)launch_after(quantize_rowwise_kernel<FMT, IN_BF16, ROUND, false, SHARED>, dim3((unsigned)blocks), dim3(NT), 0, st, a);
}

template <int FMT, bool IN_BF16>
static int launch_rowwise(const RowwiseArgs& a, int rounding, cudaStream_t st) {
  constexpr bool FP4 = Fmt<FMT>::FP4;
  if (rounding == ALTOB200_ROUND_RTN)
    launch_rowwise_kernel<FMT, IN_BF16, ALTOB200_ROUND_RTN, false>(a, st);
  else if (rounding == ALTOB200_ROUND_SR_BITS && FP4 && rowwise_shares_words(a, IN_BF16))
    launch_rowwise_kernel<FMT, IN_BF16, FP4 ? ALTOB200_ROUND_SR_BITS : ALTOB200_ROUND_RTN, FP4>(a, st);
  else if (rounding == ALTOB200_ROUND_SR_BITS && FP4)
    launch_rowwise_kernel<FMT, IN_BF16, FP4 ? ALTOB200_ROUND_SR_BITS : ALTOB200_ROUND_RTN, false>(a, st);
  else if (rounding == ALTOB200_ROUND_SR_PHILOX && FP4)
    launch_rowwise_kernel<FMT, IN_BF16, FP4 ? ALTOB200_ROUND_SR_PHILOX : ALTOB200_ROUND_RTN, false>(a, st);
  else
    return ALTOB200_EUNSUPPORTED;
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

template <int FMT, bool IN_BF16, int ROUND, bool RHT>
static void launch_colwise_kernel(const ColwiseArgs& a, cudaStream_t st) {
  const dim3 grid((unsigned)ceil_div(a.cols, COL_TN), (unsigned)ceil_div(a.rows, COL_NT)), block(COL_NT);
  constexpr bool CAN_MACRO = FMT == ALTOB200_FMT_MXFP4 && IN_BF16 && (ROUND == ALTOB200_ROUND_RTN || ROUND == ALTOB200_ROUND_SR_SLOTS);
  if constexpr (CAN_MACRO && !RHT) {
    if (a.dense != nullptr) {
      if (a.macro_codes != nullptr) (void)launch_after(quantize_colwise_kernel<FMT, IN_BF16, ROUND, false, true, true>, grid, block, 0, st, a);
      else (void)launch_after(quantize_colwise_kernel<FMT, IN_BF16, ROUND, false, false, true>, grid, block, 0, st, a);
      return;
    }
  }
  if (CAN_MACRO && a.macro_codes != nullptr)
    (void)launch_after(quantize_colwise_kernel<FMT, IN_BF16, ROUND, RHT, CAN_MACRO>, grid, block, 0, st, a);
  else
    (void)launch_after(quantize_colwise_kernel<FMT, IN_BF16, ROUND, RHT, false>, grid, block, 0, st, a);
}

template <int FMT, bool IN_BF16>
static int launch_colwise(const ColwiseArgs& a, int rounding, cudaStream_t st) {
  constexpr bool FP4 = Fmt<FMT>::FP4;
  const bool rht = a.rht.n != 0;
  if (!FP4 && (rht || rounding != ALTOB200_ROUND_RTN)) return ALTOB200_EUNSUPPORTED;
  constexpr int BITS = FP4 ? ALTOB200_ROUND_SR_BITS : ALTOB200_ROUND_RTN;
  constexpr int PHILOX = FP4 ? ALTOB200_ROUND_SR_PHILOX : ALTOB200_ROUND_RTN;
  constexpr int SLOTS = FP4 ? ALTOB200_ROUND_SR_SLOTS : ALTOB200_ROUND_RTN;
  switch (rounding) {
    case ALTOB200_ROUND_RTN:
      if (rht) launch_colwise_kernel<FMT, IN_BF16, ALTOB200_ROUND_RTN, FP4>(a, st);
      else launch_colwise_kernel<FMT, IN_BF16, ALTOB200_ROUND_RTN, false>(a, st);
      break;
    case ALTOB200_ROUND_SR_BITS:
      if (rht) launch_colwise_kernel<FMT, IN_BF16, BITS, FP4>(a, st);
      else launch_colwise_kernel<FMT, IN_BF16, BITS, false>(a, st);
      break;
    case ALTOB200_ROUND_SR_PHILOX:
      if (rht) launch_colwise_kernel<FMT, IN_BF16, PHILOX, FP4>(a, st);
      else launch_colwise_kernel<FMT, IN_BF16, PHILOX, false>(a, st);
      break;
    case ALTOB200_ROUND_SR_SLOTS:
      if (rht) launch_colwise_kernel<FMT, IN_BF16, SLOTS, FP4>(a, st);
      else launch_colwise_kernel<FMT, IN_BF16, SLOTS, false>(a, st);
      break;
    default:
      return ALTOB200_EUNSUPPORTED;
  }
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

template <int FMT, bool IN_BF16, int ROUND, bool BATCHED>
static void launch_2d_kernel(const Quant2dArgs& a, cudaStream_t st) {
  constexpr int TC = Fmt<FMT>::FP4 ? 64 : 128, TR = Fmt<FMT>::FP4 ? 64 : 32;   // a warp's tile
  constexpr bool CAN_MACRO = FMT == ALTOB200_FMT_MXFP4 && IN_BF16;
  const bool macro = CAN_MACRO && a.macro_codes != nullptr;
  const int64_t tiles = (macro ? ceil_div(a.cols, 128) * ceil_div(a.rows, 128) * 4
                               : ceil_div(a.cols, TC) * ceil_div(a.rows, TR)) * a.batch;
  const dim3 blocks((unsigned)ceil_div(tiles, WARPS_2D)), block(WARPS_2D * 32);
  if (macro) (void)launch_after(quantize_2d_kernel<FMT, IN_BF16, ROUND, BATCHED, CAN_MACRO>, blocks, block, 0, st, a);
  else (void)launch_after(quantize_2d_kernel<FMT, IN_BF16, ROUND, BATCHED, false>, blocks, block, 0, st, a);
}

template <int FMT, bool IN_BF16>
static int launch_2d(const Quant2dArgs& a, int rounding, cudaStream_t st) {
  constexpr int SR = Fmt<FMT>::FP4 ? ALTOB200_ROUND_SR_BITS : ALTOB200_ROUND_RTN;
  const bool batched = a.batch > 1;
  if (rounding == ALTOB200_ROUND_RTN) {
    if (batched) launch_2d_kernel<FMT, IN_BF16, ALTOB200_ROUND_RTN, true>(a, st);
    else launch_2d_kernel<FMT, IN_BF16, ALTOB200_ROUND_RTN, false>(a, st);
  } else if (rounding == ALTOB200_ROUND_SR_BITS && Fmt<FMT>::FP4) {
    if (batched) launch_2d_kernel<FMT, IN_BF16, SR, true>(a, st);
    else launch_2d_kernel<FMT, IN_BF16, SR, false>(a, st);
  } else {
    return ALTOB200_EUNSUPPORTED;
  }
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

#define DISPATCH_FMT_DT(fmt, dt, CALL)                                                      \
  do {                                                                                      \
    const bool _bf = (dt) == ALTOB200_DT_BF16;                                              \
    switch (fmt) {                                                                          \
      case ALTOB200_FMT_NVFP4:                                                              \
        return _bf ? CALL(ALTOB200_FMT_NVFP4, true) : CALL(ALTOB200_FMT_NVFP4, false);      \
      case ALTOB200_FMT_MXFP4:                                                              \
        return _bf ? CALL(ALTOB200_FMT_MXFP4, true) : CALL(ALTOB200_FMT_MXFP4, false);      \
      case ALTOB200_FMT_MXFP8_E4M3:                                                         \
        return _bf ? CALL(ALTOB200_FMT_MXFP8_E4M3, true) : CALL(ALTOB200_FMT_MXFP8_E4M3, false); \
      case ALTOB200_FMT_MXFP8_E5M2:                                                         \
        return _bf ? CALL(ALTOB200_FMT_MXFP8_E5M2, true) : CALL(ALTOB200_FMT_MXFP8_E5M2, false); \
      default:                                                                              \
        return ALTOB200_EUNSUPPORTED;                                                       \
    }                                                                                       \
  } while (0)

// the field is younger than the struct: read only for callers that announce it
static uint8_t* macro_codes_of(const altob200_quant_params* p) {
  return (p->scale_flags & ALTOB200_SCALE_MACRO) != 0 ? p->macro_codes : nullptr;
}

static int block_of(int fmt) { return fmt == ALTOB200_FMT_NVFP4 ? 16 : 32; }
static bool is_fp4(int fmt) { return fmt == ALTOB200_FMT_NVFP4 || fmt == ALTOB200_FMT_MXFP4; }

// Zero a packed-scale buffer when the tile grid has padding the kernels do not visit.
static int clear_packed_if_padded(void* buf, int64_t rows, int64_t ncols, cudaStream_t st) {
  if (buf == nullptr) return ALTOB200_OK;
  if ((rows & 127) == 0 && (ncols & 3) == 0) return ALTOB200_OK;
  ALTOB200_CUDA_CHECK(cudaMemsetAsync(buf, 0, altob200_packed_scale_bytes(rows, ncols), st));
  return ALTOB200_OK;
}

// The reference's stochastic-rounding words (alto/kernels/fp4/fp4_common/triton_fp4_ops.py:13-19):
// every BLOCK_M x BLOCK_N tile of the quantisation-axis-last view draws
//   r1, r2, _, _ = randint4x(seed, offset + m * (BLOCK_N / 2) + n),  m < BLOCK_M, n < BLOCK_N / 2
// with tile-local m, n and the SAME offset in every tile, r1 for the even and r2 for the odd
// element of pair n.  The words therefore form one [2][BLOCK_M][BLOCK_N/2] table that repeats over
// the matrix; this kernel writes the table (one Philox call per entry pair) and the quantizers index
// it periodically.
__global__ void __launch_bounds__(256) philox_tile_kernel(uint32_t* out, int64_t tile_rows, int64_t tile_pairs,
                                                          uint32_t offset, PhiloxKeys pk) {
  grid_dependency_wait();
  const int64_t n = tile_rows * tile_pairs;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t o[4];
    // Triton's randint4x on an int32 offset tensor: counter = (uint32(offset + i), 0, 0, 0)
    philox4x32_10_keys(offset + (uint32_t)i, 0u, pk, o);
    out[i] = o[0];
    out[n + i] = o[1];
  }
}

// The same words of a 64 x 32 table as the column-wise quantizer reads them: [position][row], where the
// positions (two per pair) of every group of 16 are in the order of the transform's slots (position pinv[k]
// is slot k; the identity without a transform).
struct SlotOrder {
  int8_t pinv[16];
};
__global__ void __launch_bounds__(256) philox_slots_kernel(uint32_t* out, uint32_t offset, PhiloxKeys pk, SlotOrder order) {
  grid_dependency_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;   // row fastest: neighbouring threads write neighbours
  const int row = i & 63, slot = i >> 6;                 // slot of the 64 positions
  const int pos = (slot & ~15) + order.pinv[slot & 15];
  uint32_t o[4];
  philox4x32_10_keys(offset + (uint32_t)(row * 32 + (pos >> 1)), 0u, pk, o);
  out[slot * 64 + row] = (pos & 1) != 0 ? o[1] : o[0];
}

// clip_mode / use_uos exist for MXFP4 only, as in the reference
static int fill_mx_opts(MxOpts* o, const altob200_quant_params* p, bool allow_dynamic) {
  o->clip = p->clip_mode;
  o->uos = p->use_uos != 0 ? 1 : 0;
  if (o->clip < ALTOB200_CLIP_NONE || o->clip > ALTOB200_CLIP_DYNAMIC) return ALTOB200_EINVAL_SHAPE;
  if ((o->clip | o->uos) != 0 && p->format != ALTOB200_FMT_MXFP4) return ALTOB200_EUNSUPPORTED;
  if (o->clip == ALTOB200_CLIP_DYNAMIC && !allow_dynamic) return ALTOB200_EUNSUPPORTED;
  return ALTOB200_OK;
}

}  // namespace altob200

using namespace altob200;

extern "C" {

int altob200_version(void) { return 1; }

const char* altob200_status_string(int status) {
  switch (status) {
    case ALTOB200_OK: return "ok";
    case ALTOB200_EINVAL_SHAPE: return "invalid shape or size contract";
    case ALTOB200_EINVAL_ALIGN: return "misaligned pointer or leading dimension";
    case ALTOB200_ETIMEOUT_DEVICE: return "bounded device-side wait timed out";
    case ALTOB200_ECUDA: return "CUDA call failed";
    case ALTOB200_EUNSUPPORTED: return "unsupported configuration";
    case ALTOB200_ELIMIT: return "size exceeds a fixed maximum";
    default: return "unknown status";
  }
}

size_t altob200_packed_scale_bytes(int64_t rows, int64_t ncols) {
  return (size_t)(ceil_div(rows, 128) * ceil_div(ncols, 4) * 512);
}

int altob200_philox_tile(uint64_t seed, uint64_t offset, int64_t tile_rows, int64_t tile_pairs, uint32_t* out,
                         void* stream) {
  if (out == nullptr || tile_rows <= 0 || tile_pairs <= 0 || tile_rows * tile_pairs > (1ll << 24))
    return ALTOB200_EINVAL_SHAPE;
  if (!aligned16(out)) return ALTOB200_EINVAL_ALIGN;
  PhiloxKeys pk;
  philox_make_keys(seed, &pk);
  const int64_t n = tile_rows * tile_pairs;
  int64_t blocks = ceil_div(n, 256);
  if (blocks > 148) blocks = 148;
  (void)launch_after(philox_tile_kernel, dim3((unsigned)blocks), dim3(256), 0, (cudaStream_t)stream, out, tile_rows, tile_pairs, (uint32_t)offset,
                                                                        pk);
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

int altob200_philox_slots(uint64_t seed, uint64_t offset, int32_t rht_n, const int32_t* rht_perm, uint32_t* out,
                          void* stream) {
  if (out == nullptr || (rht_n != 0 && (rht_n != 16 || rht_perm == nullptr))) return ALTOB200_EINVAL_SHAPE;
  if (!aligned16(out)) return ALTOB200_EINVAL_ALIGN;
  SlotOrder order;
  bool seen[16] = {false};
  for (int i = 0; i < 16; ++i) {
    const int k = rht_n != 0 ? rht_perm[i] : i;
    if (k < 0 || k > 15 || seen[k]) return ALTOB200_EINVAL_SHAPE;
    seen[k] = true;
    order.pinv[k] = (int8_t)i;
  }
  PhiloxKeys pk;
  philox_make_keys(seed, &pk);
  (void)launch_after(philox_slots_kernel, dim3(16), dim3(256), 0, (cudaStream_t)stream, out, (uint32_t)offset, pk, order);
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

int altob200_quantize_rowwise(const void* x, int64_t rows, int64_t cols, int64_t ld,
                              const altob200_quant_params* p, void* codes, void* scale_plain,
                              void* scale_packed, void* stream) {
  if (x == nullptr || p == nullptr || codes == nullptr) return ALTOB200_EINVAL_SHAPE;
  const int B = block_of(p->format);
  if (rows <= 0 || cols <= 0 || cols % B != 0 || ld < cols) return ALTOB200_EINVAL_SHAPE;
  const int esz = p->in_dtype == ALTOB200_DT_BF16 ? 2 : 4;
  if (!aligned16(x) || (ld * esz) % 16 != 0 || !aligned16(codes)) return ALTOB200_EINVAL_ALIGN;
  if (p->rounding == ALTOB200_ROUND_SR_BITS && (p->rand_bits == nullptr || !aligned16(p->rand_bits)))
    return ALTOB200_EINVAL_ALIGN;
  if (p->rht_n != 0) return ALTOB200_EUNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  RowwiseArgs a;
  a.macro_codes = macro_codes_of(p);
  if (a.macro_codes != nullptr && (p->format != ALTOB200_FMT_MXFP4 || p->in_dtype != ALTOB200_DT_BF16 ||
                                   p->rounding == ALTOB200_ROUND_SR_PHILOX))
    return ALTOB200_EUNSUPPORTED;
  a.x = x; a.rows = rows; a.cols = cols; a.ld = ld;
  a.codes = (uint8_t*)codes; a.scale_plain = scale_plain; a.scale_packed = (uint8_t*)scale_packed;
  a.ncol_tiles = ceil_div(cols / B, 4);
  a.outer = p->outer_scale; a.rand_bits = p->rand_bits;
  a.tile_rows = p->rand_tile_rows; a.tile_pairs = p->rand_tile_pairs;
  if ((a.tile_rows != 0) != (a.tile_pairs != 0) || a.tile_rows < 0 || a.tile_pairs % 8 != 0)
    return ALTOB200_EINVAL_SHAPE;
  if (a.tile_rows != 0 && (rows >= (1ll << 32) || cols >= (1ll << 32))) return ALTOB200_ELIMIT;
  a.philox_seed = p->philox_seed; a.philox_offset = p->philox_offset;
  philox_make_keys(p->philox_seed, &a.pk);
  int rc = fill_mx_opts(&a.mx, p, true);
  if (rc != ALTOB200_OK) return rc;
  rc = clear_packed_if_padded(scale_packed, rows, cols / B, st);
  if (rc != ALTOB200_OK) return rc;
  const int rounding = p->rounding;
#define CALL_ROW(F, BF) launch_rowwise<F, BF>(a, rounding, st)
  DISPATCH_FMT_DT(p->format, p->in_dtype, CALL_ROW);
#undef CALL_ROW
}

int altob200_quantize_colwise(const void* x, int64_t rows, int64_t cols, int64_t ld,
                              const altob200_quant_params* p, void* codes, void* scale_plain,
                              void* scale_packed, void* stream) {
  if (x == nullptr || p == nullptr || codes == nullptr) return ALTOB200_EINVAL_SHAPE;
  const int B = block_of(p->format);
  if (rows <= 0 || cols <= 0 || rows % B != 0 || cols % 8 != 0 || ld < cols) return ALTOB200_EINVAL_SHAPE;
  if (p->rht_n != 0 && rows % p->rht_n != 0) return ALTOB200_EINVAL_SHAPE;
  // every output row must start on a 16-byte boundary
  const int64_t out_row_bytes = is_fp4(p->format) ? rows / 2 : rows;
  if (out_row_bytes % 8 != 0) return ALTOB200_EINVAL_SHAPE;
  const int esz = p->in_dtype == ALTOB200_DT_BF16 ? 2 : 4;
  if (!aligned16(x) || (ld * esz) % 16 != 0 || !aligned16(codes) || out_row_bytes % 16 != 0)
    return ALTOB200_EINVAL_ALIGN;
  if (p->rounding == ALTOB200_ROUND_SR_BITS && p->rand_bits == nullptr) return ALTOB200_EINVAL_SHAPE;
  if (p->rounding == ALTOB200_ROUND_SR_SLOTS) {
    // one word pair per lane and slot: the table has 64 rows, and column c of an 8-byte load is even
    if (p->rand_bits == nullptr || p->rand_tile_rows != 64 || p->rand_tile_pairs != 32) return ALTOB200_EINVAL_SHAPE;
    if (!aligned16(p->rand_bits)) return ALTOB200_EINVAL_ALIGN;
  }
  cudaStream_t st = (cudaStream_t)stream;
  ColwiseArgs a;
  a.macro_codes = macro_codes_of(p);
  if (a.macro_codes != nullptr &&
      (p->format != ALTOB200_FMT_MXFP4 || p->in_dtype != ALTOB200_DT_BF16 ||
       (p->rounding != ALTOB200_ROUND_RTN && p->rounding != ALTOB200_ROUND_SR_SLOTS)))
    return ALTOB200_EUNSUPPORTED;
  a.dense = (p->scale_flags & ALTOB200_RHT_DENSE32) != 0 ? p->rht_dense : nullptr;
  a.dense_scale = 1.0f / (float)sqrt(32.0);
  if ((p->scale_flags & ALTOB200_RHT_DENSE32) != 0) {
    if (a.dense == nullptr || p->rht_n != 0) return ALTOB200_EINVAL_SHAPE;
    if (p->format != ALTOB200_FMT_MXFP4 || p->in_dtype != ALTOB200_DT_BF16 ||
        (p->rounding != ALTOB200_ROUND_RTN && p->rounding != ALTOB200_ROUND_SR_SLOTS))
      return ALTOB200_EUNSUPPORTED;
    if (!aligned16(a.dense)) return ALTOB200_EINVAL_ALIGN;
  }
  a.x = x; a.rows = rows; a.cols = cols; a.ld = ld;
  a.codes = (uint8_t*)codes; a.scale_plain = scale_plain; a.scale_packed = (uint8_t*)scale_packed;
  a.ncol_tiles = ceil_div(rows / B, 4);
  a.outer = p->outer_scale; a.rand_bits = p->rand_bits;
  a.tile_rows = p->rand_tile_rows; a.tile_pairs = p->rand_tile_pairs;
  if ((a.tile_rows != 0) != (a.tile_pairs != 0) || a.tile_rows < 0 || a.tile_pairs < 0) return ALTOB200_EINVAL_SHAPE;
  if (a.tile_rows != 0 && (rows >= (1ll << 32) || cols >= (1ll << 32) || a.tile_rows >= (1ll << 32) ||
                           a.tile_pairs >= (1ll << 32)))
    return ALTOB200_ELIMIT;
  // rows are a multiple of 32 here (see out_row_bytes): planes start and continue on 16-word boundaries
  a.rand_vec = aligned16(a.rand_bits) && (a.tile_rows == 0 || a.tile_pairs % 8 == 0);
  a.philox_seed = p->philox_seed; a.philox_offset = p->philox_offset;
  philox_make_keys(p->philox_seed, &a.pk);
  int rc = fill_rht(&a.rht, p->rht_n, p->rht_perm, p->rht_sign);
  if (rc != ALTOB200_OK) return rc;
  fill_rht_row_offsets(&a.rht, ld, p->in_dtype == ALTOB200_DT_BF16 ? 2 : 4);
  rc = fill_mx_opts(&a.mx, p, true);
  if (rc != ALTOB200_OK) return rc;
  rc = clear_packed_if_padded(scale_packed, cols, rows / B, st);
  if (rc != ALTOB200_OK) return rc;
  const int rounding = p->rounding;
#define CALL_COL(F, BF) launch_colwise<F, BF>(a, rounding, st)
  DISPATCH_FMT_DT(p->format, p->in_dtype, CALL_COL);
#undef CALL_COL
}

int altob200_quantize_2d(const void* w, int64_t rows, int64_t cols, int64_t ld,
                         const altob200_quant_params* p, void* codes_k, void* codes_t,
                         void* scale_plain, void* scale_packed_k, void* scale_packed_t,
                         void* stream) {
  return altob200_quantize_2d_batched(w, 1, rows * ld, rows, cols, ld, p, codes_k, codes_t, scale_plain,
                                      scale_packed_k, scale_packed_t, stream);
}

int altob200_quantize_2d_batched(const void* w, int64_t batch, int64_t batch_stride, int64_t rows, int64_t cols,
                                 int64_t ld, const altob200_quant_params* p, void* codes_k, void* codes_t,
                                 void* scale_plain, void* scale_packed_k, void* scale_packed_t, void* stream) {
  if (w == nullptr || p == nullptr || codes_k == nullptr || batch <= 0) return ALTOB200_EINVAL_SHAPE;
  const int B = block_of(p->format);
  if (rows <= 0 || cols <= 0 || rows % B != 0 || cols % B != 0 || ld < cols) return ALTOB200_EINVAL_SHAPE;
  if (p->rht_n != 0) return ALTOB200_EUNSUPPORTED;
  if (p->rounding != ALTOB200_ROUND_RTN && p->rounding != ALTOB200_ROUND_SR_BITS) return ALTOB200_EUNSUPPORTED;
  if (p->rounding == ALTOB200_ROUND_SR_BITS && (p->rand_bits == nullptr || !aligned16(p->rand_bits)))
    return ALTOB200_EINVAL_SHAPE;
  const int esz = p->in_dtype == ALTOB200_DT_BF16 ? 2 : 4;
  if (!aligned16(w) || (ld * esz) % 16 != 0 || !aligned16(codes_k)) return ALTOB200_EINVAL_ALIGN;
  if (codes_t != nullptr && !aligned16(codes_t)) return ALTOB200_EINVAL_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  Quant2dArgs a;
  a.macro_codes = macro_codes_of(p);
  if (a.macro_codes != nullptr && (p->format != ALTOB200_FMT_MXFP4 || p->in_dtype != ALTOB200_DT_BF16))
    return ALTOB200_EUNSUPPORTED;
  a.w = w; a.rows = rows; a.cols = cols; a.ld = ld;
  a.codes_k = (uint8_t*)codes_k; a.codes_t = (uint8_t*)codes_t; a.scale_plain = scale_plain;
  a.packed_k = (uint8_t*)scale_packed_k; a.packed_t = (uint8_t*)scale_packed_t;
  a.nct_k = ceil_div(cols / B, 4); a.nct_t = ceil_div(rows / B, 4);
  a.batch = batch; a.batch_stride = batch_stride;
  a.packed_k_bytes = altob200_packed_scale_bytes(rows, cols / B);
  a.packed_t_bytes = altob200_packed_scale_bytes(cols, rows / B);
  if (batch > 1 && ((batch_stride * (p->in_dtype == ALTOB200_DT_BF16 ? 2 : 4)) % 16 != 0 ||
                    (rows * (is_fp4(p->format) ? cols / 2 : cols)) % 16 != 0))
    return ALTOB200_EINVAL_ALIGN;
  a.outer = p->outer_scale;
  a.rand_bits = p->rand_bits; a.tile_rows = p->rand_tile_rows; a.tile_pairs = p->rand_tile_pairs;
  if ((a.tile_rows != 0) != (a.tile_pairs != 0) || a.tile_rows < 0 || a.tile_pairs < 0 || (a.tile_pairs & 3) != 0)
    return ALTOB200_EINVAL_SHAPE;
  if (a.tile_rows >= (1ll << 32) || a.tile_pairs >= (1ll << 32)) return ALTOB200_ELIMIT;
  int rc = fill_mx_opts(&a.mx, p, true);
  if (rc != ALTOB200_OK) return rc;
  // padding entries of the packed layouts are zero (the kernel does not visit them)
  if (scale_packed_k != nullptr && ((rows & 127) != 0 || ((cols / B) & 3) != 0))
    ALTOB200_CUDA_CHECK(cudaMemsetAsync(scale_packed_k, 0, (size_t)(batch * a.packed_k_bytes), st));
  if (scale_packed_t != nullptr && ((cols & 127) != 0 || ((rows / B) & 3) != 0))
    ALTOB200_CUDA_CHECK(cudaMemsetAsync(scale_packed_t, 0, (size_t)(batch * a.packed_t_bytes), st));
  const int rounding = p->rounding;
#define CALL_2D(F, BF) launch_2d<F, BF>(a, rounding, st)
  DISPATCH_FMT_DT(p->format, p->in_dtype, CALL_2D);
#undef CALL_2D
}

int altob200_amax(const void* x, int32_t in_dtype, int64_t rows, int64_t cols, int64_t ld,
                  int32_t rht_n, const int32_t* rht_perm, const int32_t* rht_sign,
                  uint32_t* amax_bits, float* outer_scale, void* scratch, void* stream) {
  if (x == nullptr || amax_bits == nullptr || scratch == nullptr) return ALTOB200_EINVAL_SHAPE;
  if (rows <= 0 || cols <= 0 || cols % 8 != 0 || ld < cols) return ALTOB200_EINVAL_SHAPE;
  if (rht_n != 0 && rows % rht_n != 0) return ALTOB200_EINVAL_SHAPE;
  const int esz = in_dtype == ALTOB200_DT_BF16 ? 2 : 4;
  if (!aligned16(x) || (ld * esz) % 16 != 0) return ALTOB200_EINVAL_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  AmaxArgs a;
  a.x = x; a.rows = rows; a.cols = cols; a.ld = ld;
  a.amax_bits = amax_bits; a.outer_scale = outer_scale; a.counter = (uint32_t*)scratch;
  int rc = fill_rht(&a.rht, rht_n, rht_perm, rht_sign);
  if (rc != ALTOB200_OK) return rc;
  fill_rht_row_offsets(&a.rht, ld, esz);
  const int64_t work = rht_n ? (rows / 16) * ceil_div(cols, 64) / 8 + 1
                             : rows * cols / (16 / esz) / 256 + 1;
  int64_t blocks = work;
  const int64_t cap = (int64_t)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  const int64_t vecs = rows * (cols * esz / 16), steps = ceil_div(vecs, blocks * 256);
  a.steps = (int32_t)(vecs >= 9 * blocks * 256 ? 8 : steps < 4 ? steps : 4);
  const bool bf = in_dtype == ALTOB200_DT_BF16;
  if (rht_n) {
    if (bf) (void)launch_after(amax_kernel<true, true>, dim3((unsigned)blocks), dim3(256), 0, st, a);
    else (void)launch_after(amax_kernel<false, true>, dim3((unsigned)blocks), dim3(256), 0, st, a);
  } else {
    const auto kernel = a.steps == 8 ? (bf ? amax_kernel<true, false, 8> : amax_kernel<false, false, 8>)
                                     : (bf ? amax_kernel<true, false, 4> : amax_kernel<false, false, 4>);
    (void)launch_after(kernel, dim3((unsigned)blocks), dim3(256), 0, st, a);
  }
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

int altob200_dequantize(const void* codes, const void* scale_plain, const float* outer_scale,
                        int32_t format, int32_t is_2d, int64_t rows, int64_t cols,
                        int32_t out_dtype, void* out, int64_t ld_out, void* stream) {
  if (codes == nullptr || scale_plain == nullptr || out == nullptr) return ALTOB200_EINVAL_SHAPE;
  const int B = block_of(format);
  if (rows <= 0 || cols <= 0 || cols % B != 0 || ld_out < cols) return ALTOB200_EINVAL_SHAPE;
  if ((is_2d & 1) && rows % B != 0) return ALTOB200_EINVAL_SHAPE;
  const int esz = out_dtype == ALTOB200_DT_BF16 ? 2 : 4;
  if (!aligned16(codes) || !aligned16(out) || (ld_out * esz) % 16 != 0) return ALTOB200_EINVAL_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  DequantArgs a;
  a.codes = (const uint8_t*)codes; a.scales = scale_plain; a.outer = outer_scale;
  a.rows = rows; a.cols = cols; a.ld_out = ld_out; a.out = out; a.is_2d = is_2d & 1;
  a.static_clip = (is_2d >> 1) & 1;
  if (a.static_clip && format != ALTOB200_FMT_MXFP4) return ALTOB200_EUNSUPPORTED;
  // (a vector per thread before any thread takes several: 1024 x 1024 FP8 -> bf16 1.6 us, 2.3 the other way round)
  int64_t blocks = ceil_div(rows * (cols * esz / 16), 256);
  const int64_t cap = (int64_t)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  const bool bf = out_dtype == ALTOB200_DT_BF16;
#define LAUNCH_DQ(F)                                                              \
  if (bf) (void)launch_after(dequantize_kernel<F, true>, dim3((unsigned)blocks), dim3(256), 0, st, a);        \
  else (void)launch_after(dequantize_kernel<F, false>, dim3((unsigned)blocks), dim3(256), 0, st, a);          \
  break;
  switch (format) {
    case ALTOB200_FMT_NVFP4: LAUNCH_DQ(ALTOB200_FMT_NVFP4)
    case ALTOB200_FMT_MXFP4: LAUNCH_DQ(ALTOB200_FMT_MXFP4)
    case ALTOB200_FMT_MXFP8_E4M3: LAUNCH_DQ(ALTOB200_FMT_MXFP8_E4M3)
    case ALTOB200_FMT_MXFP8_E5M2: LAUNCH_DQ(ALTOB200_FMT_MXFP8_E5M2)
    default: return ALTOB200_EUNSUPPORTED;
  }
#undef LAUNCH_DQ
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

int altob200_rht(const void* x, int32_t dtype, int64_t rows, int64_t cols, int64_t ld,
                 int32_t rht_n, const int32_t* rht_perm, const int32_t* rht_sign, void* y,
                 int64_t ld_y, void* stream) {
  if (x == nullptr || y == nullptr) return ALTOB200_EINVAL_SHAPE;
  if (rht_n != 16) return ALTOB200_EUNSUPPORTED;
  if (rows <= 0 || cols <= 0 || rows % 16 != 0 || cols % 8 != 0 || ld < cols || ld_y < cols)
    return ALTOB200_EINVAL_SHAPE;
  const int esz = dtype == ALTOB200_DT_BF16 ? 2 : 4;
  if (!aligned16(x) || !aligned16(y) || (ld * esz) % 16 != 0 || (ld_y * esz) % 16 != 0)
    return ALTOB200_EINVAL_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  RhtArgs a;
  a.x = x; a.y = y; a.rows = rows; a.cols = cols; a.ld = ld; a.ld_y = ld_y;
  int rc = fill_rht(&a.rht, rht_n, rht_perm, rht_sign);
  if (rc != ALTOB200_OK) return rc;
  int64_t blocks = (rows / 16) * ceil_div(cols, 64) / 8 + 1;
  const int64_t cap = (int64_t)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  if (dtype == ALTOB200_DT_BF16) (void)launch_after(rht_kernel<true>, dim3((unsigned)blocks), dim3(256), 0, st, a);
  else (void)launch_after(rht_kernel<false>, dim3((unsigned)blocks), dim3(256), 0, st, a);
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

int altob200_amax_noalloc(const void* x, int32_t in_dtype, int64_t rows, int64_t cols, int64_t ld,
                          uint32_t* amax_bits, float* outer_scale, void* stream) {
  if (x == nullptr || amax_bits == nullptr) return ALTOB200_EINVAL_SHAPE;
  if (rows <= 0 || cols <= 0 || cols % 8 != 0 || ld < cols) return ALTOB200_EINVAL_SHAPE;
  if (in_dtype != ALTOB200_DT_BF16 && in_dtype != ALTOB200_DT_F32) return ALTOB200_EUNSUPPORTED;
  const int esz = in_dtype == ALTOB200_DT_BF16 ? 2 : 4;
  if (!aligned16(x) || (ld * esz) % 16 != 0) return ALTOB200_EINVAL_ALIGN;
  // the fixed array has one slot per block of 64 KiB of input
  if (rows > ALTOB200_NOALLOC_MAX_BYTES / esz / cols) return ALTOB200_ELIMIT;
  // Set-up, once per device, with that device current: the array's name is only a host-side
  // handle, the kernel needs the device address behind it.
  // The cache is atomic because the first calls on a device may come from two host threads at
  // once (they would store the same address).  The address stays valid for the life of the
  // device's context; after cudaDeviceReset it must not be used, so a process that resets a
  // device must not call this entry point on it again.
  static std::atomic<void*> scratch_of_device[64];
  int dev = 0;
  ALTOB200_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return ALTOB200_ELIMIT;
  void* cached = scratch_of_device[dev].load(std::memory_order_acquire);
  if (cached == nullptr) {
    void* ptr = nullptr;
    ALTOB200_CUDA_CHECK(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    if (ptr == nullptr) return ALTOB200_ECUDA;
    scratch_of_device[dev].store(ptr, std::memory_order_release);
    cached = ptr;
  }
  NoallocScratch* scratch = reinterpret_cast<NoallocScratch*>(cached);
  cudaStream_t st = (cudaStream_t)stream;
  // the counter must start at zero even if an earlier launch never finished
  ALTOB200_CUDA_CHECK(cudaMemsetAsync(&scratch->counter, 0, sizeof(uint32_t), st));
  AmaxNoallocArgs a;
  a.x = x; a.rows = rows; a.cols = cols; a.ld = ld;
  a.amax_bits = amax_bits; a.outer_scale = outer_scale; a.scratch = scratch;
  const int64_t total_vec = rows * (cols / (16 / esz));
  const int64_t blocks = ceil_div(total_vec, 256 * NOALLOC_VEC_PER_THREAD);
  if (blocks > NOALLOC_MAX_BLOCKS) return ALTOB200_ELIMIT;
  if (in_dtype == ALTOB200_DT_BF16) amax_noalloc_kernel<true><<<(unsigned)blocks, 256, 0, st>>>(a);
  else amax_noalloc_kernel<false><<<(unsigned)blocks, 256, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? ALTOB200_OK : ALTOB200_ECUDA;
}

}  // extern "C"
