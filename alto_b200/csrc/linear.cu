// Backward pass of one dense block-scaled linear behind one call: the launches that alto_b200/_linear.py makes for it
// (alto/kernels/fp4/nvfp4/nvfp_linear.py:160-278, alto/kernels/fp4/mxfp4/mxfp_linear.py:431-570,
// alto/kernels/mxfp8/mxfp8_linear.py:378-439), in the same order and with the same arguments.  Host code only.
// What it is for: a small layer's step is bound by the host.  At 256 x 512 x 384 (NVFP4, transform, stochastic
// rounding) the nine launches took 154 us through one Python call each with its allocations; the kernels take 29.
#include "common.cuh"

namespace {

struct Carver {             // pieces of one allocation, each on a 256-byte boundary
  uint8_t* base;
  int64_t used = 0;
  uint8_t* take(int64_t bytes) {
    uint8_t* p = base == nullptr ? nullptr : base + used;
    used += (bytes + 255) / 256 * 256;
    return p;
  }
};

struct Work {
  uint8_t *gn_codes, *gn_scales, *gm_codes, *gm_scales;
  uint32_t* amax;           // two words, then the two outer scales
  float* outer;
  uint32_t *words_n, *words_m;
};

bool fp4(int32_t f) { return f == ALTOB200_FMT_NVFP4 || f == ALTOB200_FMT_MXFP4; }

int64_t carve(const altob200_linear_backward_args& a, uint8_t* base, Work* w) {
  Carver c{base};
  const int64_t block = a.format == ALTOB200_FMT_NVFP4 ? 16 : 32, code_bytes = fp4(a.format) ? a.M * a.N / 2 : a.M * a.N;
  if (a.use_outer) {
    w->amax = (uint32_t*)c.take(16);
    w->outer = w->amax == nullptr ? nullptr : (float*)(w->amax + 2);
  }
  if (a.dx != nullptr) {
    w->gn_codes = c.take(code_bytes);
    w->gn_scales = c.take((int64_t)altob200_packed_scale_bytes(a.M, a.N / block));
    if (a.use_sr) w->words_n = (uint32_t*)c.take(64 * 64 * 4);
  }
  if (a.dw != nullptr) {
    w->gm_codes = c.take(code_bytes);
    w->gm_scales = c.take((int64_t)altob200_packed_scale_bytes(a.N, a.M / block));
    if (a.use_sr) w->words_m = (uint32_t*)c.take(64 * 64 * 4);
  }
  return c.used;
}

// the reference quantizer's (BLOCK_M, BLOCK_N / 2) for an axis-last view
void sr_tile(int64_t rows, int64_t cols, int64_t* tile_rows, int64_t* tile_pairs) {
  *tile_rows = rows >= 64 ? 64 : rows;
  *tile_pairs = (cols >= 64 ? 64 : cols) / 2;
}

}  // namespace

extern "C" int64_t altob200_linear_backward_work_bytes(const altob200_linear_backward_args* a) {
  Work w = {};
  return a == nullptr ? 0 : carve(*a, nullptr, &w);
}

extern "C" int altob200_linear_backward(const altob200_linear_backward_args* args, void* work, void* stream) {
  if (args == nullptr || work == nullptr || args->dy == nullptr || (args->use_outer && args->scratch == nullptr))
    return ALTOB200_EINVAL_SHAPE;
  const altob200_linear_backward_args& a = *args;
  if ((a.dx != nullptr && (a.wt_codes == nullptr || a.wt_scales == nullptr)) ||
      (a.dw != nullptr && (a.xm_codes == nullptr || a.xm_scales == nullptr)) || a.M <= 0 || a.K <= 0 || a.N <= 0 ||
      a.M % 32 != 0 || a.N % 32 != 0 || a.K % 32 != 0)
    return ALTOB200_EINVAL_SHAPE;
  // (the GEMMs would take a missing outer scale for 1)
  if (a.use_outer && ((a.dx != nullptr && a.wt_outer == nullptr) || (a.dw != nullptr && a.xm_outer == nullptr)))
    return ALTOB200_EINVAL_SHAPE;
  if (reinterpret_cast<uintptr_t>(work) & 15) return ALTOB200_EINVAL_ALIGN;
  Work w = {};
  carve(a, (uint8_t*)work, &w);
  int rc = ALTOB200_OK;
  if (a.use_outer) {
    rc = altob200_amax(a.dy, a.dtype, a.M, a.N, a.ld, a.rht_n, a.rht_perm, a.rht_sign, w.amax, w.outer, a.scratch, stream);
    if (rc != ALTOB200_OK) return rc;
  }
  altob200_quant_params p = {};
  p.format = a.format;
  p.in_dtype = a.dtype;
  p.scale_flags = ALTOB200_SCALE_PACKED;
  if (a.dx != nullptr) {
    altob200_quant_params q = p;
    q.outer_scale = w.outer;
    if (a.use_sr) {
      sr_tile(a.M, a.N, &q.rand_tile_rows, &q.rand_tile_pairs);
      rc = altob200_philox_tile(a.sr_words[0], a.sr_words[1], q.rand_tile_rows, q.rand_tile_pairs, w.words_n, stream);
      if (rc != ALTOB200_OK) return rc;
      q.rounding = ALTOB200_ROUND_SR_BITS;
      q.rand_bits = w.words_n;
    }
    rc = altob200_quantize_rowwise(a.dy, a.M, a.N, a.ld, &q, w.gn_codes, nullptr, w.gn_scales, stream);
    if (rc != ALTOB200_OK) return rc;
  }
  if (a.dw != nullptr) {
    altob200_quant_params q = p;
    q.outer_scale = w.outer == nullptr ? nullptr : w.outer + (a.rht_n != 0 ? 1 : 0);
    q.rht_n = a.rht_n;
    q.rht_perm = a.rht_perm;
    q.rht_sign = a.rht_sign;
    if (a.use_sr) {
      sr_tile(a.N, a.M, &q.rand_tile_rows, &q.rand_tile_pairs);
      const bool slots = q.rand_tile_rows == 64 && q.rand_tile_pairs == 32;
      rc = slots ? altob200_philox_slots(a.sr_words[2], a.sr_words[3], a.rht_n, a.rht_perm, w.words_m, stream)
                 : altob200_philox_tile(a.sr_words[2], a.sr_words[3], q.rand_tile_rows, q.rand_tile_pairs, w.words_m, stream);
      if (rc != ALTOB200_OK) return rc;
      q.rounding = slots ? ALTOB200_ROUND_SR_SLOTS : ALTOB200_ROUND_SR_BITS;
      q.rand_bits = w.words_m;
    }
    rc = altob200_quantize_colwise(a.dy, a.M, a.N, a.ld, &q, w.gm_codes, nullptr, w.gm_scales, stream);
    if (rc != ALTOB200_OK) return rc;
  }
  if (a.dx != nullptr) {
    rc = altob200_gemm_blockscaled(a.format, a.format, a.M, a.K, a.N, w.gn_codes, w.gn_scales, a.wt_codes, a.wt_scales,
                                   w.outer, a.wt_outer, a.dtype, a.dx, a.K, stream);
    if (rc != ALTOB200_OK) return rc;
  }
  if (a.dw != nullptr)
    rc = altob200_gemm_blockscaled(a.format, a.format, a.N, a.K, a.M, w.gm_codes, w.gm_scales, a.xm_codes, a.xm_scales,
                                   w.outer == nullptr ? nullptr : w.outer + (a.rht_n != 0 ? 1 : 0), a.xm_outer, a.dtype,
                                   a.dw, a.K, stream);
  return rc;
}
