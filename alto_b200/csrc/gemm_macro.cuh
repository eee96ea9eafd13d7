// MXFP4 block-scaled GEMM with two-level ("macro-block") scaling, for sm_100a.
//
//   D[m, n] = out_scale * sum over 128-wide chunks c of K of
//             (1 / fa[m, c]) * (1 / fb[n, c]) * sum_{k in chunk c} A[m, k] * B[n, k]
//
// A and B are MXFP4 operands (E2M1 codes, one E8M0 scale per 32 elements) that were quantised AFTER
// every block of 128 elements along K had been multiplied by a factor in [1, 2) (fa, fb: eight
// mantissa bits each, alto/kernels/fp4/mxfp4/macro_block_scaling.py:70-85).  The factors are not
// powers of two, so they cannot ride on the E8M0 scales of the block-scaled MMA; they are constant
// over a chunk of 128, so the tensor cores accumulate one chunk at a time into tensor memory and
// CUDA cores fold each finished chunk into the running fp32 result, which lives in registers.
// This replaces the reference's emulation of the recipe, dequantise -> descale -> bf16 matmul
// (alto/kernels/fp4/mxfp4/mxfp_linear.py:337-356, mxfp_grouped_gemm/cg_backward.py:668-690).
//
// One CTA (512 threads = four warpgroups, persistent over 128 x 2 HN output tiles, each two halves of HN = 128
// or 64 columns that share the A operand; `macro_half` in gemm_sm100.cu chooses):
//   warpgroup 0   warp 0: producer - per stage (128 bytes of K = two chunks) three tiled TMA loads and the
//                 bulk copies of the stage's scale tiles; warps 1 and 3: MMA issuers of the two halves - two
//                 tcgen05.mma per chunk into one of the chunk accumulators in tensor memory (HN = 128: three for
//                 both halves; 64: three for each), then a commit to that accumulator's "full" barrier; warp 2 idle;
//   warpgroup 1   scale transfer shared memory -> tensor memory (as in the plain kernel), and the macro
//                 factors: the codes of the tile's rows (and columns) for the next stage's two chunks are read
//                 a stage ahead and their reciprocals left in a shared-memory ring;
//   warpgroups 2-3  fold + epilogue of one half each: four warps, one per tensor-memory lane quarter, 32 rows
//                 x HN columns in HN registers per thread.  A chunk is read in pieces of 16 columns; HN = 128: one
//                 piece is always on its way from tensor memory while another is folded; 64: the registers hold
//                 the whole chunk, and each piece is requested for the next chunk as soon as it is folded.
//                 acc += P * (1/fa[row]) * (1/fb[col]) in packed fp32x2 arithmetic.  After the last chunk the
//                 registers are scaled, converted, staged and TMA-stored.
//
// What bounds it: HN = 128: the hand-over of the chunk accumulators between the MMAs and the fold (three fit beside
// the scales), then the fold itself, 64 (128 with per-column factors) packed operations of two cycles per scheduler
// and 128 x 128 x 128 block whose MMAs take 128 cycles.  HN = 64: the latency of a stage's barriers and of the fold
// (650 cycles a chunk of 128 x 128 with a CTA to itself), and where the whole chip works the shared-memory port,
// whose 17 KB of loads per block, against 13, took 284 cycles alone.
// Measured at 8192 x 4096 x 14336, one factor per tile of B / one per column: 451 / 571 us (HN = 128);
// with 128 x 128 tiles, sixteen fold warps of 32 columns that each looked up their factors, and one issuer:
// 572 / 924 us.  (Pieces of 32 columns: a few spilled registers more in the chunk loop of the per-column variant,
// local memory that this kernel's small L1 does not hold: + 10 %.)
// The warpgroups re-divide the register file with setmaxnreg (512 threads x 128 at launch -> 56 for the
// small roles, 200 for the fold warps; the two must balance exactly, see CfgMacro).
// Rows grouped by expert (`group_expert`) and K ranges per batch entry (`k_offs`) work as in the
// plain kernel; every K range starts on a multiple of 128 elements, so chunks never straddle one.
#pragma once
// (included by gemm_sm100.cu inside namespace altob200, after the plain kernels it shares helpers with)

struct MacroSide {
  const uint8_t* codes;     // factor codes: element (row r, chunk c) at ((r >> shift) * row_stride + c * chunk_stride)
  int64_t row_stride, chunk_stride;
  int64_t expert_stride;    // B only: added per expert in row-group mode
  int shift;                // 0: one factor per row; 7: one factor per 128 rows (2-D macro blocks)
};

// Quotients of tile numbers by a divisor fixed per launch: t / d = t * m >> s for t < 2^31, with
// s = 31 + ceil(log2 d) and m = floor(2^s / d) + 1.  A tile's coordinates are on the critical path of every role;
// with three 64-bit divides a weight gradient of 128 rows per expert (one chunk per tile) took 26 % longer
// (8 experts, 2880 x 2880: 64.5 us, now 51.4).
struct TileDiv {
  uint32_t d, m;
  int s;
  __device__ __forceinline__ uint32_t quotient(uint32_t t) const { return (uint32_t)(((uint64_t)t * m) >> s); }
};
static TileDiv make_tile_div(int64_t d) {
  TileDiv v;
  v.d = (uint32_t)d;
  v.s = 31;
  while ((1ll << (v.s - 31)) < d) ++v.s;
  v.m = (uint32_t)(((unsigned __int128)1 << v.s) / (uint64_t)d + 1);
  return v;
}

struct MacroGemmArgs {
  GemmArgs g;
  MacroSide ma, mb;
  TileDiv per_batch, per_group, rows_full, rows_last;   // tiles per batch, per raster group; row tiles of a group
  float out_scale;
};

constexpr int NUM_THREADS_MACRO = 512;

// HN: columns of a half.  128: the halves share three accumulators; 64: each half has three of its own.
template <int HN_>
struct CfgMacro {
  static constexpr int HN = HN_;                                // columns of a half (one chunk accumulator)
  static_assert(HN == 128 || HN == 64, "halves");
  static constexpr int BN = 2 * HN;
  static constexpr int SF_TILES = Kind<KIND_MXF4>::SF_TILES;
  static constexpr int A_BYTES = BM * STAGE_K_BYTES;
  static constexpr int B_BYTES = HN * STAGE_K_BYTES;            // per half
  static constexpr int SF_BYTES = SF_TILES * 512;               // per 128 rows of either operand
  static constexpr int SFB_BLOCKS = BN / 128;                   // 128-row blocks of B's scales under a tile
  static constexpr int SF_OFF = A_BYTES + 2 * B_BYTES;          // scales of A, then of B's blocks
  static constexpr int STAGE_BYTES = SF_OFF + (1 + SFB_BLOCKS) * SF_BYTES;
  static_assert(STAGE_BYTES % 1024 == 0, "stages must keep the 128-byte swizzle atom aligned");
  static constexpr int SF_COLS = SF_TILES * 4;                  // tensor-memory columns of SF_BYTES
  static constexpr int STAGE_SF_COLS = (1 + SFB_BLOCKS) * SF_COLS;
  static constexpr int STAGES = HN == 128 ? 3 : 4;
  static constexpr int RING = 3;                                // chunk barriers per half, each way
  static constexpr bool OWN_BUFS = HN == 64;
  static constexpr int P_BUFS = OWN_BUFS ? 2 * RING : 3;        // chunk accumulators in tensor memory
  static constexpr int PIECES = HN / 16;
  static constexpr int FOLD_WARPS = 8;                          // four per half
  static constexpr int EPI_UNIT = 2048;                         // 16 rows x 128 bytes
  static constexpr int EPI_WARP_BYTES = 2 * EPI_UNIT;
  static constexpr int EPI_BYTES = FOLD_WARPS * EPI_WARP_BYTES;
  // Ring of reciprocal factors, per chunk 128 rows and BN columns (B_UNIFORM: the products of both, 128 rows per
  // 128 columns).  No barrier guards its reuse: a slot is rewritten FAC_STAGES stages after its last use, once
  // that stage's operands have landed, so the MMAs of the stage STAGES earlier are done, and with them (see
  // the issuers) both halves have read out every chunk up to two before (three with accumulators of their own) -
  // at least one after the slot's own, which has therefore been folded.
  static constexpr int FAC_STAGES = 8;
  static constexpr int FAC_STRIDE = BM + BN + 4;                // floats per chunk; + 4 spreads the banks
  static constexpr int FAC_BYTES = 2 * FAC_STAGES * FAC_STRIDE * 4;
  static_assert(FAC_STAGES >= STAGES + (OWN_BUFS ? 4 : 3), "factors are overwritten while they are in use");
  static constexpr int RCP_BYTES = 256 * 4;                     // 1 / factor for every code
  static constexpr int TMEM_SF_BASE = P_BUFS * HN;
  static constexpr int TMEM_COLS_USED = TMEM_SF_BASE + STAGES * STAGE_SF_COLS;
  static_assert(TMEM_COLS_USED <= 512, "tensor memory budget");
  static constexpr int NUM_BARS = 3 * STAGES + 4 * RING;
  static constexpr int SMEM_BYTES =
      STAGES * STAGE_BYTES + EPI_BYTES + FAC_BYTES + RCP_BYTES + 1024 /*align*/ + 512 /*barriers*/;
  static_assert(NUM_BARS * 8 + 16 <= 512, "barrier area");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  // Registers per thread after the warpgroups have re-divided the file.  The CTA is launched with 128
  // registers per thread (65536 / 512); setmaxnreg.inc can only take what setmaxnreg.dec has released
  // INSIDE the CTA and blocks for ever otherwise, so the two must balance exactly.
  static constexpr int REGS_LAUNCH = 128;
  static constexpr int REGS_SMALL = 56, REGS_FOLD = 200;
  static_assert(2 * 128 * REGS_SMALL + 2 * 128 * REGS_FOLD == NUM_THREADS_MACRO * REGS_LAUNCH,
                "setmaxnreg budget must balance");
  static_assert(NUM_THREADS_MACRO == (8 + FOLD_WARPS) * 32, "role layout");
};

// Tile description plus what the chunk loop needs: the first chunk of the K range, the number of
// chunks, and MMAs per stage limited to the bytes that exist (also without K ranges).
struct MacroTile {
  TileInfo t;
  int64_t chunk0;
  int n_chunks;
  int expert;
  int halves;       // 1 when the tile's second half lies outside the matrix
};

// (the raster of decode_tile: groups of `group_m` row tiles, each swept across all column tiles, row tile fastest)
template <class C>
__device__ __forceinline__ MacroTile decode_macro_tile(const MacroGemmArgs& margs, uint32_t tile, int k_stages_dense) {
  const GemmArgs& args = margs.g;
  MacroTile m;
  TileInfo& t = m.t;
  const uint32_t e = args.k_offs != nullptr ? margs.per_batch.quotient(tile) : 0u;
  const uint32_t rem = tile - e * margs.per_batch.d;
  const uint32_t g = margs.per_group.quotient(rem);
  const uint32_t in_group = rem - g * margs.per_group.d;
  const bool last_group = (uint64_t)(g + 1) * margs.per_group.d >= margs.per_batch.d;
  const TileDiv rows = last_group ? margs.rows_last : margs.rows_full;
  const uint32_t nb = rows.quotient(in_group);
  t.nb = nb;
  t.mb = (int64_t)g * args.group_m + (in_group - nb * rows.d);
  t.batch = (int)e;
  t.k_byte0 = 0;
  t.sf_tile0 = 0;
  t.b_row0 = t.nb * C::BN;
  t.sfb = args.sfb;
  t.skip = false;
  m.expert = 0;
  m.chunk0 = 0;
  int64_t bytes = args.k_bytes;
  if (args.k_offs != nullptr) {
    const int64_t k0 = e > 0 ? __ldg(args.k_offs + e - 1) : 0;
    const int64_t k1 = __ldg(args.k_offs + e);
    bytes = (k1 - k0) / 2;
    t.skip = bytes <= 0;
    t.k_stages = (int)((bytes + STAGE_K_BYTES - 1) / STAGE_K_BYTES);
    t.k_byte0 = k0 / 2;
    t.sf_tile0 = k0 >> 7;
    m.chunk0 = k0 >> 7;
  } else {
    t.k_stages = k_stages_dense;
    if (args.num_experts > 0) {
      const int ex = __ldg(args.group_expert + t.mb);
      t.skip = ex < 0;
      if (!t.skip) {
        m.expert = ex;
        t.b_row0 += (int64_t)ex * args.N;
        t.sfb += (int64_t)ex * args.sfb_expert_stride;
      }
    }
  }
  const int64_t tail = bytes - (int64_t)(t.k_stages - 1) * STAGE_K_BYTES;
  t.last_mmas = (int)((tail + 31) / 32);
  m.n_chunks = bytes > 0 ? (int)((bytes + 63) / 64) : 0;
  m.halves = args.N - t.nb * C::BN > C::HN ? 2 : 1;
  return m;
}

// One piece of a chunk accumulator: 16 columns of a warp's 32 rows, as two tensor-memory loads of 16 rows in
// the 16 x 256-bit layout.  A lane gets, per group of eight columns, columns 2 (lane % 4) and + 1 of rows
// lane / 4 and + 8 of each load: four rows and four columns of the piece, so that it needs eight factors,
// where the layout of one row per lane needs 17 and the broadcast of the column factors out of shared memory
// (128 bytes per register and warp) took longer than the multiply-adds.
struct Piece {
  uint32_t r[16];   // [row half 2][column group 2][row 2][column 2]
};
__device__ __forceinline__ void tc_ld_piece(uint32_t taddr, Piece& p) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t* r = p.r + 8 * h;
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x2.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr + ((uint32_t)(16 * h) << 16))
        : "memory");
  }
}
// tcgen05.wait::ld that the values in p depend on: nothing that uses them can move above it
__device__ __forceinline__ void tc_wait_piece(Piece& p) {
#define ALTOB200_RW8(o) "+r"(p.r[o]), "+r"(p.r[o + 1]), "+r"(p.r[o + 2]), "+r"(p.r[o + 3]), "+r"(p.r[o + 4]), \
                        "+r"(p.r[o + 5]), "+r"(p.r[o + 6]), "+r"(p.r[o + 7])
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : ALTOB200_RW8(0), ALTOB200_RW8(8)
               :
               : "memory");
}
// the same for a piece whose load an earlier wait has covered
__device__ __forceinline__ void tc_landed_piece(Piece& p) { asm volatile("" : ALTOB200_RW8(0), ALTOB200_RW8(8)); }
#undef ALTOB200_RW8
__device__ __forceinline__ float ld_shared_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float2 ld_shared_f32x2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint64_t* generic_bar(uint32_t addr) {
  return reinterpret_cast<uint64_t*>(__cvta_shared_to_generic(addr));
}

// One look at a barrier's phase, without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// acc += P * ra[row] * fb[col]; B_UNIFORM: one B factor for the half and chunk, already multiplied into ra.
// `acc` and `p` are laid out alike; fb: shared-memory address of this lane's first column factor.
template <bool B_UNIFORM>
__device__ __forceinline__ void fold_piece(float2* acc, const Piece& p, const float (&ra)[4], uint32_t fb) {
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    float2 f = make_float2(1.0f, 1.0f);
    if (!B_UNIFORM) f = ld_shared_f32x2(fb + 32 * g);
#pragma unroll
    for (int q = 0; q < 4; ++q) {   // row half q / 2, row 8 (q % 2)
      const int i = (q >> 1) * 4 + g * 2 + (q & 1);
      float2 w = make_float2(ra[q], ra[q]);
      if (!B_UNIFORM) w = __fmul2_rn(w, f);
      acc[i] = __ffma2_rn(make_float2(u2f(p.r[2 * i]), u2f(p.r[2 * i + 1])), w, acc[i]);
    }
  }
}

// B_UNIFORM: B's macro blocks are 128 x 128 tiles (one factor per half and chunk), else per column.
template <int HN, bool B_UNIFORM>
__global__ void __launch_bounds__(NUM_THREADS_MACRO, 1)
gemm_macro_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_d, const MacroGemmArgs margs) {
  using C = CfgMacro<HN>;
  const GemmArgs& args = margs.g;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi = smem + C::STAGES * C::STAGE_BYTES;
  float* fac = reinterpret_cast<float*>(epi + C::EPI_BYTES);
  float* rcp_tab = reinterpret_cast<float*>(epi + C::EPI_BYTES + C::FAC_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi + C::EPI_BYTES + C::FAC_BYTES + C::RCP_BYTES);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::STAGES;
  uint64_t* sf_full = bars + 2 * C::STAGES;
  uint64_t* p_full = bars + 3 * C::STAGES;        // [half][chunk % RING]
  uint64_t* p_empty = p_full + 2 * C::RING;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(p_empty + 2 * C::RING);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (an output of 2^31 tiles would not fit any memory)
  const int n_tiles = (int)(margs.per_batch.d * (args.k_offs != nullptr ? args.num_batches : 1));
  const int k_stages = (int)((args.k_bytes + STAGE_K_BYTES - 1) / STAGE_K_BYTES);

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 2);
      mbar_init(&sf_full[s], 4);
    }
    for (int p = 0; p < 2 * C::RING; ++p) {
      mbar_init(&p_full[p], 1);
      mbar_init(&p_empty[p], C::FOLD_WARPS / 2);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // scale staging starts from zero: a ragged last stage never feeds uninitialised scale bytes
  for (int s = 0; s < C::STAGES; ++s) {
    uint32_t* z = reinterpret_cast<uint32_t*>(smem + s * C::STAGE_BYTES + C::SF_OFF);
    for (int i = threadIdx.x; i < (1 + C::SFB_BLOCKS) * C::SF_BYTES / 4; i += NUM_THREADS_MACRO) z[i] = 0u;
  }
  // 1 / factor(code), factor = 1 + code / 256 (exact), correctly rounded
  if (threadIdx.x < 256) rcp_tab[threadIdx.x] = __frcp_rn(u2f((threadIdx.x << 15) + (127u << 23)));
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_wait();   // set-up done; global memory from here on (programmatic dependent launch)

  if (warp < 4) {
    setmaxnreg_dec<C::REGS_SMALL>();
    // Producer and MMA issuer: the WHOLE warp runs the loop and waits on the barriers, one elected lane
    // issues the TMA / tcgen05 instructions.  Those instructions take their operands (descriptors,
    // addresses, coordinates) from uniform registers; computed by a converged warp from kernel parameters
    // and loop counters they are uniform values from the start, whereas the same arithmetic inside an
    // `if (lane == 0)` region yields per-thread values that have to be moved to uniform registers one by
    // one in front of every instruction (measured: ~270 cycles per tcgen05.mma).
    if (warp == 0) {
      // ------------------------------ producer ------------------------------
      const bool elected = elect_one();
      uint32_t it = 0;
      bool alive = true;
      for (int tile = (int)blockIdx.x; tile < n_tiles && alive; tile += (int)gridDim.x) {
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
        const TileInfo& ti = mt.t;
        if (ti.skip) continue;
        const int64_t mb = ti.mb, nb = ti.nb;
        for (int ks = 0; ks < ti.k_stages; ++ks, ++it) {
          const int s = it % C::STAGES;
          alive = __all_sync(0xFFFFFFFFu,
                             mbar_wait(&empty_bar[s], ((it / C::STAGES) & 1) ^ 1, abort_flag, 21, args.wait_ns));
          if (!alive) break;
          uint8_t* st = smem + s * C::STAGE_BYTES;
          const int64_t cb0 = ti.sf_tile0 + (int64_t)ks * C::SF_TILES;
          int64_t sf_tiles = args.nct - cb0;
          if (sf_tiles > C::SF_TILES) sf_tiles = C::SF_TILES;
          const uint32_t sf_bytes = (uint32_t)sf_tiles * 512u;
          const int32_t kx = (int32_t)(ti.k_byte0 + (int64_t)ks * STAGE_K_BYTES);
          if (elected) {
            const uint32_t n_b = (uint32_t)mt.halves, n_sfb = C::SFB_BLOCKS == 2 ? n_b : 1u;
            mbar_expect_tx(&full_bar[s], C::A_BYTES + n_b * C::B_BYTES + (1u + n_sfb) * sf_bytes);
            tma_load_2d(st, &tmap_a, kx, (int32_t)(mb * BM), &full_bar[s]);
            bulk_load(st + C::SF_OFF, args.sfa + (mb * args.nct + cb0) * 512, sf_bytes, &full_bar[s]);
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
              if (h < n_b)
                tma_load_2d(st + C::A_BYTES + h * C::B_BYTES, &tmap_b, kx, (int32_t)(ti.b_row0 + h * HN), &full_bar[s]);
              if (h < n_sfb)
                bulk_load(st + C::SF_OFF + (1 + h) * C::SF_BYTES, ti.sfb + ((nb * C::SFB_BLOCKS + h) * args.nct + cb0) * 512,
                          sf_bytes, &full_bar[s]);
            }
          }
        }
      }
    } else if (warp == 1 || warp == 3) {
      // ------------------------------ MMA issuers ------------------------------
      // One per half: a tcgen05.mma does not run ahead of its thread's other instructions, so while one
      // issuer waits for its barriers (~150 cycles even when they are complete) the other one's MMAs keep the
      // tensor pipe busy.
      // Chunk n of half h goes to accumulator (2 n + h) % 3, which held chunk n - 2 of half 1 (h = 0) or
      // chunk n - 1 of half 0 (h = 1); with accumulators of their own to 2 (n % 3) + h, which held chunk n - 3 of
      // the same half.  The barriers count the chunks of one half, so that whoever waits on one has waited for
      // all its earlier phases.  A half outside the matrix runs the protocol without MMAs.
      static_assert(C::RING == 3 && (C::OWN_BUFS ? C::P_BUFS == 6 : C::P_BUFS == 3), "order of the accumulators");
      const bool elected = elect_one();
      const int h = warp >> 1;
      uint32_t it = 0, n = 0;         // stages and chunks so far
      bool alive = true;
      const uint32_t smem_base = smem_u32(smem);
      uint64_t* const my_full = p_full + h * C::RING;
      uint64_t* const drained = p_empty + (C::OWN_BUFS ? h : h ^ 1) * C::RING;
      const uint32_t back = C::OWN_BUFS ? 3u : h == 0 ? 2u : 1u;
      for (int tile = (int)blockIdx.x; tile < n_tiles && alive; tile += (int)gridDim.x) {
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
        const TileInfo& ti = mt.t;
        if (ti.skip) continue;
        const bool mine = h < mt.halves;
        for (int ks = 0; ks < ti.k_stages; ++ks, ++it) {
          const int n_mma = (ks == ti.k_stages - 1) ? ti.last_mmas : 4;
          const int s = it % C::STAGES;
          const uint32_t sfa_t = tmem_base + C::TMEM_SF_BASE + s * C::STAGE_SF_COLS;
          // (a block of 128 rows is four columns per 128 bytes of K, 32 rows each: row 64 is two columns on)
          const uint32_t sfb_t = sfa_t + C::SF_COLS + (HN == 128 ? h * C::SF_COLS : 2 * h);
          const uint32_t a_lo = ((smem_base + (uint32_t)s * C::STAGE_BYTES) >> 4) | 0x10000u;
          const uint32_t b_lo = a_lo + ((C::A_BYTES + h * C::B_BYTES) >> 4);
          // operands and scales of the stage are in place; the three barriers are looked at together, since the
          // answer of one takes as long as that of all
          const uint32_t st_phase = (it / C::STAGES) & 1, m0 = n - back;
          const bool s0 = mbar_test(smem_u32(&sf_full[s]), st_phase), s1 = mbar_test(smem_u32(&full_bar[s]), st_phase);
          const bool s2 = n < back || mbar_test(smem_u32(&drained[m0 % C::RING]), (m0 / C::RING) & 1);
          const uint32_t m1 = n + 1 - back;
          const bool s3 = n + 1 < back || mbar_test(smem_u32(&drained[m1 % C::RING]), (m1 / C::RING) & 1);
          bool ok = s0 || mbar_wait(&sf_full[s], st_phase, abort_flag, 25, args.wait_ns);
          ok = ok && (s1 || mbar_wait(&full_bar[s], st_phase, abort_flag, 23, args.wait_ns));
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (2 * c >= n_mma) break;
            // the chunk's accumulator is drained
            if (n >= back && !(c == 0 ? s2 : s3)) {
              const uint32_t m = n - back;
              ok = ok && mbar_wait(&drained[m % C::RING], (m / C::RING) & 1, abort_flag, 22, args.wait_ns);
            }
            alive = __all_sync(0xFFFFFFFFu, ok);
            if (!alive) break;
            tc_fence_after();
            if (elected) {
              if (mine) {
                const uint32_t acc_t = tmem_base + (C::OWN_BUFS ? 2 * (n % C::RING) + (uint32_t)h : (2 * n + (uint32_t)h) % 3u) * HN;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                  if (2 * c + j < n_mma)
                    tc_mma<KIND_MXF4>(acc_t, desc_of(DESC_SW128_HI, a_lo + 4 * c + 2 * j),
                                      desc_of(DESC_SW128_HI, b_lo + 4 * c + 2 * j), args.idesc[j], (uint32_t)j,
                                      sfa_t + c * 4, sfb_t + c * 4);
                }
              }
              tc_commit(&my_full[n % C::RING]);
            }
            ++n;
          }
          if (!alive) break;
          if (elected) tc_commit(&empty_bar[s]);   // both issuers
          __syncwarp();
        }
      }
    }
  } else if (warp < 8) {
    // ------------------------------ scale transfer and macro factors ------------------------------
    setmaxnreg_dec<C::REGS_SMALL>();
    const int quad = warp & 3;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    // factors: lane = (row of sixteen, chunk of the stage); the warp serves 32 rows of A and BN / 4 columns of B
    const int fc = lane & 1, fr = lane >> 1;
    uint32_t it = 0;
    bool alive = true;
    for (int tile = (int)blockIdx.x; tile < n_tiles && alive; tile += (int)gridDim.x) {
      const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
      const TileInfo& ti = mt.t;
      if (ti.skip) continue;
      const int64_t m0 = ti.mb * BM, n0 = ti.nb * C::BN;
      const uint8_t* pa = margs.ma.codes + (mt.chunk0 + fc) * margs.ma.chunk_stride +
                          (m0 >> margs.ma.shift) * margs.ma.row_stride;
      const uint8_t* pb = margs.mb.codes + (int64_t)mt.expert * margs.mb.expert_stride +
                          (mt.chunk0 + fc) * margs.mb.chunk_stride + (n0 >> margs.mb.shift) * margs.mb.row_stride;
      // offsets of the lane's rows from the tile's first (a row beyond the matrix reads the last one)
      constexpr int NB = B_UNIFORM ? C::SFB_BLOCKS : C::BN / 64;
      int64_t off_a[2], off_b[NB];
      const uint32_t m_last = (uint32_t)(args.M - m0 < BM ? args.M - m0 : BM) - 1u;
      const uint32_t n_last = (uint32_t)(args.N - n0 < C::BN ? args.N - n0 : C::BN) - 1u;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t r = (uint32_t)(quad * 32 + 16 * i + fr);
        off_a[i] = (int64_t)((r < m_last ? r : m_last) >> margs.ma.shift) * margs.ma.row_stride;
      }
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const uint32_t r = (uint32_t)(B_UNIFORM ? 128 * i : quad * (C::BN / 4) + 16 * i + fr);
        off_b[i] = (int64_t)((r < n_last ? r : n_last) >> (B_UNIFORM ? 7 : 0)) * margs.mb.row_stride;
      }
      uint32_t ca[2], cb[NB];
      auto load_codes = [&](int ks) {
        const bool have = 2 * ks + fc < mt.n_chunks;
#pragma unroll
        for (int i = 0; i < 2; ++i) ca[i] = have ? __ldg(pa + off_a[i]) : 0u;
#pragma unroll
        for (int i = 0; i < NB; ++i) cb[i] = have ? __ldg(pb + off_b[i]) : 0u;
        pa += 2 * margs.ma.chunk_stride;
        pb += 2 * margs.mb.chunk_stride;
      };
      load_codes(0);
      for (int ks = 0; ks < ti.k_stages; ++ks, ++it) {
        const int s = it % C::STAGES;
        if (!mbar_wait(&full_bar[s], (it / C::STAGES) & 1, abort_flag, 26, args.wait_ns)) { alive = false; break; }
        const uint8_t* sf = smem + s * C::STAGE_BYTES + C::SF_OFF + lane * 16;
        const uint32_t sf_t = tmem_base + lane_base + C::TMEM_SF_BASE + s * C::STAGE_SF_COLS;
#pragma unroll
        for (int t = 0; t < (1 + C::SFB_BLOCKS) * C::SF_TILES; ++t) {
          const uint4 a = *reinterpret_cast<const uint4*>(sf + t * 512);
          tc_st4(sf_t + t * 4, a.x, a.y, a.z, a.w);
        }
        float* dst = fac + (2 * (it % C::FAC_STAGES) + fc) * C::FAC_STRIDE + fr;
        if (B_UNIFORM) {
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            const float rb = rcp_tab[cb[j]];
#pragma unroll
            for (int i = 0; i < 2; ++i) dst[BM * j + quad * 32 + 16 * i] = __fmul_rn(rcp_tab[ca[i]], rb);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 2; ++i) dst[quad * 32 + 16 * i] = rcp_tab[ca[i]];
#pragma unroll
          for (int i = 0; i < NB; ++i) dst[BM + quad * (C::BN / 4) + 16 * i] = rcp_tab[cb[i]];
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sf_full[s]);
        if (ks + 1 < ti.k_stages) load_codes(ks + 1);
      }
    }
  } else {
    // ------------------------------ fold + epilogue ------------------------------
    setmaxnreg_inc<C::REGS_FOLD>();
    // Of the 200 registers, 160 are accumulators and pieces in flight: what else lives across the chunk loop is
    // kept in 32 bits (shared-memory addresses, tile numbers).
    const int quad = warp & 3;                        // tensor-memory lane quarter this warp may read
    const int half = (warp - 8) >> 2;                 // columns [HN half, HN half + HN) of the tile
    const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16);
    // this lane's first row and column factor in a chunk's slot
    const uint32_t fac_a = smem_u32(fac) + 4u * (uint32_t)((B_UNIFORM && C::SFB_BLOCKS == 2 ? half * BM : 0) + quad * 32 + (lane >> 2));
    const uint32_t fac_b = smem_u32(fac) + 4u * (uint32_t)(BM + half * HN + 2 * (lane & 3));
    const uint32_t my_full = smem_u32(p_full + half * C::RING), my_empty = smem_u32(p_empty + half * C::RING);
    uint32_t store_it = 0;                            // store units so far
    uint32_t slot = 0;                                // byte offset of the chunk's factors, always of an even slot at a tile's start
    // ring positions of the half's next chunk: its barriers (n % 3), their phase, its accumulator (see the issuers)
    uint32_t ring = 0, phase = 0, acc_i = (uint32_t)half;
    constexpr uint32_t SLOT_BYTES = C::FAC_STRIDE * 4, SLOTS_END = 2 * C::FAC_STAGES * SLOT_BYTES;
    bool alive = true;
    for (int tile = (int)blockIdx.x; tile < n_tiles && alive; tile += (int)gridDim.x) {
      int left, row0, col0, batch;                    // chunks left, this warp's part of the output
      bool mine;
      {
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
        left = mt.t.skip ? 0 : mt.n_chunks;
        mine = half < mt.halves;
        row0 = (int)mt.t.mb * BM + quad * 32;
        col0 = (int)mt.t.nb * C::BN + half * HN;
        batch = mt.t.batch;
      }
      auto step = [&]() {
        if (++ring == C::RING) {
          ring = 0;
          phase ^= 1u;
        }
        acc_i = C::OWN_BUFS ? 2u * ring + (uint32_t)half : acc_i == 0u ? 2u : acc_i - 1u;   // (+ 2 mod 3)
        slot = slot + SLOT_BYTES == SLOTS_END ? 0u : slot + SLOT_BYTES;
      };
      float2 acc[HN / 2];                             // [PIECES][Piece]
#pragma unroll
      for (int j = 0; j < HN / 2; ++j) acc[j] = make_float2(0.0f, 0.0f);
      const bool odd = (left & 1) != 0;
      if (left > 0) {
        alive = mbar_wait(generic_bar(my_full + 8 * ring), phase, abort_flag, 24, args.wait_ns);
        if (!alive) break;
      }
      if (!mine) {                                    // nothing to read, only the hand-over
        while (left > 0 && alive) {
          __syncwarp();
          if (lane == 0) mbar_arrive(generic_bar(my_empty + 8 * ring));
          step();
          if (--left > 0) alive = mbar_wait(generic_bar(my_full + 8 * ring), phase, abort_flag, 24, args.wait_ns);
        }
      } else if (left > 0) {
        uint32_t t_acc = t_row + acc_i * HN;
        tc_fence_after();
        if constexpr (C::OWN_BUFS) {
          // the whole chunk at once: a piece's registers take the next chunk's piece as soon as it is folded
          Piece pc[C::PIECES];
#pragma unroll
          for (int p = 0; p < C::PIECES; ++p) tc_ld_piece(t_acc + 16 * p, pc[p]);
          while (true) {
            const uint32_t fb = fac_b + slot;
            float ra[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) ra[q] = ld_shared_f32(fac_a + slot + 32 * q);
            const uint32_t gone = my_empty + 8 * ring;
            step();
            const bool ready = __all_sync(0xFFFFFFFFu, mbar_test(my_full + 8 * ring, phase)) && left > 1;
            tc_wait_piece(pc[0]);           // all of them
#pragma unroll
            for (int p = 1; p < C::PIECES; ++p) tc_landed_piece(pc[p]);
            tc_fence_before();
            if (lane == 0) mbar_arrive(generic_bar(gone));
            t_acc = t_row + acc_i * HN;
            if (ready) {
              tc_fence_after();
#pragma unroll
              for (int p = 0; p < C::PIECES; ++p) {
                fold_piece<B_UNIFORM>(acc + 8 * p, pc[p], ra, fb + 64 * p);
                tc_ld_piece(t_acc + 16 * p, pc[p]);
              }
              --left;
              continue;
            }
#pragma unroll
            for (int p = 0; p < C::PIECES; ++p) fold_piece<B_UNIFORM>(acc + 8 * p, pc[p], ra, fb + 64 * p);
            if (--left == 0) break;
            alive = mbar_wait(generic_bar(my_full + 8 * ring), phase, abort_flag, 24, args.wait_ns);
            if (!alive) break;
            tc_fence_after();
#pragma unroll
            for (int p = 0; p < C::PIECES; ++p) tc_ld_piece(t_acc + 16 * p, pc[p]);
          }
        } else {
          Piece p0, p1;                                 // one arrives while the other is folded
          tc_ld_piece(t_acc, p0);
          while (true) {
            const uint32_t fb = fac_b + slot;
            float ra[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) ra[q] = ld_shared_f32(fac_a + slot + 32 * q);
            const uint32_t gone = my_empty + 8 * ring;
            step();
            // the next chunk's barrier is looked at here, where the answer has time to arrive (a wait on a
            // barrier that is already complete costs ~150 cycles when the code depends on it at once)
            const bool ready = __all_sync(0xFFFFFFFFu, mbar_test(my_full + 8 * ring, phase));
#pragma unroll
            for (int p = 0; p < C::PIECES - 1; ++p) {
              tc_wait_piece(p & 1 ? p1 : p0);
              tc_ld_piece(t_acc + 16 * (p + 1), p & 1 ? p0 : p1);
              fold_piece<B_UNIFORM>(acc + 8 * p, p & 1 ? p1 : p0, ra, fb + 64 * p);
            }
            static_assert(C::PIECES % 2 == 0, "the last piece is in p1");
            tc_wait_piece(p1);              // the chunk has left tensor memory (a warp-wide wait)
            tc_fence_before();
            if (lane == 0) mbar_arrive(generic_bar(gone));
            if (--left > 0) {
              if (!ready) {
                alive = mbar_wait(generic_bar(my_full + 8 * ring), phase, abort_flag, 24, args.wait_ns);
                if (!alive) break;
              }
              t_acc = t_row + acc_i * HN;
              tc_fence_after();
              tc_ld_piece(t_acc, p0);
            }
            fold_piece<B_UNIFORM>(acc + 8 * (C::PIECES - 1), p1, ra, fb + 64 * (C::PIECES - 1));
            if (left == 0) break;
          }
        }
      }
      if (!alive) break;
      if (odd) slot = slot + SLOT_BYTES == SLOTS_END ? 0u : slot + SLOT_BYTES;   // a stage has two slots
      if (!mine) continue;
      // ---- epilogue of the tile: this warp's 32 rows x HN columns, in units of 16 rows x 128 bytes ----
      const float os = margs.out_scale;
      const bool out_bf16 = args.out_bf16 != 0;
      uint8_t* epi_warp = epi + (warp - 8) * C::EPI_WARP_BYTES;
      const int lr = lane >> 2, lc = lane & 3;
#pragma unroll
      for (int q = 0; q < HN / 32; ++q) {
        if (out_bf16 && (q & 1) != 0) continue;
#pragma unroll
        for (int rh = 0; rh < 2; ++rh) {
          if (lane == 0) bulk_wait_read<1>();  // the store issued two units ago has finished reading this buffer
          __syncwarp();
          uint8_t* unit = epi_warp + (store_it & 1u) * C::EPI_UNIT;
          const uint32_t base = smem_u32(unit);
#pragma unroll
          for (int g = 0; g < 8; ++g) {                 // column groups of eight: 16 bytes of bf16, 32 of fp32
            if (!out_bf16 && g >= 4) continue;
#pragma unroll
            for (int e = 0; e < 2; ++e) {               // row lr + 8 e of the unit
              const int cg = (q * 4 + g) & (HN / 8 - 1);   // (the mask keeps the unreachable fp32 case inside acc)
              const float2 v = acc[(cg >> 1) * 8 + rh * 4 + (cg & 1) * 2 + e];
              const uint32_t row = (uint32_t)(lr + 8 * e);
              const float x = __fmul_rn(v.x, os), y = __fmul_rn(v.y, os);
              if (out_bf16) {
                const __nv_bfloat162 p2 = __floats2bfloat162_rn(x, y);
                st_shared_u32(base + row * 128u + ((((uint32_t)g) ^ (row & 7u)) << 4) + lc * 4u,
                              *reinterpret_cast<const uint32_t*>(&p2));
              } else {
                const uint32_t chunk = (uint32_t)(2 * g) + (uint32_t)(lc >> 1);
                st_shared_v2(base + row * 128u + ((chunk ^ (row & 7u)) << 4) + (lc & 1) * 8u, f2u(x), f2u(y));
              }
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          const int col = col0 + 32 * q, r0 = row0 + 16 * rh;
          if (lane == 0) {
            if (r0 < args.M && col < args.N) tma_store_3d(unit, &tmap_d, col, r0, batch);
            bulk_commit();  // one group per unit, empty or not: the waits above count groups
          }
          ++store_it;
        }
      }
    }
    if (lane == 0) bulk_wait_all();
  }

  // ------------------------------ teardown ------------------------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}
