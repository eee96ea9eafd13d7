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
// One CTA (512 threads = four warpgroups, persistent over tiles of 128 x BN, BN = 128 or 192; `macro_tile_n` in
// gemm_sm100.cu chooses):
//   warpgroup 0   warp 0: producer - per stage (128 bytes of K = two chunks) two tiled TMA loads and the bulk copies
//                 of the stage's scale tiles; warps 1 and 3: MMA issuers of alternate chunks - two tcgen05.mma into
//                 one of the three (BN = 192: two) chunk accumulators in tensor memory, then a commit to that
//                 accumulator's "full" barrier; warp 2: waits for these and releases the fold warps;
//   warpgroup 1   scale transfer shared memory -> tensor memory (as in the plain kernel), and the macro
//                 factors: their codes are read three stages ahead and the reciprocals left in a shared-memory ring;
//   warpgroups 2-3  fold + epilogue: per tensor-memory lane quarter two warps of 32 rows x BN / 2 columns, the sums in
//                 registers.  A warp reads its part of the chunk into registers, 64 columns at a time, gives the
//                 accumulator back and then does acc += P * (1/fa[row]) * (1/fb[col]) in packed fp32x2 arithmetic.
//                 After the last chunk the registers are scaled, converted, staged and TMA-stored.
//
// What bounds it: the way of a chunk accumulator around the roles (MMA 128 or 192 cycles of 440 with issue and commit,
// wait warp, read, fold, issuer; about 1300 cycles over the accumulators that fit in tensor memory).  Nothing is
// saturated: the MMAs of a block of 128 x 128 x 128 take 128 cycles, its loads 200 to 256 at 64 bytes a cycle, reading
// it out of tensor memory 75, its multiply-adds 140, and with one B factor per tile it takes 420.  So what counts
// is latency: few instructions and fewer branches in the loops (a taken branch costs 25 to 40 cycles among so much
// different code), waits of a few instructions, and issue slots left free by the fold.
// Measured at 8192 x 4096 x 14336, one factor per tile of B / one per column: 349 / 519 us.  Before: 451 / 612 us with
// 128 x 256 tiles of two halves, chunks read in the 16 x 256-bit layout (three times the time of the present ones)
// in pieces of 16 columns, inlined bounded waits in every loop.  On the way, one factor per tile: the new layouts alone
// 411, 128 x 128 tiles 410, waits as small loops and the fold released at named barriers 377, packed arithmetic 362.
// One issuer behind a wait warp 420, two register sets for the chunks 593 (spills), one issuer that waits itself 480.
// The warpgroups re-divide the register file with setmaxnreg (512 threads x 128 at launch, see CfgMacro).
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

struct MacroGemmArgs {
  GemmArgs g;
  MacroSide ma, mb;
  float out_scale;
};

constexpr int NUM_THREADS_MACRO = 512;

// BN: columns of a tile.
template <int BN_>
struct CfgMacro {
  static constexpr int BN = BN_;
  static_assert(BN == 192 || BN == 128, "tile widths");
  static constexpr int SF_TILES = Kind<KIND_MXF4>::SF_TILES;
  static constexpr int A_BYTES = BM * STAGE_K_BYTES;
  static constexpr int B_BYTES = BN * STAGE_K_BYTES;
  static constexpr int SF_BYTES = SF_TILES * 512;               // per 128 rows of either operand
  static constexpr int SFB_BLOCKS = BN == 192 ? 2 : 1;          // 128-row blocks of B's scales under a tile
  static constexpr int SF_OFF = A_BYTES + B_BYTES;              // scales of A, then of B's blocks
  static constexpr int STAGE_BYTES = SF_OFF + (1 + SFB_BLOCKS) * SF_BYTES;
  static_assert(STAGE_BYTES % 1024 == 0, "stages must keep the 128-byte swizzle atom aligned");
  static constexpr int SF_COLS = SF_TILES * 4;                  // tensor-memory columns of SF_BYTES
  static constexpr int STAGE_SF_COLS = (1 + SFB_BLOCKS) * SF_COLS;
  static constexpr int STAGES = BN == 192 ? 4 : 5;
  static constexpr int P_BUFS = BN == 192 ? 2 : 3;              // chunk accumulators in tensor memory
  static constexpr int FOLD_WARPS = 8;                          // two per tensor-memory lane quarter
  static constexpr int WN = BN / 2;                             // columns of a fold warp
  static constexpr int PIECES = WN / 16;
  static constexpr int FLIGHT = 4;                              // pieces in registers at a time
  // staged units of 32 rows: 64 columns of bf16 where they divide a warp's, else 32; 32 of fp32
  static constexpr int EPI_COLS = WN % 64 == 0 ? 64 : 32;
  static constexpr int EPI_WARP_BYTES = 4096;
  static constexpr int EPI_BYTES = FOLD_WARPS * EPI_WARP_BYTES;
  // Ring of reciprocal factors, per chunk 128 rows and BN columns (B_UNIFORM: the products of both, 128 rows per
  // 128 columns).  No barrier guards its reuse: a slot is rewritten FAC_STAGES stages after its last use, once
  // that stage's operands have landed, so the MMAs of the stage STAGES earlier are done, and with them every chunk
  // up to P_BUFS before has been read out, in order - all but the latest of these have therefore been folded (that
  // one's column factors are read after its accumulator was given back).  A stage may hold a single chunk (K ranges of
  // 128), so P_BUFS chunks are as many stages.
  static constexpr int FAC_STAGES = BN == 192 ? 8 : 9;
  static constexpr int FAC_STRIDE = BM + (BN == 192 ? 192 : 128) + 4;   // floats per chunk; + 4 spreads the banks
  static_assert(FAC_STRIDE >= SFB_BLOCKS * BM && FAC_STRIDE >= BM + BN, "factors of a chunk");
  static constexpr int FAC_BYTES = 2 * FAC_STAGES * FAC_STRIDE * 4;
  static_assert(FAC_STAGES >= STAGES + P_BUFS + 1, "factors are overwritten while they are in use");
  static constexpr int RCP_BYTES = 256 * 4;                     // 1 / factor for every code
  static constexpr int TMEM_SF_BASE = P_BUFS * BN;
  static constexpr int TMEM_COLS_USED = TMEM_SF_BASE + STAGES * STAGE_SF_COLS;
  static_assert(TMEM_COLS_USED <= 512, "tensor memory budget");
  // named barrier that hands chunk accumulator `buf` to a group of four fold warps
  __device__ static constexpr int chunk_barrier(int group, int buf) { return 1 + 2 * buf + group; }
  static constexpr int NUM_BARS = 3 * STAGES + 2 * P_BUFS;
  static constexpr int SMEM_BYTES =
      STAGES * STAGE_BYTES + EPI_BYTES + FAC_BYTES + RCP_BYTES + 1024 /*align*/ + 512 /*barriers*/;
  static_assert(NUM_BARS * 8 + 16 <= 512, "barrier area");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  // Registers per thread after the warpgroups have re-divided the file.  The CTA is launched with 128
  // registers per thread (65536 / 512); setmaxnreg.inc can only take what setmaxnreg.dec has released
  // INSIDE the CTA and blocks for ever otherwise, so the two must balance exactly.
  static constexpr int REGS_LAUNCH = 128;
  static constexpr int REGS_SMALL = BN == 192 ? 72 : 96, REGS_FOLD = 256 - REGS_SMALL;
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
};

template <class C>
__device__ __forceinline__ MacroTile decode_macro_tile(const MacroGemmArgs& margs, uint32_t tile, int k_stages_dense) {
  const GemmArgs& args = margs.g;
  MacroTile m;
  TileInfo& t = m.t;
  const TileCoord coord = tile_coord(args, tile);
  const uint32_t e = coord.batch;
  t.nb = coord.nb;
  t.mb = coord.mb;
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
  return m;
}

// One piece of a chunk accumulator: 16 columns of a warp's 32 rows.
// One B factor per chunk: one row per lane (32 x 32-bit layout), so that a chunk needs one factor a lane.
// Per-column factors: two loads of 16 rows in the 16 x 128-bit layout, where a lane gets columns lane % 4 + 4 g of
// rows lane / 4 and + 8 of each load: four rows and four columns, eight factors, where a row per lane needs 17, and
// the broadcast of the column factors out of shared memory (128 bytes per register and warp) took 550 cycles.
// Reading a block of 128 x 128 takes 75 cycles in the 32 x 32-bit layout, 131 in the 16 x 128-bit one and 257 in the
// 16 x 256-bit one (all warps reading, nothing else running).
struct Piece {
  uint32_t r[16];   // [column 16], or [row half 2][column group 4][row 2]
};
template <bool B_UNIFORM>
__device__ __forceinline__ void tc_ld_piece(uint32_t taddr, Piece& p) {
  if constexpr (B_UNIFORM) {
    uint32_t* r = p.r;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t* r = p.r + 8 * h;
      asm volatile(
          "tcgen05.ld.sync.aligned.16x128b.x4.b32 "
          "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
          : "r"(taddr + ((uint32_t)(16 * h) << 16))
          : "memory");
    }
  }
}
// The values in p have landed (tcgen05.wait::ld came before): nothing that uses them can move above this.
__device__ __forceinline__ void tc_landed_piece(Piece& p) {
#define ALTOB200_RW8(o) "+r"(p.r[o]), "+r"(p.r[o + 1]), "+r"(p.r[o + 2]), "+r"(p.r[o + 3]), "+r"(p.r[o + 4]), \
                        "+r"(p.r[o + 5]), "+r"(p.r[o + 6]), "+r"(p.r[o + 7])
  asm volatile("" : ALTOB200_RW8(0), ALTOB200_RW8(8));
#undef ALTOB200_RW8
}
__device__ __forceinline__ void st_shared_u16(uint32_t addr, unsigned short v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}
__device__ __forceinline__ float ld_shared_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 ld_shared_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
// tcgen05 instructions of one lane, without a branch around them
__device__ __forceinline__ void tc_mma_mxf4_if(bool pred, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate, uint32_t sfa, uint32_t sfb) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %7, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb), "r"((uint32_t)pred)
      : "memory");
}
__device__ __forceinline__ void tc_commit_if(bool pred, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(bar), "r"((uint32_t)pred)
      : "memory");
}
// acc += P * ra[row] * fb[col]; B_UNIFORM: one B factor for the columns and chunk, already multiplied into ra[0].
// `acc` and `p` are laid out alike; fb: shared-memory address of this lane's first column factor.  Packed arithmetic
// takes as long as scalar but half the issue slots: beside scalar multiply-adds on every scheduler the warp that
// issues the MMAs took 1380 cycles for a pair and the wait for it, beside packed ones 550 (alone 490).
template <bool B_UNIFORM>
__device__ __forceinline__ void fold_piece(float2* acc, const Piece& p, const float2 (&ra)[B_UNIFORM ? 1 : 2], uint32_t fb) {
  if constexpr (B_UNIFORM) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      acc[i] = __ffma2_rn(make_float2(u2f(p.r[2 * i]), u2f(p.r[2 * i + 1])), ra[0], acc[i]);
  } else {
    const float4 f4 = ld_shared_f32x4(fb);
    const float f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
      for (int h = 0; h < 2; ++h) {     // rows 16 h and 16 h + 8 of the lane's
        const int i = h * 4 + g;
        const float2 w = __fmul2_rn(ra[h], make_float2(f[g], f[g]));
        acc[i] = __ffma2_rn(make_float2(u2f(p.r[2 * i]), u2f(p.r[2 * i + 1])), w, acc[i]);
      }
  }
}

// B_UNIFORM: B's macro blocks are 128 x 128 tiles (one factor per 128 columns and chunk), else per column.
template <int BN, bool B_UNIFORM>
__global__ void __launch_bounds__(NUM_THREADS_MACRO, 1)
gemm_macro_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_d, const MacroGemmArgs margs) {
  using C = CfgMacro<BN>;
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
  uint64_t* p_full = bars + 3 * C::STAGES;        // [chunk % P_BUFS]
  uint64_t* p_empty = p_full + C::P_BUFS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(p_empty + C::P_BUFS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* never = abort_flag + 1;           // an abort flag that nothing raises

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (an output of 2^31 tiles would not fit any memory)
  const int n_tiles = (int)(margs.g.per_batch.d * (args.k_offs != nullptr ? args.num_batches : 1));
  const int k_stages = (int)((args.k_bytes + STAGE_K_BYTES - 1) / STAGE_K_BYTES);

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 2);
      mbar_init(&sf_full[s], 4);
    }
    for (int p = 0; p < C::P_BUFS; ++p) {
      mbar_init(&p_full[p], 1);
      mbar_init(&p_empty[p], C::FOLD_WARPS);
    }
    *abort_flag = 0;
    *never = 0;
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
  const uint32_t abort_addr = smem_u32(const_cast<int*>(abort_flag));
  const uint64_t limit = args.wait_ns * 2ull;   // cycles, see the waits
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
      const int n_row_blocks = (int)((args.N + 127) >> 7);
      uint32_t s = 0, phase = 1;
      bool alive = true;
      for (int tile = (int)blockIdx.x; tile < n_tiles && alive; tile += (int)gridDim.x) {
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
        const TileInfo& ti = mt.t;
        if (ti.skip) continue;
        const int64_t mb = ti.mb;
        const int sfb_blk0 = (int)((ti.nb * BN) >> 7);       // first 128-row block of B's scales under this tile
        const uint32_t n_sfb = (uint32_t)(n_row_blocks - sfb_blk0 < C::SFB_BLOCKS ? n_row_blocks - sfb_blk0 : C::SFB_BLOCKS);
        for (int ks = 0; ks < ti.k_stages; ++ks) {
          alive = __all_sync(0xFFFFFFFFu, mbar_wait_tight(smem_u32(&empty_bar[s]), phase, abort_addr, limit));
          if (!alive) break;
          uint8_t* st = smem + s * C::STAGE_BYTES;
          const int64_t cb0 = ti.sf_tile0 + (int64_t)ks * C::SF_TILES;
          int64_t sf_tiles = args.nct - cb0;
          if (sf_tiles > C::SF_TILES) sf_tiles = C::SF_TILES;
          const uint32_t sf_bytes = (uint32_t)sf_tiles * 512u;
          const int32_t kx = (int32_t)(ti.k_byte0 + (int64_t)ks * STAGE_K_BYTES);
          if (elected) {
            mbar_expect_tx(&full_bar[s], C::A_BYTES + C::B_BYTES + (1u + n_sfb) * sf_bytes);
            tma_load_2d(st, &tmap_a, kx, (int32_t)(mb * BM), &full_bar[s]);
            tma_load_2d(st + C::A_BYTES, &tmap_b, kx, (int32_t)ti.b_row0, &full_bar[s]);
            bulk_load(st + C::SF_OFF, args.sfa + (mb * args.nct + cb0) * 512, sf_bytes, &full_bar[s]);
#pragma unroll
            for (uint32_t h = 0; h < C::SFB_BLOCKS; ++h)
              if (h < n_sfb)
                bulk_load(st + C::SF_OFF + (1 + h) * C::SF_BYTES, ti.sfb + ((int64_t)(sfb_blk0 + h) * args.nct + cb0) * 512,
                          sf_bytes, &full_bar[s]);
          }
          if (++s == C::STAGES) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
      if (!alive) report_timeout(abort_flag, 21);
    } else if (warp == 1 || warp == 3) {
      // ------------------------------ MMA issuers ------------------------------
      // Two, for alternate chunks: while one waits for its barriers the other one's MMAs keep the tensor pipe busy.
      // Chunk m goes to accumulator m % P_BUFS, which held chunk m - P_BUFS.  Its issuer cannot mistake the phase
      // before for the one it waits for: it has waited until chunk m - 2 - P_BUFS was drained, and chunks are drained
      // in order, so that m - 2 P_BUFS was too (P_BUFS >= 2).
      // A branch costs about 25 cycles here and a stage has 400, so the loop's only one is on the vote; the issuing
      // lane's instructions are predicated.
      const bool elected = elect_one();
      const uint32_t i = (uint32_t)(warp >> 1);
      uint32_t s = 0, st_phase = 0, odd = 0;      // odd: chunks so far, modulo 2
      uint32_t buf = i, drained = 1;              // this issuer's next accumulator and the phase it waits for
      bool alive = true;
      const uint32_t smem_base = smem_u32(smem);
      const uint32_t bar_full = smem_u32(full_bar), bar_sf = smem_u32(sf_full), bar_acc = smem_u32(p_empty);
      for (int tile = (int)blockIdx.x; tile < n_tiles && alive; tile += (int)gridDim.x) {
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
        const TileInfo& ti = mt.t;
        if (ti.skip) continue;
        // scale columns of B start at word 0 of the first block, or 64 rows (2 words) into it
        const uint32_t sfb_off = C::SFB_BLOCKS == 2 ? (uint32_t)((ti.nb * BN) & 127) >> 5 : 0u;
        for (int ks = 0; ks < ti.k_stages; ++ks) {
          const int n_mma = (ks == ti.k_stages - 1) ? ti.last_mmas : 4;
          const int c = (int)(odd ^ i);           // this issuer's chunk of the stage
          const bool mine = 2 * c < n_mma;
          // operands and scales of the stage are in place, the accumulator is drained
          const uint32_t b0 = bar_sf + 8 * s, b1 = bar_full + 8 * s;
          const uint32_t b2 = mine ? bar_acc + 8 * buf : b1, p2 = mine ? drained : st_phase;
          alive = __all_sync(0xFFFFFFFFu, mbar_wait3_tight(b0, b1, st_phase, b2, p2, abort_addr, limit));
          if (!alive) break;
          tc_fence_after();
          const uint32_t sfa_t = tmem_base + C::TMEM_SF_BASE + s * C::STAGE_SF_COLS + c * 4;
          const uint32_t sfb_t = tmem_base + C::TMEM_SF_BASE + s * C::STAGE_SF_COLS + C::SF_COLS + c * 4 * C::SFB_BLOCKS + sfb_off;
          const uint32_t a_lo = (((smem_base + s * C::STAGE_BYTES) >> 4) | 0x10000u) + 4 * c;
          const uint32_t b_lo = a_lo + (C::A_BYTES >> 4);
#pragma unroll
          for (int j = 0; j < 2; ++j)
            tc_mma_mxf4_if(elected && 2 * c + j < n_mma, tmem_base + buf * BN, desc_of(DESC_SW128_HI, a_lo + 2 * j),
                           desc_of(DESC_SW128_HI, b_lo + 2 * j), args.idesc[j], (uint32_t)j, sfa_t, sfb_t);
          tc_commit_if(elected && mine, smem_u32(p_full) + 8 * buf);
          tc_commit_if(elected, smem_u32(empty_bar) + 8 * s);      // both issuers
          if (mine) {                             // two chunks on
            if (C::P_BUFS == 2 || buf != 0) drained ^= 1u;
            if (C::P_BUFS == 3) buf = buf == 0 ? 2u : buf - 1;
          }
          odd ^= n_mma <= 2 ? 1u : 0u;
          if (++s == C::STAGES) {
            s = 0;
            st_phase ^= 1u;
          }
        }
      }
      if (!alive) report_timeout(abort_flag, !mbar_complete(bar_full + 8 * s, st_phase) ? 23 : !mbar_complete(bar_sf + 8 * s, st_phase) ? 25 : 22);
    } else {
      // ------------------------------ wait warp of the fold ------------------------------
      // It waits for the finished chunks and releases the two groups of fold warps, each at its own named barrier of
      // the accumulator: 20 cycles a chunk for a fold warp, where a look at an mbarrier and the branch on its answer
      // took 75 of 260.  A barrier cannot be met twice ahead of the fold: the accumulator's next chunk is finished only
      // after all fold warps have given it back.  After a failure the chunks left are handed over one by one without
      // waiting for them, so that the fold warps come to their end (they store nothing then).
      uint32_t buf = 0, phase = 0;
      bool alive = true;
      for (int tile = (int)blockIdx.x; tile < n_tiles; tile += (int)gridDim.x) {
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
        int left = mt.t.skip ? 0 : mt.n_chunks;
        for (; left > 0; --left) {
          if (alive) {
            alive = __all_sync(0xFFFFFFFFu, mbar_wait_tight(smem_u32(p_full) + 8 * buf, phase, abort_addr, limit));
            if (!alive) report_timeout(abort_flag, 24);
          }
          if (alive) {
            named_barrier_arrive(C::chunk_barrier(0, (int)buf), 160);
            named_barrier_arrive(C::chunk_barrier(1, (int)buf), 160);
          } else {
            // (the fold is past the accumulator's chunk before: its barriers are free)
            (void)mbar_wait_tight(smem_u32(p_empty) + 8 * buf, phase ^ 1u, smem_u32(const_cast<int*>(never)), limit);
            __syncwarp();
            named_barrier_sync(C::chunk_barrier(0, (int)buf), 160);
            named_barrier_sync(C::chunk_barrier(1, (int)buf), 160);
          }
          if (++buf == C::P_BUFS) {
            buf = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp < 8) {
    // ------------------------------ scale transfer and macro factors ------------------------------
    setmaxnreg_dec<C::REGS_SMALL>();
    const int quad = warp & 3;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    // factors: lane = (row of sixteen, chunk of the stage); the warp serves 32 rows of A and BN / 4 columns of B
    // (columns c, c + 4, c + 8 and c + 12 of a piece lie together, see Piece)
    const int fc = lane & 1, fr = lane >> 1, fr_col = (fr & 3) * 4 + (fr >> 2) - fr;
    constexpr int NB = B_UNIFORM ? C::SFB_BLOCKS : BN / 64;
    struct Codes {
      uint32_t a[2], b[NB];
    };
    // The codes of a stage are requested AHEAD stages before it: read one stage ahead, their latency was what a
    // stage took (900 cycles, with no operand loaded, no MMA issued and nothing folded).
    const uint8_t *pa[2], *pb[NB];
    int next_tile = (int)blockIdx.x, stages_left = 0, chunks_left = 0;
    auto request = [&](Codes& q) -> bool {
      while (stages_left == 0) {
        if (next_tile >= n_tiles) return false;
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)next_tile, k_stages);
        next_tile += (int)gridDim.x;
        if (mt.t.skip) continue;
        stages_left = mt.t.k_stages;
        chunks_left = mt.n_chunks - fc;
        const int64_t m0 = mt.t.mb * BM, n0 = mt.t.nb * BN;
        const uint8_t* a0 = margs.ma.codes + (mt.chunk0 + fc) * margs.ma.chunk_stride + (m0 >> margs.ma.shift) * margs.ma.row_stride;
        const uint8_t* b0 = margs.mb.codes + (int64_t)mt.expert * margs.mb.expert_stride +
                            (mt.chunk0 + fc) * margs.mb.chunk_stride + (n0 >> margs.mb.shift) * margs.mb.row_stride;
        // (a row beyond the matrix reads the last one)
        const uint32_t m_last = (uint32_t)(args.M - m0 < BM ? args.M - m0 : BM) - 1u;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t r = (uint32_t)(quad * 32 + 16 * i + fr);
          pa[i] = a0 + (int64_t)((r < m_last ? r : m_last) >> margs.ma.shift) * margs.ma.row_stride;
        }
        const uint32_t n_last = B_UNIFORM ? (uint32_t)(((args.N - 1) >> 7) - (n0 >> 7))   // of the 128-row blocks
                                          : (uint32_t)(args.N - n0 < BN ? args.N - n0 : BN) - 1u;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const uint32_t r = (uint32_t)(B_UNIFORM ? i : quad * (BN / 4) + 16 * i + fr);
          pb[i] = b0 + (int64_t)(r < n_last ? r : n_last) * margs.mb.row_stride;
        }
      }
      const bool have = chunks_left > 0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        q.a[i] = have ? __ldg(pa[i]) : 0u;
        pa[i] += 2 * margs.ma.chunk_stride;
      }
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        q.b[i] = have ? __ldg(pb[i]) : 0u;
        pb[i] += 2 * margs.mb.chunk_stride;
      }
      --stages_left;
      chunks_left -= 2;
      return true;
    };
    uint32_t s = 0, phase = 0, slot = 0;          // operand stage and its phase, factor stage
    auto transfer = [&](const Codes& q) -> bool {
      if (!mbar_wait_tight(smem_u32(full_bar) + 8 * s, phase, abort_addr, limit)) return false;
      const uint8_t* sf = smem + s * C::STAGE_BYTES + C::SF_OFF + lane * 16;
      const uint32_t sf_t = tmem_base + lane_base + C::TMEM_SF_BASE + s * C::STAGE_SF_COLS;
#pragma unroll
      for (int t = 0; t < C::SF_TILES; ++t) {
        const uint4 a = *reinterpret_cast<const uint4*>(sf + t * 512);
        tc_st4(sf_t + t * 4, a.x, a.y, a.z, a.w);
#pragma unroll
        for (int h = 0; h < C::SFB_BLOCKS; ++h) {            // the blocks of a K tile lie together
          const uint4 b = *reinterpret_cast<const uint4*>(sf + (1 + h) * C::SF_BYTES + t * 512);
          tc_st4(sf_t + C::SF_COLS + (t * C::SFB_BLOCKS + h) * 4, b.x, b.y, b.z, b.w);
        }
      }
      float* dst = fac + (2 * slot + fc) * C::FAC_STRIDE + fr;
      if (B_UNIFORM) {
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const float rb = rcp_tab[q.b[j]];
#pragma unroll
          for (int i = 0; i < 2; ++i) dst[BM * j + quad * 32 + 16 * i] = __fmul_rn(rcp_tab[q.a[i]], rb);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i) dst[quad * 32 + 16 * i] = rcp_tab[q.a[i]];
#pragma unroll
        for (int i = 0; i < NB; ++i) dst[BM + quad * (BN / 4) + 16 * i + fr_col] = rcp_tab[q.b[i]];
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_lane0(smem_u32(sf_full) + 8 * s, lane);
      if (++slot == C::FAC_STAGES) slot = 0;
      if (++s == C::STAGES) {
        s = 0;
        phase ^= 1u;
      }
      return true;
    };
    constexpr int AHEAD = 3;
    Codes q[AHEAD];
    bool have[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) have[i] = request(q[i]);
    bool alive = true;
    while (alive && have[0]) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        if (alive && have[i]) {
          alive = transfer(q[i]);
          have[i] = request(q[i]);
        }
      }
    }
    if (!alive) report_timeout(abort_flag, 26);
  } else {
    // ------------------------------ fold + epilogue ------------------------------
    setmaxnreg_inc<C::REGS_FOLD>();
    // (What lives across the chunk loop beside the sums and the pieces is kept in 32 bits: local memory does not fit
    // beside 228 128 bytes of shared memory (232 192 with 192 columns), a few spilled registers in this loop or the transfer's cost a tenth.)
    const int quad = warp & 3;                        // tensor-memory lane quarter this warp may read
    const int side = (warp - 8) >> 2;                 // columns [WN side, WN side + WN) of the tile
    const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(side * C::WN);
    // this lane's first row and column factor in a chunk's slot
    const uint32_t fac_a = smem_u32(fac) + 4u * (uint32_t)(quad * 32 + (B_UNIFORM ? lane : lane >> 2));
    const uint32_t fac_b = smem_u32(fac) + 4u * (uint32_t)(BM + side * C::WN + 4 * (lane & 3));
    const uint32_t bar_empty = smem_u32(p_empty);
    uint32_t store_it = 0;                            // store units so far
    uint32_t slot = 0;                                // byte offset of the chunk's factors, always of an even slot at a tile's start
    uint32_t ring = 0;                                // accumulator of the next chunk
    constexpr uint32_t SLOT_BYTES = C::FAC_STRIDE * 4, SLOTS_END = 2 * C::FAC_STAGES * SLOT_BYTES;
    constexpr int PIECES = C::PIECES, FLIGHT = C::FLIGHT, RA = B_UNIFORM ? C::SFB_BLOCKS : 2;
    for (int tile = (int)blockIdx.x; tile < n_tiles; tile += (int)gridDim.x) {
      int left, row0, col0, batch;                    // chunks left, this warp's part of the output
      int split = PIECES;                             // B_UNIFORM: pieces under the first of the tile's 128-column blocks
      {
        const MacroTile mt = decode_macro_tile<C>(margs, (uint32_t)tile, k_stages);
        left = mt.t.skip ? 0 : mt.n_chunks;
        row0 = (int)mt.t.mb * BM + quad * 32;
        col0 = (int)mt.t.nb * BN + side * C::WN;
        batch = mt.t.batch;
        if (C::SFB_BLOCKS == 2) split = (128 - ((int)(mt.t.nb * BN) & 127) - side * C::WN) / 16;
      }
      float2 acc[C::WN / 2];                          // [PIECES][Piece]
#pragma unroll
      for (int j = 0; j < C::WN / 2; ++j) acc[j] = make_float2(0.0f, 0.0f);
      const bool odd = (left & 1) != 0;
      for (; left > 0; --left) {
        named_barrier_sync(C::chunk_barrier(side, (int)ring), 160);   // the chunk is finished
        tc_fence_after();
        // As much of the chunk as the registers take, so that its accumulator is given back before most of the
        // multiply-adds.
        Piece pc[FLIGHT];
        const uint32_t t_acc = t_row + ring * BN;
#pragma unroll
        for (int p = 0; p < FLIGHT; ++p) tc_ld_piece<B_UNIFORM>(t_acc + 16 * p, pc[p]);
        const uint32_t fb = fac_b + slot;
        float2 ra[RA];
#pragma unroll
        for (int q = 0; q < RA; ++q) {
          if (B_UNIFORM) {
            ra[q].x = ra[q].y = ld_shared_f32(fac_a + slot + 4 * BM * q);
          } else {
            ra[q].x = ld_shared_f32(fac_a + slot + 64 * q);
            ra[q].y = ld_shared_f32(fac_a + slot + 64 * q + 32);
          }
        }
        const uint32_t gone = bar_empty + 8 * ring;
        if (++ring == C::P_BUFS) ring = 0;
        slot = slot + SLOT_BYTES == SLOTS_END ? 0u : slot + SLOT_BYTES;
        auto fold = [&](int p) {
          if constexpr (B_UNIFORM) {
            const float2 r[1] = {RA == 1 || p < split ? ra[0] : ra[RA - 1]};
            fold_piece<true>(acc + 8 * p, pc[p % FLIGHT], r, 0u);
          } else {
            fold_piece<false>(acc + 8 * p, pc[p % FLIGHT], ra, fb + 64 * p);
          }
        };
        auto landed = [&]() {
#pragma unroll
          for (int p = 0; p < FLIGHT; ++p) tc_landed_piece(pc[p]);
        };
        if (FLIGHT < PIECES) {
          tc_wait_ld();
          landed();
        }
#pragma unroll
        for (int p = FLIGHT; p < PIECES; ++p) {
          fold(p - FLIGHT);
          tc_ld_piece<B_UNIFORM>(t_acc + 16 * p, pc[p - FLIGHT]);
        }
        tc_wait_ld();
        tc_fence_before();
        mbar_arrive_lane0(gone, lane);
        landed();                       // (after the arrival: no multiply-add moves in front of it)
#pragma unroll
        for (int p = PIECES - FLIGHT; p < PIECES; ++p) fold(p);
      }
      if (odd) slot = slot + SLOT_BYTES == SLOTS_END ? 0u : slot + SLOT_BYTES;   // a stage has two slots
      // ---- epilogue of the tile: this warp's 32 rows x WN columns ----
      // Units of 128 bytes a row in one buffer, or of 64 (32 columns of bf16) in two.  A unit costs 600 cycles beside its
      // conversions, for the wait for the last store and the proxy fence, so it is as wide as it can be (a warp's 64
      // columns as two: wgrad of 69 632 rows, 5760 x 2880, in 32 ranges 1508 us).  A row per lane straight to global
      // memory was slower yet: 378 us for 356, forward at 8192 x 4096 x 14336.
      // Executed once a tile, this code is not in the instruction caches: its instructions count (1400 to 2500 cycles,
      // in which the MMAs get no further than the free accumulators).
      if (margs.out_scale != 1.0f) {
        const float2 os = make_float2(margs.out_scale, margs.out_scale);
#pragma unroll
        for (int j = 0; j < C::WN / 2; ++j) acc[j] = __fmul2_rn(acc[j], os);
      }
      const bool out_bf16 = args.out_bf16 != 0, failed = *abort_flag != 0;
      uint8_t* const epi_warp = epi + (warp - 8) * C::EPI_WARP_BYTES;
      constexpr bool NARROW = C::EPI_COLS == 32;          // bf16 units of 64 bytes a row
#pragma unroll
      for (int q = 0; q < C::WN / 32; ++q) {              // 32 columns
        if (!NARROW && out_bf16 && (q & 1) != 0) continue;
        if (lane == 0) {                                  // the last store has finished reading this buffer
          if (NARROW && out_bf16) bulk_wait_read<1>();
          else bulk_wait_read<0>();
        }
        __syncwarp();
        uint8_t* const unit = epi_warp + (NARROW && out_bf16 ? (store_it & 1u) * 2048u : 0u);
        const uint32_t base = smem_u32(unit);
        if constexpr (B_UNIFORM) {
          const uint32_t row = (uint32_t)lane;
          if (out_bf16) {
#pragma unroll
            for (int g = 0; g < C::EPI_COLS / 8; ++g) {
              uint32_t o[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 v = acc[(q * 16 + g * 4 + e) % (C::WN / 2)];   // (never beyond: an even q where units have 64)
                const __nv_bfloat162 p2 = __floats2bfloat162_rn(v.x, v.y);
                o[e] = *reinterpret_cast<const uint32_t*>(&p2);
              }
              const uint32_t at = NARROW ? row * 64u + ((((uint32_t)g) ^ ((row >> 1) & 3u)) << 4)
                                         : row * 128u + ((((uint32_t)g) ^ (row & 7u)) << 4);
              st_shared_v4(base + at, o[0], o[1], o[2], o[3]);
            }
          } else {
#pragma unroll
            for (int g = 0; g < 8; ++g) {
              const float2 v = acc[q * 16 + g * 2], w = acc[q * 16 + g * 2 + 1];
              st_shared_v4(base + row * 128u + ((((uint32_t)g) ^ (row & 7u)) << 4), f2u(v.x), f2u(v.y), f2u(w.x), f2u(w.y));
            }
          }
        } else {
          static_assert(B_UNIFORM || !NARROW, "units of per-column factors");
          const uint32_t lr = (uint32_t)(lane >> 2), lc = (uint32_t)(lane & 3);
#pragma unroll
          for (int g = 0; g < 16; ++g) {                // column lc + 4 g of the unit
            if (!out_bf16 && g >= 8) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {               // rows lr + 16 h and + 8
              const float2 v = acc[((q * 2 + (g >> 2)) * 8 + h * 4 + (g & 3)) % (C::WN / 2)];
              const uint32_t row_at = base + (lr + 16u * h) * 128u;   // (the swizzle of both rows is that of lr)
              if (out_bf16) {
                const __nv_bfloat162 p2 = __floats2bfloat162_rn(v.x, v.y);
                const uint32_t w = *reinterpret_cast<const uint32_t*>(&p2);
                const uint32_t at = row_at + ((((uint32_t)g >> 1) ^ lr) << 4) + (g & 1) * 8u + lc * 2u;
                st_shared_u16(at, (unsigned short)w);
                st_shared_u16(at + 8u * 128u, (unsigned short)(w >> 16));
              } else {
                const uint32_t at = row_at + ((((uint32_t)g) ^ lr) << 4) + lc * 4u;
                st_shared_u32(at, f2u(v.x));
                st_shared_u32(at + 8u * 128u, f2u(v.y));
              }
            }
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        const int col = col0 + 32 * q;
        if (lane == 0) {
          if (row0 < args.M && col < args.N && !failed) tma_store_3d(unit, &tmap_d, col, row0, batch);
          bulk_commit();  // one group per unit, empty or not: the waits above count groups
        }
        ++store_it;
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
