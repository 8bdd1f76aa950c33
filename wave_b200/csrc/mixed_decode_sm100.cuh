// Decode (M <= 128) GEMM of 8-bit activations with packed 4-bit weights, weights on the N side of the MMA.
//
// The whole-tile decode kernel (skinny_whole_sm100.cuh) puts 128 weight rows on the 128 lanes of the accumulator and the few
// activation rows on its columns. An MMA of 128 lanes and 16 columns takes about 100 clocks, as long as one of 128 lanes and
// 200 columns (what it costs to bring 128 rows of the first operand in), so that kernel cannot multiply more than
// 128 rows x 32 bytes of weights per 100 clocks. For 4-bit weights that is what bounded it: a stage brings 64 bytes per weight
// row from memory but takes the MMAs of 128 (the 8-bit containers), and with the loads left out the kernel ran no faster:
// 34.8 of 34.2 us at M = 16, N = 28672, K = 8192. Here the activations take the lanes (M of 128 are real) and up to 208 weight
// rows the columns: half the MMAs per weight row. The activation tile is also fetched half as often.
// N = 28672, K = 8192 (117 MB of weights), per launch: M = 1 / 16 / 64 / 128: 34.2 / 34.2 / 36.9 / 40.2 -> 25.2 / 25.6 / 27.7 /
// 30.9 us; what remains is the rate at which the copy engine expands (26.7 us with the MMAs left out before).
//   * one CTA per SM walks tiles blockIdx.x, + gridDim.x, ..: the tile height is chosen on the host so that every SM gets the
//     same number of tiles (wb200_mixed_decode_tile_rows);
//   * a tile of more than 128 rows has two rows of scale atoms (rows 0 .. 127 and 128 .. of the tile);
//   * the MMA reads 128 activation rows from the stage: what follows the NP loaded ones are weight bytes, whose lanes are
//     never read;
//   * a lane of the epilogue holds consecutive columns of one output row: 16-byte stores, no transposition.
#pragma once
#include "gemm_sm100.cuh"

namespace wb {

constexpr int kMixedTileRowsMax = 208;  // two accumulators of 208 columns and the scale ring share 512 columns

template <int NP_>
struct MixedDecodeCfg {
  static constexpr int NP = NP_;  // activation rows a stage holds
  static constexpr int X_BYTES = NP * 128;
  static constexpr int W_BYTES = kMixedTileRowsMax * 128;
  static constexpr int SFX_OFFSET = X_BYTES + W_BYTES;
  static constexpr int SFW_OFFSET = SFX_OFFSET + 512;
  static constexpr int STAGE_BYTES = (SFW_OFFSET + 2 * 512 + 1023) / 1024 * 1024;
  static constexpr int SMEM_LIMIT = 232448;
  static constexpr int STAGES = (SMEM_LIMIT - 1024 - 512) / STAGE_BYTES;
  static constexpr int NUM_BARRIERS = 2 * STAGES + 4;
  static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + NUM_BARRIERS * 8 + 64;
  static constexpr int TMEM_COLS = 512;
  static constexpr int SF_COL = 2 * kMixedTileRowsMax;
  static constexpr int SF_SET_COLS = 16;  // activations 4 (8 reserved), weights 2 blocks x 4
  static constexpr int SF_SETS = 4;
  static_assert(SF_COL + SF_SETS * SF_SET_COLS <= TMEM_COLS, "tensor memory");
  static_assert(STAGES >= 4 && SMEM_BYTES <= SMEM_LIMIT, "shared memory");
  static_assert(STAGE_BYTES >= 128 * 128, "the MMA reads 128 rows from the head of a stage");
};

struct MixedDecodeMaps {
  CUtensorMap w, sfw, x, sfx;
};
struct MixedDecodeParams {
  void* c;
  int M, N;
  int ldc;
  int tiles_n;    // ceil(N / tile_rows)
  int tile_rows;  // a multiple of 8, at most kMixedTileRowsMax
  int num_kb;     // K / 128
  int accumulate;
  int dependent;  // kFirst, or kDependent: behind the kernel that writes the activations' packed scales
  int elem_format;
  int vec_ok;
  int* status;
};

template <int NP, typename OutT>
__global__ void __launch_bounds__(192, 1)
mixed_decode_kernel(const __grid_constant__ MixedDecodeMaps maps, const MixedDecodeParams p) {
  using Cfg = MixedDecodeCfg<NP>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (p.dependent) pdl_launch_dependents();
  if (warp == 0 && lane < 4)  // the copy engine fetches a descriptor on first use: start that now
    prefetch_tensormap(lane == 0 ? &maps.w : lane == 1 ? &maps.sfw : lane == 2 ? &maps.x : &maps.sfx);
  const uint32_t bar_base = smem_base + STAGES * Cfg::STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto acc_full_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };
  auto acc_empty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + 2 + s); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_gen + STAGES * Cfg::STAGE_BYTES + Cfg::NUM_BARRIERS * 8);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  WaitCtx ctx{abort_flag, p.status};
  const int row_warps = (p.M + 31) >> 5;  // epilogue warps with real rows

  uint32_t p_stage = 0, p_phase = 0;
  uint64_t stream_policy = 0, keep_policy = 0;
  const int blocks = (p.tile_rows + 127) >> 7;  // scale atom rows per tile
  // part 0: all loads of a stage; 1: the weights and their scales only; 2: the byte count, the activations and their scales
  auto load_stage = [&](int tile, int kb, uint32_t stage, int part) {
    const uint32_t sX = smem_base + stage * Cfg::STAGE_BYTES;
    const uint32_t fb = full_bar(stage);
    if (elect_one()) {
      // (weights that the copy engine expands count with their packed size, 64 bytes per row)
      if (part != 1) mbar_expect_tx(fb, uint32_t(Cfg::X_BYTES + 512 + blocks * 512 + p.tile_rows * 64));
      if (part != 2) {
        tma_load_2d_hint(sX + Cfg::X_BYTES, &maps.w, kb * 128, tile * p.tile_rows, fb, stream_policy);
        tma_load_2d(sX + Cfg::SFW_OFFSET, &maps.sfw, kb * 128, tile * blocks, fb);
      }
      if (part != 1) {
        tma_load_2d_hint(sX, &maps.x, kb * 128, 0, fb, keep_policy);
        tma_load_2d(sX + Cfg::SFX_OFFSET, &maps.sfx, kb * 128, 0, fb);
      }
    }
    __syncwarp();
  };
  int head = 0;
  if (warp == 0) {
    for (int b = lane; b < Cfg::NUM_BARRIERS; b += 32) mbar_init(bar_base + 8u * b, b >= 2 * STAGES + 2 ? uint32_t(row_warps) : 1u);
    if (lane == 0) *abort_flag = 0u;
    fence_mbar_init();
    __syncwarp();
    stream_policy = l2_policy_evict_first();  // weights are read once
    keep_policy = l2_policy_evict_last();     // activations are re-read by every CTA
    if (!p.dependent) {
      pdl_wait();
      pdl_launch_dependents();
    }
    head = min(STAGES, p.num_kb);
    for (int i = 0; i < head; ++i) load_stage(int(blockIdx.x), i, uint32_t(i), p.dependent ? 1 : 0);
  }
  if (warp == 1) {
    tmem_alloc<1>(smem_u32(tmem_slot), Cfg::TMEM_COLS);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (p.dependent) pdl_wait();
    for (int tile = blockIdx.x; tile < p.tiles_n; tile += gridDim.x) {
      for (int kb = 0; kb < p.num_kb; ++kb) {
        if (head > 0) {  // this stage's weights are already on their way
          --head;
          if (p.dependent) load_stage(tile, kb, p_stage, 2);
        } else {
          mbar_wait(empty_bar(p_stage), p_phase ^ 1u, ctx, WB_DEV_TIMEOUT_PRODUCER);
          load_stage(tile, kb, p_stage, 0);
        }
        if (++p_stage == STAGES) { p_stage = 0; p_phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc = make_idesc_mxf8(128, (p.tile_rows + 15) & ~15, act_format_of(p.elem_format), weight_format_of(p.elem_format));
    uint32_t stage = 0, phase = 0, sf_set = 0;
    int it = 0;
    for (int tile = blockIdx.x; tile < p.tiles_n; tile += gridDim.x, ++it) {
      const int as = it & 1;
      if (it >= 2) mbar_wait(acc_empty_bar(as), uint32_t((it - 2) >> 1) & 1u, ctx, WB_DEV_TIMEOUT_MMA_ACC);
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + as * kMixedTileRowsMax;
      for (int kb = 0; kb < p.num_kb; ++kb) {
        const uint32_t t_sfx = tmem_base + Cfg::SF_COL + sf_set * Cfg::SF_SET_COLS;
        const uint32_t t_sfw = t_sfx + 8;
        if (++sf_set == Cfg::SF_SETS) sf_set = 0;
        mbar_wait(full_bar(stage), phase, ctx, WB_DEV_TIMEOUT_MMA_FULL);
        tc_fence_after_sync();
        const uint32_t sX = smem_base + stage * Cfg::STAGE_BYTES;
        const uint64_t x_desc = make_desc_k_sw128(sX), w_desc = make_desc_k_sw128(sX + Cfg::X_BYTES);
        const uint64_t sfx_desc = make_desc_sf_atom(sX + Cfg::SFX_OFFSET), sfw_desc = make_desc_sf_atom(sX + Cfg::SFW_OFFSET);
        if (elect_one()) {
          utccp_sf_atom<1>(t_sfx, sfx_desc);
          utccp_sf_atom<1>(t_sfw, sfw_desc);
          if (blocks == 2) utccp_sf_atom<1>(t_sfw + 4, sfw_desc + uint64_t(32));
#pragma unroll
          for (int k = 0; k < 4; ++k)  // 32 values per instruction, one scale each: byte k of the atom's column
            mma_mxf8<1>(d_tmem, x_desc + uint64_t(k * 2), w_desc + uint64_t(k * 2), idesc_with_sf_id(idesc, k), t_sfx, t_sfw,
                        (kb > 0 || k > 0) ? 1u : 0u);
          tc_commit<1>(empty_bar(stage));
          if (kb == p.num_kb - 1) tc_commit<1>(acc_full_bar(as));
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if ((warp & 3) < row_warps) {
    // ------------------------------------------------------------------ epilogue: warp quad q holds output rows 32 q ..
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    pdl_wait();  // C may still be read by the kernels before this one
    int it = 0;
    for (int tile = blockIdx.x; tile < p.tiles_n; tile += gridDim.x, ++it) {
      const int as = it & 1;
      mbar_wait(acc_full_bar(as), uint32_t(it >> 1) & 1u, ctx, WB_DEV_TIMEOUT_EPILOGUE);
      tc_fence_after_sync();
      const uint32_t t_acc = tmem_base + (uint32_t(quad * 32) << 16) + as * kMixedTileRowsMax;
#pragma unroll 1
      for (int c0 = 0; c0 < p.tile_rows; c0 += 32) {
        uint32_t r[32];
        // the last chunk of the second accumulator reads on into the scale columns; what it finds there is not stored
        tmem_ld_32x32(t_acc + c0, r);
        tmem_ld_wait();
        if (c0 + 32 >= p.tile_rows) {  // accumulator fully read: hand it back to the MMA warp
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty_bar(as));
        }
        const int col = tile * p.tile_rows + c0;
        const int ncols = min(min(32, p.tile_rows - c0), p.N - col);
        if (row < p.M && ncols > 0 && WB_CHECK(col >= 0 && col + ncols <= p.N, kCheckOutputIndex, (long long)row << 32 | unsigned(col))) {
          OutT* dst = reinterpret_cast<OutT*>(p.c) + size_t(row) * p.ldc + col;
          if (p.accumulate) add_old_chunk32<OutT>(dst, r, ncols, p.vec_ok != 0);
          store_chunk32<OutT>(dst, r, ncols, p.vec_ok != 0);
        }
      }
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, Cfg::TMEM_COLS);
  }
}

}  // namespace wb
