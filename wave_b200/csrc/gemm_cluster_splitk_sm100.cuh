// MXFP4 x MXFP4 block-scaled GEMM for few output tiles and a long K: the K range of one tile is cut into 2 to 4 slices
// that run on the CTA pairs of ONE cluster and meet in distributed shared memory.
//
// The tile kernel (gemm_sm100.cuh) gives one tile to one CTA pair. With fewer tiles than pairs (the shapes the reference's
// split-K templates are for, wave_lang/kernel/wave/templates/tagged_mxfp4_gemm.py:611-947) most SMs idle while a pair
// walks all of K. Here
//   * a cluster holds `slices` pairs (4, 6 or 8 CTAs); pair s multiplies its share of the K blocks with the pipeline of the
//     tile kernel (same stages, same descriptors, one accumulator);
//   * when every pair of the cluster has finished, each 32-column chunk of the f32 accumulator goes to the pair that owns it
//     (chunk c: pair c mod slices) with 16-byte stores into that CTA's shared memory, where the ring of stages has become
//     free, and the owner adds the slices in slice order: the same bits on every run, no workspace, no atomics, no
//     second launch and no table of tensor maps per slice (which makes the workspace form too dear on the host to
//     be taken by eager calls).
// A thread holds one row; a piece of 4 columns is 16 bytes at [piece][row], so that the 32 lanes of a warp write and
// read 512 contiguous bytes.
// What bounds a plain launch of such a shape is what one SM can fetch (about 64 bytes a clock from L2: 0.19 us per 256 K of a
// 256 x 128 tile); a cluster spreads that over its SMs and pays ~3 us for its wider start and the exchange.
// 512 x 2048 x 16000: 18.5 -> 15.4 us with 2 slices; 512 x 512 x 16000: 17.8 -> 14.0 / 12.8 / 11.7 us with 2 / 3 / 4.
#pragma once
#include "gemm_sm100.cuh"

namespace wb {

constexpr int kMaxClusterSlices = 4;

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// 32 columns of one row of C as they are in memory (16-byte aligned, read through L2).
template <typename OutT>
struct OldChunk {
  static constexpr int V = 32 * int(sizeof(OutT)) / 16;
  uint4 v[V];
  __device__ __forceinline__ void load(const OutT* p) {
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = __ldcg(reinterpret_cast<const uint4*>(p) + j);
  }
  __device__ __forceinline__ void add_to(uint32_t (&r)[32]) const {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if constexpr (sizeof(OutT) == 4) {
          r[4 * j + i] = __float_as_uint(__uint_as_float(r[4 * j + i]) + __uint_as_float(w[i]));
        } else {
          r[8 * j + 2 * i] = __float_as_uint(__uint_as_float(r[8 * j + 2 * i]) + __uint_as_float(w[i] << 16));
          r[8 * j + 2 * i + 1] = __float_as_uint(__uint_as_float(r[8 * j + 2 * i + 1]) + __uint_as_float(w[i] & 0xffff0000u));
        }
      }
    }
  }
};

template <int BN, typename OutT>
struct ClusterSplitCfg {
  using Base = GemmCfg<2, BN, int(sizeof(OutT))>;
  static constexpr int STAGES = Base::STAGES;
  static constexpr int NUM_BARRIERS = 2 * STAGES + 1;
  static constexpr int SMEM_BYTES = 1024 + STAGES * Base::STAGE_BYTES + NUM_BARRIERS * 8 + 64;
  static constexpr int CHUNKS = BN / 32;
  static constexpr int OWNED = (CHUNKS + 1) / 2;  // chunks that a pair owns at most: with two slices
  static constexpr int CHUNK_BYTES = 128 * 128;  // 128 rows x 32 columns of f32
  // what the other slices deposit here: at most (slices - 1) * ceil(CHUNKS / slices) chunks
  static_assert(3 * ((CHUNKS + 3) / 4) * CHUNK_BYTES <= STAGES * Base::STAGE_BYTES && 2 * ((CHUNKS + 2) / 3) * CHUNK_BYTES <= STAGES * Base::STAGE_BYTES &&
                    ((CHUNKS + 1) / 2) * CHUNK_BYTES <= STAGES * Base::STAGE_BYTES, "the deposits fit in the ring");
};

template <int BN, typename OutT>
__global__ void __launch_bounds__(192, 1)
mxfp4_gemm_cluster_splitk_kernel(const __grid_constant__ PlainMaps maps, const GemmParams p, const int slices) {
  using Cfg = GemmCfg<2, BN, int(sizeof(OutT))>;
  using Split = ClusterSplitCfg<BN, OutT>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment for the 128-byte swizzle; identical offset in all CTAs of the cluster
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cluster_rank = cluster_ctarank();
  const int slice = int(cluster_rank >> 1);
  const uint32_t rank = cluster_rank & 1u;  // in the pair
  const uint32_t leader_rank = cluster_rank & ~1u;
  const bool leader = rank == 0;

  const uint32_t bar_base = smem_base + STAGES * Cfg::STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  const uint32_t acc_full_bar = bar_base + 8u * (2 * STAGES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_gen + STAGES * Cfg::STAGE_BYTES + Split::NUM_BARRIERS * 8);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  WaitCtx ctx{abort_flag, p.status};

  if (threadIdx.x == 0) {
    for (int b = 0; b < Split::NUM_BARRIERS; ++b) mbar_init(bar_base + 8u * b, 1);
    *abort_flag = 0u;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc<2>(smem_u32(tmem_slot), Cfg::TMEM_COLS);
    tmem_relinquish<2>();
  }
  if (warp == 0 && lane == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) prefetch_tensormap(maps.map(0, i));
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();  // the barriers of every CTA exist before anyone signals them
  cluster_wait();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  int mt, nt;
  raster_tile(int(blockIdx.x) / (2 * slices), p.tiles_m, p.tiles_n, p.group_n, mt, nt);
  const int num_kb = (p.K + Cfg::BK - 1) / Cfg::BK;
  const int kb0 = num_kb * slice / slices, kb1 = num_kb * (slice + 1) / slices;  // num_kb >= slices: never empty

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    uint32_t stage = 0, phase = 0;
    pdl_wait();  // the packed activation scales may be written by the kernel launched just before this one
    const int a_row = (mt * 2 + int(rank)) * Cfg::BM;
    const int b_row = nt * BN + int(rank) * Cfg::B_ROWS;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(empty_bar(stage), phase ^ 1u, ctx, WB_DEV_TIMEOUT_PRODUCER);
      const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES;
      const uint32_t sB = sA + Cfg::A_BYTES;
      const uint32_t sSFA = sB + Cfg::B_BYTES;
      const uint32_t sSFB = sSFA + Cfg::SFA_BYTES;
      const uint32_t fb = mapa_shared(full_bar(stage), leader_rank);  // the loads of both CTAs report to the pair's leader
      if (elect_one()) {
        if (leader) mbar_expect_tx(full_bar(stage), Cfg::LOAD_BYTES * 2);
        tma_load_2d<2>(sA, maps.map(0, 0), kb * 128, a_row, fb);
        tma_load_2d<2>(sB, maps.map(0, 1), kb * 128, b_row, fb);
        tma_load_2d<2>(sSFA, maps.map(0, 2), kb * (Cfg::SF_ATOMS * 128), mt * 2 + int(rank), fb);
        tma_load_2d<2>(sSFB, maps.map(0, 3), kb * (Cfg::SF_ATOMS * 128), (nt * BN) / 128, fb);
      }
      __syncwarp();
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
    pdl_launch_dependents();  // (as in gemm_sm100.cuh)
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader of each pair)
    if (leader) {
      const uint32_t idesc = make_idesc_mxf4(Cfg::BM * 2, BN);
      const uint32_t peer = leader_rank + 1;
      const uint32_t peer_empty0 = mapa_shared(empty_bar(0), peer), peer_acc_full = mapa_shared(acc_full_bar, peer);
      uint32_t stage = 0, phase = 0, sf_set = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        const uint32_t t_sfa = tmem_base + Cfg::SF_COL + sf_set * Cfg::SF_SET_COLS;
        const uint32_t t_sfb = t_sfa + 8;
        if (++sf_set == Cfg::SF_SETS) sf_set = 0;
        mbar_wait(full_bar(stage), phase, ctx, WB_DEV_TIMEOUT_MMA_FULL);
        tc_fence_after_sync();
        const uint32_t sA = smem_base + stage * Cfg::STAGE_BYTES;
        const uint32_t sB = sA + Cfg::A_BYTES;
        const uint32_t sSFA = sB + Cfg::B_BYTES;
        const uint64_t a_desc = make_desc_k_sw128(sA), b_desc = make_desc_k_sw128(sB);
        const uint64_t sfa_desc = make_desc_sf_atom(sSFA), sfb_desc = make_desc_sf_atom(sSFA + Cfg::SFA_BYTES);
        if (elect_one()) {
#pragma unroll
          for (int a = 0; a < Cfg::SF_ATOMS; ++a) utccp_sf_atom<2>(t_sfa + a * 4, sfa_desc + uint64_t(a * 32));
#pragma unroll
          for (int j = 0; j < Cfg::SFB_BLOCKS; ++j)
#pragma unroll
            for (int a = 0; a < Cfg::SF_ATOMS; ++a)
              utccp_sf_atom<2>(t_sfb + a * (Cfg::SFB_BLOCKS * 4) + j * 4, sfb_desc + uint64_t((j * Cfg::SF_ATOMS + a) * 32));
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_mxf4<2>(tmem_base, a_desc + uint64_t(k * 2), b_desc + uint64_t(k * 2), idesc_with_sf_id(idesc, (k & 1) * 2),
                        t_sfa + (k >> 1) * 4, t_sfb + (k >> 1) * (Cfg::SFB_BLOCKS * 4), (kb > kb0 || k > 0) ? 1u : 0u);
          tc_commit<2>(empty_bar(stage));
          tc_commit<2>(peer_empty0 + 8u * stage);
          if (kb == kb1 - 1) {
            tc_commit<2>(acc_full_bar);
            tc_commit<2>(peer_acc_full);
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else {
    // this pair's MMAs are done: they have read every stage, and every load they needed has landed
    mbar_wait(acc_full_bar, 0u, ctx, WB_DEV_TIMEOUT_EPILOGUE);
  }
  __syncwarp();
  tc_fence_before_sync();
  cluster_arrive();  // once all have come here the rings of all CTAs of the cluster are free

  const int quad = warp & 3;  // tensor-memory lane quadrant (warps 2 .. 5)
  const uint32_t t_acc = tmem_base + (uint32_t(quad * 32) << 16);
  const int lane_row = quad * 32 + lane;
  const int row = (mt * 2 + int(rank)) * Cfg::BM + lane_row;
  const int per_owner = (Split::CHUNKS + slices - 1) / slices;  // chunks a pair can own
  // What C holds under this pair's chunks is fetched while the slices are exchanged (whole chunks of 16-byte aligned rows).
  OldChunk<OutT> old[Split::OWNED];
  const bool early = p.accumulate && p.vec_ok && row < p.M;
  if (warp >= 2) {
    pdl_wait();  // C may still be used by the kernels before this one
#pragma unroll
    for (int i = 0; i < Split::OWNED; ++i) {
      const int c = slice + i * slices, col = nt * BN + c * 32;
      if (early && c < Split::CHUNKS && col + 32 <= p.N) old[i].load(reinterpret_cast<const OutT*>(p.c) + size_t(row) * p.ldc + col);
    }
  }
  cluster_wait();
  tc_fence_after_sync();

  if (warp >= 2) {
#pragma unroll 1
    for (int c = 0; c < Split::CHUNKS; ++c) {
      const int owner = c % slices;
      if (owner == slice || nt * BN + c * 32 >= p.N) continue;
      uint32_t r[32];
      tmem_ld_32x32(t_acc + c * 32, r);
      tmem_ld_wait();
      const int slot = (slice < owner ? slice : slice - 1) * per_owner + c / slices;
      const uint32_t dst = mapa_shared(smem_base + uint32_t(slot) * Split::CHUNK_BYTES + uint32_t(lane_row) * 16u, uint32_t(owner) * 2u + rank);
#pragma unroll
      for (int j = 0; j < 8; ++j) st_cluster_v4(dst + j * 2048u, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
    }
  }
  __syncwarp();
  cluster_arrive();  // release: the deposits are visible to their owners after the wait
  cluster_wait();

  if (warp >= 2) {
#pragma unroll
    for (int i = 0; i < Split::OWNED; ++i) {
      const int c = slice + i * slices, col = nt * BN + c * 32;
      if (c >= Split::CHUNKS || col >= p.N) break;
      uint32_t own[32];
      tmem_ld_32x32(t_acc + c * 32, own);
      tmem_ld_wait();
      uint32_t r[32];
#pragma unroll 1
      for (int s = 0; s < slices; ++s) {
        if (s == slice) {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = s == 0 ? own[j] : __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(own[j]));
        } else {
          const uint32_t src = smem_base + uint32_t((s < slice ? s : s - 1) * per_owner + c / slices) * Split::CHUNK_BYTES + uint32_t(lane_row) * 16u;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint4 v = ld_shared_v4(src + j * 2048u);
            if (s == 0) {
              r[4 * j] = v.x; r[4 * j + 1] = v.y; r[4 * j + 2] = v.z; r[4 * j + 3] = v.w;
            } else {
              r[4 * j] = __float_as_uint(__uint_as_float(r[4 * j]) + __uint_as_float(v.x));
              r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + __uint_as_float(v.y));
              r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + __uint_as_float(v.z));
              r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + __uint_as_float(v.w));
            }
          }
        }
      }
      if (row < p.M && WB_CHECK(row >= 0 && col >= 0 && col < p.N, kCheckOutputIndex, (long long)row << 32 | unsigned(col))) {
        OutT* dst = reinterpret_cast<OutT*>(p.c) + size_t(row) * p.ldc + col;
        const int ncols = min(32, p.N - col);
        if (early && ncols == 32) old[i].add_to(r);
        else if (p.accumulate) add_old_chunk32<OutT>(dst, r, ncols, p.vec_ok != 0);
        store_chunk32<OutT>(dst, r, ncols, p.vec_ok != 0);
      }
    }
  }

  // ------------------------------------------------------------------ teardown: the pair leaves together
  tc_fence_before_sync();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<2>(tmem_base, Cfg::TMEM_COLS);
  }
}

}  // namespace wb
