// Activation scales of a decode GEMM (M <= 32) taken row-major by the GEMM kernel itself.
//
// The reference-facing call hands over a_scale as [M, K/32]. Packing it into the layout tcgen05.cp reads
// (scales.cuh) by a kernel of its own costs a launch on the host and, on the device, about a microsecond in front of every
// GEMM. Here one extra warp of the decode kernels brings the scales of every pipeline stage straight into the stage's
// atoms: a lane reads the eight scale bytes (one stage = 256 K) of its row and writes two 16-byte lines, exactly what the
// packed array holds there. It runs as far ahead as the ring of stages allows.
// M = 16, N = 28672, K = 8192, replayed from a graph: 23.6 -> 22.6 us, launched eagerly 26.2 -> 24.2; 16 x 4096 x 4096 eagerly
// 24.8 -> 19.5. Up to 32 rows only: the fence that hands a stage to the tensor core and the loads cost up to a microsecond a
// stage when four rows per lane are read (128 x 8192 x 8192: 31.4 -> 42.0 us), and the 128-row stages of the tile kernel
// cannot wait for that either (8192^3: 178 -> 500 us).
#pragma once
#include "ptx.cuh"
#include "scales.cuh"

namespace wb {

struct RowScales {
  const uint8_t* base;  // [rows, kblocks] bytes
  long long stride;     // bytes between rows
  int rows, kblocks;
  int vec;              // base and stride are multiples of 8: whole 8-byte loads
};

// The scales of K blocks 8 kb .. 8 kb + 7 of one row; the padding byte outside the matrix. The 8-byte load is predicated and
// nothing selects on its result, so that it stays in flight until the stage it belongs to is written.
__device__ __forceinline__ uint2 row_scales_of(const RowScales& s, int row, int kb) {
  uint2 v = make_uint2(0x01010101u * WB_SF_PAD, 0x01010101u * WB_SF_PAD);
  const int left = s.kblocks - kb * 8;
  const uint8_t* p = s.base + (long long)row * s.stride + kb * 8;
  if (s.vec && left >= 8) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p ld.global.v2.b32 {%0, %1}, [%2];\n\t}"
                 : "+r"(v.x), "+r"(v.y) : "l"(p), "r"(int(row < s.rows)) : "memory");
    return v;
  }
  if (row >= s.rows || left <= 0) return v;
  uint32_t w[2] = {v.x, v.y};
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < left) w[j >> 2] = (w[j >> 2] & ~(0xffu << (8 * (j & 3)))) | (uint32_t(p[j]) << (8 * (j & 3)));
  return make_uint2(w[0], w[1]);
}

constexpr int kRowScaleRows = 32;  // one row per lane

// Feeds `count` stages; stage i takes K block (kb0 + i) mod num_kb (in stages of 256 K), so that a run over several tiles is
// one sequence: the loads for the next tile's stages are not held up at its start. atoms(stage): shared address of its two
// atoms; wait(stage, phase): the stage is free; signal(stage): by one lane, the scales are there.
template <int STAGES, typename Atoms, typename Wait, typename Signal>
__device__ __forceinline__ void feed_row_scales(const RowScales& s, int lane, int kb0, int num_kb, int count, uint32_t& stage, uint32_t& phase,
                                                Atoms atoms, Wait wait, Signal signal) {
  // The loads of D stages go out together, between two fences: a fence waits for the loads before it.
  constexpr int D = 8;
  constexpr uint32_t kPad = 0x01010101u * WB_SF_PAD;
  int kb = kb0;
  for (int i = 0; i < count; i += D) {
    uint2 v[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      v[d] = (i + d < count) ? row_scales_of(s, lane, kb) : make_uint2(kPad, kPad);
      if (++kb == num_kb) kb = 0;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (i + d >= count) break;
      wait(stage, phase);
      const uint32_t line = atoms(stage) + uint32_t(lane) * 16u;  // rows lane, lane + 32, .. of the atom
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %2, %2};" ::"r"(line), "r"(v[d].x), "r"(kPad) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %2, %2};" ::"r"(line + 512u), "r"(v[d].y), "r"(kPad) : "memory");
      fence_proxy_async_smem();  // the tensor core's copy reads them through the async proxy
      __syncwarp();
      if (lane == 0) signal(stage);
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
  }
}

}  // namespace wb
