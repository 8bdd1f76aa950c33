// Activation scales taken row-major by the GEMM kernels themselves.
//
// The reference-facing call hands over a_scale as [M, K/32]. Packing it into the layout tcgen05.cp reads
// (scales.cuh) by a kernel of its own costs a launch on the host and, on the device, its own start and end in front
// of every GEMM: 2 to 3 us, a tenth of a decode step. Here one extra warp of the GEMM brings the scales of every pipeline
// stage straight into the stage's atoms: a lane reads the eight scale bytes (one stage = 256 K) of rows lane, lane + 32, ..
// and writes two 16-byte lines, exactly what the packed array holds there. It runs as far ahead as the ring of stages allows;
// a row's bytes of four consecutive stages share a 32-byte sector.
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

// Feeds stages with the scales of K blocks [kb0, kb1) (in stages of 256 K) of rows row0 .. row0 + 32 R - 1. atoms(stage): shared
// address of the stage's two atoms; wait(stage, phase): the stage is free; signal(stage): by one lane, the scales are there.
template <int R, int STAGES, typename Atoms, typename Wait, typename Signal>
__device__ __forceinline__ void feed_row_scales(const RowScales& s, int row0, int lane, int kb0, int kb1, uint32_t& stage, uint32_t& phase,
                                                Atoms atoms, Wait wait, Signal signal) {
  // The loads of D stages go out together, between two fences: a fence waits for the loads before it, so one that is
  // in flight across the fence of a stage costs that stage its whole latency (1.1 us a stage instead of ~0.25).
  constexpr int D = 8;
  constexpr uint32_t kPad = 0x01010101u * WB_SF_PAD;
  for (int kb = kb0; kb < kb1; kb += D) {
    uint2 v[D][R];
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
      for (int r = 0; r < R; ++r) v[d][r] = (kb + d < kb1) ? row_scales_of(s, row0 + r * 32 + lane, kb + d) : make_uint2(kPad, kPad);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (kb + d >= kb1) break;
      wait(stage, phase);
      const uint32_t line = atoms(stage) + uint32_t(lane) * 16u;
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(line), "r"(v[d][0].x), "r"(R > 1 ? v[d][1 % R].x : kPad),
                   "r"(R > 2 ? v[d][2 % R].x : kPad), "r"(R > 3 ? v[d][3 % R].x : kPad) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(line + 512u), "r"(v[d][0].y), "r"(R > 1 ? v[d][1 % R].y : kPad),
                   "r"(R > 2 ? v[d][2 % R].y : kPad), "r"(R > 3 ? v[d][3 % R].y : kPad) : "memory");
      fence_proxy_async_smem();  // the tensor core's copy reads them through the async proxy
      __syncwarp();
      if (lane == 0) signal(stage);
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
  }
}

}  // namespace wb
