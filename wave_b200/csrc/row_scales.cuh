// Activation scales of a decode GEMM (M <= 32) taken row-major by the GEMM kernel itself.
//
// The reference-facing call hands over a_scale as [M, K/32]. Packing it into the layout tcgen05.cp reads
// (scales.cuh) by a kernel of its own costs a launch on the host and, on the device, about a microsecond in front of every
// GEMM. Here one extra warp of the decode kernels brings the scales of every pipeline stage straight into the stage's
// atoms: a lane reads the eight scale bytes (one stage = 256 K) of its row and writes two 16-byte lines, exactly what the
// packed array holds there. It runs as far ahead as the ring of stages allows.
// M = 16, N = 28672, K = 8192, 24 calls on as many weights in one graph: 23.8 -> 22.8 us a call, launched eagerly 32.4 -> 28.9;
// 16 x 14336 x 4096 14.1 -> 13.4, eagerly 20.8 -> 17.4. (A graph of one call each gains 0.2 to 0.3 us.) Up to 32 rows only: the fence that hands a stage to the tensor core and the loads cost up to a microsecond a
// stage when four rows per lane are read (128 x 8192 x 8192: 31.4 -> 42.0 us), and the 128-row stages of the tile kernel
// cannot wait for that either (8192^3: 178 -> 500 us).
#pragma once
#include "ptx.cuh"
#include "scales.cuh"

namespace wb {

struct RowScales {
  const uint8_t* base;  // [rows, kblocks] bytes; a multiple of 8
  long long stride;     // bytes between rows; a multiple of 8
  int rows, kblocks;
};

// The scales of K blocks 8 kb .. 8 kb + 7 of one row; the padding byte outside the matrix. The 8-byte load is predicated and
// nothing selects on its result, so that it stays in flight until the stage it belongs to is written.
__device__ __forceinline__ uint2 row_scales_of(const RowScales& s, int row, int kb) {
  uint2 v = make_uint2(0x01010101u * WB_SF_PAD, 0x01010101u * WB_SF_PAD);
  const int left = s.kblocks - kb * 8;
  const uint8_t* p = s.base + (long long)row * s.stride + kb * 8;
  if (left >= 8) {
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

// Feeds the scale atoms of `count` stages. load(): the next stage's piece (its loads only issued); lines(piece, l0, l1): this
// lane's 16-byte line of either atom; atoms(stage): shared address of the two atoms; wait(stage, phase): the stage is free;
// signal(stage): by one lane, the scales are there.
template <int STAGES, typename Piece, typename Load, typename Lines, typename Atoms, typename Wait, typename Signal>
__device__ __forceinline__ void feed_scales(int lane, int count, uint32_t& stage, uint32_t& phase, Load load, Lines lines, Atoms atoms, Wait wait,
                                            Signal signal) {
  // The loads of D stages go out together, between two fences: a fence waits for the loads before it.
  constexpr int D = 8;
  for (int i = 0; i < count; i += D) {
    Piece v[D];
#pragma unroll
    for (int d = 0; d < D; ++d)
      if (i + d < count) v[d] = load();
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (i + d >= count) break;
      wait(stage, phase);
      uint4 l0, l1;
      lines(v[d], l0, l1);
      const uint32_t line = atoms(stage) + uint32_t(lane) * 16u;  // rows lane, lane + 32, .. of the atom
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(line), "r"(l0.x), "r"(l0.y), "r"(l0.z), "r"(l0.w) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(line + 512u), "r"(l1.x), "r"(l1.y), "r"(l1.z), "r"(l1.w) : "memory");
      fence_proxy_async_smem();  // the tensor core's copy reads them through the async proxy
      __syncwarp();
      if (lane == 0) signal(stage);
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
  }
}

// Row-major scales: stage i takes K block (kb0 + i) mod num_kb (in stages of 256 K), so that a run over several tiles is one
// sequence: the loads for the next tile's stages are not held up at its start.
template <int STAGES, typename Atoms, typename Wait, typename Signal>
__device__ __forceinline__ void feed_row_scales(const RowScales& s, int lane, int kb0, int num_kb, int count, uint32_t& stage, uint32_t& phase,
                                                Atoms atoms, Wait wait, Signal signal) {
  constexpr uint32_t kPad = 0x01010101u * WB_SF_PAD;
  int kb = kb0;
  feed_scales<STAGES, uint2>(
      lane, count, stage, phase,
      [&] {
        const uint2 v = row_scales_of(s, lane, kb);
        if (++kb == num_kb) kb = 0;
        return v;
      },
      [&](const uint2& v, uint4& l0, uint4& l1) {
        l0 = make_uint4(v.x, kPad, kPad, kPad);
        l1 = make_uint4(v.y, kPad, kPad, kPad);
      },
      atoms, wait, signal);
}

// Scales of a tile of 64 gate rows and the 64 up rows of the same hidden columns, from the usual packing of an expert's
// [2 inter, K] matrix (`gate`, `up`: this lane's eight bytes, half a line, of the two row blocks' first atoms). A copy of the scales in the
// tile's row order would have to be kept in step with weights that a caller may write at any time; the half lines are
// joined here instead, where a lane's four loads per stage stay as far ahead as the ring of stages allows.
struct GateUpScales {
  uint2 gate0, up0, gate1, up1;  // atoms 0 and 1 of a stage
};
template <int STAGES, typename Atoms, typename Wait, typename Signal>
__device__ __forceinline__ void feed_gate_up_scales(const uint8_t* gate, const uint8_t* up, int lane, int num_kb, uint32_t& stage, uint32_t& phase,
                                                    Atoms atoms, Wait wait, Signal signal) {
  auto half_line = [](const uint8_t* p) {
    uint2 v;
    asm volatile("ld.global.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
  };
  feed_scales<STAGES, GateUpScales>(
      lane, num_kb, stage, phase,
      [&] {
        const GateUpScales v{half_line(gate), half_line(up), half_line(gate + 512), half_line(up + 512)};
        gate += 1024;
        up += 1024;
        return v;
      },
      [](const GateUpScales& v, uint4& l0, uint4& l1) {
        l0 = make_uint4(v.gate0.x, v.gate0.y, v.up0.x, v.up0.y);
        l1 = make_uint4(v.gate1.x, v.gate1.y, v.up1.x, v.up1.y);
      },
      atoms, wait, signal);
}

}  // namespace wb
