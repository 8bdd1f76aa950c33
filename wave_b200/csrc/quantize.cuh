// Activation quantiser: f32 or bf16 [rows, K] -> packed E2M1 codes [rows, K/2] plus E8M0 scales,
// written row-major ([rows, K/32], the reference's a_scale layout) and/or directly in the tcgen05
// scale-factor layout, so that the GEMM needs no separate repack pass over the scales.
//
// The reference only has this as a stated direction ("fused dynamic quantization",
// wave_lang/kernel/wave/templates/test_kernels.py:74; its tests feed random codes,
// wave_lang/kernel/wave/utils/mxfp_utils.py:20-57). Rule, per 32-element block:
//   e = floor(log2(amax)) - 2 (E2M1's largest value is 6 = 1.5 * 2^2), scale byte clamp(e + 127, 0, 254),
//   amax == 0 -> byte 127; y = x * 2^-(byte - 127), clamped to [-6, 6], rounded to the nearest E2M1
//   value, a value on a midpoint going to the neighbour with the even code; even k in the low nibble.
//   A block that holds a NaN or an infinity gets scale byte 255 (E8M0's NaN: the OCP MX rule, and what the
//   reference's dequantisation reads as NaN, mxfp_utils.py:86-95) and codes 0, so that the GEMM's outputs for
//   that row are NaN instead of plausible finite numbers.
//
// HBM-bound. What bounded the first form (one block per 4 lanes and thread, 8 values each) was instruction issue: index
// arithmetic, two f32 maxima per pair and one scattered byte per scale. Here a warp takes 32 consecutive blocks, so that
//   * all of a lane's loads are in flight before any arithmetic, and a load covers whole lines;
//   * the block maximum of bf16 input is taken on packed pairs, two values per instruction;
//   * four scale bytes leave as one 32-bit word, row-major and in the packed layout alike (a word of an atom is four K blocks of one
//     row), and padding bytes are written by the same pass.
// 28672 x 8192 bf16, codes and both scale layouts (602 MB): 94.5 us (6.4 TB/s, the rate of a copy); 16384 x 8192 f32 (612 MB): 87 us;
// 3000 x 8192 bf16 with packed scales only: 12.5 us.
#pragma once
#include "ptx.cuh"
#include "scales.cuh"
#include <cuda_bf16.h>

namespace wb {

// Two f32 -> one byte of E2M1 codes (lo in the low nibble), by the hardware conversion: round to
// nearest with ties to the even code (of the magnitudes {0, .5, 1, 1.5, 2, 3, 4, 6}: 0.25 -> 0, 0.75 -> 1,
// 1.25 -> 1, 1.75 -> 2, 2.5 -> 2, 3.5 -> 4, 5 -> 4), saturating at +-6, sign in bit 3.
__device__ __forceinline__ uint32_t e2m1x2_code(float lo, float hi) {
  uint16_t r;
  asm("{ .reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; mov.b16 %0, {t, 0}; }" : "=h"(r) : "f"(hi), "f"(lo));
  return uint32_t(r);
}

// silu(g) * u = g / (1 + exp(-g)) * u in f32 with the fast exponential and division (~1e-6 relative).
__device__ __forceinline__ float silu_mul(float g, float u) { return __fdividef(g, 1.0f + __expf(-g)) * u; }
// The same for two packed bf16 pairs.
__device__ __forceinline__ void silu_mul_bf16x2(uint32_t g, uint32_t u, float& lo, float& hi) {
  lo = silu_mul(__uint_as_float(g << 16), __uint_as_float(u << 16));
  hi = silu_mul(__uint_as_float(g & 0xffff0000u), __uint_as_float(u & 0xffff0000u));
}

// Bit pattern of the largest |v| over the 32 values held by a group of 32 / VPL neighbouring lanes. For
// non-negative floats the unsigned order of the bit patterns is the numeric order, with the infinity above
// every finite value and every NaN above the infinity: an integer maximum keeps a NaN that fmaxf would drop.
template <int VPL>
__device__ __forceinline__ uint32_t block_amax_bits(const float (&v)[VPL]) {
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < VPL; ++j) m = max(m, __float_as_uint(fabsf(v[j])));
#pragma unroll
  for (int o = 1; o < 32 / VPL; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// Scale byte and codes of the 32 values held by a group of 32 / VPL neighbouring lanes (v: the VPL consecutive
// values of this lane; VPL = 4 or 8). All lanes of a warp must call it together (shuffles).
template <int VPL>
__device__ __forceinline__ void mxfp4_encode_values(const float (&v)[VPL], uint32_t& packed, int& sb) {
  static_assert(VPL == 4 || VPL == 8, "4 or 8 values per lane");
  const uint32_t amax_bits = block_amax_bits<VPL>(v);
  if ((amax_bits >> 23) == 0xffu) {  // an infinity or a NaN somewhere in the block
    sb = 255;
    packed = 0;
    return;
  }
  // floor(log2(amax)) is the unbiased exponent field for normal numbers; subnormal maxima fall
  // below the clamp at 0 either way
  sb = 127;
  if (amax_bits != 0u) {
    sb = int(amax_bits >> 23) - 2;
    sb = max(0, min(254, sb));
  }
  // y = x * 2^(127 - sb), exact; 2^127 and 2^-127 are both representable
  const int ie = 127 - sb;  // -127 .. 127
  const float inv = (ie == -127) ? __int_as_float(0x00400000) : __int_as_float((ie + 127) << 23);
  packed = 0;
#pragma unroll
  for (int j = 0; j < VPL / 2; ++j) packed |= e2m1x2_code(v[2 * j] * inv, v[2 * j + 1] * inv) << (8 * j);
}

// Stores what mxfp4_encode_values produced for row r, K block kb (lane `sub` of the group).
template <int VPL>
__device__ __forceinline__ void mxfp4_store_block(uint32_t packed, int sb, int r, int kb, int sub, int K, int kblocks,
                                                  int k_atoms, uint8_t* __restrict__ q, uint8_t* __restrict__ scale_rm,
                                                  uint8_t* __restrict__ scale_packed) {
  uint8_t* dst = q + (long long)r * (K / 2) + kb * 16;
  if constexpr (VPL == 4) reinterpret_cast<uint16_t*>(dst)[sub] = uint16_t(packed);
  else reinterpret_cast<uint32_t*>(dst)[sub] = packed;
  if (sub == 0) {
    if (scale_rm) scale_rm[(long long)r * kblocks + kb] = uint8_t(sb);
    if (scale_packed) {
      const size_t off = (size_t(r >> 7) * k_atoms + (kb >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (kb & 3);
      scale_packed[off] = uint8_t(sb);
    }
  }
}

// Quantises the 32 values of row r, K block kb held by a group of 32 / VPL neighbouring lanes and stores codes
// and scale. All lanes of a warp must call it together; inactive groups pass active = false and store nothing.
template <int VPL>
__device__ __forceinline__ void mxfp4_encode_group(const float (&v)[VPL], bool active, int r, int kb, int sub, int K,
                                                   int kblocks, int k_atoms, uint8_t* __restrict__ q,
                                                   uint8_t* __restrict__ scale_rm, uint8_t* __restrict__ scale_packed) {
  uint32_t packed;
  int sb;
  mxfp4_encode_values<VPL>(v, packed, sb);
  if (active) mxfp4_store_block<VPL>(packed, sb, r, kb, sub, K, kblocks, k_atoms, q, scale_rm, scale_packed);
}

// 8 consecutive values from 16-byte aligned memory.
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 t = *reinterpret_cast<const uint4*>(p);
  v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xffff0000u);
  v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xffff0000u);
  v[4] = __uint_as_float(t.z << 16); v[5] = __uint_as_float(t.z & 0xffff0000u);
  v[6] = __uint_as_float(t.w << 16); v[7] = __uint_as_float(t.w & 0xffff0000u);
}

__device__ __forceinline__ void raw8_values(const uint4& t, float (&v)[8]) {
  v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xffff0000u);
  v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xffff0000u);
  v[4] = __uint_as_float(t.z << 16); v[5] = __uint_as_float(t.z & 0xffff0000u);
  v[6] = __uint_as_float(t.w << 16); v[7] = __uint_as_float(t.w & 0xffff0000u);
}

// 32 bytes. `wide`: the address is a multiple of 32 (otherwise of 16).
struct Raw32 { uint32_t w[8]; };
__device__ __forceinline__ void load_raw32(const void* p, bool wide, Raw32& v) {
  if (wide) {
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p));
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(v.w[4 * i]), "=r"(v.w[4 * i + 1]), "=r"(v.w[4 * i + 2]), "=r"(v.w[4 * i + 3]) : "l"(static_cast<const uint4*>(p) + i));
  }
}

// Scale byte of a block whose largest magnitude has the f32 pattern `amax_bits` (the rule at the head of this file) and
// the factor that brings its values to codes: 2^(127 - byte). (Byte 255, a block with a NaN or an infinity, has none: the callers
// write codes 0 there whatever the product is.)
__device__ __forceinline__ int mxfp4_scale_byte(uint32_t amax_bits) {
  const int e = int(amax_bits >> 23);
  if (e == 255) return 255;
  return amax_bits == 0u ? 127 : max(0, e - 2);
}
__device__ __forceinline__ float mxfp4_code_factor(int sb) {
  // 127 - sb is -127 .. 127; 2^-127 is subnormal
  return sb >= 254 ? __int_as_float(0x00400000) : __int_as_float((254 - sb) << 23);
}

// The 32 K blocks of one warp: blocks kb0 .. kb0 + 31 of the row at `row` (nullptr: all padding); all loads are in flight before any
// arithmetic. Maxima are taken on bit patterns: the unsigned order of magnitudes is numeric order, infinity above every
// finite value and NaN above infinity. `word[i]` is the scale word of atom kb0 / 4 + atom(i, lane) (padding bytes for blocks at or past
// kblocks), held by the lanes where writes(lane).
template <typename InT>
struct WarpQuant;

// bf16: a block is 64 bytes, half a line. Two loads of 32 bytes per lane, each 1 KB of the row without a gap, two neighbouring lanes per
// block (with four blocks per four lanes a load took half lines; 28672 x 8192: 102.7 -> 94.5 us).
template <>
struct WarpQuant<__nv_bfloat16> {
  static constexpr int kWords = 2;
  uint32_t codes[2][2];  // of load u: this lane's half of block kb0 + 16 u + lane / 2
  uint32_t word[2];
  static __device__ __forceinline__ int atom(int i, int lane) { return (i * 16 + lane / 2) >> 2; }
  static __device__ __forceinline__ bool writes(int lane) { return lane % 8 == 0; }

  // wide: rows start on 32 bytes (otherwise on 16)
  __device__ __forceinline__ void run(const __nv_bfloat16* __restrict__ row, bool wide, int kb0, int kblocks, int lane) {
    Raw32 raw[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (row != nullptr && kb0 + u * 16 + (lane >> 1) < kblocks) {
        load_raw32(reinterpret_cast<const uint8_t*>(row + (long long)(kb0 + u * 16) * 32) + lane * 32, wide, raw[u]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) raw[u].w[i] = 0u;  // an all-zero block has the padding byte as its scale
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t p = raw[u].w[0] & 0x7fff7fffu;
#pragma unroll
      for (int i = 1; i < 8; ++i) p = __vmaxu2(p, raw[u].w[i] & 0x7fff7fffu);
      uint32_t m = max(p & 0xffffu, p >> 16) << 16;  // the f32 pattern of the largest magnitude
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
      const int sb = mxfp4_scale_byte(m);
      const float f = mxfp4_code_factor(sb);
      uint32_t w = uint32_t(sb) << (8 * ((lane >> 1) & 3));
      w |= __shfl_xor_sync(0xffffffffu, w, 2);
      word[u] = w | __shfl_xor_sync(0xffffffffu, w, 4);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float lo = __uint_as_float(raw[u].w[4 * i + j] << 16), hi = __uint_as_float(raw[u].w[4 * i + j] & 0xffff0000u);
          c |= e2m1x2_code(lo * f, hi * f) << (8 * j);
        }
        codes[u][i] = (sb == 255) ? 0u : c;
      }
    }
  }
  // The codes to the row's code bytes; vec: they start on 16 bytes (otherwise on 4).
  __device__ __forceinline__ void store_codes(uint8_t* __restrict__ q_row, bool vec, int kb0, int kblocks, int lane) const {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (kb0 + u * 16 + (lane >> 1) >= kblocks) continue;
      uint8_t* d = q_row + (kb0 + u * 16) * 16 + lane * 8;
      if (vec) {
        *reinterpret_cast<uint2*>(d) = make_uint2(codes[u][0], codes[u][1]);
      } else {
        reinterpret_cast<uint32_t*>(d)[0] = codes[u][0];
        reinterpret_cast<uint32_t*>(d)[1] = codes[u][1];
      }
    }
  }
};

// f32: a block is a line. Lane l belongs to group g = l / 4, whose blocks are kb0 + 4 g .. + 3 = one scale word.
template <>
struct WarpQuant<float> {
  static constexpr int kWords = 1;
  uint4 codes;  // of block kb0 + lane
  uint32_t word[1];
  static __device__ __forceinline__ int atom(int, int lane) { return lane >> 2; }
  static __device__ __forceinline__ bool writes(int lane) { return (lane & 3) == 0; }

  __device__ __forceinline__ void run(const float* __restrict__ row, bool, int kb0, int kblocks, int lane) {
    const int g = lane >> 2, sub = lane & 3;
    Raw32 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int kb = kb0 + g * 4 + u;
      if (row != nullptr && kb < kblocks) {
        load_raw32(row + kb * 32 + sub * 8, false, raw[u]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) raw[u].w[i] = 0u;
      }
    }
    uint32_t w[4], scales = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) m = max(m, raw[u].w[i] & 0x7fffffffu);
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
      const int sb = mxfp4_scale_byte(m);
      scales |= uint32_t(sb) << (8 * u);
      const float f = mxfp4_code_factor(sb);
      w[u] = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        w[u] |= e2m1x2_code(__uint_as_float(raw[u].w[2 * j]) * f, __uint_as_float(raw[u].w[2 * j + 1]) * f) << (8 * j);
      if (sb == 255) w[u] = 0u;
    }
    word[0] = scales;
    // 4 x 4 transpose over the group: lane `sub` ends with the four words of block 4 g + sub
    const bool b1 = sub & 1, b2 = sub & 2;
    const uint32_t s0 = __shfl_xor_sync(0xffffffffu, b1 ? w[0] : w[1], 1), s1 = __shfl_xor_sync(0xffffffffu, b1 ? w[2] : w[3], 1);
    const uint32_t x0 = b1 ? s0 : w[0], x1 = b1 ? w[1] : s0, x2 = b1 ? s1 : w[2], x3 = b1 ? w[3] : s1;
    const uint32_t t0 = __shfl_xor_sync(0xffffffffu, b2 ? x0 : x2, 2), t1 = __shfl_xor_sync(0xffffffffu, b2 ? x1 : x3, 2);
    codes.x = b2 ? t0 : x0;
    codes.y = b2 ? t1 : x1;
    codes.z = b2 ? x2 : t0;
    codes.w = b2 ? x3 : t1;
  }
  __device__ __forceinline__ void store_codes(uint8_t* __restrict__ q_row, bool vec, int kb0, int kblocks, int lane) const {
    if (kb0 + lane >= kblocks) return;
    uint8_t* d = q_row + (kb0 + lane) * 16;
    if (vec) {
      *reinterpret_cast<uint4*>(d) = codes;
    } else {
      uint32_t* d4 = reinterpret_cast<uint32_t*>(d);
      d4[0] = codes.x; d4[1] = codes.y; d4[2] = codes.z; d4[3] = codes.w;
    }
  }
};

// The scale bytes of a warp's blocks to the row's at `scale_row`; words: every row of them starts on 4 bytes.
template <typename Quant>
__device__ __forceinline__ void store_scale_row(const Quant& w, uint8_t* __restrict__ scale_row, bool words, int kb0, int kblocks, int lane) {
  if (!Quant::writes(lane)) return;
#pragma unroll
  for (int i = 0; i < Quant::kWords; ++i) {
    const int kb = kb0 + Quant::atom(i, lane) * 4;
    if (words) {
      if (kb < kblocks) *reinterpret_cast<uint32_t*>(scale_row + kb) = w.word[i];
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (kb + j < kblocks) scale_row[kb + j] = uint8_t(w.word[i] >> (8 * j));
    }
  }
}
// Rows of x start on 32 bytes.
template <typename InT>
__device__ __forceinline__ bool rows_on_32(const InT* x, long long ldx) {
  return ((reinterpret_cast<uintptr_t>(x) | uintptr_t(ldx * (long long)sizeof(InT))) & 31) == 0;
}

// Word (row r, atom) of a packed scale array: the four K blocks of that atom.
__device__ __forceinline__ uint32_t* packed_scale_word(uint8_t* base, int k_atoms, int r, int atom) {
  return reinterpret_cast<uint32_t*>(base + (size_t(r >> 7) * k_atoms + atom) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4);
}

// One warp per (row, 32 K blocks). The 8 warps of a CTA take the same 32 K blocks of 8 rows of a 128-row block: two
// neighbouring rows of each of its four 32-row groups. Their scale words of one atom are 32 consecutive bytes of the packed
// layout, so the words are exchanged through shared memory and every 32-byte sector is written once (a warp that writes its
// own 8 words touches 8 sectors with 4 bytes each). Rows past `rows` (the padding rows of the packed scales) get the padding byte
// only. x rows are 16-byte aligned; q rows 16-byte aligned when q_vec. Grid: 16 x row blocks x chunks of 32 K blocks.
// release: the library launches this kernel's programmatic dependent right behind it, which waits before it reads a scale
// or a code. Otherwise it does not let dependents start early: what it writes may be the WEIGHTS of a GEMM two launches
// on, which WB200_OVERLAP_PREVIOUS allows to be read before that GEMM's wait.
// (bf16: 32 registers, so that an SM holds 2048 threads; a form that took 38 needed 100 us for 28672 x 8192.)
template <typename InT>
__global__ void __launch_bounds__(256)
quantize_mxfp4_kernel(const InT* __restrict__ x, long long ldx, int rows, int K, uint8_t* __restrict__ q, int q_vec,
                      uint8_t* __restrict__ scale_rm, uint8_t* __restrict__ scale_packed, int k_atoms, int release) {
  __shared__ uint32_t words[8][8];  // [atom of the chunk][word of the sector]
  pdl_wait();
  if (release) pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kblocks = K >> 5;
  const unsigned chunks = unsigned(k_atoms + 7) >> 3;
  const unsigned group = blockIdx.x / chunks;  // 8 rows
  const int kb0 = int(blockIdx.x - group * chunks) * 32;
  const int r = int(group >> 4) * 128 + (warp & 3) * 32 + int(group & 15) * 2 + (warp >> 2);
  const bool real = r < rows;
  using Quant = WarpQuant<InT>;
  Quant w;
  w.run(real ? x + (long long)r * ldx : static_cast<const InT*>(nullptr), rows_on_32(x, ldx), kb0, kblocks, lane);
  if (real) {
    w.store_codes(q + (long long)r * (K / 2), q_vec, kb0, kblocks, lane);
    if (scale_rm) store_scale_row(w, scale_rm + (long long)r * kblocks, (kblocks & 3) == 0 && (reinterpret_cast<uintptr_t>(scale_rm) & 3) == 0, kb0, kblocks, lane);
  }
  if (scale_packed) {
    if (Quant::writes(lane)) {
#pragma unroll
      for (int i = 0; i < Quant::kWords; ++i) words[Quant::atom(i, lane)][warp] = w.word[i];  // word (row of the pair, 32-row group) of the sector
    }
    __syncthreads();
    const int atom = (kb0 >> 2) + (threadIdx.x >> 3);
    if (threadIdx.x < 64 && atom < k_atoms) {
      uint8_t* d = scale_packed + (size_t(group >> 4) * k_atoms + atom) * 512 + (group & 15) * 32 + (threadIdx.x & 7) * 4;
      const uint32_t word = words[threadIdx.x >> 3][threadIdx.x & 7];
      if ((reinterpret_cast<uintptr_t>(scale_packed) & 3) == 0) {
        *reinterpret_cast<uint32_t*>(d) = word;
      } else {  // an array that a caller placed at any byte
#pragma unroll
        for (int u = 0; u < 4; ++u) d[u] = uint8_t(word >> (8 * u));
      }
    }
  }
}

// MXFP8 counterpart: f32 or bf16 [rows, K] -> one byte per element (E4M3 when fmt == 0, E5M2 when fmt == 1) plus
// E8M0 scales, e = floor(log2(amax)) - 8 (E4M3: largest value 448) or - 15 (E5M2: 57344); the rounding and the
// saturation are the hardware conversion's (cvt.rn.satfinite). Same thread layout as the MXFP4 quantiser.
__device__ __forceinline__ uint32_t f8x2_code(float lo, float hi, int fmt) {
  uint16_t r;
  if (fmt == 0) asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  else asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return uint32_t(r);
}

template <typename InT>
__global__ void __launch_bounds__(256)
quantize_mxfp8_kernel(const InT* __restrict__ x, long long ldx, int rows, int K, int fmt, uint8_t* __restrict__ q,
                      uint8_t* __restrict__ scale_rm, uint8_t* __restrict__ scale_packed, int k_atoms) {
  const int sub = threadIdx.x & 3;
  const int kblocks = K >> 5;
  const int r = blockIdx.x;
  const int kb = blockIdx.y * 64 + (threadIdx.x >> 2);
  const bool active = r < rows && kb < kblocks;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (active) load8(x + (long long)r * ldx + kb * 32 + sub * 8, v);
  const uint32_t amax_bits = block_amax_bits<8>(v);
  const bool not_finite = (amax_bits >> 23) == 0xffu;  // an infinity or a NaN in the block: scale byte 255, codes 0
  int sb = not_finite ? 255 : 127;
  if (!not_finite && amax_bits != 0u) {
    sb = int(amax_bits >> 23) - (fmt == 0 ? 8 : 15);
    sb = max(0, min(254, sb));
  }
  const int ie = 127 - sb;
  const float inv = (ie <= -127) ? __int_as_float(0x00400000) : __int_as_float((ie + 127) << 23);
  if (!active) return;
  uint2 out = make_uint2(0u, 0u);
  if (!not_finite) {
    out.x = f8x2_code(v[0] * inv, v[1] * inv, fmt) | (f8x2_code(v[2] * inv, v[3] * inv, fmt) << 16);
    out.y = f8x2_code(v[4] * inv, v[5] * inv, fmt) | (f8x2_code(v[6] * inv, v[7] * inv, fmt) << 16);
  }
  *reinterpret_cast<uint2*>(q + (long long)r * K + kb * 32 + sub * 8) = out;
  if (sub == 0) {
    if (scale_rm) scale_rm[(long long)r * kblocks + kb] = uint8_t(sb);
    if (scale_packed) {
      const size_t off = (size_t(r >> 7) * k_atoms + (kb >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (kb & 3);
      scale_packed[off] = uint8_t(sb);
    }
  }
}

// Quantise-and-scatter for routed tokens: row t of x is quantised once and written to the `copies` output rows
// dst_rows[t * copies + j] (negative entries are skipped): the tokens of a mixture-of-experts layer go straight
// to their expert-sorted rows without a separate gather pass. Scales are written row-major.
template <typename InT>
__global__ void __launch_bounds__(256)
quantize_scatter_mxfp4_kernel(const InT* __restrict__ x, long long ldx, int rows, int K, int copies,
                              const int* __restrict__ dst_rows, uint8_t* __restrict__ q, int q_vec, uint8_t* __restrict__ scale_rm,
                              int k_atoms) {
  const int lane = threadIdx.x & 31;
  const int kblocks = K >> 5;
  const unsigned chunks = unsigned(k_atoms + 7) >> 3;
  const unsigned wid = blockIdx.x * 8u + (threadIdx.x >> 5);
  const int r = int(wid / chunks);
  if (r >= rows) return;
  const int kb0 = int(wid - unsigned(r) * chunks) * 32;
  WarpQuant<InT> w;
  w.run(x + (long long)r * ldx, rows_on_32(x, ldx), kb0, kblocks, lane);
  const bool words = (kblocks & 3) == 0 && (reinterpret_cast<uintptr_t>(scale_rm) & 3) == 0;
  for (int j = 0; j < copies; ++j) {
    const int dst = __ldcg(dst_rows + r * copies + j);
    if (dst < 0) continue;
    w.store_codes(q + (long long)dst * (K / 2), q_vec, kb0, kblocks, lane);
    store_scale_row(w, scale_rm + (long long)dst * kblocks, words, kb0, kblocks, lane);
  }
}

// Fills the padding bytes of a packed scale array (rows past `rows` in the last 128-row block, K blocks
// past K/32 in the last atoms) with the neutral byte; the quantiser above writes only real positions.
__global__ void __launch_bounds__(256)
fill_scale_padding_kernel(uint8_t* __restrict__ scale_packed, int rows, int kblocks, int k_atoms, int row_blocks) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)row_blocks * k_atoms * 512;
  if (idx >= total) return;
  const int within = int(idx & 511);
  const long long atom = idx >> 9;
  const int rb = int(atom / k_atoms), ka = int(atom - (long long)rb * k_atoms);
  const int r = rb * 128 + ((within >> 2) & 3) * 32 + (within >> 4);
  const int kb = ka * 4 + (within & 3);
  if (r >= rows || kb >= kblocks) scale_packed[idx] = WB_SF_PAD;
}

}  // namespace wb
