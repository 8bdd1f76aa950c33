// The steps either side of the grouped (per-expert) MXFP4 GEMM in a mixture-of-experts MLP:
//
//   moe_align_block_size   routed (token, slot) pairs -> rows sorted by expert, every expert padded to
//                          whole blocks. Same outputs as the reference's moe_align_block_size_pytorch
//                          (tests/kernel/moe/torch_kernels.py:10-97), integer work, bit-exact.
//   moe_gather_rows        copy the packed codes / scales of each routed token to its sorted row.
//   silu_and_mul           out = x1 / (1 + exp(-x1)) * x2, the reference's get_silu_and_mul_kernel
//                          (wave_lang/kernel/wave/templates/moe.py:89-145; checked there against
//                          gate * up / (1 + exp(-gate)), tests/kernel/moe_test.py:39-40), optionally
//                          quantised to MXFP4 in the same pass so that the down projection reads codes.
//   moe_combine            out[t] = sum_j weight[t, j] * y[row of (t, j)]: the weighted sum at the end of
//                          the reference's MoE (tests/kernel/moe_test.py:123-127).
//
// All four are HBM- or latency-bound integer / elementwise work: coalesced 16-byte accesses, no
// tensor cores.
#pragma once
#include "ptx.cuh"
#include "quantize.cuh"

namespace wb {

constexpr int kMoeMaxExperts = 256;

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// One CTA of 1024 threads. ids: [n] expert of every routed (token, slot) pair in flat order.
// sorted_ids [sorted_cap]: flat indices grouped by expert, ascending inside an expert, each expert's
// run padded with the value n to a multiple of block_size; the rest of the array is n as well.
// expert_ids [total / block_size]: expert of every block. inverse [n] (may be null): position of
// flat index i in sorted_ids. Ids outside [0, E) are skipped.
// Latency-bound. Every warp owns a contiguous run of ids: it counts them per expert in its own row of a table, one scan over
// the rows gives every warp its first position per expert, and a second walk over the run places the ids; positions are
// in flat order because the runs are. Three CTA barriers in all, where there was a walk in chunks of 1024 ids with a scan per
// chunk: 8192 ids of 8 experts 14.5 -> 9.2 us (calls back to back from a graph), 32768 of 256 experts 123 -> 92, 32 ids 3.4 -> 3.3.
template <typename IdT>
__global__ void __launch_bounds__(1024)
moe_align_block_size_kernel(const IdT* __restrict__ ids, int n, int E, int block_size, int sorted_cap,
                            int* __restrict__ sorted_ids, int* __restrict__ expert_ids,
                            int* __restrict__ num_tokens_post_pad, int* __restrict__ inverse) {
  __shared__ int next[32][kMoeMaxExperts];  // counts of a warp's run, then the position of its next id, per expert
  __shared__ int totals[kMoeMaxExperts];
  __shared__ int starts[kMoeMaxExperts];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < sorted_cap; i += blockDim.x) sorted_ids[i] = n;
  for (int e = lane; e < E; e += 32) next[warp][e] = 0;
  const int run = ((n + 1023) >> 10) * 32;  // ids per warp, a multiple of 32
  const int r0 = warp * run, r1 = min(n, r0 + run);
  __syncwarp();
  // lanes with the same expert: the first of them adds their number
  auto step = [&](int i, int& e, int& rank, int& same_count) {
    const long long e64 = (i < r1) ? (long long)__ldcg(ids + i) : -1;
    e = (e64 >= 0 && e64 < E) ? int(e64) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    rank = __popc(same & ((1u << lane) - 1u));
    same_count = __popc(same);
  };
  for (int base = r0; base < r1; base += 32) {
    int e, rank, count;
    step(base + lane, e, rank, count);
    if (e >= 0 && rank == 0) next[warp][e] += count;
    __syncwarp();
  }
  __syncthreads();
  // exclusive scan over the warps, one warp per expert
  for (int e = warp; e < E; e += 32) {
    const int c = next[lane][e];
    int sum = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    next[lane][e] = sum - c;
    if (lane == 31) totals[e] = sum;
  }
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the padded totals over the experts
    int at = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int padded = (e0 + lane < E) ? (totals[e0 + lane] + block_size - 1) / block_size * block_size : 0;
      int sum = padded;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (e0 + lane < E) starts[e0 + lane] = at + sum - padded;
      at += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) *num_tokens_post_pad = at;
  }
  __syncthreads();
  for (int e = warp; e < E; e += 32) {
    const int b0 = starts[e] / block_size, nb = (totals[e] + block_size - 1) / block_size;
    for (int b = lane; b < nb; b += 32) expert_ids[b0 + b] = e;
  }
  for (int base = r0; base < r1; base += 32) {
    const int i = base + lane;
    int e, rank, count;
    step(i, e, rank, count);
    int at = -1;
    if (e >= 0) at = starts[e] + next[warp][e] + rank;
    __syncwarp();
    if (e >= 0 && rank == 0) next[warp][e] += count;
    __syncwarp();
    if (e >= 0) sorted_ids[at] = i;
    if (i < r1 && inverse) inverse[i] = at;
  }
}

// Order-preserving integer of an f32, every NaN above the infinity.
__device__ __forceinline__ uint32_t order_key(float v) {
  if (v != v) return 0xffffffffu;
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// ---------------------------------------------------------------------------------------------
// Routing of an expert MLP and its first step: softmax over at most 32 experts, top-k, the sorted row of every (token, slot)
// pair with the experts' runs padded to whole blocks (the positions moe_align_block_size gives), and the tokens quantised
// to those rows.
//
// Latency-bound. As three launches (top-k, block alignment by one CTA, quantise and scatter) the chain took 24 us ahead of the first GEMM
// at 4096 tokens. A token picks an expert at most once, so the row of a pair is (first row of the expert's run) + (earlier tokens
// that picked it): moe_route_kernel leaves each pair's rank inside a block of tokens and each block's count per expert, and
// the quantising kernel adds up the counts of the at most 64 blocks in every CTA, with its loads of x in flight. Up to 128 tokens
// (a decode step) there is one launch: every CTA of the quantising kernel routes all tokens itself.
// Whole MLP, 8 experts, top-2, us per call from a graph: K = 4096, inter = 7168: 16 tokens 68.2 -> 64.3; K = inter = 2048: 1 token
// 18.3 -> 15.2, 128 tokens 29.8 -> 26.9, 600 tokens 32.7 -> 29.7, 4096 tokens 84.2 -> 80.7.
// ---------------------------------------------------------------------------------------------
constexpr int kRouteMaxExperts = 32;
constexpr int kRouteTokens = 128;  // tokens ranked at a time, one per thread
constexpr int kRouteMaxBlocks = 64;

struct RouteParams {
  const void* logits;
  long long ld;
  int tokens, E, top_k;
  int block_rows;           // rows an expert's run is padded to
  int tokens_per_block;     // a multiple of kRouteTokens
  float* weight;            // [tokens, top_k] in descending order of the logit, the lower expert first among equals
  int* slots;               // [tokens, top_k] expert | rank inside the block of tokens << 8 (more than kRouteTokens tokens)
  int* counts;              // [blocks of tokens][kRouteMaxExperts]
  int* inverse;             // [tokens, top_k] sorted row
  int* expert_ids;          // expert of every block of rows
  int* num_rows;            // padded total
  unsigned int* zero_word;  // cleared for the GEMM that follows: the tile counter of its decode form
};

// Router of one token: its choices in order, as bytes, and as a bit mask. weight may be null. EM: experts held in registers.
template <typename T, int EM>
__device__ __forceinline__ uint32_t route_token(const RouteParams& p, int t, float* __restrict__ weight, uint8_t* choice) {
  const T* row = static_cast<const T*>(p.logits) + (long long)t * p.ld;
  float v[EM];
#pragma unroll
  for (int e = 0; e < EM; ++e) v[e] = e < p.E ? to_f32<T>(row[e]) : -INFINITY;
  float mx = -INFINITY, sum = 0.f;
#pragma unroll
  for (int e = 0; e < EM; ++e)
    if (e < p.E) mx = fmaxf(mx, v[e]);
#pragma unroll
  for (int e = 0; e < EM; ++e)
    if (e < p.E) sum += expf(v[e] - mx);
  uint32_t taken = 0;
  for (int j = 0; j < p.top_k; ++j) {
    uint32_t best_key = 0;
    int best = -1;
    float best_v = 0.f;
#pragma unroll
    for (int e = 0; e < EM; ++e) {
      const uint32_t key = order_key(v[e]);
      if (e < p.E && !((taken >> e) & 1u) && (best < 0 || key > best_key)) { best = e; best_key = key; best_v = v[e]; }
    }
    taken |= 1u << best;
    if (weight) weight[j] = expf(best_v - mx) / sum;
    choice[j] = uint8_t(best);
  }
  return taken;
}

// Who picked what among kRouteTokens tokens, thread t of the first four warps holding token t.
struct RouteTable {
  uint32_t picked[kRouteTokens / 32][kRouteMaxExperts];  // tokens of a warp that picked an expert
  uint8_t choice[kRouteTokens][kRouteMaxExperts];
  __device__ __forceinline__ void enter(uint32_t taken, int E, int warp, int lane) {
    uint32_t mine = 0;
    for (int e = 0; e < E; ++e) {
      const uint32_t b = __ballot_sync(0xffffffffu, (taken >> e) & 1u);
      if (lane == e) mine = b;
    }
    picked[warp][lane] = mine;
  }
  __device__ __forceinline__ int count(int e) const {
    int n = 0;
#pragma unroll
    for (int w = 0; w < kRouteTokens / 32; ++w) n += __popc(picked[w][e]);
    return n;
  }
  __device__ __forceinline__ int rank(int t, int e) const {
    int n = __popc(picked[t >> 5][e] & ((1u << (t & 31)) - 1u));
#pragma unroll
    for (int w = 0; w < kRouteTokens / 32 - 1; ++w) n += w < (t >> 5) ? __popc(picked[w][e]) : 0;
    return n;
  }
};

template <typename T, int EM>
__global__ void __launch_bounds__(kRouteTokens)
moe_route_kernel(const RouteParams p) {
  __shared__ RouteTable table;
  __shared__ int seen[kRouteMaxExperts];  // pairs of each expert in the tokens so far
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < kRouteMaxExperts) seen[tid] = 0;
  const int t0 = blockIdx.x * p.tokens_per_block, t1 = min(t0 + p.tokens_per_block, p.tokens);
  for (int base = t0; base < t1; base += kRouteTokens) {
    const int t = base + tid;
    const uint32_t taken = t < t1 ? route_token<T, EM>(p, t, p.weight + (long long)t * p.top_k, table.choice[tid]) : 0u;
    table.enter(taken, p.E, warp, lane);
    __syncthreads();
    if (t < t1)
      for (int j = 0; j < p.top_k; ++j) {
        const int e = table.choice[tid][j];
        p.slots[(long long)t * p.top_k + j] = e | (seen[e] + table.rank(tid, e)) << 8;
      }
    __syncthreads();
    if (tid < p.E) seen[tid] += table.count(tid);
    __syncthreads();
  }
  if (tid < kRouteMaxExperts) p.counts[blockIdx.x * kRouteMaxExperts + tid] = seen[tid];
}

// Row t of x quantised once and written to the rows of its top_k pairs, scales in the packed layout. Thread layout as
// quantize_scatter_mxfp4_kernel: a warp takes 32 K blocks of a row; the warps of a CTA are in one block of tokens. HERE: this
// kernel routes too (at most kRouteTokens tokens); otherwise it is moe_route_kernel's programmatic dependent.
template <typename InT, typename T, int EM, bool HERE>
__global__ void __launch_bounds__(256)
moe_quantize_kernel(const InT* __restrict__ x, long long ldx, int K, uint8_t* __restrict__ q, uint8_t* __restrict__ scale_packed, int k_atoms,
                    const RouteParams p) {
  __shared__ RouteTable table;
  __shared__ int totals[kRouteMaxExperts], before[kRouteMaxExperts];  // pairs per expert: in all, and in earlier blocks of tokens
  __shared__ int first[kRouteMaxExperts];                             // sorted row of rank 0 in this block of tokens
  if constexpr (HERE) pdl_wait();  // (otherwise moe_route_kernel has released this one: what came before that is complete)
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kblocks = K >> 5;
  const unsigned chunks = unsigned(k_atoms + 7) >> 3;
  const unsigned wid = blockIdx.x * 8u + warp;
  const int r = int(wid / chunks);
  const bool real = r < p.tokens;
  const int kb0 = int(wid - unsigned(r) * chunks) * 32;
  using Quant = WarpQuant<InT>;
  Quant w;
  w.run(real ? x + (long long)r * ldx : static_cast<const InT*>(nullptr), rows_on_32(x, ldx), kb0, kblocks, lane);
  int slot = 0;  // of this row's pair `lane`
  if constexpr (HERE) {
    if (warp < kRouteTokens / 32) {
      const int t = threadIdx.x;
      const uint32_t taken =
          t < p.tokens ? route_token<T, EM>(p, t, blockIdx.x == 0 ? p.weight + t * p.top_k : nullptr, table.choice[t]) : 0u;
      table.enter(taken, p.E, warp, lane);
    }
    __syncthreads();
    if (warp == 0) {
      totals[lane] = lane < p.E ? table.count(lane) : 0;
      before[lane] = 0;
    }
    if (real && lane < p.top_k) {
      const int e = table.choice[r][lane];
      slot = e | table.rank(r, e) << 8;
    }
  } else {
    pdl_wait();
    if (real && lane < p.top_k) slot = __ldcg(p.slots + (long long)r * p.top_k + lane);
    const int blocks = (p.tokens + p.tokens_per_block - 1) / p.tokens_per_block;
    const int block = int(blockIdx.x * 8u / chunks) / p.tokens_per_block;
    for (int e = warp; e < kRouteMaxExperts; e += 8) {
      int sum = 0, part = 0;
      if (e < p.E)
        for (int b = lane; b < blocks; b += 32) {
          const int c = __ldcg(p.counts + b * kRouteMaxExperts + e);
          sum += c;
          part += b < block ? c : 0;
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        part += __shfl_xor_sync(0xffffffffu, part, o);
      }
      if (lane == 0) { totals[e] = sum; before[e] = part; }
    }
    __syncthreads();
  }
  if (warp == 0) {  // exclusive scan of the padded totals over the experts
    __syncwarp();
    const int run_blocks = (totals[lane] + p.block_rows - 1) / p.block_rows;
    int sum = run_blocks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    first[lane] = (sum - run_blocks) * p.block_rows + before[lane];
    if (blockIdx.x == 0) {
      for (int b = sum - run_blocks; b < sum; ++b) p.expert_ids[b] = lane;
      if (lane == 31) *p.num_rows = sum * p.block_rows;
      if (lane == 0) *p.zero_word = 0u;
    }
  }
  __syncthreads();
  if (!real) return;
  for (int j = 0; j < p.top_k; ++j) {
    const int s = __shfl_sync(0xffffffffu, slot, j);
    const int dst = first[s & 255] + (s >> 8);
    w.store_codes(q + (long long)dst * (K / 2), true, kb0, kblocks, lane);
    if (Quant::writes(lane)) {
#pragma unroll
      for (int i = 0; i < Quant::kWords; ++i) {
        const int atom = (kb0 >> 2) + Quant::atom(i, lane);
        if (atom < k_atoms) *packed_scale_word(scale_packed, k_atoms, dst, atom) = w.word[i];
      }
    }
    if (kb0 == 0 && lane == 0) p.inverse[(long long)r * p.top_k + j] = dst;
  }
}

// dst[p, :] = src[sorted_ids[p] / top_k, :] for sorted_ids[p] < n_valid, zero otherwise. Rows are
// row_bytes long; one warp per row. vec: bases, pitches and row_bytes are multiples of 16 bytes.
__global__ void __launch_bounds__(256)
moe_gather_rows_kernel(const uint8_t* __restrict__ src, long long src_pitch, int row_bytes,
                       const int* __restrict__ sorted_ids, int num_rows, int n_valid, int top_k,
                       uint8_t* __restrict__ dst, long long dst_pitch, int vec) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= num_rows) return;
  const int lane = threadIdx.x & 31;
  const int id = sorted_ids[row];
  const bool real = id >= 0 && id < n_valid;
  const uint8_t* s = src + (long long)(real ? id / top_k : 0) * src_pitch;
  uint8_t* d = dst + (long long)row * dst_pitch;
  if (vec) {
    const int nvec = row_bytes >> 4;
    for (int v = lane; v < nvec; v += 32)
      reinterpret_cast<uint4*>(d)[v] = real ? reinterpret_cast<const uint4*>(s)[v] : make_uint4(0u, 0u, 0u, 0u);
  } else {
    for (int v = lane; v < row_bytes; v += 32) d[v] = real ? s[v] : uint8_t(0);
  }
}

// 8 consecutive values from 16-byte aligned memory that an overlapping earlier kernel wrote (through L2).
__device__ __forceinline__ void load8_cg(const float* p, float (&v)[8]) {
  const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8_cg(const __nv_bfloat16* p, float (&v)[8]) { raw8_values(__ldcg(reinterpret_cast<const uint4*>(p)), v); }
__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&v)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                            pack_bf16x2(v[6], v[7]));
}

// y = x1 / (1 + exp(-x1)) * x2 in f32. Four lanes share 32 consecutive columns (8 each), as in the
// quantiser; `out` (same type as the inputs, may be null) gets y rounded once; q / scales (may be
// null; need n % 32 == 0) get y quantised to MXFP4 from the f32 value, not from the rounded one.
// VEC: all three matrices have 16-byte aligned bases and pitches, so 8 values move as one or two accesses.
// Every group of 4 lanes works on kSiluUnroll consecutive blocks of 32 columns and issues all their
// loads before any arithmetic. grid (rows, ceil(nblocks / (64 U))): a CTA covers 64 U blocks of one row.
constexpr int kSiluUnroll = 2;
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
silu_and_mul_kernel(const T* __restrict__ x1, const T* __restrict__ x2, long long ld1, long long ld2, int rows, int n,
                    T* __restrict__ out, long long ldo, uint8_t* __restrict__ q, uint8_t* __restrict__ scale_rm,
                    uint8_t* __restrict__ scale_packed, int k_atoms, const int* __restrict__ row_limit) {
  constexpr int U = kSiluUnroll;
  // rows at or past *row_limit (a device value: the padded row count of a routed batch) are left alone
  if (row_limit) rows = min(rows, __ldg(row_limit));
  const int g0 = blockIdx.y * 64 + (threadIdx.x >> 2);
  const int sub = threadIdx.x & 3;
  const int nblocks = (n + 31) >> 5;
  const int r = blockIdx.x;
  bool active[U], full[U];
  float g[U][8], u[U][8];
#pragma unroll
  for (int i = 0; i < U; ++i) {
    const int kb = g0 * U + i;
    active[i] = r < rows && kb < nblocks;
    const int c0 = kb * 32 + sub * 8;
    full[i] = VEC && c0 + 8 <= n;
#pragma unroll
    for (int j = 0; j < 8; ++j) g[i][j] = u[i][j] = 0.f;
    if (active[i]) {
      const T* p1 = x1 + (long long)r * ld1 + c0;
      const T* p2 = x2 + (long long)r * ld2 + c0;
      if (full[i]) {
        load8(p1, g[i]);
        load8(p2, u[i]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (c0 + j < n) { g[i][j] = to_f32<T>(p1[j]); u[i][j] = to_f32<T>(p2[j]); }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < U; ++i) {
    const int kb = g0 * U + i;
    const int c0 = kb * 32 + sub * 8;
    float y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = silu_mul(g[i][j], u[i][j]);
    if (out && active[i]) {
      T* po = out + (long long)r * ldo + c0;
      if (full[i]) {
        store8(po, y);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (c0 + j < n) po[j] = from_f32<T>(y[j]);
      }
    }
    if (q) mxfp4_encode_group<8>(y, active[i], r, kb, sub, n, nblocks, k_atoms, q, scale_rm, scale_packed);
  }
}

// out[t, c] = sum_j weight[t * top_k + j] * y[row_of[t * top_k + j], c], accumulated in f32 in slot
// order; pairs with row_of < 0 are skipped. One thread per (token, 8 columns); VEC: cols % 8 == 0 and 16-byte aligned
// rows of both matrices, so that a thread's columns move as 16-byte accesses.
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
moe_combine_kernel(const T* __restrict__ y, long long ldy, const int* __restrict__ row_of,
                   const float* __restrict__ weight, int tokens, int top_k, int cols, T* __restrict__ out,
                   long long ldo, int dependent) {
  if (dependent) pdl_launch_dependents();  // (in a chain of the library's own; see quantize_mxfp4_kernel)
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int cvec = (cols + 7) >> 3;
  if (dependent) pdl_wait();
  if (idx >= (long long)tokens * cvec) return;
  const int t = int(idx / cvec);
  const int c0 = int(idx - (long long)t * cvec) * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // two slots at a time: their row numbers, then their rows, are in flight together
  for (int j = 0; j < top_k; j += 2) {
    int row[2];
    float w[2], v[2][8];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      row[u] = (j + u < top_k) ? __ldcg(row_of + (long long)t * top_k + j + u) : -1;
      w[u] = (j + u < top_k) ? __ldcg(weight + (long long)t * top_k + j + u) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (row[u] < 0) continue;
      const T* src = y + (long long)row[u] * ldy + c0;
      if constexpr (VEC) {
        load8_cg(src, v[u]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[u][i] = (c0 + i < cols) ? to_f32<T>(src[i]) : 0.f;
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (row[u] < 0) continue;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += w[u] * v[u][i];
    }
  }
  T* dst = out + (long long)t * ldo + c0;
  if constexpr (VEC) {
    store8(dst, acc);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < cols) dst[i] = from_f32<T>(acc[i]);
  }
}

// out[i] = slots[0][i] + slots[1][i] + ... in slot order (f32), rounded once to the output type: the
// reduction step of the K-sharded GEMM, whose ranks deposit f32 partial tiles in one slot each.
template <typename T>
__global__ void __launch_bounds__(256)
sum_slots_kernel(const float* __restrict__ slots, int num_slots, long long slot_stride, long long count, T* __restrict__ out) {
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i >= count) return;
  if (i + 4 <= count) {
    float4 acc = *reinterpret_cast<const float4*>(slots + i);
    for (int s = 1; s < num_slots; ++s) {
      const float4 v = *reinterpret_cast<const float4*>(slots + s * slot_stride + i);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(out + i) = acc;
    } else {
      *reinterpret_cast<uint2*>(out + i) = make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
    }
  } else {
    for (long long j = i; j < count; ++j) {
      float acc = slots[j];
      for (int s = 1; s < num_slots; ++s) acc += slots[s * slot_stride + j];
      out[j] = from_f32<T>(acc);
    }
  }
}

// c[r, :] (+)= slots[0][r, :] + slots[1][r, :] + ... in slot order (f32), rounded once to the output type:
// the reduction of the tile path's split-K. Slots are dense [M, N] f32 matrices; c has row pitch ldc.
template <typename T>
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ slots, int num_slots, long long slot_stride, int M, int N, T* __restrict__ c,
                     long long ldc, int accumulate) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nvec = (N + 3) >> 2;
  if (idx >= (long long)M * nvec) return;
  const int r = int(idx / nvec), c0 = int(idx - (long long)r * nvec) * 4;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const float* src = slots + (long long)r * N + c0;
  if (c0 + 4 <= N && (N & 3) == 0) {
    for (int s = 0; s < num_slots; ++s) {
      const float4 v = *reinterpret_cast<const float4*>(src + s * slot_stride);
      acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w;
    }
  } else {
    for (int s = 0; s < num_slots; ++s)
      for (int j = 0; j < 4; ++j)
        if (c0 + j < N) acc[j] += src[s * slot_stride + j];
  }
  T* dst = c + (long long)r * ldc + c0;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (c0 + j < N) dst[j] = from_f32<T>(accumulate ? acc[j] + to_f32<T>(dst[j]) : acc[j]);
}

}  // namespace wb
