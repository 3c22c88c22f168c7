// W4A4 prefill MoE (many tokens): a ragged grouped GEMM on tcgen05.mma kind::mxf4nvf4 with TMEM accumulators. It replaces
// the third-party CUTLASS hand-off of the reference (sm120fp4/vllm_backend.py:123-168) with its own kernels and implements
// the reference's own W4A4 arithmetic (sm120fp4/kernels/bench_moe_baseline.py:53-74 with act_quant=True): x and the
// SiLU*mul activations quantised to NVFP4 by the bit-exact quantiser, fp32 accumulation, weighted sum over the top-k.
//
// Pipeline (all on the caller's stream, no host synchronisation):
//   k_plan:             router tables, per-expert row segments padded to 128-row tiles (the tile plan) and the map between
//                       token-expert pairs and operand rows (plan.cuh); for up to 1024 pairs part of the kernel after it
//   k_quantize_scatter: bf16 x -> NVFP4 "tile records" (128 rows x 256 codes in the 128-byte-swizzle shared-memory image
//                       + four 512 B scale tiles, 18 KB contiguous): every token row quantised once, stored to its pairs' rows
//   k_grouped_gemm<1>:  FC1 tiles (128 rows x [64 up | 64 gate] columns), epilogue SiLU*mul + NVFP4 re-quantisation
//                       straight into FC2's tile records (scales written in the 128x4 order)
//   k_grouped_gemm<2>:  FC2 tiles (128 rows x 128 columns), epilogue alpha * routing weight -> bf16 rows per (token, expert)
//   k_combine:          out[token] = sum over its top-k rows, in slot order (deterministic)
// Both GEMM operands are streamed as 18 KB records with one bulk copy each (weights: the records built by
// b200moe_layer_prepack), so no tensor map is needed. All launches are programmatic (each kernel is scheduled while the one
// before it drains and waits for its results with grid_dependency_wait); every kernel waits before it touches what an
// earlier one wrote, except where a comment says why that kernel must already have completed.
#include "grouped_gemm.cuh"
#include "plan.cuh"
#include <string.h>
#include <stdlib.h>
#include <type_traits>

namespace b200 {

// ------------------------------------------------------------------------------------------------ x -> records
// Blocks [0, aside) do what else the records and the GEMM behind this kernel need: block i zeroes the scale bytes of the rows of
// tile i that hold no pair (a zero scale silences whatever codes a row holds, so their codes are never written), marks these rows
// in row_pair and asks the first weight records of GEMM CTA i into L2, which is idle meanwhile.
//
// Planned (both kernels below): there is no plan kernel before this one, every block works the plan out for itself (plan.cuh).
struct GgPlanning { const int* ids; int P, E, Umax; PlanTables T; };
template <bool Planned, int ARows, int Rec>
__device__ __forceinline__ void records_aside(const GgAside& A, const GgPlanning& Q, BlockPlan& B, uint8_t* rec, int* row_pair, int tid, int nthreads) {
  constexpr int kPer = ARows == 64 ? kTerms : 1, kTile = ARows / kPer;
  const int i = blockIdx.x;
  if (Planned) block_plan<kTile>(Q.ids, Q.P, Q.E, Q.Umax, Q.T, i == 0, B);
  const int NT = Planned ? B.NT : __ldcg(A.ntiles);
  if (i < A.gemm_ctas) {
    const GgSplit s(NT, A.NBLK, A.gemm_ctas, i);
    if (s.nseg > 0) {
      const GgSplit::Segment g = s.segment(0);
      const int e = Planned ? block_plan_tile<kTile>(B, g.t).x : __ldcg(A.tile_expert + g.t);
      if (tid < kGgWarm && tid < (g.n1 - g.n0) * A.KB) l2_prefetch(A.wrec + (((long long)e * A.NBLK + g.n0) * A.KB + tid) * kRec, kRec);
    }
  }
  if (i < NT) {
    const int pairs = Planned ? block_plan_tile<kTile>(B, i).y : __ldcg(A.tile_end + i) - __ldcg(A.tile_first + i);
    const int used = min(ARows, pairs * kPer), spare = ARows - used;
    for (int j = tid; j < spare * 4 * A.KB; j += nthreads) {
      const int r = used + j % spare, q = j / spare;   // scale word q & 3 of K box q >> 2
      *reinterpret_cast<uint32_t*>(rec + ((long long)i * A.KB + (q >> 2)) * Rec + (Rec - 2048) + (q & 3) * 512 + (r & 31) * 16 + (r >> 5) * 4) = 0u;
    }
    for (int r = used + tid; r < ARows; r += nthreads) row_pair[(long long)i * ARows + r] = -1;
  }
}

// The rows of a token's pairs into s_row, and this thread's (warp 3: slot tid - 96) row and tile_first. The block synchronises.
template <bool Planned, int TILE>
__device__ __forceinline__ void token_rows(const GgPlanning& Q, BlockPlan& B, const PairTables& T, int* dst_row, int tok, int top_k, int* s_row, int* s_first,
                                           int& my_row, int& my_first) {
  const int tid = threadIdx.x, slot = tid - 96;
  if (Planned) {
    block_plan<TILE>(Q.ids, Q.P, Q.E, Q.Umax, Q.T, false, B);
    for (int j = tid >> 5; j < top_k; j += 4) {
      int first = 0;
      const int row = block_plan_row<TILE>(B, tok * top_k + j, &first);
      if ((tid & 31) == 0) s_row[j] = row, s_first[j] = first;
    }
    __syncthreads();
    if (slot >= 0 && slot < top_k) {
      my_row = s_row[slot], my_first = s_first[slot];
      dst_row[tok * top_k + slot] = my_row;
    }
  } else {
    if (slot >= 0 && slot < top_k) {
      my_row = __ldcg(dst_row + tok * top_k + slot);
      s_row[slot] = my_row;
      if (my_row >= 0) my_first = __ldcg(T.tile_first + my_row / TILE);
    }
    __syncthreads();
  }
}

// One block of 128 threads per token, one thread per 16-value block (a second round for rows of more than 2048 values):
// the token's row is read and quantised ONCE (the reference's block arithmetic, bit-exact), while the plan kernel is still
// running, and its codes and scale bytes are then stored into the record rows of each of its top_k pairs (dst_row, -1 = empty
// slot). rec [ntiles][KB][18432]; blocks beyond H inside the last K box are written as zero codes and zero scales.
template <bool Planned>
__global__ void __launch_bounds__(128) k_quantize_scatter(const __nv_bfloat16* __restrict__ x, int* dst_row, int H, int KB, int top_k, float gs,
                                                          uint8_t* rec, GgAside A, PairTables T, GgPlanning Q) {
  __shared__ typename std::conditional<Planned, BlockPlan, int>::type s_plan;
  BlockPlan& B = reinterpret_cast<BlockPlan&>(s_plan);
  if ((int)blockIdx.x < A.blocks) {
    grid_dependency_wait();
    grid_launch_dependents();
    records_aside<Planned, 128, kRec>(A, Q, B, rec, T.row_pair, threadIdx.x, 128);
    return;
  }
  __shared__ float s_scale[128];   // gs / (E4M3 value) for every scale byte: one division per table entry instead of one per block
  __shared__ int s_row[16], s_first[16];
  fill_scale_table(s_scale, gs, threadIdx.x, blockDim.x);
  const int tok = blockIdx.x - A.blocks;
  __syncthreads();
  if (Planned) grid_dependency_wait();   // x and the ids alike
  const int nblk = KB * 16;
  bool waited = false;
  const int slot = threadIdx.x - 96;   // warp 3: this token's entries of the pair tables
  int my_row = -1, my_first = 0;
#pragma unroll 1
  for (int b = threadIdx.x; b < ((nblk + 127) & ~127); b += 128) {   // whole warps stay in the loop: the shuffles below need them
    uint2 pk = make_uint2(0u, 0u);
    uint32_t sb = 0;
    if (b < nblk && b * 16 < H) {
      float v[16];
      load16(x + (long long)tok * H + b * 16, v);
      sb = quantize_block16_t(v, gs, s_scale, pk);
    }
    // the four scale bytes of one 64-value K step are adjacent in a record: lane 4i gathers them into one 32-bit store
    uint32_t sf4 = sb | (__shfl_down_sync(0xffffffffu, sb, 1) << 8);
    sf4 |= __shfl_down_sync(0xffffffffu, sf4, 2) << 16;
    const int kb = b >> 4, b16 = b & 15;
    if (!waited) {
      waited = true;
      grid_dependency_wait();
      grid_launch_dependents();
      token_rows<Planned, 128>(Q, B, T, dst_row, tok, top_k, s_row, s_first, my_row, my_first);
    }
    if (b >= nblk) continue;
#pragma unroll 4
    for (int j = 0; j < top_k; ++j) {
      const int row = s_row[j];
      if (row < 0) continue;
      uint8_t* dst = rec + ((long long)(row >> 7) * KB + kb) * kRec;
      const int r = row & 127;
      *reinterpret_cast<uint2*>(dst + rec_code_offset(r, b16)) = pk;
      if ((b & 3) == 0) *reinterpret_cast<uint32_t*>(dst + rec_scale_offset(r, b16)) = sf4;
    }
  }
  if (my_row >= 0) put_pair<128, 1>(T, tok * top_k + slot, my_row, my_first);
}

// ------------------------------------------------------------------------------------------------ x -> W4A16 records
// Mid-sized batches (17 tokens up to a few hundred) keep the decode path's W4A16 arithmetic but run as a grouped GEMM over
// per-expert gathered rows: a tile of 64 operand rows holds 16 token-expert pairs x four NVFP4 terms of the pair's token
// row (row 4p + t = term t of pair p), so that an expert's weight records are streamed once for all of its pairs.
//
// One block of 128 threads per token: token amax, then every 16-value block expanded into four NVFP4 terms ONCE and stored
// into the four term rows of each of the token's pairs (dst_row[pair] = tile * 16 + pair row); the first four threads also
// write the rows' 1 / g_t.
// The row's amax is taken while the plan kernel is still running. Blocks [0, aside): see records_aside.
template <bool Planned>
__global__ void __launch_bounds__(128) k_expand_scatter(const __nv_bfloat16* __restrict__ x, int* dst_row, int H, int KB, int top_k, uint8_t* rec,
                                                        float* rowscale, GgAside A, PairTables T, GgPlanning Q) {
  __shared__ typename std::conditional<Planned, BlockPlan, int>::type s_plan;
  BlockPlan& B = reinterpret_cast<BlockPlan&>(s_plan);
  const int tid = threadIdx.x;
  if ((int)blockIdx.x < A.blocks) {
    grid_dependency_wait();
    grid_launch_dependents();
    records_aside<Planned, 64, kMidRec>(A, Q, B, rec, T.row_pair, tid, 128);
    return;
  }
  if (Planned) grid_dependency_wait();   // x and the ids alike
  __shared__ float wm[4];
  __shared__ int s_row[16], s_first[16];
  const int tok = blockIdx.x - A.blocks;
  float m = 0.f;
  for (int i = tid * 8; i < H; i += 128 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(x + (long long)tok * H + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) m = fmaxf(m, fmaxf(fabsf(__uint_as_float(w[q] << 16)), fabsf(__uint_as_float(w[q] & 0xffff0000u))));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) wm[tid >> 5] = m;
  grid_dependency_wait();
  grid_launch_dependents();
  const int slot = tid - 96;   // warp 3: this token's entries of the pair tables
  int my_row = -1, my_first = 0;
  token_rows<Planned, 16>(Q, B, T, dst_row, tok, top_k, s_row, s_first, my_row, my_first);
  m = fmaxf(fmaxf(wm[0], wm[1]), fmaxf(wm[2], wm[3]));
  const float g1 = 2688.0f / fmaxf(m, 1e-30f);
  if (tid < kTerms) {
    float g = g1;
    for (int q = 0; q < tid; ++q) g *= 6.0f;
    for (int j = 0; j < top_k; ++j) {
      const int prow = s_row[j];
      if (prow >= 0) rowscale[(prow >> 4) * 64 + 4 * (prow & 15) + tid] = 1.0f / g;
    }
  }
  const int nblk = KB * 16;
  for (int b = tid; b < nblk; b += 128) {
    auto put = [&](int q, uint2 codes, uint8_t sf) {
      for (int j = 0; j < top_k; ++j) {
        const int prow = s_row[j];
        if (prow < 0) continue;
        uint8_t* dst = rec + ((long long)(prow >> 4) * KB + (b >> 4)) * kMidRec;
        const int r = 4 * (prow & 15) + q;
        *reinterpret_cast<uint2*>(dst + rec_code_offset(r, b & 15)) = codes;
        dst[8192 + ((b & 15) >> 2) * 512 + (r & 31) * 16 + (r >> 5) * 4 + (b & 3)] = sf;
      }
    };
    if (b * 16 < H) {
      float v[16];
      load16(x + (long long)tok * H + b * 16, v);
      expand_block16<true>(v, g1, put);
    } else {
      for (int q = 0; q < kTerms; ++q) put(q, make_uint2(0u, 0u), 0);
    }
  }
  if (my_row >= 0) put_pair<16, kTerms>(T, tok * top_k + slot, my_row, my_first);
}

// ------------------------------------------------------------------------------------------------ combine
__device__ __forceinline__ void add8(float (&acc)[8], const uint4& v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    acc[2 * q] += __uint_as_float(w[q] << 16);
    acc[2 * q + 1] += __uint_as_float(w[q] & 0xffff0000u);
  }
}

// out[tok, :] = sum_j y[dst_row[tok*k + j], :] in slot order, fp32 accumulation, one bf16 rounding (for fp32 rows, the W4A16 path,
// the only one of the layer). A thread sums eight columns; the rows of Batch slots are loaded before the first is added, so
// that the loads of a token overlap (with one row at a time: 88 us at 8192 tokens x 8 rows of 4 KB).
// The rows of a thread's first slots are looked up ahead of the wait: dst_row is complete (the kernels of this call start behind the one that has seen its writer complete).
// That is worth something where a block is there before FC2 has ended, on an SM that FC2's CTA has left: beside one there are no registers for a block.
// Blocks: resident per SM, which says how many registers a thread has. The loads are volatile, or the compiler adds as it loads to save registers: with 32
// of them about four were in flight, and a call of 333 tokens of 2816 x 704 took 71.1 us instead of 68.5, of 512 of 2048 x 768 37.8 instead of 35.2. (Volatile keeps them in their
// order; that the additions stand behind them is what the compiler does where the registers allow it. 32 registers hold the rows of four slots at most.)
template <bool F32, int Batch, int Blocks>
__global__ void __launch_bounds__(256, Blocks) k_combine(const void* yv, const int* dst_row, int M, int top_k, int H, __nv_bfloat16* out) {
  constexpr int kBatch = Batch;
  const unsigned chunks = (unsigned)H / 8, total = (unsigned)M * chunks, step = gridDim.x * 256;   // (2^32 chunks are 64 GB of x, as much of out and more of rows)
  unsigned i = blockIdx.x * 256 + threadIdx.x;
  int tok = (int)(i / chunks), c = (int)(i % chunks);
  int r[kBatch];
  auto look = [&](int j0) {
#pragma unroll
    for (int j = 0; j < kBatch; ++j) r[j] = j0 + j < top_k ? __ldcg(dst_row + tok * top_k + j0 + j) : -1;   // -1: empty slot
  };
  if (i < total) look(0);
  grid_dependency_wait();
  grid_launch_dependents();
#pragma unroll 1
  while (i < total) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int j0 = 0; j0 < top_k; j0 += kBatch) {
      if (j0) look(j0);
      uint4 v[kBatch][F32 ? 2 : 1];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
#pragma unroll
        for (int q = 0; q < (F32 ? 2 : 1); ++q)
        {
          v[j][q] = make_uint4(0u, 0u, 0u, 0u);
          if (r[j] >= 0)
            asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[j][q].x), "=r"(v[j][q].y), "=r"(v[j][q].z), "=r"(v[j][q].w)
                         : "l"(reinterpret_cast<const uint4*>(yv) + ((long long)r[j] * H + c * 8) / (F32 ? 4 : 8) + q));
        }
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (F32) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            acc[4 * q] += __uint_as_float(v[j][F32 ? q : 0].x), acc[4 * q + 1] += __uint_as_float(v[j][F32 ? q : 0].y);
            acc[4 * q + 2] += __uint_as_float(v[j][F32 ? q : 0].z), acc[4 * q + 3] += __uint_as_float(v[j][F32 ? q : 0].w);
          }
        } else {
          add8(acc, v[j][0]);
        }
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
      o[q] = *reinterpret_cast<const uint32_t*>(&h);
    }
    if (!F32) combine_columns(o, threadIdx.x & 31);
    *reinterpret_cast<uint4*>(out + (long long)tok * H + c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    i += step;
    if (i < step) break;   // (past the end of the type)
    tok = (int)(i / chunks), c = (int)(i % chunks);
    if (i < total) look(0);
  }
}

}  // namespace b200

using namespace b200;


struct PrefillLayout {
  long long experts, offsets, pairs, ntiles, tile_expert, tile_tab, row_pair, dst_row, status, xrec, arec, y, total;
  int max_tiles;
};

static inline long long pf_align(long long v) { return (v + 255) / 256 * 256; }

static PrefillLayout prefill_layout(int E, int H, int I, int top_k, int max_tokens) {
  PrefillLayout L;
  const long long P = (long long)max_tokens * top_k;
  const int KB1 = (H + 255) / 256, KB2 = (I + 255) / 256;
  L.max_tiles = (int)(P / 128 + E);   // every expert may end in a partly filled tile
  long long o = 0;
  L.experts = o, o = pf_align(o + 4LL * E);
  L.offsets = o, o = pf_align(o + 4LL * (E + 1));
  L.pairs = o, o = pf_align(o + 4 * P);
  L.ntiles = o, o += 256;
  L.tile_expert = o, o = pf_align(o + 4LL * L.max_tiles);
  L.tile_tab = o, o = pf_align(o + 8LL * L.max_tiles);   // tile_first [max_tiles], then tile_end [max_tiles]
  L.row_pair = o, o = pf_align(o + 4LL * L.max_tiles * 128);
  L.dst_row = o, o = pf_align(o + 4 * P);
  L.status = o, o += 256;
  L.xrec = o, o = pf_align(o + (long long)L.max_tiles * KB1 * kRec);
  L.arec = o, o = pf_align(o + (long long)L.max_tiles * KB2 * kRec);
  L.y = o, o = pf_align(o + (long long)L.max_tiles * 128 * H * 2);
  L.total = o;
  return L;
}

long long b200_prefill_workspace_bytes(int E, int H, int I, int top_k, int max_tokens) {
  return prefill_layout(E, H, I, top_k, max_tokens).total;
}

// Byte offsets of the tables and records inside a prefill workspace, for tools and tests that read them back:
// out[0..11] = experts, offsets, pairs, ntiles, tile_expert, tile_first, tile_end, row_pair, dst_row, x records, activation
// records, weighted rows (columns at B200MOE_WEIGHTED_ROW_COLUMN); out[12] = tile capacity, out[13] = total bytes.
void b200_prefill_workspace_map(int E, int H, int I, int top_k, int max_tokens, long long* out) {
  const PrefillLayout L = prefill_layout(E, H, I, top_k, max_tokens);
  const long long v[14] = {L.experts, L.offsets, L.pairs, L.ntiles, L.tile_expert, L.tile_tab, L.tile_tab + 4LL * L.max_tiles, L.row_pair,
                           L.dst_row, L.xrec, L.arec, L.y, L.max_tiles, L.total};
  for (int i = 0; i < 14; ++i) out[i] = v[i];
}

// One launch of the grouped GEMM (grouped_gemm.cuh): one persistent CTA per SM, programmatically behind the kernel before it so
// that its set-up and the first weight records overlap that kernel's tail.
static int launch_gemm(GroupedParams p, int phase, int sms, cudaStream_t st) {
  static const void* const kernels[5] = {(const void*)k_grouped_gemm<1>, (const void*)k_grouped_gemm<2>, (const void*)k_grouped_gemm<3>,
                                         (const void*)k_grouped_gemm<4>, (const void*)k_grouped_gemm<1, true>};
  const int which = phase == 1 && gg_ieee_silu(p.KB) ? 4 : phase - 1;
  const void* fn = kernels[which];
  static thread_local unsigned configured[5] = {0, 0, 0, 0, 0};   // bit d: device d has the attribute
  int dev = 0;
  B200_CUDA_TRY(cudaGetDevice(&dev));
  if (dev > 31 || !((configured[which] >> dev) & 1u)) {
    B200_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGgSmem));
    if (dev <= 31) configured[which] |= 1u << dev;
  }
  void* args[] = {(void*)&p};
  return launch_kernel(fn, sms, kGgThreads, kGgSmem, true, args, st);
}

// Whether both projections' tile records together are more than L2 holds (126 MB). A call may touch a few experts only, which fit: that shows
// nowhere by more than 1 % (eight experts again and again, us with and without marks: 128 experts of 2048 x 768 27.5 and 27.8 at 64 tokens,
// 39.2 and 39.1 at 512; of 4096 x 1536 41.2 and 41.2, 81.3 and 81.0), and 40 experts of 128 gain (200 skewed tokens 54.1 and 58.8).
static bool gg_stream_weights(int E, int H, int I) {
  return (long long)E * ((long long)(I / 64) * ((H + 255) / 256) + (long long)(H / 128) * ((I + 255) / 256)) * kRec > (126LL << 20);
}

// w1t / w2t: the weight tile records of b200moe_layer_prepack. gs_x / gs_a: global scales of the two activation quantisations.
// Launches: plan -> token-major quantiser -> FC1 GEMM -> FC2 GEMM -> combine.
int b200_prefill_forward(int E, int H, int I, int top_k, const uint8_t* w1t, const uint8_t* w2t, const float* alpha1, const float* alpha2,
                         const void* x, const int* ids, const float* wts, int M, void* out, void* ws, long long ws_bytes, int ws_tokens,
                         float gs_x, float gs_a, int sms, cudaStream_t st) {
  const PrefillLayout L = prefill_layout(E, H, I, top_k, ws_tokens);
  if (ws_bytes < L.total || M > ws_tokens) return B200MOE_ERR_WORKSPACE;
  uint8_t* w = (uint8_t*)ws;
  const int P = M * top_k;
  const int Umax = E < P ? E : P;
  const int KB1 = (H + 255) / 256, KB2 = (I + 255) / 256, KT1 = (H / 16 + 3) / 4, KT2 = (I / 16 + 3) / 4;
  int* experts = (int*)(w + L.experts);
  int* offsets = (int*)(w + L.offsets);
  int* pairs = (int*)(w + L.pairs);
  int* ntiles = (int*)(w + L.ntiles);
  int* tile_expert = (int*)(w + L.tile_expert);
  int* tile_first = (int*)(w + L.tile_tab);
  int* tile_end = tile_first + L.max_tiles;
  int* row_pair = (int*)(w + L.row_pair);
  int* dst_row = (int*)(w + L.dst_row);
  int* status = (int*)(w + L.status);
  if (Umax > 256) return B200MOE_ERR_LIMIT;
  const int max_tiles = P / 128 + Umax;   // tiles this batch can need (<= the workspace's capacity)
  const PlanTables tab = {experts, offsets, ntiles, tile_expert, tile_first, tile_end, dst_row};
  const PairTables ptab = {tile_first, pairs, row_pair};
  const bool planned = P <= kBlockPlanPairs;   // no plan kernel (plan.cuh)
  int rc = planned ? B200MOE_OK : launch_plan<128>(ids, P, E, Umax, tab, st);
  if (rc != B200MOE_OK) return rc;
  {
    const GgAside aside = {ntiles, tile_expert, tile_first, tile_end, w1t, I / 64, KB1, sms, max_tiles > sms ? max_tiles : sms};
    const GgPlanning planning = {ids, P, E, Umax, tab};
    const __nv_bfloat16* xp = (const __nv_bfloat16*)x;
    uint8_t* rec = w + L.xrec;
    void* args[] = {(void*)&xp, (void*)&dst_row, (void*)&H, (void*)&KB1, (void*)&top_k, (void*)&gs_x, (void*)&rec, (void*)&aside, (void*)&ptab, (void*)&planning};
    rc = launch_kernel(planned ? (const void*)k_quantize_scatter<true> : (const void*)k_quantize_scatter<false>, aside.blocks + M, 128, 0, true, args, st);
    if (rc != B200MOE_OK) return rc;
  }
  GroupedParams p;
  memset(&p, 0, sizeof(p));
  p.ntiles = ntiles, p.tile_expert = tile_expert, p.tile_first = tile_first, p.tile_end = tile_end, p.row_pair = row_pair, p.status = status, p.H = H, p.E = E;
  p.stream = gg_stream_weights(E, H, I);
  // FC1
  p.arec = w + L.xrec, p.wrec = w1t, p.alpha = alpha1, p.gs_in = gs_x, p.gs_out = gs_a, p.orec = w + L.arec;
  p.NBLK = I / 64, p.KB = KB1, p.KT = KT1, p.KB2 = KB2;
  p.wait_tables = planned;
  rc = launch_gemm(p, 1, sms, st);
  if (rc != B200MOE_OK) return rc;
  // FC2
  p.arec = w + L.arec, p.wrec = w2t, p.alpha = alpha2, p.gs_in = gs_a, p.gs_out = 0.f, p.orec = nullptr;
  p.wts = wts, p.y = (__nv_bfloat16*)(w + L.y);
  p.NBLK = H / 128, p.KB = KB2, p.KT = KT2;
  p.wait_tables = 0;
  rc = launch_gemm(p, 2, sms, st);
  if (rc != B200MOE_OK) return rc;
  const uint8_t* y = w + L.y;
  void* args[] = {(void*)&y, (void*)&dst_row, (void*)&M, (void*)&top_k, (void*)&H, (void*)&out};
  // Rows that L2 does not hold come at HBM's rate, and more threads are worth more than more loads of each: 8192 tokens of 2048 x 768 (268 MB) 304.5 us, 306 with
  // half the threads and twice the loads; 4000 (131 MB) 169 either way, 2500 142.5 and 141. (Four slots or fewer: 7500 tokens of 60 experts of 2304 x 1408 280.5, with lookups for eight 290.7.)
  const bool deep = (long long)P * H * 2 <= (126LL << 20);
  return launch_kernel(deep ? (const void*)k_combine<false, 8, 4> : (const void*)k_combine<false, 4, 8>, sms * 8, 256, 0, true, args, st);
}

int b200_prefill_status_offset(int E, int H, int I, int top_k, int max_tokens, long long* off) {
  *off = prefill_layout(E, H, I, top_k, max_tokens).status;
  return 0;
}

// ---------------------------------------------------------------------------------------------------------------------
// W4A16 layer call for mid-sized batches (the decode path's arithmetic, one pass over the touched experts' weights).
struct MidLayout {
  long long experts, offsets, pairs, ntiles, tile_expert, tile_tab, row_pair, rowscale, dst_row, status, xrec, arec, y, total;
  int max_tiles;
};

static MidLayout mid_layout(int E, int H, int I, int top_k, int max_tokens) {
  MidLayout L;
  const long long P = (long long)max_tokens * top_k;
  const int KB1 = (H + 255) / 256, KB2 = (I + 255) / 256;
  L.max_tiles = (int)(P / 16 + E);
  long long o = 0;
  L.experts = o, o = pf_align(o + 4LL * E);
  L.offsets = o, o = pf_align(o + 4LL * (E + 1));
  L.pairs = o, o = pf_align(o + 4 * P);
  L.ntiles = o, o += 256;
  L.tile_expert = o, o = pf_align(o + 4LL * L.max_tiles);
  L.tile_tab = o, o = pf_align(o + 8LL * L.max_tiles);
  L.row_pair = o, o = pf_align(o + 4LL * L.max_tiles * 64);
  L.rowscale = o, o = pf_align(o + 4LL * L.max_tiles * 64);
  L.dst_row = o, o = pf_align(o + 4 * P);
  L.status = o, o += 256;
  L.xrec = o, o = pf_align(o + (long long)L.max_tiles * KB1 * kMidRec);
  L.arec = o, o = pf_align(o + (long long)L.max_tiles * KB2 * kMidRec);
  L.y = o, o = pf_align(o + (long long)L.max_tiles * 16 * H * 4);
  L.total = o;
  return L;
}

long long b200_mid_workspace_bytes(int E, int H, int I, int top_k, int max_tokens) { return mid_layout(E, H, I, top_k, max_tokens).total; }

int b200_mid_status_offset(int E, int H, int I, int top_k, int max_tokens, long long* off) {
  *off = mid_layout(E, H, I, top_k, max_tokens).status;
  return 0;
}

int b200_mid_forward(int E, int H, int I, int top_k, const uint8_t* w1t, const uint8_t* w2t, const float* alpha1, const float* alpha2,
                     const void* x, const int* ids, const float* wts, int M, void* out, void* ws, long long ws_bytes, int ws_tokens,
                     float act_g1, int sms, cudaStream_t st) {
  const MidLayout L = mid_layout(E, H, I, top_k, ws_tokens);
  if (ws_bytes < L.total || M > ws_tokens) return B200MOE_ERR_WORKSPACE;
  uint8_t* w = (uint8_t*)ws;
  const int P = M * top_k;
  const int Umax = E < P ? E : P;
  const int KB1 = (H + 255) / 256, KB2 = (I + 255) / 256, KT1 = (H / 16 + 3) / 4, KT2 = (I / 16 + 3) / 4;
  if (Umax > 256 || KB1 > 12) return B200MOE_ERR_LIMIT;
  int* experts = (int*)(w + L.experts);
  int* offsets = (int*)(w + L.offsets);
  int* pairs = (int*)(w + L.pairs);
  int* ntiles = (int*)(w + L.ntiles);
  int* tile_expert = (int*)(w + L.tile_expert);
  int* tile_first = (int*)(w + L.tile_tab);
  int* row_pair = (int*)(w + L.row_pair);
  float* rowscale = (float*)(w + L.rowscale);
  int* dst_row = (int*)(w + L.dst_row);
  const int max_tiles = P / 16 + Umax;
  int* tile_end = tile_first + max_tiles;
  const PlanTables tab = {experts, offsets, ntiles, tile_expert, tile_first, tile_end, dst_row};
  const PairTables ptab = {tile_first, pairs, row_pair};
  // No plan kernel (plan.cuh). Wider layers keep it: without it the smallest batches lose up to 2 % and the others gain up to 2 %. us with (without) at
  // 33, 64, 96 and 128 tokens of 2816 x 704: 82.3 (82.5), 89.9 (89.8), 94.5 (92.8), 99.9 (98.3); 33, 64 and 128 of 64 experts of 2304 x 768:
  // 53.4 (54.6), 54.9 (55.0), 65.8 (65.0). At 2048 x 768 64 and 128 tokens 73.1 (72.2), 76.3 (74.2).
  const bool planned = P <= kBlockPlanPairs && KB1 <= 8;
  int rc = planned ? B200MOE_OK : launch_plan<16>(ids, P, E, Umax, tab, st);
  if (rc != B200MOE_OK) return rc;
  {
    const GgAside aside = {ntiles, tile_expert, tile_first, tile_end, w1t, I / 64, KB1, sms, max_tiles > sms ? max_tiles : sms};
    const GgPlanning planning = {ids, P, E, Umax, tab};
    const __nv_bfloat16* xp = (const __nv_bfloat16*)x;
    uint8_t* rec = w + L.xrec;
    void* args[] = {(void*)&xp, (void*)&dst_row, (void*)&H, (void*)&KB1, (void*)&top_k, (void*)&rec, (void*)&rowscale, (void*)&aside, (void*)&ptab, (void*)&planning};
    rc = launch_kernel(planned ? (const void*)k_expand_scatter<true> : (const void*)k_expand_scatter<false>, aside.blocks + M, 128, 0, true, args, st);
    if (rc != B200MOE_OK) return rc;
  }
  GroupedParams p;
  memset(&p, 0, sizeof(p));
  p.ntiles = ntiles, p.tile_expert = tile_expert, p.tile_first = tile_first, p.tile_end = tile_end, p.row_pair = row_pair, p.status = (int*)(w + L.status), p.H = H, p.E = E;
  p.stream = gg_stream_weights(E, H, I);
  p.rowscale = rowscale, p.act_g1 = act_g1;
  // FC1
  p.arec = w + L.xrec, p.wrec = w1t, p.alpha = alpha1, p.orec = w + L.arec;
  p.NBLK = I / 64, p.KB = KB1, p.KT = KT1, p.KB2 = KB2;
  p.wait_tables = planned;
  rc = launch_gemm(p, 3, sms, st);
  if (rc != B200MOE_OK) return rc;
  // FC2
  p.arec = w + L.arec, p.wrec = w2t, p.alpha = alpha2, p.orec = nullptr;
  p.wts = wts, p.yf = (float*)(w + L.y);
  p.NBLK = H / 128, p.KB = KB2, p.KT = KT2;
  p.wait_tables = 0;
  rc = launch_gemm(p, 4, sms, st);
  if (rc != B200MOE_OK) return rc;
  const uint8_t* y = w + L.y;
  void* args[] = {(void*)&y, (void*)&dst_row, (void*)&M, (void*)&top_k, (void*)&H, (void*)&out};
  // Eight slots at a time where the blocks that have work are more than one an SM and all of them fit (two an SM have the registers). Fewer leave an SM's loads short of what
  // it can have in flight either way, and looking four rows up is done sooner; of more blocks, four an SM run side by side in the form for four. us with four and eight slots at a time, by
  // blocks an SM: 2048 wide 0.99 77.5 / 78.0, 1.08 81.7 / 79.0, 1.73 96.0 / 92.6, 1.97 93.8 / 90.9, 2.4 108.6 / 109.1, 4.7 166.1 / 168.8; 2816 wide 0.66 94.9 / 95.4, 0.98 96.7 / 97.2, 1.05 100.1 / 97.3, 1.97 112.4 / 109.2, 2.4 120.8 / 121.2;
  // 3072 wide 0.98 79.9 / 80.2, 1.06 81.1 / 79.2, 1.97 117.4 / 116.1, 2.6 119.8 / 120.6. Four slots or fewer are one round of the form for four.
  const int blocks = (int)(((long long)M * (H / 8) + 255) / 256);
  const bool eight = top_k > 4 && blocks > sms && blocks <= 2 * sms;
  return launch_kernel(eight ? (const void*)k_combine<true, 8, 2> : (const void*)k_combine<true, 4, 4>, sms * 4, 256, 0, true, args, st);
}

// out[i] = g[i] / den[i], den[i] = 1 + exp(-g[i]), as FC1's epilogue divides in wide layers (gg_quotient), for tests.
static __global__ void __launch_bounds__(256) k_quotient(const float* gate, float* den, float* out, int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const float g = gate[i], d = 1.0f + __expf(-g);
  den[i] = d;
  out[i] = g < kGgQuotLo || g > kGgQuotHi ? __fdiv_rn(g, d) : gg_quotient(g, d);
}

extern "C" int b200moe_quotient_probe(const float* gate, float* den, float* out, int n, void* stream) {
  if (!gate || !den || !out || n < 0) return B200MOE_ERR_ARG;
  if (n == 0) return B200MOE_OK;
  k_quotient<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(gate, den, out, n);
  B200_LAUNCH_CHECK();
  return B200MOE_OK;
}
