// The decode-regime MoE layer on the 5th-generation tensor cores: weights are consumed as FP4 straight from shared
// memory by tcgen05.mma kind::mxf4nvf4 with their E4M3 block scales in TMEM - no CUDA-core dequantisation at all - so the
// SMs only move bytes and the kernel is bound by HBM. It keeps the contract of the reference's decode kernels
// (sm120fp4/kernels/{fc1_w4a16,fc1_mma,fc2_w4a16,fc2_mma_pf}.py: W4A16, fp32 accumulation, alpha in fp32, SiLU*mul,
// weighted combine, bit-identical from call to call).
//
// W4A16 on an FP4 x FP4 instruction: a 16-bit activation vector is written as a short sum of NVFP4 vectors,
//     x = q1*s1/g1 + q2*s2/g2 + q3*s3/g3 + q4*s4/g4 + r,   g_t = g1 * 6^(t-1),   |r| <= blockmax(x) * 6^-4 (about 2^-10.3),
// each term the NVFP4 quantisation (E2M1 codes, E4M3 scale per 16 values) of the residual left by the terms before it.
// The terms of a token are adjacent columns of the B operand; the epilogue adds the four accumulator columns with their
// 1/g_t. Four terms carry more mantissa than bf16 for the values that decide a dot product and keep the layer's error
// against the fp32 oracle below the bf16 output rounding.
//
// Structure: one CTA per SM = one worker. Warps 0-3: epilogue (tcgen05.ld of a double-buffered TMEM accumulator, term sums,
// SiLU*mul, re-expansion of the activations for FC2, fixed-order reduction of partials). Warp 4: MMA issuer - converged, one
// elected lane; it waits for a record, copies its scale tiles into TMEM (tcgen05.cp), issues the four K=64 MMAs and commits
// the ring slot: operations of one lane execute in order, so a record passes from the producer to the tensor core
// in one hand-off. Warps 5-6: producers (one bulk copy per 18 KB record into the ring, FC2 records prefetched across the gates).
// Warp 7: arrivals at the gates, warp 8: routing tables. What bounds it: at 16 tokens the weight stream (an SM's share of HBM is a record per ~740 cycles, the
// issuer needs ~300 for one), at 1 token a chain of latencies: launch, routing tables, first record, eight
// records of a unit, gate, three records of FC2, reduction. (With four warps that moved the scales through registers, and
// an issuer whose lanes left their waits one by one, a record took about 1,000 cycles of issue alone.)
#include "common.cuh"
#include "tcgen05.cuh"
#include "decode_params.h"
#include "expand.cuh"
#include "nvfp4_math.cuh"
#include <string.h>
#include <type_traits>
#include <stdlib.h>

namespace b200 {

constexpr int kTcMmaWarp = 4, kTcProd0 = 5, kTcUnitsWarp = 7, kTcTablesWarp = 8;
constexpr int kTcProducers = 2;    // producer warps: one thread's wait + issue round is ~430 cycles
constexpr int kTcThreads = 9 * 32;
constexpr int kTcStage = 18432;   // 16 KB codes + 2 KB scale tiles
constexpr int kTcMaxE = 256, kTcMaxP = 256;
constexpr int kTcPause = 100;
constexpr int kTcPace = 700, kTcAhead = 24;   // see ask_ahead

struct TcTables {
  int ids[kTcMaxP];
  float wts[kTcMaxP];
  int cnt[kTcMaxE], base[kTcMaxE], uidx[kTcMaxE], experts[kTcMaxE];
  unsigned xmax[16];           // amax bits of every token
  float xg1[16];
  float colscale[64];          // 1 / g_t of every B column of the FC1 operand (token-major, four terms per token)
  float a1[kTcMaxE], a2n[kTcMaxE];   // per touched expert (unit index): alpha1, alpha2 relative to the layer's largest alpha2
  int U;
  volatile int units_done;       // FC1 units whose activations the epilogue has written
  unsigned long long gate0[2];   // arrival counts of the two FC1 gates before this launch (a multiple of the worker count)
  volatile int abort_flag;
  uint32_t tmem_base;
  uint64_t full[12], empty[12];   // stage landed / stage consumed
  uint64_t acc_full[2], acc_empty[2];
  uint64_t xb_full, fc1_done;   // x operand landed / this worker's FC1 MMAs are complete
};

#ifdef B200_TIMERS
#define TC_T0(var) long long var = clock64()
#define TC_ADD(acc, var) acc += clock64() - var
#define TC_TRACE(j, k) do { if (P.debug && v == 5 && (threadIdx.x & 31) == 0 && (j) < 128) P.debug[148 * 16 + (j) * 8 + (k)] = clock64() - tm_begin; } while (0)
#else
#define TC_TRACE(j, k)
#define TC_T0(var)
#define TC_ADD(acc, var)
#endif

__device__ __forceinline__ float tc_silu_mul(float gate, float up) { return __fdividef(gate, 1.0f + __expf(-gate)) * up; }

// The larger of two non-negative bf16 values in one word, as the bits of a float (which order like the values). A NaN, which is what the
// packed maximum leaves where all values were NaN, counts as zero: it would pass for the largest value of the row.
__device__ __forceinline__ unsigned pair_max_bits(uint32_t w) {
  return __float_as_uint(fmaxf(fmaxf(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)), 0.f));
}

// ------------------------------------------------------------------------------------------------ x -> B operand
// One block of 256 threads per token slot (N/4 slots), a thread per 16-value block: token amax, then the block expanded into four
// NVFP4 terms. The block is small enough (registers, shared memory) to be resident next to a block of the layer kernel.
// What bounds it is latency: it starts when the kernel before it has completed and the layer kernel waits for it. So it goes
// through its code once before that, on zeros and without storing: a launch finds none of its instructions in the SM's cache, and
// fetching them took 2 of the 3 us it needed.
// xb: the FC1 B operand exactly as the kernel wants it in shared memory, so that ONE bulk copy brings it in:
//   [KB1 boxes][N rows (token*4 + term)][128 B] in the 128-byte-swizzle image (16-byte chunk c of row n sits at chunk
//   c ^ (n & 7)), followed by KT1 scale tiles of 512 B (128x4 order, rows >= N zero). colscale f32 [N] = 1/g_t.
// kHost: x, ids and weights are in page-locked host memory. This kernel reads x across the host link itself and its block 0 brings the
// routing inputs into device memory (ids_d, wts_d) before it lets the layer kernel start, which reads them at its entry: one
// kernel instead of three copies that wait for one another and for the link (13 us a call).
template <bool kHost>
__global__ void __launch_bounds__(256, 4) k_expand_x(const __nv_bfloat16* x, int M, int H, int N, int KB1, uint8_t* xb, float* colscale,
                                                     const int* ids_h, const float* wts_h, int npairs, int* ids_d, float* wts_d) {
  const int tok = blockIdx.x, tid = threadIdx.x, b = tid;
  if (!kHost) grid_launch_dependents();   // the layer kernel may start its prologue and weight prefetch now; it waits before reading xb
  uint8_t* xsf = xb + (long long)KB1 * N * 128;
  __shared__ unsigned wm[8];
  const bool live = tok < M && b * 16 < H;
  const int kb = b >> 4, chunk = (b & 15) >> 1, half = b & 1;   // 8 code bytes = half a 16-byte chunk
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    uint4 u = make_uint4(0u, 0u, 0u, 0u), v = u;
    if (pass == 1) {
      grid_dependency_wait();     // this kernel is itself launched programmatically: x (and the workspace it writes) belong to
                                  // whatever ran before it in the stream until that has completed
      if (kHost && tok != 0) grid_launch_dependents();
      if (live) {
        const uint4* src = reinterpret_cast<const uint4*>(x + (long long)tok * H + b * 16);
        u = kHost ? __ldcv(src) : src[0];
        v = kHost ? __ldcv(src + 1) : src[1];
      }
      if (kHost && tok == 0) {   // (x is in flight)
        if (tid < npairs) {
          __stcg(ids_d + tid, __ldcv(ids_h + tid));
          __stcg(wts_d + tid, __ldcv(wts_h + tid));
        }
        __threadfence();
        __syncthreads();
        grid_launch_dependents();
      }
    }
    const uint32_t w[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    __nv_bfloat162 m2 = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
    for (int i = 1; i < 8; ++i) m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
    const uint32_t bits = *reinterpret_cast<const uint32_t*>(&m2);
    const unsigned wmax = __reduce_max_sync(0xffffffffu, pair_max_bits(bits));
    if ((tid & 31) == 0) wm[tid >> 5] = wmax;
    __syncthreads();
    unsigned mb = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) mb = max(mb, wm[i]);
    const float g1 = 2688.0f / fmaxf(__uint_as_float(mb), 1e-30f);
    if (tid < kTerms) {
      float g = g1;
      for (int t = 0; t < tid; ++t) g *= 6.0f;
      if (pass == 1) colscale[tok * kTerms + tid] = tok < M ? 1.0f / g : 0.f;
    }
    float r[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) { r[2 * i] = __uint_as_float(w[i] << 16); r[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    // (a block beyond the batch or the row is all zeros, and so are its codes and scales)
    expand_block16<true>(r, g1, [&](int t, uint2 codes, uint8_t sf) {
      if (pass == 0 || b >= KB1 * 16) return;
      const int n = tok * kTerms + t;
      *reinterpret_cast<uint2*>(xb + ((long long)kb * N + n) * 128 + ((chunk ^ (n & 7)) << 4) + half * 8) = codes;
      if ((b >> 2) < (H / 16 + 3) / 4) xsf[(long long)(b >> 2) * 512 + (n & 31) * 16 + (n >> 5) * 4 + (b & 3)] = sf;
    });
    __syncthreads();   // wm is free again
  }
}

// ------------------------------------------------------------------------------------------------ weight tiles
// Kernel-native weight layout, built once per layer: every (expert, block, K box) tile is ONE contiguous 18 KB record =
// the shared-memory image of its 128 rows x 128 B of codes (128-byte swizzle) followed by its four 512 B scale tiles, so
// a single bulk copy per tile streams it at full HBM rate (one thread issues only ~2.5 M TMA operations per second,
// whatever their size; 2-D boxes from the checkpoint layout need 3-4 operations per tile).
//   FC1 record (e, cb, kb): rows 0..63 = up rows 64cb.., rows 64..127 = gate rows I+64cb..; scale rows likewise.
//   FC2 record (e, nb, kb): rows = output rows 128nb...
__global__ void __launch_bounds__(256) k_pack_tiles(const uint8_t* __restrict__ q, const uint8_t* __restrict__ sf, uint8_t* __restrict__ out,
                                                    int E, int rows_per_expert, int row_bytes, int blocks, int KB, int KT, int fc1, int I,
                                                    long long sf_expert_stride) {
  const long long records = (long long)E * blocks * KB;
  const long long total = records * (1024 + 128);   // 1024 code chunks of 16 B + 128 scale rows x 16 B
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long rec = i / 1152;
    const int w = (int)(i % 1152);
    const int kb = (int)(rec % KB), blk = (int)((rec / KB) % blocks), e = (int)(rec / ((long long)KB * blocks));
    uint8_t* dst = out + rec * kTcStage;
    if (w < 1024) {
      const int r = w >> 3, c = w & 7;
      const int src_row = fc1 ? (r < 64 ? 64 * blk + r : I + 64 * blk + (r - 64)) : 128 * blk + r;
      const int byte = kb * 128 + c * 16;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (byte < row_bytes) v = *reinterpret_cast<const uint4*>(q + ((long long)e * rows_per_expert + src_row) * row_bytes + byte);
      *reinterpret_cast<uint4*>(dst + r * 128 + ((c ^ (r & 7)) << 4)) = v;
    } else {
      const int r = w - 1024;   // scale row of the record: four K tiles x 4 bytes
      const int src_row = fc1 ? (r < 64 ? 64 * blk + r : I + 64 * blk + (r - 64)) : 128 * blk + r;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kt = 4 * kb + j;
        uint32_t v = 0;
        if (kt < KT)
          v = *reinterpret_cast<const uint32_t*>(sf + e * sf_expert_stride + ((long long)(src_row >> 7) * KT + kt) * 512 + (src_row & 31) * 16 +
                                                 ((src_row & 127) >> 5) * 4);
        *reinterpret_cast<uint32_t*>(dst + 16384 + j * 512 + (r & 31) * 16 + (r >> 5) * 4) = v;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ x -> B operand, inside the layer kernel
// Small operands (P.self: up to 256 blocks of 16 values, e.g. two tokens of 2048) every worker expands by itself, with its 128
// epilogue threads, straight into shared memory: a launch less, and nothing has to travel (one token of 2048 values: 2.7 us from
// the completion of the kernel before to the operand, against 3.5 to 4.3 with the kernel above; a layer 12.2 us against 13.5).
// Beyond that the kernel's 16 blocks are ahead: loads wait behind the weight stream here and the work per thread grows. With four blocks
// a thread a layer of 352 blocks takes 17.4 us against 16.9 with the kernel, 384 blocks 19.2 against 17.8, 512 21.6 against 20.5, and the
// longer code costs the calls of up to 256 blocks 0.3 to 0.5 us; 704 blocks, with six a thread, 27.3 against 26.0.
__device__ __forceinline__ void zero_scales(uint8_t* xsf, int KT1, int et) {   // rows that hold no token keep zero scales
  for (int i = et; i < KT1 * 32; i += 128) reinterpret_cast<uint4*>(xsf)[i] = make_uint4(0u, 0u, 0u, 0u);
}

template <int N>
__device__ __forceinline__ void expand_x_here(const DecodeTcParams& P, uint8_t* region, float* colscale, unsigned* amax, float* g1s, int et) {
  constexpr int kTok = N / kTerms, kMost = 2;   // blocks per thread
  const int nb = P.H >> 4, lane = et & 31, total = P.M * nb;
  uint8_t* xsf = region + P.KB1 * (N * 128);
  // this thread's blocks: et, et + 128, ...; all of x is loaded at once and stays in registers (a load takes 1 to 2 us here, while the
  // weight stream fills the memory system's queues)
  uint4 raw[kMost][2];
#pragma unroll
  for (int j = 0; j < kMost; ++j) {
    raw[j][0] = raw[j][1] = make_uint4(0u, 0u, 0u, 0u);
    if (et + 128 * j < total) {   // x is [M, H] without gaps: block i of the batch starts at value 16 i
      const uint4* src = reinterpret_cast<const uint4*>(P.x + (long long)(et + 128 * j) * 16);
      raw[j][0] = src[0], raw[j][1] = src[1];
    }
  }
  int tok0 = 0, b0 = et;
  while (b0 >= nb) b0 -= nb, ++tok0;
  {
    int tok = tok0, b = b0;
#pragma unroll
    for (int j = 0; j < kMost; ++j) {
      if (128 * j >= total) break;
      const uint32_t w[8] = {raw[j][0].x, raw[j][0].y, raw[j][0].z, raw[j][0].w, raw[j][1].x, raw[j][1].y, raw[j][1].z, raw[j][1].w};
      __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
      for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
      const uint32_t bits = *reinterpret_cast<const uint32_t*>(&m);
      const unsigned mine = pair_max_bits(bits);
      const int first = __shfl_sync(0xffffffffu, tok, 0), last = __shfl_sync(0xffffffffu, tok, 31);
      for (int t = first; t <= last && t < P.M; ++t) {             // the tokens this warp's 32 blocks belong to
        const unsigned wm = __reduce_max_sync(0xffffffffu, tok == t ? mine : 0u);
        if (lane == 0) atomicMax(amax + t, wm);
      }
      b += 128;
      while (b >= nb) b -= nb, ++tok;
    }
  }
  named_bar_sync(1, 128);
  if (et < kTok) g1s[et] = 2688.0f / fmaxf(__uint_as_float(amax[et]), 1e-30f);
  named_bar_sync(1, 128);
  if (et < N) {
    float g = g1s[et >> 2];
    for (int q = 0; q < (et & 3); ++q) g *= 6.0f;
    colscale[et] = (et >> 2) < P.M ? 1.0f / g : 0.f;
  }
  int tok = tok0, b = b0;
  auto expand = [&](auto two) {
    constexpr int K = decltype(two)::value;
    int tk[K], bb[K];
    float r[K][16], g[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      tk[k] = tok, bb[k] = b, g[k] = g1s[tok];
      const uint32_t w[8] = {raw[k][0].x, raw[k][0].y, raw[k][0].z, raw[k][0].w, raw[k][1].x, raw[k][1].y, raw[k][1].z, raw[k][1].w};
#pragma unroll
      for (int i = 0; i < 8; ++i) r[k][2 * i] = __uint_as_float(w[i] << 16), r[k][2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      b += 128;
      while (b >= nb) b -= nb, ++tok;
    }
    expand_blocks16<true, K>(r, g, [&](int k, int t, uint2 codes, uint8_t sf) {
      const int n = tk[k] * kTerms + t, c = bb[k];   // 8 code bytes = half a 16-byte chunk
      *reinterpret_cast<uint2*>(region + (c >> 4) * (N * 128) + n * 128 + ((((c & 15) >> 1) ^ (n & 7)) << 4) + (c & 1) * 8) = codes;
      xsf[(c >> 2) * 512 + (n & 31) * 16 + (n >> 5) * 4 + (c & 3)] = sf;
    });
  };
  const int mine = (total - et + 127) >> 7;
  if (mine == 2) expand(std::integral_constant<int, 2>());
  else if (mine == 1) expand(std::integral_constant<int, 1>());
}

// ------------------------------------------------------------------------------------------------ the layer kernel
template <int NB>   // N = 16 * NB columns of the B operand (tokens x four terms): NB = 1 (M<=4), 2 (M<=8), 4 (M<=16)
__global__ void __launch_bounds__(kTcThreads, 1) k_moe_decode_tc(const __grid_constant__ DecodeTcParams P) {
  constexpr int N = 16 * NB;
  const bool self = NB <= 2 && P.self != 0;   // the worker expands x itself
  constexpr int kSlab = N * 128 + 2048;     // FC2 activation slab of one tile: N rows x 128 B codes + 4 scale tiles
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int NS = P.NS;
  uint8_t* ring = smem;                                   // NS x [16 KB codes | 2 KB scales]
  uint8_t* region = smem + NS * kTcStage;                 // FC1: resident x operand [KB1][N x 128 B] then its scale tiles;
                                                          // FC2: NS activation slabs
  TcTables& T = *reinterpret_cast<TcTables*>(region + P.region_bytes);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (a value from lane 0 is known to be warp-uniform)
#ifdef B200_TIMERS
  if (tid == 0 && P.debug) { unsigned long long g; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g)); P.debug[blockIdx.x * 16 + 13] = (long long)g; }
#endif
  const int npairs = P.M * P.top_k;
  const int V = gridDim.x;
  const int KB1 = P.KB1, KB2 = P.KB2, CB1 = P.CB1, NB2 = P.NB2;

  // ---------------------------------------------------------------- prologue
  // Every global load of the prologue is issued at entry, each by a thread of its own, so that their latencies overlap
  // one another and the barrier / TMEM set-up: pair p is thread p's (npairs <= 256 < threads).
  int my_e = -1;
  float my_w = 0.f;
  if (tid < npairs) { my_e = __ldcg(P.ids + tid); my_w = __ldcg(P.wts + tid); }
  // the per-expert scales of ALL experts come in with the ids (no load depends on another): thread e holds expert e's
  float ex_a1 = 0.f, ex_a2 = 0.f;
  if (tid < P.E) { ex_a1 = P.alpha1[tid]; ex_a2 = P.alpha2[tid]; }
  const float a2inv = P.alpha2_ref[1];
  // The gate counters are only ever incremented, by exactly V arrivals per launch and gate (so their quotient numbers the
  // launches: what the flagged words of the partial sums carry), and a launch starts after the
  // gates of the launch before it on this workspace have opened: whatever this thread reads, rounding down to a multiple of
  // V gives the count before this launch (other workers of this launch may have arrived already).
  unsigned long long my_gate = 0;
  if (tid == kTcProd0 * 32) my_gate = ld_acquire_gpu_u64(P.gates);
  if (tid == (kTcProd0 + 1) * 32) my_gate = ld_acquire_gpu_u64(P.gates + 1);
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(&T.full[s], 1); mbar_init(&T.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&T.acc_full[b], 1); mbar_init(&T.acc_empty[b], 4); }
    mbar_init(&T.xb_full, 1);
    T.abort_flag = 0;
    T.units_done = 0;
    fence_mbar_init();
  }
  if (warp == kTcMmaWarp) {              // the MMA warp owns the TMEM allocation (all 512 columns: one CTA per SM)
    tmem_alloc(&T.tmem_base, 512);
    tmem_relinquish();
  }
  for (int i = tid; i < kTcMaxE; i += kTcThreads) T.cnt[i] = 0;
  if (tid < 16) T.xmax[tid] = 0u;
  if (tid < npairs) {   // a negative id marks an empty slot (expert-parallel shards mask the experts they do not own)
    if (my_e >= P.E) { *P.status = 4; my_e = -1; }
    if (my_e < 0) my_e = -1;
  }
  __syncthreads();
  if (tid < npairs) {
    T.ids[tid] = my_e;
    T.wts[tid] = my_w;
    if (my_e >= 0) atomicAdd(&T.cnt[my_e], 1);
  }
  __syncthreads();
  if (warp == 0) {
    int c[8], f[8], sc = 0, sf = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) { c[i] = T.cnt[lane * 8 + i]; f[i] = c[i] > 0; sc += c[i]; sf += f[i]; }
    int ic = sc, iff = sf;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, ic, o), b = __shfl_up_sync(0xffffffffu, iff, o);
      if (lane >= o) { ic += a; iff += b; }
    }
    int rc = ic - sc, rf = iff - sf;
#pragma unroll
    for (int i = 0; i < 8; ++i) { rc += c[i]; rf += f[i]; T.base[lane * 8 + i] = rc; T.uidx[lane * 8 + i] = rf; }
    if (lane == 31) T.U = iff;
  }
  __syncthreads();
  const int U = __shfl_sync(0xffffffffu, T.U, 0);
  if (tid < P.E && T.cnt[tid] > 0) {   // thread e: expert e is touched -> its slot in the tables of touched experts
    const int u = T.uidx[tid] - 1;
    T.experts[u] = tid;
    T.a1[u] = ex_a1;
    T.a2n[u] = ex_a2 * a2inv;
  }
  // One worker leaves the x operand it expanded in the workspace, for tools and tests that read it back: the last one, which has the
  // least FC1 work (at one token none: it then expands x for this alone). Its fc1_done is complete when the copy has read the
  // operand, too. (On the first worker the copy's 32 KB held up the release of its unit, and with it everybody, by 3 us.)
  const bool x_out = self && blockIdx.x == V - 1 && U > 0;
  if (tid == 0) { mbar_init(&T.fc1_done, (blockIdx.x < U * CB1 ? 1 : 0) + (x_out ? 1 : 0) > 1 ? 2 : 1); fence_mbar_init(); }
  if (tid == kTcProd0 * 32) T.gate0[0] = my_gate - my_gate % (unsigned long long)V;
  if (tid == (kTcProd0 + 1) * 32) T.gate0[1] = my_gate - my_gate % (unsigned long long)V;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // ---------------------------------------------------------------- work split (closed form, the same on every worker)
  // FC1: units q = (touched expert u, 64-column block cb), u-major; worker v takes q = v, v + V, ...: whole units (no
  // cross-CTA reduction), and all workers move through the experts in the same order, so the experts below uA (group A,
  // seven eighths of them) are finished grid-wide seven eighths of the way through FC1. Gate A opens when every worker
  // has finished its units of group A, gate B when all of FC1 is done; a worker's FC2 items of group A keep it busy
  // while gate B and the last slabs are still on their way.
  // FC2: the workers are split into NB2 groups, one per 128-row output block; inside a group, worker r takes the items
  // i = (u, kb) = r, r + W, ... in ascending order, accumulates them in one TMEM accumulator, and the group's partials
  // travel as flagged words and are added in worker order by its first workers. A worker's first items belong to group A: they run while the tail of
  // FC1, gate B and the fetch of the remaining activation slabs are still in flight elsewhere.
  const int v = blockIdx.x;
  const int Q1 = U * CB1;
  const int nu1 = v < Q1 ? (Q1 - v + V - 1) / V : 0;
  const int n1 = nu1 * KB1;
  // With at most two rounds of FC1 units (Q1 <= 2V) gate A would open hardly before gate B, so it is left out (no
  // arrivals, nobody waits) and all of FC2 waits for gate B.
  const bool use_gate_a = Q1 > 2 * V;
  const int uA = use_gate_a ? (7 * U) / 8 : 0, qA = uA * CB1;
  const int nuA = v < qA ? (qA - v + V - 1) / V : 0;   // this worker's units of group A (its first ones)
  const int I2 = U * KB2;
  const int Wb = V / NB2, Wx = V % NB2;                // groups 0..Wx-1 have Wb + 1 workers
  int nb2, r2, W2, vlo2;
  if (v < Wx * (Wb + 1)) { nb2 = v / (Wb + 1); r2 = v - nb2 * (Wb + 1); W2 = Wb + 1; vlo2 = nb2 * (Wb + 1); }
  else { const int vv = v - Wx * (Wb + 1); nb2 = Wx + vv / Wb; r2 = vv % Wb; W2 = Wb; vlo2 = Wx * (Wb + 1) + (nb2 - Wx) * Wb; }
  const int n2 = r2 < I2 ? (I2 - r2 + W2 - 1) / W2 : 0;
  const int live2 = W2 < I2 ? W2 : I2;                 // workers of the group that hold a partial: ranks 0..live2-1
  const int dU2 = W2 / KB2, dK2 = W2 % KB2;            // item step W2 as (experts, K boxes)
#ifdef B200_TIMERS
  long long tm_a = 0, tm_b = 0, tm_c = 0, tm_d = 0;
  const long long tm_begin = clock64();
  if (tid == 0 && P.debug) { unsigned long long g; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g)); P.debug[blockIdx.x * 16 + 15] = (long long)g;
    unsigned sm; asm volatile("mov.u32 %0, %%smid;" : "=r"(sm)); P.debug[blockIdx.x * 16 + 11] = sm; }
#endif
  const unsigned call = (unsigned)(T.gate0[1] / (unsigned long long)V) + 1u;   // number of this launch on the workspace, from 1
  const uint32_t tmem = __shfl_sync(0xffffffffu, T.tmem_base, 0);
  // accumulators 2 x 64 | weight scales, 4 x 16 in rotation | scales of the resident x operand, 16 per K box (<= 16 boxes) | of FC2's slabs, 4 x 16
  const uint32_t tm_acc = tmem, tm_sfa = tmem + 128, tm_sfx = tmem + 192, tm_sfs = tmem + 448;
  uint8_t* xb_sf = region + KB1 * (N * 128);   // scale tiles of the resident x operand (same bulk copy)

  if (warp == kTcProd0 || warp == kTcProd0 + 1) {
    // ============================================================== TMA producers (one thread each)
    // Both producers walk the worker's whole tile sequence with incremental indices (no divisions in the loop) and
    // issue the tiles whose position is theirs (position mod kTcProducers).
    if (lane == 0) {
      const int pw = warp - kTcProd0;
      const uint64_t pol = policy_evict_first();
      // (The resident B operand of FC1 is fetched by an epilogue thread: it has to wait for the expansion kernel, and a
      // producer that waited with it would leave half of the ring empty while the weights could already be streaming.)
      bool passed[2] = {!use_gate_a, false};
      int pend_slot[16], pend_idx[16], pend_g[16] = {0}, npend = 0, pend_head = 0;   // ring of 16: at most NS (<= 12) entries wait at a time
      int slot_g[12];                                                          // gate of the FC2 tile in each ring slot
      auto load_slab = [&](int slot, int idx) {   // activation slab (u, kb) of FC2: N x 128 B codes image + 4 scale tiles
        bulk_load(region + slot * kSlab, P.aslab + (long long)idx * kSlab, kSlab, &T.full[slot]);
      };
      // An activation slab may land only when (a) the gate of its expert group is open and (b) this worker's own FC1 MMAs
      // are complete: the slabs share their shared memory with the resident x operand, and their scale columns in TMEM
      // with the x operand's. Weight tiles of FC2 are prefetched regardless; only the slab loads wait.
      bool local_ok = n1 == 0 && !x_out;
      auto flush = [&]() {   // issue the parked slab loads whose conditions hold now
        while (pend_head < npend && local_ok && passed[pend_g[pend_head & 15]]) { load_slab(pend_slot[pend_head & 15], pend_idx[pend_head & 15]); ++pend_head; }
      };
      // While this worker can issue nothing - the x operand comes from another kernel and is not there yet, or activations are
      // awaited, and the ring is full - its next records are asked into L2, one per kTcPace cycles, about the rate at which HBM
      // delivers them: HBM would be idle meanwhile. (Not while the worker expands x itself: that waits for loads of its own,
      // which the stream delays. 16 tokens: 48 -> 46 us a layer with it; 4 tokens, asking during the expansion: 29 -> 31.)
      int pf_next = 0;          // position of the next record to ask for
      long long pf_last = 0;
      auto record_at = [&](int j) {   // the weight record of position j of this worker's sequence
        if (j < n1) {
          const int t = j / KB1, q = v + t * V, u = q / CB1;
          return P.w1t + (((long long)T.experts[u] * CB1 + (q - u * CB1)) * KB1 + (j - t * KB1)) * kTcStage;
        }
        const int i = r2 + (j - n1) * W2, u = i / KB2;
        return P.w2t + (((long long)T.experts[u] * NB2 + nb2) * KB2 + (i - u * KB2)) * kTcStage;
      };
      auto ask_ahead = [&](int pos) {   // pos: the position this producer will issue next
        const long long now = clock64();
        if (now - pf_last < kTcProducers * kTcPace) return;
        if (pf_next < pos) pf_next = pos;
        if (pf_next >= n1 + n2 || pf_next > pos + kTcAhead) return;
        l2_prefetch(record_at(pf_next), kTcStage);
        pf_next += kTcProducers;
        pf_last = now;
      };
      auto open_gate = [&](int g, int pos) {   // blocking: wait for (b) and for gate g and every gate before it; issue what waited for them
        if (!local_ok) {
          if (!mbar_wait(&T.fc1_done, 0, &T.abort_flag)) *P.status = 9;
          local_ok = true;
        }
        for (int gg = 0; gg <= g; ++gg) {
          if (passed[gg]) continue;
          bool ok = false;
          for (uint32_t it = 0; it < (1u << 24); ++it) {
            if (ld_acquire_gpu_u64(P.gates + gg) - T.gate0[gg] >= (unsigned long long)V) { ok = true; break; }
            if (T.abort_flag) break;
            ask_ahead(pos);
            __nanosleep(kTcPause);   // 296 threads that spin on one line hold up the arrivals they wait for
          }
          if (!ok) { T.abort_flag = 1; *P.status = 3; }
          passed[gg] = true;
          fence_proxy_async();   // the slabs were written through the generic proxy and are read by bulk copies
        }
        flush();
      };
      auto peek_gate = [&](int g) {   // one look, no waiting: gates usually opened long before the tile that needs them is issued
        if (!local_ok && mbar_test_wait(&T.fc1_done, 0)) local_ok = true;
        for (int gg = 0; gg <= g && !passed[gg]; ++gg)
          if (ld_acquire_gpu_u64(P.gates + gg) - T.gate0[gg] >= (unsigned long long)V) { passed[gg] = true; fence_proxy_async(); }
          else break;
        flush();
      };
      int slot = 0, use = 0, mine = pw == 0 ? 0 : kTcProducers - pw;   // `mine` counts down to this producer's next tile
      bool x_there = n1 == 0;
      auto acquire = [&](int gate, int pos) {   // the ring slot of the current position, free of its previous occupant
        if (use >= 1) {
          if (!x_there) {
            for (uint32_t it = 0; it < (1u << 22) && !self && !mbar_test_wait(&T.xb_full, 0) && !T.abort_flag; ++it) ask_ahead(pos);
            x_there = true;
          }
          if (gate >= 0) open_gate(gate, pos);   // that occupant may be an FC2 tile still waiting for its activations
          if (!mbar_wait(&T.empty[slot], (use - 1) & 1, &T.abort_flag)) *P.status = 2;
        }
      };
      auto advance = [&]() {
        if (++slot == NS) { slot = 0; ++use; }
        mine = mine == 0 ? kTcProducers - 1 : mine - 1;
      };
      // ---- FC1 tiles: units v, v + V, ... x KB1 boxes; the KB1 records of a unit are contiguous
      for (int t = 0, j = 0; t < nu1; ++t) {
        const int q = v + t * V, u = q / CB1, cb = q - u * CB1;
        const uint8_t* src = P.w1t + ((long long)T.experts[u] * CB1 + cb) * KB1 * kTcStage;
        for (int kb = 0; kb < KB1; ++kb, ++j) {
          if (mine == 0) {
            acquire(-1, j);
            TC_TRACE(j, 0);
            mbar_expect_tx(&T.full[slot], kTcStage);
            bulk_load_hint(ring + slot * kTcStage, src + (long long)kb * kTcStage, kTcStage, &T.full[slot], pol);
          }
          advance();
        }
      }
      // ---- FC2 tiles: items (u, kb) = r2, r2 + W2, ... of output block nb2; weights (expert of u, nb2, kb), slab (u, kb)
      {
        int u = r2 / KB2, kb = r2 % KB2;
        for (int j = 0; j < n2; ++j) {
          const int g = u < uA ? 0 : 1;
          const int prev_g = j >= NS ? slot_g[slot] : -1;   // gate of the FC2 tile that holds this slot now, if any
          slot_g[slot] = g;
          if (mine == 0) {
            acquire(prev_g, n1 + j);
            TC_TRACE(n1 + j, 0);
            mbar_expect_tx(&T.full[slot], kTcStage + kSlab);
            bulk_load_hint(ring + slot * kTcStage, P.w2t + (((long long)T.experts[u] * NB2 + nb2) * KB2 + kb) * kTcStage, kTcStage, &T.full[slot], pol);
            peek_gate(g);
            if (local_ok && passed[g]) load_slab(slot, u * KB2 + kb);
            else { pend_slot[npend & 15] = slot; pend_idx[npend & 15] = u * KB2 + kb; pend_g[npend & 15] = g; ++npend; }
          }
          kb += dK2, u += dU2;
          if (kb >= KB2) { kb -= KB2; ++u; }
          advance();
        }
      }
      if (pend_head < npend) open_gate(1, n1 + n2);
      if (pw == 0) {
        // The kernel after this one in the stream, if it was launched programmatically (the activation expansion of the
        // next layer call is), may be scheduled once every worker has seen gate B open: its blocks start as SMs free up
        // and wait for this grid's completion before they touch any data. Not earlier: a next call on the same workspace
        // reads the gate words at its entry, and they are final only when the last gate of this launch has opened.
        open_gate(1, n1 + n2);
        grid_launch_dependents();
      }
#ifdef B200_TIMERS
      if (P.debug && pw == 0) P.debug[v * 16 + 9] = clock64() - tm_begin;
#endif
    }
    __syncwarp();
  } else if (warp == kTcUnitsWarp) {
    // ============================================================== arrivals at the gates of FC1
    // Everything this worker wrote for the experts of the gate's group is visible to the bulk loads of every worker that sees the
    // gate open (the producers are the only waiters, and they fence the proxies). A warp of its own does it, so that nobody in
    // the epilogue waits for the stores to be acknowledged (1 to 2 us while the weight stream runs).
    if (lane == 0) {
      auto arrive = [&](int g, int units) {   // when that many units are done
        for (uint32_t it = 0; T.units_done < units && !T.abort_flag; ++it)
          if (it > 64) __nanosleep(20);
        __threadfence_block();
        red_add_release_gpu_u64(P.gates + g, 1ull);   // nothing to wait for: the gate is open when V have arrived
      };
      if (use_gate_a) arrive(0, nuA);
      arrive(1, nu1);
    }
    __syncwarp();
  } else if (warp == kTcTablesWarp) {
    // ============================================================== x operand copies, routing tables
    if (x_out) {
      if (!mbar_wait_warp(smem_u32(&T.xb_full), 0, &T.abort_flag)) *P.status = 6;
      if (lane == 0) {
        bulk_store(P.xb, region, KB1 * (N * 128) + P.KT1 * 512);
        mbar_arrive(&T.fc1_done);   // the store has read the region
      }
      __syncwarp();
    }
    // The routing tables in the router's padded form, for callers that ask for them: written by this warp of the
    // last worker (the one with the least FC1 work), off every critical path.
    if (blockIdx.x == V - 1 && P.experts_out) {
      grid_dependency_wait();   // the tables of the previous call on this workspace may still be read by its tail
      const int t4 = lane;
      for (int e = t4; e < P.E; e += 32)
        if (T.cnt[e] > 0) { P.experts_out[T.uidx[e] - 1] = e; P.offsets_out[T.uidx[e] - 1] = T.base[e] - T.cnt[e]; }
      for (int u = U + t4; u < P.Umax; u += 32) { P.experts_out[u] = -1; P.offsets_out[u + 1] = T.base[kTcMaxE - 1]; }
      if (t4 == 0) P.offsets_out[U] = T.base[kTcMaxE - 1];
      for (int p = t4; p < npairs; p += 32) {
        const int e = T.ids[p];
        if (e < 0) continue;
        int r = 0;
        for (int q = 0; q < p; ++q) r += T.ids[q] == e;
        P.pairs_out[T.base[e] - T.cnt[e] + r] = p;
      }
    }
  } else if (warp == kTcMmaWarp) {
    // ============================================================== MMA issuer: the whole warp stays converged
    const uint32_t el = elect_one();
    const uint32_t idesc = idesc_mxf4nvf4(128, N);
    const uint32_t r16 = kDescLoSw128 + (smem_u32(ring) >> 4), g16 = kDescLoSw128 + (smem_u32(region) >> 4);   // descriptor low words
    const uint32_t xsf16 = smem_u32(xb_sf) >> 4;
    const uint32_t full_u = smem_u32(T.full), empty_u = smem_u32(T.empty), accf_u = smem_u32(T.acc_full), acce_u = smem_u32(T.acc_empty);
    const int nkt_last1 = P.KT1 - 4 * (KB1 - 1), nkt_last2 = P.KT2 - 4 * (KB2 - 1);
    int si = 0, piece = 0;
    uint32_t ph = 0, rot = 0;
    auto take = [&]() {   // the record in ring slot si has landed
      if (!mbar_wait_warp(full_u + 8 * si, ph, &T.abort_flag)) *P.status = 1;
      tc_fence_after();
    };
    auto copy_scales = [&](uint32_t dst, uint32_t src16) {   // four 512-byte tiles -> 16 TMEM columns
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) tmem_cp_sf_lo(dst + 4 * jj, src16 + 32 * jj, el);
    };
    auto issue = [&](uint32_t acc, uint32_t b_lo, uint32_t sfb, int nkt, bool fresh) {   // scales and MMAs of the record in slot si
      const uint32_t a_lo = r16 + si * (kTcStage >> 4), sfa = tm_sfa + 16 * rot;
      copy_scales(sfa, a_lo - kDescLoSw128 + 1024);
      if (nkt == 4) {
        umma_mxf4nvf4_lo(acc, a_lo, b_lo, idesc, sfa, sfb, fresh ? 0u : 1u, el);
#pragma unroll
        for (int jj = 1; jj < 4; ++jj) umma_mxf4nvf4_lo(acc, a_lo + 2 * jj, b_lo + 2 * jj, idesc, sfa + 4 * jj, sfb + 4 * jj, 1u, el);
      } else {
        for (int jj = 0; jj < nkt; ++jj) umma_mxf4nvf4_lo(acc, a_lo + 2 * jj, b_lo + 2 * jj, idesc, sfa + 4 * jj, sfb + 4 * jj, fresh && jj == 0 ? 0u : 1u, el);
      }
      umma_commit_u32(empty_u + 8 * si, el);
      rot = (rot + 1) & 3u;
      if (++si == NS) { si = 0; ph ^= 1u; }
    };
    auto open_piece = [&]() {   // first record of a piece: the epilogue must have drained this accumulator buffer
      if (piece >= 2 && !mbar_wait_warp(acce_u + 8 * (piece & 1), (uint32_t)((piece >> 1) - 1) & 1u, &T.abort_flag)) *P.status = 5;
      return tm_acc + 64 * (piece & 1);
    };
    auto close_piece = [&]() {
      umma_commit_u32(accf_u + 8 * (piece & 1), el);
      ++piece;
    };
    if (n1 > 0 && !mbar_wait_warp(smem_u32(&T.xb_full), 0, &T.abort_flag)) *P.status = 6;
    for (int t = 0; t < nu1; ++t) {   // units: K boxes 0..KB1-1 into one accumulator
      const uint32_t acc = open_piece();
      for (int kb = 0; kb < KB1; ++kb) {
        take();
        // the scales of the resident x operand: once per K box (a short last box copies what follows its tiles; no MMA reads it)
        if (t == 0) copy_scales(tm_sfx + 16 * kb, xsf16 + 128 * kb);
        issue(acc, g16 + kb * ((N * 128) >> 4), tm_sfx + 16 * kb, kb == KB1 - 1 ? nkt_last1 : 4, kb == 0);
      }
      close_piece();
    }
    if (n1 > 0) umma_commit_p(&T.fc1_done, el);   // the x operand's shared memory may be reused from here on
    if (n2 > 0) {   // one piece: all of this worker's items of output block nb2 go into one accumulator
      const uint32_t acc = open_piece();
      int kb = r2 % KB2;
      for (int j = 0; j < n2; ++j) {
        take();
        const uint32_t b_lo = g16 + si * (kSlab >> 4), sfb = tm_sfs + 16 * rot;
        copy_scales(sfb, b_lo - kDescLoSw128 + ((N * 128) >> 4));
        issue(acc, b_lo, sfb, kb == KB2 - 1 ? nkt_last2 : 4, j == 0);
        kb += dK2;
        if (kb >= KB2) kb -= KB2;
      }
      close_piece();
    }
#ifdef B200_TIMERS
    if (P.debug && lane == 0) { P.debug[v * 16 + 6] = clock64() - tm_begin; P.debug[v * 16 + 12] = n1 + n2; }
#endif
  } else {
    // ============================================================== epilogue: 4 warps, thread = accumulator row
    const int et = tid;                            // 0..127
    const int quad = warp;                     // TMEM lane quadrant this warp may read
    const int row = quad * 32 + lane;              // accumulator row (MMA M index)
    __shared__ float s_up[N / 4][68], s_gate[N / 4][68];   // one unit's FC1 sums: [token][intermediate column]
    __shared__ float s_w[16];
    __shared__ unsigned s_mask;
    __shared__ int s_tok[16];                      // the routed tokens
    if (self && (n1 > 0 || x_out)) zero_scales(region + KB1 * (N * 128), P.KT1, et);
    grid_dependency_wait();   // everything before this kernel in the stream is complete and visible from here on
    if (self) {
      if (n1 > 0 || x_out) {
        if constexpr (NB <= 2) expand_x_here<N>(P, region, T.colscale, T.xmax, T.xg1, et);
        fence_proxy_async();
        named_bar_sync(1, 128);
        if (et == 0) mbar_arrive(&T.xb_full);
        if (x_out && et < N) P.xscale[et] = T.colscale[et];
      }
    } else if (et == 0 && n1 > 0) {
      // the resident B operand of FC1 (x expanded into NVFP4 terms by the kernel launched just before this one) and its
      // scale tiles: one bulk copy
      mbar_expect_tx(&T.xb_full, KB1 * (N * 128) + P.KT1 * 512);
      bulk_load(region, P.xb, KB1 * (N * 128) + P.KT1 * 512, &T.xb_full);
    }
    if (!self && et < N) T.colscale[et] = __ldcg(P.xscale + et);
    // The routing inputs were read at entry, before the wait above, so that the weight stream could start early. If they
    // were still being written then (a producer kernel that lets its successors start before it has written them), the
    // copies used here are stale: say so instead of returning a wrong result silently.
    for (int p = et; p < npairs; p += 128) {
      int e2 = (int)ld_acquire_gpu(reinterpret_cast<const unsigned*>(P.ids) + p);
      if (e2 < 0 || e2 >= P.E) e2 = -1;
      const unsigned w2 = ld_acquire_gpu(reinterpret_cast<const unsigned*>(P.wts) + p);
      if (e2 != T.ids[p] || w2 != __float_as_uint(T.wts[p])) P.status[2] = 1;
    }
    named_bar_sync(1, 128);
    int ab = 0;
    uint32_t aph[2] = {0, 0};
    auto load_terms = [&](float (&val)[16], const float* cs, bool per_column) {   // sum the four term columns of every token
      TC_T0(t0);
      if (!mbar_wait_warp(smem_u32(&T.acc_full[ab]), aph[ab], &T.abort_flag)) *P.status = 7;
      TC_ADD(tm_a, t0);
#ifdef B200_TIMERS
      if (tm_d == 0) tm_d = clock64() - tm_begin;   // first accumulator ready
#endif
      tc_fence_after();
      uint32_t r[NB][16];   // all columns in flight before the one wait
#pragma unroll
      for (int c = 0; c < NB; ++c) tmem_ld_32x32b_x16(tm_acc + 64 * ab + ((uint32_t)(quad * 32) << 16) + 16 * c, r[c]);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < NB; ++c) {
#pragma unroll
        for (int tk = 0; tk < 4; ++tk) {
          const int o = per_column ? 16 * c + 4 * tk : 0;
          val[4 * c + tk] = __uint_as_float(r[c][4 * tk]) * cs[o] + __uint_as_float(r[c][4 * tk + 1]) * cs[o + 1] +
                            __uint_as_float(r[c][4 * tk + 2]) * cs[o + 2] + __uint_as_float(r[c][4 * tk + 3]) * cs[o + 3];
        }
      }
#pragma unroll
      for (int i = N / 4; i < 16; ++i) val[i] = 0.f;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&T.acc_empty[ab]);
      aph[ab] ^= 1u;
      ab ^= 1;
    };
    // ---- FC1 pieces
    {
      for (int t = 0; t < nu1; ++t) {
        const int q = v + t * V, u = q / CB1, cb = q - u * CB1;   // a whole unit: K boxes 0..KB1-1 of (expert u, block cb)
        const int e = T.experts[u];
        // s_w[tk]: routing weight of token tk on this expert folded with alpha2 (relative to the layer's largest), 0 when the
        // token is not routed here - only routed tokens cost any arithmetic below (bit tk of s_mask).
        if (warp == 0) {
          float wsum = 0.f;
          if (lane < P.M)
            for (int sidx = 0; sidx < P.top_k; ++sidx)
              if (T.ids[lane * P.top_k + sidx] == e) wsum += T.wts[lane * P.top_k + sidx];
          wsum *= T.a2n[u];
          const unsigned mask = __ballot_sync(0xffffffffu, wsum != 0.f);
          if (lane < 16) s_w[lane] = wsum;
          if (wsum != 0.f) s_tok[__popc(mask & ((1u << lane) - 1u))] = lane;
          if (lane == 0) s_mask = mask;
        }
        float val[16];
        load_terms(val, T.colscale, true);
        TC_T0(tfix);
        {
          // rows 0..63 hold the up columns 64cb.., rows 64..127 the gate columns: exchange through shared memory
          const float alpha = T.a1[u];
          float* mine = row < 64 ? &s_up[0][row] : &s_gate[0][row - 64];
#pragma unroll
          for (int tk = 0; tk < N / 4; ++tk) mine[tk * 68] = val[tk] * alpha;
          named_bar_sync(1, 128);
          const unsigned mask = s_mask;
          const int cnt = __popc(mask);
          uint8_t* slab = P.aslab + ((long long)u * KB2 + (cb >> 2)) * kSlab;   // slab of K box cb/4
          uint8_t* sfp = slab + N * 128 + (cb & 3) * 512;
          // a token that is not routed here only gets zero scale bytes (a zero scale silences whatever codes the row holds)
          if (et < N && !((mask >> (et >> 2)) & 1u)) *reinterpret_cast<uint32_t*>(sfp + (et & 31) * 16 + (et >> 5) * 4) = 0u;
          // SiLU*mul and re-expansion, four lanes per (routed token, 16-column block): four NVFP4 terms of the FC2 operand. (With a
          // thread per block, in two passes through shared memory, a unit's epilogue took 2.4 us; several of them stand between
          // FC1's last MMA and its gate.)
#pragma unroll 1
          for (int i0 = warp * 8; i0 < 4 * cnt; i0 += 32) {
            const int i = i0 + (lane >> 2), blk = i & 3;
            const bool live = i < 4 * cnt;
            const int tk = live ? s_tok[i >> 2] : 0;
            const int col = blk * 16 + 4 * (lane & 3);
            const float4 up = *reinterpret_cast<const float4*>(&s_up[tk][col]), gt = *reinterpret_cast<const float4*>(&s_gate[tk][col]);
            const float wf = s_w[tk];
            float r[4] = {tc_silu_mul(gt.x, up.x) * wf, tc_silu_mul(gt.y, up.y) * wf, tc_silu_mul(gt.z, up.z) * wf, tc_silu_mul(gt.w, up.w) * wf};
            const int chunk = 2 * (cb & 3) + (blk >> 1);                        // 16-byte chunk of the row's 128 bytes
            const bool clipped = expand_quad(r, P.act_g1, [&](int t, uint16_t codes, uint8_t sf) {
              const int n = tk * kTerms + t;
              if (!live) return;
              *reinterpret_cast<uint16_t*>(slab + n * 128 + ((chunk ^ (n & 7)) << 4) + (blk & 1) * 8 + 2 * (lane & 3)) = codes;
              if ((lane & 3) == 0) sfp[(n & 31) * 16 + (n >> 5) * 4 + blk] = sf;
            });
            if (clipped && live) P.status[1] = 1;   // beyond the range of the fixed activation scale
          }
          named_bar_sync(1, 128);
          if (et == 0) { __threadfence_block(); T.units_done = t + 1; }
        }
        TC_ADD(tm_b, tfix);
      }
#ifdef B200_TIMERS
      tm_c = clock64() - tm_begin;
#endif
    }
    // ---- FC2: this worker's items of output block nb2, summed over experts and K boxes inside the tensor core
    if (n2 > 0) {
      float cs[kTerms];   // 1 / g_t of the activation terms, times the alpha2 the operand was normalised by
      {
        float g = P.act_g1;
        const float a2ref = P.alpha2_ref[0];
#pragma unroll
        for (int t = 0; t < kTerms; ++t) { cs[t] = a2ref / g; g *= 6.0f; }
      }
      float val[16];
      load_terms(val, cs, false);
      // Publish the partial as flagged words ([worker][token pair][row], 16 bytes each); the first workers of the group add the
      // block's outputs, in worker order. Nothing is fenced or counted: a word that carries this launch's number has its value.
      // One adder per two token pairs, and the others leave at once, so that the next launch's blocks can start on their SMs.
      // (With a counter whose last arriver adds: 0.9 us more for its round trip, and nobody leaves before it. With every worker of
      // the group adding a share: all leave 2 us later, 12 % more per layer at one token.)
      const int tpairs = (P.M + 1) >> 1;
      uint4* words = reinterpret_cast<uint4*>(P.partials);
#pragma unroll
      for (int tp = 0; tp < N / 8; ++tp)
        if (tp < tpairs) st_flagged2(words + ((long long)v * 8 + tp) * 128 + row, val[2 * tp], val[2 * tp + 1], call);
      const int tasks = 128 * tpairs, adders = min(live2, (tpairs + 1) >> 1);
      const int first = r2 < adders ? tasks * r2 / adders : 0, last = r2 < adders ? tasks * (r2 + 1) / adders : 0;
      for (int i = first + et; i < last; i += 128) {
        const uint4* src = words + (long long)vlo2 * 1024 + i;
        float s0 = 0.f, s1 = 0.f;
        constexpr int kBatch = 8;
        for (int p0 = 0; p0 < live2; p0 += kBatch) {
          float a[kBatch], b[kBatch];
          for (uint32_t it = 0;; ++it) {
            bool ok = true;
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
              if (p0 + k < live2) ok &= ld_flagged2(src + (long long)(p0 + k) * 1024, call, a[k], b[k]);
            if (ok) break;
            if (T.abort_flag || it >= (1u << 22)) { T.abort_flag = 1; *P.status = 10; break; }
            __nanosleep(50);
          }
#pragma unroll
          for (int k = 0; k < kBatch; ++k)
            if (p0 + k < live2) s0 += a[k], s1 += b[k];
        }
        const int tk = 2 * (i >> 7);
        __nv_bfloat16* dst = P.out + (long long)tk * P.H + 128 * nb2 + (i & 127);
        dst[0] = __float2bfloat16_rn(s0);
        if (tk + 1 < P.M) dst[P.H] = __float2bfloat16_rn(s1);
      }
    } else if (I2 == 0 && r2 == 0) {   // every slot of the batch is empty: the layer's output is zero
      for (int tk = 0; tk < P.M; ++tk) P.out[(long long)tk * P.H + 128 * nb2 + row] = __float2bfloat16_rn(0.f);
    }
#ifdef B200_TIMERS
    if (P.debug && et == 0) { P.debug[v * 16 + 0] = tm_a; P.debug[v * 16 + 1] = tm_b; P.debug[v * 16 + 2] = tm_c; P.debug[v * 16 + 3] = tm_d; P.debug[v * 16 + 7] = clock64() - tm_begin; }
#endif
  }
  tc_fence_before();
  __syncthreads();
#ifdef B200_TIMERS
  if (tid == 0 && P.debug) { unsigned long long g; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g)); P.debug[blockIdx.x * 16 + 14] = (long long)g; }
#endif
  if (warp == kTcMmaWarp) tmem_dealloc(tmem, 512);
  if (T.abort_flag)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

}  // namespace b200

using namespace b200;

int b200_decode_tc_smem_bytes(int NS, int region_bytes) { return 1024 + NS * kTcStage + region_bytes + (int)sizeof(TcTables); }

// static shared memory of the kernel for N operand columns: FC1's sums [N / 4][68] of up and of gate, and a few words
int b200_decode_tc_static_bytes(int N) { return 2 * (N / 4) * 68 * 4 + 256; }

static bool pdl_chain_enabled() {   // B200MOE_PDL_CHAIN=0: launch the expansion kernel as an ordinary stream-ordered kernel
  static const bool on = [] { const char* c = getenv("B200MOE_PDL_CHAIN"); return !(c && c[0] == '0'); }();
  return on;
}

int b200_expand_x_launch(const void* x, int M, int H, int N, int KB1, void* xb, float* colscale, const HostRouting* host, bool chained, cudaStream_t st) {
  // programmatic launch: the blocks may be scheduled while the previous kernel of the stream drains (if that kernel
  // allows it, as this library's layer kernel does); griddepcontrol.wait at their top keeps stream order for all data
  const HostRouting h = host ? *host : HostRouting{nullptr, nullptr, 0, nullptr, nullptr};
  void* args[] = {(void*)&x, (void*)&M, (void*)&H, (void*)&N, (void*)&KB1, (void*)&xb, (void*)&colscale,
                  (void*)&h.ids_h, (void*)&h.wts_h, (void*)&h.npairs, (void*)&h.ids_d, (void*)&h.wts_d};
  return launch_kernel(host ? (const void*)k_expand_x<true> : (const void*)k_expand_x<false>, N / kTerms, 256, 0, chained && pdl_chain_enabled(), args, st);
}

// x, ids and weights of a call from page-locked host memory into device memory. Block 0 brings the routing inputs, which the
// layer kernel reads at its entry, before it lets that kernel start; the others bring x.
__global__ void __launch_bounds__(128) k_host_stage(const uint4* x, int n16, const int* ids_h, const float* wts_h, int npairs, uint4* x_d, int* ids_d, float* wts_d) {
  const int tid = threadIdx.x;
  grid_dependency_wait();   // a kernel before this one may still read the copies it replaces
  if (blockIdx.x != 0) {
    grid_launch_dependents();
    const int i = (blockIdx.x - 1) * 128 + tid;
    if (i < n16) __stcg(x_d + i, __ldcv(x + i));
    return;
  }
  int id[2];
  float wt[2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (tid + 128 * j < npairs) { id[j] = __ldcv(ids_h + tid + 128 * j); wt[j] = __ldcv(wts_h + tid + 128 * j); }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (tid + 128 * j < npairs) { __stcg(ids_d + tid + 128 * j, id[j]); __stcg(wts_d + tid + 128 * j, wt[j]); }
  __threadfence();
  __syncthreads();
  grid_launch_dependents();
}

int b200_host_stage_launch(const void* x, int n16, const HostRouting& h, void* x_d, bool chained, cudaStream_t st) {
  void* args[] = {(void*)&x, (void*)&n16, (void*)&h.ids_h, (void*)&h.wts_h, (void*)&h.npairs, (void*)&x_d, (void*)&h.ids_d, (void*)&h.wts_d};
  return launch_kernel((const void*)k_host_stage, 1 + (n16 + 127) / 128, 128, 0, chained && pdl_chain_enabled(), args, st);
}

// q u8 [E, rows, row_bytes], sf = 128x4-swizzled scales per expert -> tile records (see k_pack_tiles)
int b200_pack_tiles_launch(const void* q, const void* sf, void* out, int E, int rows_per_expert, int row_bytes, int blocks, int KB, int KT,
                           int fc1, int I, long long sf_stride, cudaStream_t st) {
  const long long total = (long long)E * blocks * KB * 1152;
  long long g = (total + 255) / 256;
  if (g > 148 * 32) g = 148 * 32;
  k_pack_tiles<<<(int)g, 256, 0, st>>>((const uint8_t*)q, (const uint8_t*)sf, (uint8_t*)out, E, rows_per_expert, row_bytes, blocks, KB, KT, fc1,
                                       I, sf_stride);
  B200_LAUNCH_CHECK();
  return B200MOE_OK;
}

int b200_decode_tc_launch(const DecodeTcParams& p, int grid, int smem_bytes, bool chained, cudaStream_t st) {
  void* args[] = {(void*)&p};
  const void* fn = p.M <= 4 ? (const void*)k_moe_decode_tc<1> : p.M <= 8 ? (const void*)k_moe_decode_tc<2> : (const void*)k_moe_decode_tc<4>;
  static thread_local int configured[3] = {0, 0, 0};
  const int which = p.M <= 4 ? 0 : p.M <= 8 ? 1 : 2;
  if (configured[which] < smem_bytes) {
    B200_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    configured[which] = smem_bytes;
  }
  // programmatic dependent launch: this kernel's prologue and weight prefetch overlap the activation-expansion kernel
  return launch_kernel(fn, grid, kTcThreads, smem_bytes, chained, args, st);
}
