// Ragged grouped GEMM on tcgen05.mma kind::mxf4nvf4: row tiles of gathered tokens (up to 128 rows of one expert) times the
// expert's weight records. Four forms share the main loop:
//   PHASE 1  W4A4 FC1:  128 rows x [64 up | 64 gate] columns, epilogue SiLU*mul + NVFP4 re-quantisation into FC2's records
//   PHASE 2  W4A4 FC2:  128 rows x 128 columns, epilogue alpha * routing weight -> bf16 rows per (token, expert)
//   PHASE 3  W4A16 FC1: 64 rows (16 pairs x four NVFP4 terms), epilogue term sum + SiLU*mul + four-term re-expansion
//   PHASE 4  W4A16 FC2: the same rows, epilogue term sum + alpha * routing weight -> fp32 rows
//
// What bounds it. Per weight record (128 columns x 256 K values, 18 KB) the tensor core needs 4 x 64 cycles (measured:
// 128 x 128 x 64 in 64 cycles) plus 8 cycles per tcgen05.cp of a 512-byte scale tile; an SM takes in 63 bytes per cycle from
// L2 (17.3 TB/s over the chip, from four 18 KB copies in flight on), i.e. 288 cycles per record; HBM delivers a record per
// SM every ~700 cycles (7.1 TB/s). A batch that touches every expert with few rows is bound by HBM. In a large one no unit is
// near its peak over the whole kernel (FC1 of 8192 tokens: tensor pipe 48 %, shared memory 51 %, L2 24 %, HBM 30 %), but two streams of nearly the same length share the SM. Cycles a record of
// FC1 at 8192 tokens and seven boxes: 560 as it is, 500 without the epilogue, 430 with the ring alone (no MMA, scale copy or epilogue; 305 if every CTA reads one expert's records), 420 with
// the MMAs alone on one expert's records. In a loop of its own a round of four scale copies and four MMAs takes 290 (257 without the copies) with 100 bytes a cycle landing beside it, so
// neither the tensor pipe nor shared memory is the limit; where the ring's waits lengthen it to 420 is not known. The clock counts too: 1965 MHz without MMAs, 1750 in FC1, 1350 in that loop. Slots
// count for little: launch time at four to eight boxes 78.5, 87.3, 99.1, 111.9 and 131.0 us with eight, seven, six, five and four; the same with five, 2 to 5 % more with four, 13 to 19 % with three.
// Everything else has to stay out of the way of that stream: ONE warp waits for a record, copies its scale tiles into TMEM (tcgen05.cp) and issues its MMAs - operations of one lane execute in order, so nothing is handed from
// warp to warp between a record's arrival and its math. (Before, four warps moved the scales through registers and handed every
// record to the MMA warp over a barrier: 870 cycles a record at 8192 tokens.)
//
// A CTA keeps the records of the first NR K boxes of its row tile resident for all column blocks of the tile; boxes beyond NR
// come through the ring with the weights (gg_plan).
#pragma once
#include "common.cuh"
#include "tcgen05.cuh"
#include "nvfp4_math.cuh"
#include "expand.cuh"

namespace b200 {

constexpr int kRec = 18432;          // one tile record: 16 KB codes image + 4 x 512 B scale tiles
// W4A16 phases: the operand tile holds 64 rows (16 token-expert pairs x four terms) in 10 KB records (8 KB codes image +
// four 512-byte scale tiles whose row groups 2 and 3 stay zero). The MMA still spans 128 rows: rows 64..127 read whatever
// follows the record in shared memory, with zero scales, and their accumulator rows are ignored.
constexpr int kMidRec = 8192 + 2048;

constexpr int kGgThreads = 12 * 32;  // warps 0-7 epilogue (two groups of four), 8 row-tile producer, 9-10 ring producers, 11 MMA issuer
constexpr int kGgMaxRing = 12;
constexpr int kGgSmem = 227 * 1024 - 1024;   // dynamic shared memory of a CTA (1 KB is left to the static part)

// byte offset inside a tile record of 8 consecutive code bytes (one 16-value block) of row r, K block b16 (0..15)
__device__ __forceinline__ int rec_code_offset(int r, int b16) { return r * 128 + ((((b16 >> 1) ^ (r & 7))) << 4) + (b16 & 1) * 8; }
__device__ __forceinline__ int rec_scale_offset(int r, int b16) { return 16384 + (b16 >> 2) * 512 + (r & 31) * 16 + (r >> 5) * 4 + (b16 & 3); }

struct GroupedParams {
  const uint8_t* arec;        // operand records [ntiles][KB][kRec or kMidRec]
  const uint8_t* wrec;        // weight records [E][NBLK][KB][kRec]
  const int* ntiles;          // tiles, experts that they are of
  const int* tile_expert;
  const int* tile_first;      // first and end index of the tile's rows in the router's pair list
  const int* tile_end;
  const int* row_pair;        // [ntiles*rows] pair index or -1
  const float* alpha;         // per-expert weight scale
  float gs_in;                // PHASE 1/2: global scale the A operand was quantised with
  float gs_out;               // PHASE 1: global scale for the activation re-quantisation
  const float* wts;           // PHASE 2/4: routing weights [P]
  uint8_t* orec;              // PHASE 1/3: FC2 operand records [ntiles][KB2][...]
  __nv_bfloat16* y;           // PHASE 2: weighted rows [ntiles*128][H], columns at B200MOE_WEIGHTED_ROW_COLUMN
  float* yf;                  // PHASE 4: weighted rows [ntiles*16][H] in fp32 (one rounding only, in the combine)
  int* status;
  const float* rowscale;      // PHASE 3: 1 / g_t of every term row of the x operand [ntiles*64]
  float act_g1;               // PHASE 3/4: global scale of the first term of the SiLU*mul activations
  int NBLK, KB, KT, KB2, H, E;
  int stream;                 // the layer's weights do not fit in L2
  int wait_tables;            // the kernel before this one writes the tile tables
};

struct GgShared {
  uint64_t a_full[12], a_empty[12];                    // per resident K box
  uint64_t full[kGgMaxRing], empty[kGgMaxRing];        // per ring slot
  uint64_t acc_full[2], acc_empty[2];
  float scale[128];                                    // PHASE 1: gs_out / (E4M3 value), per scale byte
  uint32_t tmem_base;
  int max_rows;                                        // most operand rows of any tile this CTA works on
  volatile int abort_flag;
};

constexpr int kGgHead = 1024;   // barriers ahead of the records
static_assert(sizeof(GgShared) <= kGgHead, "the records start on a 1 KB boundary");

// How a CTA divides its shared memory, from the most rows its tiles hold: a resident operand record keeps only those rows (rounded
// up to 8) and its scale tiles; the rest is the ring. A tile of 64 rows over 8 K boxes takes 80 KB and leaves eight slots,
// one of 128 rows 144 KB and four. Depth matters when the weights come from HBM: four 18 KB records in flight are worth about
// 1.7 us of an SM's share, less than HBM latency plus the hand-offs. NR boxes stay resident; if not all of them do, the
// ring carries operand records as well and should hold kGgMinShared slots, or kGgMinStream where the weights' way from HBM counts for more than the
// operand's from L2: us with 6, 8, 9, 10, 11 slots: 333 skewed tokens of 2816 x 704 73.8, 72.1, 72.4, 71.6, 71.8; 2000 of it 154.5, 152, 151.5, 151, 151.5; 300
// skewed of 4096 x 1536 148, 141.5, 142.5, 139, 141; 800 of it 262, 254, 254, 253, 254; 2050 of it 371, 362, 360, 359, 356.
// That goes by how often a weight record is read (tiles by the experts they are of) and by what the four boxes fewer add to a column block's copies (a third at
// nine boxes, 15 % at 16). us with 6 and 10 slots, at tiles / experts: 10 boxes 1.47 137.8 / 136.7, 1.65 146.5 / 146.7, 1.99 162.5 / 165.6; 11 boxes 1.52 161.6 / 159.5, 2.0 219.7 / 221.4, 3.0
// 152.8 / 156.2, 8.0 61.0 / 62.4; 12 boxes 1.98 146.3 / 145.0, 2.25 53.2 / 52.5, 8.0 75.6 / 77.1; 14 boxes 2.33 74.0 / 71.9, 3.0 192.0 / 187.3, 8.0 67.7 / 69.1; 16 boxes
// 1.98 513 / 508, 3.0 61.0 / 60.2, 8.0 131.5 / 132.4. (By the layer's experts alone a batch on a few of them streamed: 3500 tokens on eight of 2816 x 704 190.2 instead of 184.4.)
// Where every expert has three tiles six slots are the better ones at all sizes (12 boxes 210.4 / 216.0, 16 boxes 761 / 770): at most two a layer's expert.
// TMEM: 256 accumulator columns + 16 per resident box
// + 64 for the rotating weight scales + 64 more for streamed operand scales.
//
// Once (no more tiles than the layer has experts): most weight records are then read once or twice, and the CTAs share what HBM delivers by the bytes each has in flight; one
// with few rows and a deep ring takes from one with many - at 333 tokens of 2816 x 704 a record took 300 ns with ten slots and 420 with four. Six slots a
// CTA are enough for the stream. (A batch on few experts, whose records are read many times, is indifferent: on eight of 128, 512 tokens of 2048 x 768 34.5 and 34.3 with all slots, W4A16 96 tokens
// 39.0 and 39.3.) us with all slots, eight, seven, six and five: 333 skewed tokens of 2816 x 704 75.7, 74.8, 74.2, 73.7, 72.4; 128 of it 93.7, 92.9, 92.2,
// 91.8, 91.7; 400 of 256 experts of 2048 x 1536 238.8, 236.0, 230.2, 227.5, 228.8; 700 skewed of 60 experts of 2304 x 1408 64.7, 64.2, 63.4, 62.6, 63.1; 300 skewed of
// 4096 x 1536 151.5, 149.6, 148.0, 147.8, 147.7. With more tiles than experts records come from L2 as well, and depth is worth something: 2500 of 2048 x 768
// 147.1, 147.2, 147.4, 147.9, 149.7; W4A16, 200 skewed of the 60 experts 65.8, 65.5, 65.4, 66.0, 68.2.
constexpr int kGgMinRing = 4, kGgMinShared = 6, kGgMinStream = 10, kGgMostOnce = 6;
struct GgPlan { int astride, NR, NS; };
__host__ __device__ inline GgPlan gg_plan(int KB, int max_rows, int tiles, int touched, int experts) {   // touched: experts that the tiles are of
  GgPlan p;
  const bool stream = tiles <= 2 * experts && 2 * tiles <= touched * (KB > 10 ? KB - 7 : 3);
  const int room = kGgSmem - 1024 - kGgHead;
  p.astride = ((max_rows + 7) & ~7) * 128 + 2048;
  p.NR = KB < 12 ? KB : 12;
  if ((room - p.NR * p.astride) / kRec < kGgMinRing || p.NR < KB) {
    p.NR = (room - (stream ? kGgMinStream : kGgMinShared) * kRec) / p.astride;
    if (p.NR > 8) p.NR = 8;
  }
  p.NS = (room - p.NR * p.astride) / kRec;
  const int most = tiles <= experts && p.NR == KB ? kGgMostOnce : kGgMaxRing;
  if (p.NS > most) p.NS = most;
  return p;
}

// A CTA's work: segments (row tile t, column blocks [n0, n1)). Whole tiles are dealt round-robin for as many full rounds as there
// are (tiles t and t + 1 of one expert then run on neighbouring CTAs at the same time and in the same block order, so the
// second reader of a weight record finds it in L2); the tiles left over are cut into equal ranges of column blocks so that
// every CTA gets a share of them.
struct GgSplit {
  int G, cta, NBLK, rounds, T0, ra, rb, nseg;
  struct Segment { int t, n0, n1; };
  __device__ GgSplit(int NT, int nblk, int g, int c) : G(g), cta(c), NBLK(nblk) {
    rounds = NT / G, T0 = rounds * G;
    const int rem = (NT - T0) * NBLK;
    ra = (int)((long long)rem * cta / G), rb = (int)((long long)rem * (cta + 1) / G);
    nseg = rounds + (rb > ra ? (rb - 1) / NBLK - ra / NBLK + 1 : 0);
  }
  __device__ Segment segment(int ord) const {
    if (ord < rounds) return {ord * G + cta, 0, NBLK};
    const int q = ra / NBLK + (ord - rounds);
    return {T0 + q, ord == rounds ? ra - q * NBLK : 0, min(NBLK, rb - q * NBLK)};
  }
};

// What the kernel ahead of FC1 does beside its records (records_aside): `blocks` extra thread blocks in front of its grid.
constexpr int kGgWarm = 8;   // weight records per GEMM CTA asked into L2 ahead of the GEMM
struct GgAside {
  const int *ntiles, *tile_expert, *tile_first, *tile_end;
  const uint8_t* wrec;       // FC1 weight records
  int NBLK, KB, gemm_ctas, blocks;
};

// W4A4 FC1 divides with IEEE rounding where the operand has more than nine K boxes (hidden sizes above 2304): the results of these
// layers were defined that way, and an approximate quotient moves an activation on the edge of two FP4 codes to the other one (1.4e-4
// of a layer's output at 4096 x 1536). Up to nine boxes it has always been the approximate one.
inline bool gg_ieee_silu(int KB1) { return KB1 > 9; }
// g / d rounded to nearest for d = 1 + exp(-g) and -44 <= g <= 2^64: Markstein's method (IBM J. Res. Dev. 34, 1990) - the approximate
// reciprocal, one Newton step, the quotient and one correction by its exact residual. In that range d is below 2^64 and no step leaves
// the normal numbers (below 2^-24 d is exactly 2); a zero keeps its sign. The caller takes __fdiv_rn elsewhere. (333 tokens of 2816 x
// 704: 76 us, 74 with the approximate quotient. With __fdiv_rn throughout 103: an empty row of a tile holds zeros, and a zero
// numerator takes its special path.)
__device__ __forceinline__ float gg_quotient(float g, float d) {
  float y = rcp_approx(d);
  y = __fmaf_rn(__fmaf_rn(-d, y, 1.0f), y, y);
  const float q = __fmul_rn(g, y);
  return g == 0.f ? g : __fmaf_rn(__fmaf_rn(-d, q, g), y, q);
}
constexpr float kGgQuotLo = -44.f, kGgQuotHi = 0x1p64f;   // (a NaN may go either way)

// ---- epilogues: one warp, 32 accumulator rows x 128 columns at taddr (thread = row). `release` frees the accumulator buffer
// once its values are in registers.

// W4A4 FC1: columns 0..63 = up, 64..127 = gate of intermediate columns 64n..; SiLU*mul, re-quantise four blocks of 16 and store
// the row's 32 code bytes (two 16-byte chunks of one sector) and four scale bytes into FC2's record `dst`.
template <bool Ieee, class F>
__device__ __forceinline__ void gg_epilogue_fc1(uint32_t taddr, float s, float gs_out, const float* scale_table, uint8_t* dst, int row, bool store,
                                                int n, F&& release) {
  uint32_t sfw = 0;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    uint32_t up[2][16], gt[2][16];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tmem_ld_32x32b_x16(taddr + 32 * h + 16 * b, up[b]);
      tmem_ld_32x32b_x16(taddr + 64 + 32 * h + 16 * b, gt[b]);
    }
    tmem_ld_wait();
    if (h == 1) release();
    uint2 pk[2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      float a[16];
      float lo = 0.f, hi = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float g = __uint_as_float(gt[b][i]) * s, u = __uint_as_float(up[b][i]) * s;
        const float d = 1.0f + __expf(-g);
        if (Ieee) lo = fminf(lo, g), hi = fmaxf(hi, g);
        a[i] = (Ieee ? gg_quotient(g, d) : __fdividef(g, d)) * u;
      }
      if (Ieee && (lo < kGgQuotLo || hi > kGgQuotHi) && store) {   // (not in the dry pass, on whatever the accumulator holds)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float g = __uint_as_float(gt[b][i]) * s, u = __uint_as_float(up[b][i]) * s;
          a[i] = __fdiv_rn(g, 1.0f + __expf(-g)) * u;
        }
      }
      sfw |= (uint32_t)quantize_block16_t(a, gs_out, scale_table, pk[b]) << (16 * h + 8 * b);
    }
    if (store) *reinterpret_cast<uint4*>(dst + rec_code_offset(row, 4 * (n & 3) + 2 * h)) = make_uint4(pk[0].x, pk[0].y, pk[1].x, pk[1].y);
  }
  if (store) *reinterpret_cast<uint32_t*>(dst + rec_scale_offset(row, 4 * (n & 3))) = sfw;
}

// W4A4 FC2: scale, round to bf16 and store. The accumulator is read in the fragment layout of mma (eight rows x four lanes), so that the four lanes
// of a row hold 64 columns between them and an instruction stores 64-byte halves of eight rows' segments; nothing goes through shared
// memory. The columns of a segment lie as the lanes hold them: 16-byte chunk 4j + q has columns 32j + 8w + 2q + {0, 1}, w = 0..3 (combine_columns
// puts them right; B200MOE_WEIGHTED_ROW_COLUMN tells callers). s[i]: scale of row 8i + lane / 4 of the warp; the first `rows` rows hold a pair. A block's epilogue takes 920 cycles at 1024
// tokens of the 2048 x 768 layer and 1290 at 8192 (FC2 73 us there); with a thread per row and a transposition through shared memory 2680 and 3170 (84 us, the
// epilogue was the bound), with that and bulk stores 4040 and 3850: a store waits behind the ring's loads in the copy engine.
template <class F>
__device__ __forceinline__ void gg_epilogue_fc2(uint32_t taddr, const float (&s)[4], int rows, __nv_bfloat16* ybase, int H, int lane, F&& release) {
  __nv_bfloat16* yrow = ybase + (long long)(lane >> 2) * H + (lane & 3) * 8;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    uint32_t r[2][32];
    tmem_ld_16x256b_x8(taddr + 64 * half, r[0]);
    tmem_ld_16x256b_x8(taddr + 64 * half + (16u << 16), r[1]);
    tmem_ld_wait();
    if (half == 1) release();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool store = 8 * i + (lane >> 2) < rows;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t o[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint32_t* v = &r[i >> 1][4 * (4 * j + w) + 2 * (i & 1)];
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[0]) * s[i], __uint_as_float(v[1]) * s[i]);
          o[w] = *reinterpret_cast<const uint32_t*>(&h);
        }
        if (store) *reinterpret_cast<uint4*>(yrow + (long long)(8 * i) * H + 64 * half + 32 * j) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}
// The four lanes of a quad hold chunks 4j..4j+3 of a segment: afterwards lane q holds columns 32j + 8q .. + 7 in their order.
__device__ __forceinline__ void combine_columns(uint32_t (&w)[4], int lane) {
  const unsigned quad = 0xfu << (lane & 28);
  uint32_t a = __shfl_xor_sync(quad, lane & 1 ? w[0] : w[1], 1), b = __shfl_xor_sync(quad, lane & 1 ? w[2] : w[3], 1);
  if (lane & 1) w[0] = a, w[2] = b;
  else w[1] = a, w[3] = b;
  a = __shfl_xor_sync(quad, lane & 2 ? w[0] : w[2], 2), b = __shfl_xor_sync(quad, lane & 2 ? w[1] : w[3], 2);
  if (lane & 2) w[0] = a, w[1] = b;
  else w[2] = a, w[3] = b;
}

// W4A16 FC1: rows 4p..4p+3 are the four terms of pair p, each scaled by its 1/g_t. A reduce-scatter over the pair's four lanes
// leaves lane q with the sums of the q-th 16-column block (up, then gate), so that SiLU*mul and the expansion of the activations
// into four terms run once per block with every lane at work; the lane writes its block of all four term rows of FC2's operand
// record. (With two blocks at a time and every second lane idle in the expansion an epilogue took 12,500 cycles, more than the
// eight weight records of a block take to arrive.) Returns whether a block lay beyond the range of the activation scale.
// Fused: whether the lane's own product is rounded before the add. Which of the two a phase does is part of its results: a bf16 output
// in a few thousand moves by one step with the other.
template <bool Fused>
__device__ __forceinline__ void gg_reduce_scatter16(uint32_t taddr, float rs, int tq, float (&o)[16]) {
  uint32_t r[4][16];
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x16(taddr + 16 * c, r[c]);
  tmem_ld_wait();
  const int hi = tq >> 1, lo = tq & 1;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float k2[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float mine = __uint_as_float(hi ? r[2 + j][i] : r[j][i]), other = __fmul_rn(__uint_as_float(hi ? r[j][i] : r[2 + j][i]), rs);
      const float got = __shfl_xor_sync(0xffffffffu, other, 2);   // the lane two over keeps the other two blocks and sends these
      k2[j] = Fused ? __fmaf_rn(mine, rs, got) : __fadd_rn(__fmul_rn(mine, rs), got);
    }
    const float keep = lo ? k2[1] : k2[0], send = lo ? k2[0] : k2[1];
    o[i] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
  }
}

template <class F>
__device__ __forceinline__ bool gg_epilogue_fc1_a16(uint32_t taddr, float s, float rs, float act_g1, uint8_t* dst, int row, bool used, bool store, int n,
                                                    int lane, F&& release) {
  const int tq = lane & 3;
  float up[16], a[16];
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {   // the up columns, then the gate columns
#pragma unroll
    for (int i = 0; i < 16; ++i) up[i] = a[i];
    gg_reduce_scatter16<false>(taddr + 64 * half, rs, tq, a);
  }
  release();
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float g = a[i] * s, u = up[i] * s;
    a[i] = __fdividef(g, 1.0f + __expf(-g)) * u;
  }
  bool clipped = false;
  if (used) {
    const int r0 = row & ~3;
    clipped = expand_block16<true>(a, act_g1, [&](int q, uint2 codes, uint8_t sf) {
      if (!store) return;
      *reinterpret_cast<uint2*>(dst + rec_code_offset(r0 + q, 4 * (n & 3) + tq)) = codes;
      dst[8192 + (n & 3) * 512 + ((r0 + q) & 31) * 16 + ((r0 + q) >> 5) * 4 + tq] = sf;
    });
  }
  return clipped && store;
}

// W4A16 FC2: the four term rows of a pair are scaled and added; lane t of the pair stores columns 16t..16t+15 of each 64-column
// half, so the four lanes write contiguous 256-byte segments of the pair's row.
template <class F>
__device__ __forceinline__ void gg_epilogue_fc2_a16(uint32_t taddr, float s, float rs, bool store, float* yrow, int lane, F&& release) {
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const int tq = lane & 3;
    float o[16];
    gg_reduce_scatter16<true>(taddr + 64 * half, rs, tq, o);
    if (half == 1) release();
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] *= s;
    if (store) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(yrow + 64 * half + 16 * tq + 4 * i) = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
    }
  }
}

// Ieee (PHASE 1): SiLU divides with IEEE rounding instead of __fdividef; see gg_ieee_silu.
template <int PHASE, bool Ieee = false>
__global__ void __launch_bounds__(kGgThreads, 1) k_grouped_gemm(const __grid_constant__ GroupedParams P) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int kARec = PHASE >= 3 ? kMidRec : kRec;            // bytes of one operand record in global memory
  constexpr int kACodes = PHASE >= 3 ? 8192 : 16384;            // ... of which codes; the scale tiles follow
  constexpr int kARows = PHASE >= 3 ? 64 : 128;                 // operand rows per tile
  constexpr int kRowsPerPair = PHASE >= 3 ? kTerms : 1;
  const int KB = P.KB, NBLK = P.NBLK;
  GgShared& S = *reinterpret_cast<GgShared*>(smem);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);       // (a value from lane 0 is known to be warp-uniform)
  // Without wait_tables the tile tables are read without waiting for the kernel before this one: the tables' own producer is at least
  // two kernels back, and the kernel in between lets this one start only after it has seen that producer complete.
  int2 ntiles = P.wait_tables ? make_int2(0, 0) : __ldcg(reinterpret_cast<const int2*>(P.ntiles));
  if (tid == 0) {
    for (int k = 0; k < 12; ++k) { mbar_init(&S.a_full[k], 1); mbar_init(&S.a_empty[k], 1); }
    for (int s = 0; s < kGgMaxRing; ++s) { mbar_init(&S.full[s], 1); mbar_init(&S.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&S.acc_full[b], 1); mbar_init(&S.acc_empty[b], 4); }
    S.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 11) { tmem_alloc(&S.tmem_base, 512); tmem_relinquish(); }
  if (PHASE == 1) fill_scale_table(S.scale, P.gs_out, tid, kGgThreads);
  if (P.wait_tables) { grid_dependency_wait(); ntiles = __ldcg(reinterpret_cast<const int2*>(P.ntiles)); }
  grid_launch_dependents();   // the next kernel of the chain may take over SMs as this one's CTAs leave
  const int NT = __shfl_sync(0xffffffffu, ntiles.x, 0), touched = __shfl_sync(0xffffffffu, ntiles.y, 0);
  const GgSplit split(NT, NBLK, (int)gridDim.x, (int)blockIdx.x);
  const int nseg = split.nseg;
  auto for_each_segment = [&](auto&& body) {   // body(t, n0, n1, ordinal), one call site: a copy of a role's code per launch is enough
#pragma unroll 1
    for (int ord = 0; ord < nseg; ++ord) {
      const GgSplit::Segment g = split.segment(ord);
      body(g.t, g.n0, g.n1, ord);
    }
  };
  auto tile_rows = [&](int t) {   // operand rows that hold something, rounded up to the 8-row groups of the record image
    return min(kARows, ((__ldcg(P.tile_end + t) - __ldcg(P.tile_first + t)) * kRowsPerPair + 7) & ~7);
  };
  if (warp == 10) {   // the most rows of this CTA's tiles
    int m = 8;
    for (int i = lane; i < nseg; i += 32) m = max(m, tile_rows(split.segment(i).t));
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) S.max_rows = m;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const GgPlan plan = gg_plan(KB, __shfl_sync(0xffffffffu, S.max_rows, 0), NT, touched, P.E);
  const int NR = plan.NR, NS = plan.NS, astride = plan.astride, acodes = astride - 2048;
  uint8_t* abuf = smem + kGgHead;                  // NR records of the current row tile
  uint8_t* ring = abuf + NR * astride;                          // NS slots
  const uint32_t tmem = __shfl_sync(0xffffffffu, S.tmem_base, 0);
  const uint32_t tm_acc = tmem, tm_sfa = tmem + 256, tm_sfb = tmem + 256 + 16 * NR, tm_sfs = tm_sfb + 64;   // 2 x 128 | NR x 16 | 4 x 16 | 4 x 16
  const int nkt_last = P.KT - 4 * (KB - 1);

  if (warp == 8) {
    // ============================================================== resident operand records: once per segment, box by box
    const uint32_t el = elect_one();
    const uint32_t full_u = smem_u32(S.a_full), empty_u = smem_u32(S.a_empty), abuf_u = smem_u32(abuf);
    grid_dependency_wait();   // the records are written by the kernel before this one
    for_each_segment([&](int t, int, int, int ord) {
      const int codes = tile_rows(t) * 128;   // only the rows in use, then the scale tiles
      for (int kb = 0; kb < NR; ++kb) {
        if (ord >= 1 && !mbar_wait_warp(empty_u + 8 * kb, (uint32_t)((ord - 1) & 1), &S.abort_flag)) *P.status = 2;
        const uint8_t* src = P.arec + ((long long)t * KB + kb) * kARec;
        mbar_expect_tx_u32(full_u + 8 * kb, codes + 2048, el);
        bulk_load_u32(abuf_u + kb * astride, src, codes, full_u + 8 * kb, el);
        bulk_load_u32(abuf_u + kb * astride + acodes, src + kACodes, 2048, full_u + 8 * kb, el);
      }
    });
    __syncwarp();
  } else if (warp == 9 || warp == 10) {
    // ============================================================== ring: weight records (and operand records of boxes >= NR).
    // Two producers walk the same sequence and issue alternate slots. The warps stay converged and an elected lane issues: a copy takes a producer 320 cycles beside its
    // wait, 470 from a branch that a single lane takes (8192 tokens of 2048 x 768 348 -> 341 us, 2050 of 4096 x 1536 425 -> 411).
    // Weight records are the first to leave L2 again, so that what the layer writes stays there: layers one after the other, each with its
    // own weights, take 76 us (78 without) at 96 tokens (W4A16), 86.4 (88.1) at 1024, 65.9 (68.1) at 24. Not so the records of an
    // expert with several tiles, which are read again: with those as well 3000 tokens take 167.8 us instead of 162.5, and in W4A16, where a
    // tile is 16 pairs, skewed batches 178 instead of 145 (195 tokens of 3072 x 1536), 113 instead of 96 (256 of 60 experts of 2304 x 1408) and 120 instead of 104
    // (150 of 256 experts of 2048 x 1536); at most 3 % were gained with those as well (256 of 2816 x 704: 95.8 instead of 98.5). Nor the weights of a layer that
    // fits in L2, which the next call on it may find there (113 MB, one layer again and again: 43.2 us marked, 42.7 not).
    const uint64_t once = policy_evict_first();
    const uint32_t el = elect_one();
    const uint32_t full_u = smem_u32(S.full), empty_u = smem_u32(S.empty), ring_u = smem_u32(ring);
    int slot = 0;
    uint32_t ph = 1;          // parity that a free slot's `empty` barrier has completed: the first pass finds all slots free
    bool mine = warp == 9, waited = NR == KB;
    auto next = [&]() { mine = !mine; if (++slot == NS) { slot = 0; ph ^= 1u; } };
    auto acquire = [&]() { if (!mbar_wait_warp(empty_u + 8 * slot, ph, &S.abort_flag)) *P.status = 2; };
    for_each_segment([&](int t, int n0, int n1, int) {
      // (the three loads in flight together: nothing else starts before them)
      const int expert = __ldcg(P.tile_expert + t), before = t > 0 ? __ldcg(P.tile_expert + t - 1) : -1, after = t + 1 < NT ? __ldcg(P.tile_expert + t + 1) : -1;
      const uint8_t* src = P.wrec + ((long long)__shfl_sync(0xffffffffu, expert, 0) * NBLK + n0) * KB * kRec;   // consecutive column blocks are contiguous
      const bool stay = __shfl_sync(0xffffffffu, (int)(!P.stream || before == expert || after == expert), 0) != 0;
      const uint8_t* asrc = P.arec + (long long)t * KB * kARec;
      const int codes = NR < KB ? tile_rows(t) * 128 : 0;
      for (int n = n0; n < n1; ++n)
        for (int kb = 0; kb < KB; ++kb, src += kRec) {
          if (kb >= NR) {
            if (mine) {
              acquire();
              if (!waited) { grid_dependency_wait(); waited = true; }
              mbar_expect_tx_u32(full_u + 8 * slot, codes + 2048, el);
              bulk_load_u32(ring_u + slot * kRec, asrc + (long long)kb * kARec, codes, full_u + 8 * slot, el);
              bulk_load_u32(ring_u + slot * kRec + kACodes, asrc + (long long)kb * kARec + kACodes, 2048, full_u + 8 * slot, el);
            }
            next();
          }
          if (mine) {
            acquire();
            mbar_expect_tx_u32(full_u + 8 * slot, kRec, el);
            if (stay) bulk_load_u32(ring_u + slot * kRec, src, kRec, full_u + 8 * slot, el);
            else bulk_load_hint_u32(ring_u + slot * kRec, src, kRec, full_u + 8 * slot, once, el);
          }
          next();
        }
    });
    __syncwarp();
  } else if (warp == 11) {
    // ============================================================== MMA issuer: the warp stays converged (all values are
    // warp-uniform) and one elected lane issues. Measured per record (wait, 4 scale copies, 4 MMAs, commit; dynamic slots): 320
    // cycles this way - the MMAs themselves are 256 - against 450 to 620 from inside a branch that a single lane takes.
    const uint32_t el = elect_one();
    const uint32_t idesc = idesc_mxf4nvf4(128, 128);
    const uint32_t a16 = kDescLoSw128 + (smem_u32(abuf) >> 4), r16 = kDescLoSw128 + (smem_u32(ring) >> 4);   // descriptor low words
    const uint32_t full_u = smem_u32(S.full), empty_u = smem_u32(S.empty), afull_u = smem_u32(S.a_full), aempty_u = smem_u32(S.a_empty);
    const uint32_t accf_u = smem_u32(S.acc_full), acce_u = smem_u32(S.acc_empty);
    int slot = 0, seq = 0;
    uint32_t ph = 0, rot = 0;
    auto take = [&]() {   // the next ring slot, landed
      if (!mbar_wait_warp(full_u + 8 * slot, ph, &S.abort_flag)) *P.status = 1;
      const int s = slot;
      if (++slot == NS) { slot = 0; ph ^= 1u; }
      return s;
    };
    auto copy_scales = [&](uint32_t dst, uint32_t rec_lo, int codes16) {   // four 512-byte tiles -> 16 TMEM columns
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) tmem_cp_sf_lo(dst + 4 * jj, rec_lo - kDescLoSw128 + codes16 + 32 * jj, el);
    };
    for_each_segment([&](int, int n0, int n1, int ord) {
      for (int n = n0; n < n1; ++n, ++seq) {
        const int ab = seq & 1;
        const bool first = n == n0, last = n == n1 - 1;
        if (seq >= 2 && !mbar_wait_warp(acce_u + 8 * ab, (uint32_t)((seq >> 1) - 1) & 1u, &S.abort_flag)) *P.status = 5;
        const uint32_t acc = tm_acc + 128 * ab;
        for (int kb = 0; kb < KB; ++kb) {
          uint32_t a_lo, sfa;
          int aslot = -1;
          if (kb < NR) {
            a_lo = a16 + kb * (astride >> 4), sfa = tm_sfa + 16 * kb;
            if (first) {
              if (!mbar_wait_warp(afull_u + 8 * kb, (uint32_t)(ord & 1), &S.abort_flag)) *P.status = 1;
              tc_fence_after();
              copy_scales(sfa, a_lo, acodes >> 4);
            }
          } else {
            aslot = take();
            a_lo = r16 + aslot * (kRec >> 4), sfa = tm_sfs + 16 * rot;
            tc_fence_after();
            copy_scales(sfa, a_lo, kACodes >> 4);
          }
          const int bslot = take();
          const uint32_t b_lo = r16 + bslot * (kRec >> 4), sfb = tm_sfb + 16 * rot;
          rot = (rot + 1) & 3u;
          tc_fence_after();
          copy_scales(sfb, b_lo, 1024);   // a short last box has zero scale tiles behind its last K step: copying them is harmless
          if (kb < KB - 1 || nkt_last == 4) {
            umma_mxf4nvf4_lo(acc, a_lo, b_lo, idesc, sfa, sfb, kb != 0 ? 1u : 0u, el);
#pragma unroll
            for (int jj = 1; jj < 4; ++jj) umma_mxf4nvf4_lo(acc, a_lo + 2 * jj, b_lo + 2 * jj, idesc, sfa + 4 * jj, sfb + 4 * jj, 1u, el);
          } else {
            for (int jj = 0; jj < nkt_last; ++jj)
              umma_mxf4nvf4_lo(acc, a_lo + 2 * jj, b_lo + 2 * jj, idesc, sfa + 4 * jj, sfb + 4 * jj, kb + jj != 0 ? 1u : 0u, el);
          }
          umma_commit_u32(empty_u + 8 * bslot, el);
          if (aslot >= 0) umma_commit_u32(empty_u + 8 * aslot, el);
          else if (last) umma_commit_u32(aempty_u + 8 * kb, el);   // the next segment's record of this box may land
        }
        umma_commit_u32(accf_u + 8 * ab, el);
      }
    });
    __syncwarp();
  } else {
    // ============================================================== epilogue: group g = warps 4g..4g+3 takes every second block
    // (accumulator buffer g), so a block's epilogue may last as long as two blocks of MMAs; thread = accumulator row.
    const int grp = warp >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;
    int seq = 0;
    uint32_t aph = 0;
    // The first pass through a block is a dry one, on whatever the accumulator holds and without storing: it brings the epilogue's
    // instructions into the SM while the first records are still on their way. (Without it the first block's epilogue
    // took 16,000 cycles against 3,000 later on, and the MMAs of the third block waited for it.)
    bool dry = true;
    for_each_segment([&](int t, int n0, int n1, int) {
#pragma unroll 1
     for (int pass = dry ? 0 : 1; pass < 2; ++pass) {
      if (dry && pass == 1) {
        dry = false;
        grid_dependency_wait();   // what is read and written from here on belongs to the kernels before this one until they are complete
      }
      const int rows = tile_rows(t);
      float s = P.alpha[__ldcg(P.tile_expert + t)];
      if (PHASE <= 2) s /= P.gs_in;
      int pr = -1;
      float rs = 0.f;   // W4A16 phases: 1 / g_t of this operand row's term
      // (not in the dry pass: the kernel that writes row_pair and rowscale may still be running, and what an earlier, larger call left in
      // row_pair would index beyond this call's weights)
      if (!dry && (PHASE == 2 || (PHASE == 4 && row < kARows))) {   // FC2: times the row's routing weight
        pr = __ldcg(P.row_pair + (long long)t * kARows + row);
        s = pr >= 0 ? s * P.wts[pr] : 0.f;
      }
      if (PHASE == 3 && !dry && row < rows) rs = __ldcg(P.rowscale + (long long)t * kARows + row);
      if (PHASE == 4) {
        float g = P.act_g1;
        for (int q = 0; q < (lane & 3); ++q) g *= 6.0f;
        rs = 1.0f / g;
      }
      const int held = PHASE == 2 ? __popc(__ballot_sync(0xffffffffu, pr >= 0)) : 0;   // rows of this quadrant that hold a pair: the first ones
      float s4[4];
      if (PHASE == 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s4[i] = __shfl_sync(0xffffffffu, s, 8 * i + (lane >> 2));
      }
      const bool work = quad * 32 < rows;   // warp-uniform: this quadrant holds rows of the tile
#pragma unroll 1
      for (int n = n0; n < n1; ++n, ++seq) {
        if (!dry) {
          if ((seq & 1) != grp) continue;
          if (!mbar_wait(&S.acc_full[grp], aph, &S.abort_flag)) *P.status = 7;
          aph ^= 1u;
          tc_fence_after();
        }
        const uint32_t taddr = tm_acc + 128 * grp + ((uint32_t)(quad * 32) << 16);
        auto release = [&]() {   // the accumulator is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0 && !dry) mbar_arrive(&S.acc_empty[grp]);
        };
        if (!work && !dry) {
          release();
        } else if (PHASE == 1) {
          gg_epilogue_fc1<Ieee>(taddr, s, P.gs_out, S.scale, P.orec + ((long long)t * P.KB2 + (n >> 2)) * kRec, row, row < rows && !dry, n, release);
        } else if (PHASE == 2) {
          gg_epilogue_fc2(taddr, s4, dry ? 0 : held, P.y + ((long long)t * 128 + quad * 32) * P.H + 128 * n, P.H, lane, release);
        } else if (PHASE == 3) {
          if (gg_epilogue_fc1_a16(taddr, s, rs, P.act_g1, P.orec + ((long long)t * P.KB2 + (n >> 2)) * kMidRec, row, row < rows, !dry, n, lane, release))
            P.status[1] = 1;   // beyond the range of the fixed activation scale
        } else {
          gg_epilogue_fc2_a16(taddr, s, rs, pr >= 0 && !dry, P.yf + ((long long)t * 16 + (row >> 2)) * P.H + 128 * n, lane, release);
        }
        if (dry) break;
      }
     }
    });
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 11) tmem_dealloc(tmem, 512);
  if (S.abort_flag)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

}  // namespace b200
