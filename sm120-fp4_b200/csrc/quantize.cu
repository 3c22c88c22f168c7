// NVFP4 quantisation with the group's own global scale (2688 / amax): the amax pass and the quantising pass in ONE launch. Same
// bytes as b200moe_global_scale_grouped followed by b200moe_quantize_nvfp4 (sm120fp4/reference.py:68-90).
//
// Small inputs (up to 64 rows of 2048) stay in the registers of one thread-block cluster between the two passes: what bounds
// them is launches and round trips, and this is one launch with one exchange of maxima over distributed shared memory.
// Large ones are bound by HBM: the input has to be read twice, but the second read of a group comes right after the first, when
// the group is still in L2. Work units (64 KB of input) are taken round-robin in an order that keeps a window of groups open:
// amax(0) .. amax(W-1), then amax(g + W), quantise(g) in turn. A quantising unit waits until its group's amax units have
// published their maxima; they all stand earlier in the order, and every block takes its units in that order.
#include "common.cuh"
#include "nvfp4_math.cuh"
#include "tcgen05.cuh"
#include <type_traits>

namespace b200 {

constexpr int kQThreads = 512;                                   // of the small form
constexpr int kQgThreads = 256;                                  // of the large form, two blocks per SM (three of 32 KB units: 3 % slower; four, or the next unit's loads ahead of this one's math: 15 % and more)
constexpr int kQSmallPerThread = 2;                              // 16-value blocks a thread keeps in registers
constexpr int kQSmallMaxBlocks = 8 * kQThreads * kQSmallPerThread;
template <typename T> constexpr int kQPerThread = sizeof(T) == 2 ? 8 : 4;   // 16-value blocks a thread takes of one work unit (64 KB of input)
// Input bytes between a group's two passes. Of large inputs what is read for the second time and the codes are marked to leave L2 first, so
// that L2 holds about this and what is in flight: 60 x 1024 x 1536 fp32 take 91.5 us (20 MB 96, 12 MB 114, 45 MB 92.5; unmarked 98 to 100).
constexpr long long kQWindowBytes = 30ll << 20;
// Above this an input is large in any case; below, one whose groups do not all lie in a window is (8 x 1472 x 1344 fp32, 60 MB, 21.3 us with the marks and
// 22.3 without; 16 x 768 x 1024 fp32 behind a copy of it 32.2 and 33.0). 8192 x 4096 fp32 (128 MB) 58.7 us on new inputs with the marks and 63.2
// without. What is left L2 holds as a whole, and the next kernel finds it there: 2048 x 4096 bf16 again and again on the same input 12.2 us with
// marks and 10.7 without, 4096 x 4096 18.5 and 18.0, 8192 x 2048 fp32 24.4 and 23.7.
constexpr long long kQMarkFrom = 64ll << 20;

struct QuantGeom {
  int rows, bpr;           // rows of a group, 16-value blocks per row
  int layout;              // 0: scales row-major [groups * rows][bpr]; 1: 128x4 swizzle per group, padded to 128 rows x 4 columns
  long long sf_stride;     // scale bytes of a group
  int nkt;
  bool wide;               // x is 32-byte aligned
  bool mark;               // what is not needed again leaves L2 first
  // i / bpr = i * bpr_inv >> bpr_shift with bpr_inv = ceil(2^shift / bpr): exact while i * (bpr_inv * bpr - 2^shift) < 2^shift, which
  // i < 2^30 and shift = 30 + the bits of bpr grant
  unsigned long long bpr_inv;
  int bpr_shift;
  int step_r, step_c;      // kQgThreads blocks on, as rows and columns
};

__device__ __forceinline__ long long sf_swizzled(int r, int c, int nkt) {
  return ((long long)(r >> 7) * nkt + (c >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (c & 3);
}

// global_scale = reciprocal(max(amax, 1e-12)) * 2688 with the reference's two roundings (see k_global_scale)
__device__ __forceinline__ float scale_of(float amax) { return __fmul_rn(__frcp_rn(fmaxf(amax, 1e-12f)), 2688.0f); }

// 16 values as loaded
template <typename T> struct Raw16 { uint4 r[sizeof(T)]; };
// wide: the address is 32-byte aligned, so that a thread's 32 (64) bytes are one (two) 256-bit loads and every sector is asked for once.
// last: nobody reads the values again, so they leave L2 first
template <typename T> __device__ __forceinline__ void load_raw(const T* p, bool wide, bool last, Raw16<T>& v) {
  if (wide && last) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); i += 2)
      asm volatile("ld.global.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(v.r[i].x), "=r"(v.r[i].y), "=r"(v.r[i].z), "=r"(v.r[i].w), "=r"(v.r[i + 1].x), "=r"(v.r[i + 1].y), "=r"(v.r[i + 1].z), "=r"(v.r[i + 1].w)
                   : "l"(reinterpret_cast<const uint4*>(p) + i));
  } else if (wide) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); i += 2)
      asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(v.r[i].x), "=r"(v.r[i].y), "=r"(v.r[i].z), "=r"(v.r[i].w), "=r"(v.r[i + 1].x), "=r"(v.r[i + 1].y), "=r"(v.r[i + 1].z), "=r"(v.r[i + 1].w)
                   : "l"(reinterpret_cast<const uint4*>(p) + i));
  } else {
#pragma unroll
    for (int i = 0; i < (int)sizeof(T); ++i) v.r[i] = reinterpret_cast<const uint4*>(p)[i];
  }
}
__device__ __forceinline__ void st_policy(uint2* p, uint2 v, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.v2.b32 [%0], {%1, %2}, %3;" ::"l"(p), "r"(v.x), "r"(v.y), "l"(policy) : "memory");
}
// largest magnitude of the 16 values; NaNs are passed over, as fmaxf does, unless there is nothing else (a block of NaNs then gets the
// largest block scale, as quantize_block16 gives it)
__device__ __forceinline__ float amax_raw(const Raw16<__nv_bfloat16>& v) {
  // the larger magnitude of either half, with the product of the signs: those go at the end
  auto larger = [](uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  };
  const uint32_t b = larger(larger(larger(v.r[0].x, v.r[0].y), larger(v.r[0].z, v.r[0].w)), larger(larger(v.r[1].x, v.r[1].y), larger(v.r[1].z, v.r[1].w)));
  return fmaxf(fabsf(__uint_as_float(b << 16)), fabsf(__uint_as_float(b & 0xffff0000u)));
}
__device__ __forceinline__ float amax_raw(const Raw16<float>& v) {
  float m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    m[i] = fmaxf(fmaxf(fabsf(__uint_as_float(v.r[i].x)), fabsf(__uint_as_float(v.r[i].y))),
                 fmaxf(fabsf(__uint_as_float(v.r[i].z)), fabsf(__uint_as_float(v.r[i].w))));
  return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}
__device__ __forceinline__ void floats(const Raw16<__nv_bfloat16>& v, float (&f)[16]) {
  const uint32_t w[8] = {v.r[0].x, v.r[0].y, v.r[0].z, v.r[0].w, v.r[1].x, v.r[1].y, v.r[1].z, v.r[1].w};
#pragma unroll
  for (int i = 0; i < 8; ++i) { f[2 * i] = __uint_as_float(w[i] << 16); f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}
__device__ __forceinline__ void floats(const Raw16<float>& v, float (&f)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[4 * i] = __uint_as_float(v.r[i].x), f[4 * i + 1] = __uint_as_float(v.r[i].y), f[4 * i + 2] = __uint_as_float(v.r[i].z), f[4 * i + 3] = __uint_as_float(v.r[i].w);
  }
}

__device__ __forceinline__ float amax16(const float (&v)[16]) {
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(v[i]));
  return m;
}

// amax / 6 rounded to nearest for a bf16 amax: quotient by the rounded reciprocal, one residual correction (Markstein's division
// step). Exact for every bf16 value from 2^-100 up; below that the block's scale is zero whatever the quotient (the largest
// global scale is 2688 / 1e-12), so nothing depends on it. An fp32 amax takes the IEEE division.
__device__ __forceinline__ float sixth(float amax, __nv_bfloat16) {
  const float q = __fmul_rn(amax, 1.0f / 6.0f);
  return __fmaf_rn(__fmaf_rn(-6.0f, q, amax), 1.0f / 6.0f, q);
}
__device__ __forceinline__ float sixth(float amax, float) { return __fdiv_rn(amax, 6.0f); }

// quantize_block16 on values as loaded and their largest magnitude, its second division looked up and two products per instruction
template <typename T>
__device__ __forceinline__ uint32_t quantize_raw(const Raw16<T>& v, float amax, float gs, const float* table, uint2& packed) {
  const float sf_f = fminf(__fmul_rn(sixth(amax, T()), gs), 448.0f);
  uint16_t sb;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(sb) : "f"(0.0f), "f"(sf_f));
  const float scale = table[sb & 127];
  float f[16];
  floats(v, f);
#pragma unroll
  for (int i = 0; i < 16; i += 2)
    asm("{\n .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %2};\n mul.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}\n"
        : "+f"(f[i]), "+f"(f[i + 1]) : "f"(scale));
  packed = make_uint2(e2m1x8_rn(f), e2m1x8_rn(f + 8));
  return sb;
}

// maximum over the block's threads, in every thread
__device__ __forceinline__ float block_max(float m, float* wm) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
  __syncthreads();
  m = wm[threadIdx.x & 15];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// Each unit of a group does its part: with all of it in one unit the blocks of the resident form, which keep step with one another, waited
// for that one (60 x 1472 x 1984 bf16 118 us, 99 in parts; 128 x 1472 x 2048 239 and 202).
__device__ __forceinline__ void zero_padding(uint8_t* sf, const QuantGeom& q, int first, int step) {   // 128x4: rows and columns beyond the matrix
  const int prow = (q.rows + 127) & ~127, pcol = q.nkt * 4;
  const int spare = pcol - q.bpr;
  for (int i = first; i < (prow - q.rows) * pcol; i += step) sf[sf_swizzled(q.rows + i / pcol, i % pcol, q.nkt)] = 0;
  if (spare > 0)
    for (int i = first; i < q.rows * spare; i += step) sf[sf_swizzled(i / spare, q.bpr + i % spare, q.nkt)] = 0;
}

template <typename T>
__global__ void __launch_bounds__(kQThreads) k_quantize_small(const T* x, QuantGeom q, float* gs_out, uint8_t* packed, uint8_t* sf) {
  __shared__ float wm[kQThreads / 32];
  __shared__ int s_max;
  const int tid = threadIdx.x, rank = (int)cluster_ctarank(), C = (int)gridDim.x, nblk = q.rows * q.bpr;
  grid_dependency_wait();
  grid_launch_dependents();
  float v[kQSmallPerThread][16], m = 0.f;
#pragma unroll
  for (int j = 0; j < kQSmallPerThread; ++j) {
    const int i = rank * kQThreads + tid + j * C * kQThreads;
    if (i < nblk) {
      load16(x + (long long)i * 16, v[j]);
      m = fmaxf(m, amax16(v[j]));
    }
  }
  m = block_max(m, wm);
  if (tid == 0) s_max = __float_as_int(m);
  cluster_sync_all();
  int mb = 0;   // non-negative floats order like their bit patterns
  for (int c = 0; c < C; ++c) {
    int o;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(o) : "r"(mapa_shared(smem_u32(&s_max), (uint32_t)c)) : "memory");
    mb = max(mb, o);
  }
  cluster_arrive();
  const float gs = scale_of(__int_as_float(mb));
  if (rank == 0 && tid == 0) *gs_out = gs;
#pragma unroll
  for (int j = 0; j < kQSmallPerThread; ++j) {
    const int i = rank * kQThreads + tid + j * C * kQThreads;
    if (i < nblk) {
      uint2 pk;
      const uint8_t sb = quantize_block16(v[j], gs, pk);
      *reinterpret_cast<uint2*>(packed + (long long)i * 8) = pk;
      if (q.layout == 0) sf[i] = sb;
      else sf[sf_swizzled(i / q.bpr, i % q.bpr, q.nkt)] = sb;
    }
  }
  if (q.layout == 1) zero_padding(sf, q, rank * kQThreads + tid, C * kQThreads);
  cluster_wait();
}

// scratch: [0] number of the calls that have used it, [1] blocks of this call that have left (zero between calls); then one 8-byte
// word {call number + 1, bits of the largest magnitude} per amax unit. A word is stored whole, so whoever reads this call's
// number in it has the maximum: nothing is counted and nothing is fenced, and a unit's only round trip to L2 overlaps its loads.
// A quantising unit looks `polls` times for the words of its group; then its block works out what is missing by itself.
// (With a ticket per unit and counters behind a fence: 330 to 400 us for 128 x 1536 x 2048 bf16.)
template <typename T>
__global__ void __launch_bounds__(kQgThreads, 2) k_quantize_grouped(const T* x, int groups, int units, int window, QuantGeom q, float* gs_out,
                                                                    uint8_t* packed, uint8_t* sf, unsigned* scratch, int polls) {
  constexpr int kWarps = kQgThreads / 32, kPer = kQPerThread<T>;
  __shared__ unsigned wm[2][kWarps], late[kWarps];
  __shared__ float s_table[128];
  __shared__ int3 s_next[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = q.rows * q.bpr;             // 16-value blocks of a group
  const unsigned total = 2u * (unsigned)groups * (unsigned)units;
  unsigned long long* words = reinterpret_cast<unsigned long long*>(scratch + 2);
  const uint64_t once = policy_evict_first();
  grid_dependency_wait();
  grid_launch_dependents();
  const unsigned call = __ldcg(scratch) + 1u;   // nobody advances it before every block of this call has left
  float gs_table = -1.f;                        // the global scale s_table was filled for
  int k = 0;
  // maximum over the block, one barrier (the buffer of the unit before may still be read)
  auto unit_max = [&](unsigned m) {
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) wm[k][warp] = m;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, wm[k][lane & (kWarps - 1)]);
    k ^= 1;
    return m;
  };
  // place t in the order -> (group, unit, pass). One thread works it out for the next unit while the block is at the current one.
  auto place = [&](unsigned t) {
    const unsigned head = (unsigned)window * (unsigned)units, n = (unsigned)units;
    if (t >= total) return make_int3(-1, 0, 0);
    if (t < head) return make_int3((int)(t / n), (int)(t % n), 0);
    const unsigned r = t - head, pairs = (unsigned)(groups - window);
    if (r < pairs * 2u * n) {
      const unsigned p = r / (2u * n), o = r - p * 2u * n;
      return o < n ? make_int3((int)p + window, (int)o, 0) : make_int3((int)p, (int)(o - n), 1);
    }
    const unsigned o = r - pairs * 2u * n;
    return make_int3((int)(pairs + o / n), (int)(o % n), 1);
  };
  if (tid == 0) s_next[0] = place(blockIdx.x);
  __syncthreads();
  unsigned t1 = blockIdx.x + gridDim.x;        // the place that is worked out next
  auto load = [&](const int3& at, Raw16<T> (&v)[kPer]) {
    if (at.x < 0) return;
    const int i0 = at.y * (kPer * kQgThreads), left = nblk - i0 - tid;   // this thread's blocks: i0 + tid + j * threads while j * threads < left
    const T* src = x + ((long long)at.x * nblk + i0 + tid) * 16;
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if (j * kQgThreads < left) load_raw(src + j * kQgThreads * 16, q.wide, q.mark && at.z != 0, v[j]);
  };
  // The maximum of group g by this block alone, for units whose blocks have not run for a long time (another kernel holds their SMs:
  // nothing says that the grid is resident as a whole). What it finds out it publishes, so that others need not.
  constexpr unsigned kMissing = ~0u;   // above the bits of every magnitude
  auto group_max = [&](int g) {
    unsigned all = 0u;
#pragma unroll 1
    for (int w = 0; w < units; ++w) {
      unsigned long long* at = words + (long long)g * units + w;
      const unsigned long long word = ld_relaxed_gpu_u64(at);
      if (__syncthreads_and((unsigned)(word >> 32) == call)) { all = max(all, (unsigned)word); continue; }
      float m = 0.f;
      const int i1 = min(nblk, (w + 1) * (kPer * kQgThreads));
#pragma unroll 1
      for (int i = w * (kPer * kQgThreads) + tid; i < i1; i += kQgThreads) {
        Raw16<T> raw;
        load_raw(x + ((long long)g * nblk + i) * 16, q.wide, false, raw);
        m = fmaxf(m, amax_raw(raw));
      }
      unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
      if (lane == 0) late[warp] = mb;      // (read before the next round's barrier)
      __syncthreads();
      mb = __reduce_max_sync(0xffffffffu, late[lane & (kWarps - 1)]);
      if (tid == 0) __stcg(at, ((unsigned long long)call << 32) | mb);
      all = max(all, mb);
    }
    return all;
  };
  auto process = [&](const int3& at, Raw16<T> (&v)[kPer]) {
    const int g = at.x, u = at.y;
    const bool second = at.z != 0;
    unsigned long long* gw = words + (long long)g * units;
    const int i0 = u * (kPer * kQgThreads), left = nblk - i0 - tid;
    const long long first = (long long)g * nblk + i0 + tid;
    if (!second) {
      float m = 0.f;
#pragma unroll
      for (int j = 0; j < kPer; ++j)
        if (j * kQgThreads < left) m = fmaxf(m, amax_raw(v[j]));
      const unsigned mb = unit_max(__float_as_uint(m));
      if (tid == 0) __stcg(gw + u, ((unsigned long long)call << 32) | mb);
      return;
    }
    unsigned m = 0u;
    int looks = polls;
    for (int w = tid; w < units; w += kQgThreads) {
      bool ok = false;
      for (; looks > 0; --looks) {
        const unsigned long long word = ld_relaxed_gpu_u64(gw + w);
        ok = (unsigned)(word >> 32) == call;
        if (ok) { m = max(m, (unsigned)word); break; }
        __nanosleep(100);
      }
      if (!ok) { m = kMissing; break; }
    }
    m = unit_max(m);
    if (m == kMissing) {
      m = group_max(g);
      load(at, v);
    }
    const float gs = scale_of(__uint_as_float(m));
    if (gs != gs_table) {
      fill_scale_table(s_table, gs, tid, kQgThreads);
      gs_table = gs;
      __syncthreads();
    }
    uint8_t* sfg = sf + (long long)g * q.sf_stride;
    uint2* codes = reinterpret_cast<uint2*>(packed) + first;
    uint8_t* sfl = sfg + i0 + tid;                                    // row-major place
    int r = 0, c = 0;                                                 // 128x4: (row, scale column) of the block
    if (q.layout == 1) {
      r = (int)(((unsigned long long)(unsigned)(i0 + tid) * q.bpr_inv) >> q.bpr_shift);
      c = i0 + tid - r * q.bpr;
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (j * kQgThreads < left) {
        uint2 pk;
        const uint32_t sb = quantize_raw(v[j], amax_raw(v[j]), gs, s_table, pk);
        if (q.mark) st_policy(codes + j * kQgThreads, pk, once);
        else __stcg(codes + j * kQgThreads, pk);
        if (q.layout == 0) {
          sfl[j * kQgThreads] = (uint8_t)sb;
        } else {
          sfg[((r >> 7) * q.nkt + (c >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (c & 3)] = (uint8_t)sb;
          r += q.step_r, c += q.step_c;
          if (c >= q.bpr) { c -= q.bpr; ++r; }
        }
      }
    }
    if (u == 0 && tid == 0) gs_out[g] = gs;
    if (q.layout == 1) zero_padding(sfg, q, u * kQgThreads + tid, units * kQgThreads);
  };
  for (;;) {
    const int3 at = s_next[k];
    if (at.x < 0) break;
    if (tid == kQgThreads - 1) s_next[k ^ 1] = place(t1);   // read behind this unit's barrier
    t1 += gridDim.x;
    Raw16<T> v[kPer];
    load(at, v);
    process(at, v);
  }
  __syncthreads();
  if (tid == 0 && atomicAdd(scratch + 1, 1u) == gridDim.x - 1u) { scratch[1] = 0u; scratch[0] = call; }
}

// The same for bf16 groups of which the shared memory of all SMs holds more than one (one block per SM, 32 KB units taken round-robin): a
// unit is copied into shared memory once, its maximum is published, and it is quantised from there one unit of its worker later,
// when the maxima of its group have normally all been published. A block is three workers of eight warps, a copying warp and one that
// looks for the maxima. The kernel above reads every value twice into registers and is held up by latency with the 16 warps an SM that
// its registers allow (issue slots 50 % busy, DRAM 47 %); here what bounds it is the issue of about 165 instructions per 16 values (61 to 67 %
// busy), 190 before what is kept from one pass to the other: a thread's block maxima and the unit's place stay in registers, and magnitudes are compared without
// being taken first (220 us before, 208 with them, 205 with the order of load_shared, which takes 13 of 21 million conflict cycles away). 128 x 1536 x 2048 bf16, swizzled scales: 232 above; with two workers 13 % more. (fp32 has half the arithmetic per byte, and its 64-byte blocks
// meet a quarter of the banks: 60 x 1024 x 1536 take 96 us either way, or 115 here without instructions that avoid the conflicts.)
constexpr int kQcUnit = 32768, kQcSlots = 7, kQcWorkers = 3, kQcWorkerThreads = 256;
constexpr int kQcThreads = kQcWorkers * kQcWorkerThreads + 64;
constexpr int kQcLooks = 8;        // maxima that may wait for their worker
// Words of a group that a lane has in flight together, also the last few: a look at a group takes one to three round trips. (With the words of the
// last incomplete four one after the other it took up to five, and with more than three the blocks waited for it: 320 MB of bf16 in groups
// of 102 units 107 us, now 91; of 240 units 117, now 93; of 192 units 91 both. All of a group's words at once:
// 90, 93 and 92, but 128 x 1536 x 2048 with swizzled scales 210 instead of 206.6.)
constexpr int kQcWords = 4;
constexpr int kQcBlocks = kQcUnit / 32;   // 16-value blocks of a unit
struct QcShared {
  uint64_t full[kQcSlots], empty[kQcSlots], known[kQcLooks], taken[kQcLooks];
  unsigned gmax[kQcLooks];
  float table[kQcWorkers][128];
  unsigned wm[kQcWorkers][2][8], late[kQcWorkers][8];
  int abort_flag;
};
constexpr int kQcSmem = kQcSlots * kQcUnit + (int)sizeof(QcShared) + 128;

// 16 values of a thread from shared memory, the half at `first` (0 or 16) first. Neighbouring threads' blocks are 32 bytes apart: with every second four of a warp's
// threads starting with the other half, eight threads meet all banks once. A maximum does not mind the order, and two words of codes are put right more cheaply
// than eight of values.
__device__ __forceinline__ void load_shared(uint32_t at, uint32_t first, Raw16<__nv_bfloat16>& v) { v.r[0] = lds128(at ^ first), v.r[1] = lds128(at ^ first ^ 16u); }

// A wait inside the block gives up after `tries`. The warp that gave up works without what it waited for to the end of the call (a
// barrier's parity tells only whether the phase before has passed): values come from global memory, group maxima from the worker itself. The
// bytes are the same, and the block does not leave before its copies have landed.
__global__ void __launch_bounds__(kQcThreads, 1) k_quantize_resident(const __nv_bfloat16* x, int groups, int units, QuantGeom q, float* gs_out, uint8_t* packed, uint8_t* sf,
                                                                     unsigned* scratch, int polls, unsigned tries) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
  QcShared& S = *reinterpret_cast<QcShared*>(smem + kQcSlots * kQcUnit);
  constexpr int kUnitBlocks = kQcBlocks, kPer = kUnitBlocks / kQcWorkerThreads;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int nblk = q.rows * q.bpr;             // 16-value blocks of a group
  const unsigned total = (unsigned)groups * (unsigned)units, G = gridDim.x;
  const int n = (int)((total - blockIdx.x + G - 1u) / G);   // this block's units: places blockIdx.x + k * G in the order (group, unit)
  unsigned long long* words = reinterpret_cast<unsigned long long*>(scratch + 2);
  if (tid == 0) {
    for (int s = 0; s < kQcSlots; ++s) { mbar_init(&S.full[s], 1); mbar_init(&S.empty[s], 8); }
    for (int s = 0; s < kQcLooks; ++s) { mbar_init(&S.known[s], 1); mbar_init(&S.taken[s], 1); }
    S.abort_flag = 0;
    fence_mbar_init();
  }
  grid_dependency_wait();
  grid_launch_dependents();
  const unsigned call = __ldcg(scratch) + 1u;   // nobody advances it before every block of this call has left
  __syncthreads();
  constexpr unsigned kMissing = ~0u;            // above the bits of every magnitude
  auto place = [&](int k) { const unsigned p = blockIdx.x + (unsigned)k * G; return make_int2((int)(p / (unsigned)units), (int)(p % (unsigned)units)); };
  if (warp == 8 * kQcWorkers) {
    // ============================================================== copies
    if (lane == 0) {
      const uint64_t once = policy_evict_first();
      int slot = 0;
      uint32_t ph = 1;   // parity that a free slot's barrier has completed: the first pass finds all slots free
      int k = 0;
      for (; k < n; ++k) {
        const int2 at = place(k);
        const int i0 = at.y * kUnitBlocks, bytes = min(kUnitBlocks, nblk - i0) * 32;
        if (!mbar_wait(&S.empty[slot], ph, &S.abort_flag, tries)) break;
        mbar_expect_tx(&S.full[slot], bytes);
        bulk_load_hint(smem + slot * kQcUnit, x + ((long long)at.x * nblk + i0) * 16, bytes, &S.full[slot], once);
        if (++slot == kQcSlots) { slot = 0; ph ^= 1u; }
      }
      for (int j = max(0, k - kQcSlots); j < k; ++j)   // the copies that may still be under way
        for (int i = 0; i < (1 << 20) && !mbar_try_wait(&S.full[j % kQcSlots], (uint32_t)((j / kQcSlots) & 1)); ++i) {}
    }
  } else if (warp == 8 * kQcWorkers + 1) {
    // ============================================================== the maximum of each unit's group, looked at `polls` times
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
      const unsigned long long* gw = words + (long long)place(k).x * units;
      unsigned m = 0u;
      bool ok = false;
      int looks = polls;
#pragma unroll 1
      for (;;) {
        m = 0u, ok = looks > 0;
#pragma unroll 1
        for (int w0 = lane; w0 < units; w0 += 32 * kQcWords) {
          unsigned long long word[kQcWords];
#pragma unroll
          for (int i = 0; i < kQcWords; ++i)
            if (w0 + 32 * i < units) word[i] = ld_relaxed_gpu_u64(gw + w0 + 32 * i);
#pragma unroll
          for (int i = 0; i < kQcWords; ++i)
            if (w0 + 32 * i < units) { ok &= (unsigned)(word[i] >> 32) == call; m = max(m, (unsigned)word[i]); }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (ok || looks <= 0) break;
        --looks;
        __nanosleep(500);
      }
      m = __reduce_max_sync(0xffffffffu, m);
      // What a worker learns of unit k also tells it that units up to k have landed. It waits for unit k + 7 later on, in the same slot: the parity of
      // the slot's barrier says something only once the phase before is over. (That the maxima are there does not tell: another block may
      // have worked them out. Ahead of the looks this wait holds them up: 16000 x 128 x 64 93.1 us instead of 90.8.)
      if (!mbar_wait_warp(smem_u32(&S.full[k % kQcSlots]), (uint32_t)((k / kQcSlots) & 1), &S.abort_flag, tries)) break;
      if (k >= kQcLooks && !mbar_wait_warp(smem_u32(&S.taken[k % kQcLooks]), (uint32_t)((k / kQcLooks - 1) & 1), &S.abort_flag, tries)) break;
      if (lane == 0) {
        S.gmax[k % kQcLooks] = ok ? m : kMissing;
        mbar_arrive(&S.known[k % kQcLooks]);
      }
      __syncwarp();
    }
  } else {
    // ============================================================== workers: unit k belongs to worker k % kQcWorkers
    const int grp = warp >> 3, wt = tid & (kQcWorkerThreads - 1), ww = wt >> 5;
    auto sync = [&]() { named_bar_sync(1 + grp, kQcWorkerThreads); };
    const uint64_t once = policy_evict_first();
    const uint32_t ring = smem_u32(smem), first_half = (lane & 4) << 2;
    float gs_table = -1.f;
    bool copied = true, told = true;   // this warp has not given up on the copies, on the maxima
    // The largest magnitudes of this thread's blocks, of the unit that is read and of the one before, which is quantised behind it.
    float seen[kPer] = {}, kept[kPer] = {};
    // body(j, block, whether it comes from the slot) for this thread's blocks i0 + wt + j * threads of a unit. (Once a warp reads global memory it does so to the
    // end, and keeps nothing.)
    auto blocks = [&](int g, int slot, int i0, auto&& body) {
      const int left = nblk - i0 - wt;
      if (copied) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          if (j * kQcWorkerThreads < left) {
            Raw16<__nv_bfloat16> v;
            load_shared(ring + slot * kQcUnit + (wt + j * kQcWorkerThreads) * 32, first_half, v);
            body(j, v, std::true_type());
          }
        }
      } else {
#pragma unroll 1
        for (int j = 0; j < kPer && j * kQcWorkerThreads < left; ++j) {
          Raw16<__nv_bfloat16> v;
          load_raw(x + ((long long)g * nblk + i0 + wt + j * kQcWorkerThreads) * 16, q.wide, false, v);
          body(j, v, std::false_type());
        }
      }
    };
    // The maximum of group g by this worker alone, for units whose blocks have not run for a long time (another kernel holds their
    // SMs: nothing says that the grid is resident as a whole). What it finds out it publishes, so that others need not.
    auto group_max = [&](int g) {
      unsigned all = 0u;
#pragma unroll 1
      for (int w = 0; w < units; ++w) {
        unsigned long long* at = words + (long long)g * units + w;
        const unsigned long long word = ld_relaxed_gpu_u64(at);
        const bool there = (unsigned)(word >> 32) == call;   // (threads may see it differently: they agree below)
        float m = 0.f;
        const int i1 = min(nblk, (w + 1) * kUnitBlocks);
        if (!there) {
#pragma unroll 1
          for (int i = w * kUnitBlocks + wt; i < i1; i += kQcWorkerThreads) {
            Raw16<__nv_bfloat16> raw;
            load_raw(x + ((long long)g * nblk + i) * 16, q.wide, false, raw);
            m = fmaxf(m, amax_raw(raw));
          }
        }
        unsigned mb = there ? (unsigned)word : __float_as_uint(m);   // the larger of a published maximum and a part of it is the maximum
        mb = __reduce_max_sync(0xffffffffu, mb);
        if (lane == 0) S.late[grp][ww] = mb;
        sync();
        mb = __reduce_max_sync(0xffffffffu, S.late[grp][lane & 7]);
        sync();
        if (wt == 0) __stcg(at, ((unsigned long long)call << 32) | mb);
        all = max(all, mb);
      }
      return all;
    };
    int buf = 0;
    int2 next = make_int2(0, 0);
#pragma unroll 1
    for (int k = grp; k < n + kQcWorkers; k += kQcWorkers) {
      const int2 last = next;   // of unit k - kQcWorkers
#pragma unroll
      for (int j = 0; j < kPer; ++j) kept[j] = seen[j];
      if (k < n) {
        const int2 at = next = place(k);
        const int slot = k % kQcSlots;
        copied = copied && told && mbar_wait_warp(smem_u32(&S.full[slot]), (uint32_t)((k / kQcSlots) & 1), &S.abort_flag, tries);
        float m = 0.f;
        blocks(at.x, slot, at.y * kUnitBlocks, [&](int j, const Raw16<__nv_bfloat16>& v, auto held) {
          const float a = amax_raw(v);
          if constexpr (held.value) seen[j] = a;
          m = fmaxf(m, a);
        });
        __syncwarp();
        unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
        if (lane == 0) S.wm[grp][buf][ww] = mb;
        sync();
        if (ww == 0) {
          mb = __reduce_max_sync(0xffffffffu, S.wm[grp][buf][lane & 7]);
          if (lane == 0) __stcg(words + (long long)at.x * units + at.y, ((unsigned long long)call << 32) | mb);
        }
        buf ^= 1;
      }
      const int kq = k - kQcWorkers;
      if (kq < 0) continue;
      const int g = last.x, u = last.y, slot = kq % kQcSlots, i0 = u * kUnitBlocks;
      told = told && mbar_wait_warp(smem_u32(&S.known[kq % kQcLooks]), (uint32_t)((kq / kQcLooks) & 1), &S.abort_flag, tries);
      unsigned m = told ? S.gmax[kq % kQcLooks] : kMissing;
      const bool all = named_bar_and(1 + grp, kQcWorkerThreads, m != kMissing);   // (and nobody is at the table any more)
      if (wt == 0 && told) mbar_arrive(&S.taken[kq % kQcLooks]);
      if (!all) m = group_max(g);
      const float gs = scale_of(__uint_as_float(m));
      if (gs != gs_table) fill_scale_table(S.table[grp], gs, wt, kQcWorkerThreads);
      gs_table = gs;
      sync();
      uint8_t* sfg = sf + (long long)g * q.sf_stride;
      uint2* codes = reinterpret_cast<uint2*>(packed) + (long long)g * nblk + i0 + wt;
      uint8_t* sfl = sfg + i0 + wt;                                    // row-major place
      int r = 0, c = 0;                                                // 128x4: (row, scale column) of the block
      if (q.layout == 1) {
        r = (int)(((unsigned long long)(unsigned)(i0 + wt) * q.bpr_inv) >> q.bpr_shift);
        c = i0 + wt - r * q.bpr;
      }
      blocks(g, slot, i0, [&](int j, const Raw16<__nv_bfloat16>& v, auto held) {
        uint2 pk;
        float amax;
        if constexpr (held.value) amax = kept[j];
        else amax = amax_raw(v);
        const uint32_t sb = quantize_raw(v, amax, gs, S.table[grp], pk);
        if (held.value && first_half) pk = make_uint2(pk.y, pk.x);
        st_policy(codes + j * kQcWorkerThreads, pk, once);
        if (q.layout == 0) {
          sfl[j * kQcWorkerThreads] = (uint8_t)sb;
        } else {
          sfg[((r >> 7) * q.nkt + (c >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (c & 3)] = (uint8_t)sb;
          r += q.step_r, c += q.step_c;
          if (c >= q.bpr) { c -= q.bpr; ++r; }
        }
      });
      __syncwarp();
      if (lane == 0 && copied) mbar_arrive(&S.empty[slot]);
      if (u == 0 && wt == 0) gs_out[g] = gs;
      if (q.layout == 1) zero_padding(sfg, q, u * kQcWorkerThreads + wt, units * kQcWorkerThreads);
    }
  }
  __syncthreads();
  if (tid == 0 && atomicAdd(scratch + 1, 1u) == G - 1u) { scratch[1] = 0u; scratch[0] = call; }
}

}  // namespace b200

using namespace b200;

extern "C" int b200moe_global_scale(const void* x, int dtype, long long n, void* amax_scratch_u32, float* gs_out, void* stream);
extern "C" int b200moe_quantize_nvfp4(const void* x, int dtype, const int* src_row, int rows, int K, const float* global_scale, int gs_rows, void* packed,
                                      void* sf, int sf_layout, void* stream);

static int quant_resident_units(int dtype, int rows, int K) {
  return dtype == 0 ? (int)(((long long)rows * (K / 16) + kQcBlocks - 1) / kQcBlocks) : 0;
}

static int quant_units(int dtype, int rows, int K) {
  const long long nblk = (long long)rows * (K / 16), unit = kQgThreads * (dtype == 0 ? kQPerThread<__nv_bfloat16> : kQPerThread<float>);
  return (int)((nblk + unit - 1) / unit);
}

// Inputs beyond L2 take the resident form: below the line the other one is ahead, but for the smallest groups (new inputs, swizzled scales, us in this form and
// in the other: 16 x 1536 x 2048, 96 MB, 38.2 and 35.5; 60 x 704 x 1536, 124 MB, 46.5 and 45.5; 4000 x 500 x 16, 61 MB, 40.3 and 66.3), somewhat above it too
// (64 x 1024 x 1024, 128 MB, 47.6 and 45.0; 24 x 1536 x 2048, 144 MB, 51.0 and 50.1; 8400 x 500 x 16, 128 MB, 76.5 and 144), then this one is (128 x 448
// x 2048, 224 MB, 71.6 and 74.9; 128 x 1536 x 2048, 768 MB, 204 and 232).
constexpr long long kQResidentFrom = 126ll << 20;
constexpr unsigned kQTries = 1u << 20;   // of a wait inside a block, for another warp or a copy
constexpr int kQPolls = 2048;   // looks of ~0.7 us: a unit takes 5 to 10 us, so the words are there long before unless the grid is held up

static bool quant_one_cluster(int groups, int rows, int K) { return groups == 1 && (long long)rows * (K / 16) <= kQSmallMaxBlocks; }

extern "C" long long b200moe_quantize_own_scale_workspace_bytes(int dtype, int groups, int rows, int K) {
  if (groups <= 0 || rows < 0 || K <= 0 || (dtype != 0 && dtype != 1)) return B200MOE_ERR_ARG;
  if (quant_one_cluster(groups, rows, K)) return 0;
  const int a = quant_units(dtype, rows, K), b = quant_resident_units(dtype, rows, K);
  return 8 + 8LL * groups * (a > b ? a : b);
}

// Matrices beyond what the one launch can index: amax, scale and codes of one group after the other, in launches of their own.
static int quant_separate(const void* x, int dtype, int groups, int rows, int K, float* gs_out, uint8_t* packed, uint8_t* sf, int sf_layout,
                          long long sf_stride, unsigned* word, void* stream) {
  const long long n = (long long)rows * K;
  for (int g = 0; g < groups; ++g) {
    const void* xg = (const uint8_t*)x + g * n * (dtype == 0 ? 2 : 4);
    int rc = b200moe_global_scale(xg, dtype, n, word, gs_out + g, stream);
    if (rc == B200MOE_OK) rc = b200moe_quantize_nvfp4(xg, dtype, nullptr, rows, K, gs_out + g, 0, packed + g * (n / 2), sf + g * sf_stride, sf_layout, stream);
    if (rc != B200MOE_OK) return rc;
  }
  return B200MOE_OK;
}

// x [groups, rows, K] (dtype 0 bf16, 1 f32) -> gs_out f32 [groups], packed u8 [groups, rows, K/2], sf u8: sf_layout 0 row-major
// [groups, rows, K/16], 1 the 128x4 swizzle per group ([groups, pad128(rows) * pad4(K/16)], padding written 0). workspace: zeroed once,
// then only ever passed to this function; two calls that may overlap on the GPU (a replay of a captured call is one) need one each.
// Null where b200moe_quantize_own_scale_workspace_bytes says 0.
static int quantize_own_scale(const void* x, int dtype, int groups, int rows, int K, float* gs_out, void* packed, void* sf, int sf_layout, void* workspace,
                              long long workspace_bytes, int polls, unsigned tries, void* stream) {
  if (!x || !gs_out || !packed || !sf || groups <= 0 || groups > 65535 || rows < 0) return B200MOE_ERR_ARG;
  if (K <= 0 || K % 16) return B200MOE_ERR_SHAPE;
  if ((dtype != 0 && dtype != 1) || (sf_layout != 0 && sf_layout != 1)) return B200MOE_ERR_ARG;
  if (((uintptr_t)x & 15) || ((uintptr_t)packed & 7) || ((uintptr_t)workspace & 7)) return B200MOE_ERR_ARG;
  if (!workspace && !quant_one_cluster(groups, rows, K)) return B200MOE_ERR_ARG;
  if (workspace_bytes < b200moe_quantize_own_scale_workspace_bytes(dtype, groups, rows, K)) return B200MOE_ERR_WORKSPACE;
  if (rows == 0) return B200MOE_OK;
  cudaStream_t st = (cudaStream_t)stream;
  QuantGeom q;
  q.rows = rows, q.bpr = K / 16, q.layout = sf_layout, q.nkt = (q.bpr + 3) / 4;
  q.sf_stride = sf_layout == 0 ? (long long)rows * q.bpr : ((rows + 127LL) / 128 * 128) * q.nkt * 4;
  q.wide = ((uintptr_t)x & 31) == 0;
  q.bpr_shift = 30;
  for (int b = q.bpr; b; b >>= 1) ++q.bpr_shift;
  q.bpr_inv = ((1ULL << q.bpr_shift) + q.bpr - 1) / q.bpr;
  q.step_r = kQgThreads / q.bpr, q.step_c = kQgThreads % q.bpr;
  const long long nblk = (long long)rows * q.bpr;
  unsigned* scratch = (unsigned*)workspace;
  // 2^30 blocks a group and 2 GB of scales are what the kernels' 32-bit offsets hold. (The word lent here is a unit's: its flag half
  // stays as it is, so no later call takes the value for a maximum of its own.)
  if (q.sf_stride > 0x7fffffffLL || nblk > (1LL << 30))
    return quant_separate(x, dtype, groups, rows, K, gs_out, (uint8_t*)packed, (uint8_t*)sf, sf_layout, q.sf_stride, scratch + 2, stream);
  if (quant_one_cluster(groups, rows, K)) {
    int C = 1;   // CTAs: one block per thread, then two
    while (C < 8 && C * kQThreads < nblk) C *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C), cfg.blockDim = dim3(kQThreads), cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 2;
    if (dtype == 0) B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_quantize_small<__nv_bfloat16>, (const __nv_bfloat16*)x, q, gs_out, (uint8_t*)packed, (uint8_t*)sf));
    else B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_quantize_small<float>, (const float*)x, q, gs_out, (uint8_t*)packed, (uint8_t*)sf));
    return B200MOE_OK;
  }
  const int units = quant_units(dtype, rows, K);
  if (2LL * groups * units > 0x7fffffffLL) return B200MOE_ERR_LIMIT;
  long long w = kQWindowBytes / (nblk * (dtype == 0 ? 32 : 64));
  const int window = (int)(w < 1 ? 1 : w > groups ? groups : w);
  q.mark = groups > window || groups * nblk * (dtype == 0 ? 32 : 64) > kQMarkFrom;
  static int sms = 0;   // of the first device used: all devices of a machine are alike, and any grid size is correct
  if (!sms) {
    int dev = 0, n = 0;
    B200_CUDA_TRY(cudaGetDevice(&dev));
    B200_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    sms = n;
  }
  if (dtype == 0 && groups * nblk * 32 > kQResidentFrom) {
    // The resident form where a group's units are at most 1.75 rounds of the grid: beyond, the blocks wait for maxima that stand up to three rounds
    // ahead of the unit to be quantised, as many as lie between a worker's two passes over it. 320 MB of bf16, us in this form (in the other): groups of 256
    // units 93.4 (95.6), 272 109.3 (97.6), 288 106.7 (98.2), 320 102.7 (95.1), 352 102.5 (93.7).
    const int ru = quant_resident_units(dtype, rows, K);
    const long long all = (long long)groups * ru;
    const int G = (int)(all < sms ? all : sms);
    if (4LL * ru <= 7LL * G && all < 0x7fffffffLL) {
      static thread_local unsigned configured = 0;   // bit d: device d has the attribute
      int dev = 0;
      B200_CUDA_TRY(cudaGetDevice(&dev));
      if (dev > 31 || !((configured >> dev) & 1u)) {
        B200_CUDA_TRY(cudaFuncSetAttribute((const void*)k_quantize_resident, cudaFuncAttributeMaxDynamicSharedMemorySize, kQcSmem));
        if (dev <= 31) configured |= 1u << dev;
      }
      const int trips = (ru + 32 * kQcWords - 1) / (32 * kQcWords), looks = (polls + trips) / (1 + trips);   // a look takes that much longer here, with its pause
      void* args[] = {(void*)&x, (void*)&groups, (void*)&ru, (void*)&q, (void*)&gs_out, (void*)&packed, (void*)&sf, (void*)&scratch, (void*)&looks, (void*)&tries};
      return launch_kernel((const void*)k_quantize_resident, G, kQcThreads, kQcSmem, true, args, st);
    }
  }
  const long long most = 2LL * groups * units;
  const int grid = (int)(most < 2LL * sms ? most : 2LL * sms);
  void* args[] = {(void*)&x, (void*)&groups, (void*)&units, (void*)&window, (void*)&q, (void*)&gs_out, (void*)&packed, (void*)&sf, (void*)&scratch, (void*)&polls};
  return launch_kernel(dtype == 0 ? (const void*)k_quantize_grouped<__nv_bfloat16> : (const void*)k_quantize_grouped<float>, grid, kQgThreads, 0, true, args, st);
}

extern "C" int b200moe_quantize_nvfp4_own_scale(const void* x, int dtype, int groups, int rows, int K, float* gs_out, void* packed, void* sf, int sf_layout,
                                                void* workspace, long long workspace_bytes, void* stream) {
  return quantize_own_scale(x, dtype, groups, rows, K, gs_out, packed, sf, sf_layout, workspace, workspace_bytes, kQPolls, kQTries, stream);
}

// The same call that looks `polls` times for a unit's maximum before it works it out again (0: never waits), for tests of that way. Below
// zero it never waits for other blocks, and a wait inside a block gives up after -1 - polls tries.
extern "C" int b200moe_quantize_own_scale_probe(const void* x, int dtype, int groups, int rows, int K, float* gs_out, void* packed, void* sf, int sf_layout,
                                                void* workspace, long long workspace_bytes, int polls, void* stream) {
  return quantize_own_scale(x, dtype, groups, rows, K, gs_out, packed, sf, sf_layout, workspace, workspace_bytes, polls < 0 ? 0 : polls, polls < 0 ? (unsigned)(-1 - polls) : kQTries, stream);
}
