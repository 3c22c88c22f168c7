// The plan of one grouped layer call in ONE launch: router tables (experts, offsets, pairs - the same as b200moe_route, bit for
// bit), tile tables and the map between token-expert pairs and operand rows. It replaced five launches (clear, histogram,
// scan, placement, row map: 35 us of a 127 us call at 1024 tokens, most of it launch gaps).
//
// A cluster of up to eight CTAs. Every warp of the cluster owns a contiguous run of pairs and walks it in index order, 32 at a time:
// pairs of one expert are ranked by lane (match.any) on top of a running count per (warp, expert) in shared memory, so a pair's
// position is known up to the start of its warp's run. Per expert the counts are then scanned over the warps, over the CTAs
// (distributed shared memory) and over the experts; no atomic decides a position. Bound by latency (a few dependent passes of
// a microsecond each). What is scattered by row (`pairs`, `row_pair`) is written by the kernel behind this one (put_pair, one thread
// per pair on every SM): eight SMs take one 32-byte sector a cycle each, and with those stores in here a plan of
// 65536 pairs took 27 us instead of 16. A warp keeps its run's positions in registers between the two passes, up to 256 pairs.
#pragma once
#include "common.cuh"
#include "tcgen05.cuh"

namespace b200 {

constexpr int kPlanMaxE = 256;

__device__ __forceinline__ int ld_shared_cluster(uint32_t addr) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// TILE pairs per row tile (at most P / TILE + Umax tiles: the tables have room for them), ROWS operand rows per pair. row_pair
// [tiles*TILE*ROWS] = pair of every operand row of a tile (-1: none),
// dst_row[pair] = tile * TILE + slot (-1: empty slot, or an id >= E). tile_first / tile_end: first and end index into `pairs`.
struct PlanTables {   // ntiles: how many tiles, and how many experts they are of
  int *experts, *offsets, *ntiles, *tile_expert, *tile_first, *tile_end, *dst_row;
};

// The scattered tables, written behind the plan kernel. `first` = tile_first of the pair's tile (read ahead by the caller).
struct PairTables {
  const int* tile_first;
  int *pairs, *row_pair;
};
template <int TILE, int ROWS>
__device__ __forceinline__ void put_pair(const PairTables& T, int pair, int row, int first) {
  T.pairs[first + row % TILE] = pair;
  if (ROWS == 4) *reinterpret_cast<int4*>(T.row_pair + 4LL * row) = make_int4(pair, pair, pair, pair);
  else T.row_pair[row] = pair;
}

template <int TILE>
__global__ void __launch_bounds__(1024) k_plan(const int* ids, int P, int E, int Umax, PlanTables T) {
  __shared__ int wc[32][kPlanMaxE];     // pairs of expert e in warp w's run, then the start of the run in `pairs`
  __shared__ int tot[kPlanMaxE];        // ... in this CTA (read by the other CTAs)
  __shared__ int cnt[kPlanMaxE], off[kPlanMaxE], tb[kPlanMaxE];   // all pairs of expert e, its first index in `pairs`, its first tile
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = (int)cluster_ctarank();
  int C;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
  for (int i = tid; i < 32 * kPlanMaxE / 4; i += 1024) reinterpret_cast<int4*>(&wc[0][0])[i] = make_int4(0, 0, 0, 0);
  grid_dependency_wait();      // the ids, and whoever still reads the tables of the previous call
  grid_launch_dependents();    // from here on everything before this kernel is complete: the next kernel may read the call's inputs at once
  __syncthreads();
  const int L = ((P + C * 32 - 1) / (C * 32) + 31) & ~31;   // pairs per warp
  const int p0 = (rank * 32 + warp) * L, p1 = min(P, p0 + L);
  // ---- positions inside the warp's run. (expert, position) is kept in `held` until the run's start is known, or in dst_row by runs that do
  // not fit
  constexpr int kHeld = 8;
  const bool fits = L <= 32 * kHeld;
  int held[kHeld];
#pragma unroll 1
  for (int s = p0; s < p1; s += 32 * kHeld) {
#pragma unroll
    for (int k = 0; k < kHeld; ++k) held[k] = s + 32 * k + lane < p1 ? __ldcg(ids + s + 32 * k + lane) : -1;   // in flight together
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
      if (s + 32 * k >= p1) break;
      const int e = held[k] < 0 || held[k] >= E ? -1 : held[k];
      const unsigned peers = __match_any_sync(0xffffffffu, e);
      const int r = __popc(peers & ((1u << lane) - 1u));
      const int before = e >= 0 ? wc[warp][e] : 0;
      __syncwarp();
      if (e >= 0 && r == 0) wc[warp][e] = before + __popc(peers);
      held[k] = e >= 0 ? (e << 22) | (before + r) : -1;
      const int p = s + 32 * k + lane;
      if (!fits && p < p1) __stcg(T.dst_row + p, held[k]);
      __syncwarp();
    }
  }
  __syncthreads();
  if (tid < kPlanMaxE) {   // thread e: exclusive scan of expert e's counts over the warps of this CTA
    int c = 0;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) { const int v = wc[w][tid]; wc[w][tid] = c; c += v; }
    tot[tid] = c;
  }
  cluster_sync_all();
  int mine = 0;            // thread e: pairs of expert e in the CTAs before this one
  if (tid < kPlanMaxE) {
    int c = 0;
    for (int q = 0; q < C; ++q) {
      const int v = ld_shared_cluster(mapa_shared(smem_u32(&tot[tid]), (uint32_t)q));
      if (q < rank) mine += v;
      c += v;
    }
    cnt[tid] = c;
  }
  cluster_arrive();        // `tot` of every CTA has been read (waited for before exit)
  __syncthreads();
  if (warp == 0) {         // scans over the experts, eight per lane: first pair, index among the touched experts, first tile
    int c[8], sc = 0, su = 0, st = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) { c[i] = cnt[lane * 8 + i]; sc += c[i]; su += c[i] > 0; st += (c[i] + TILE - 1) / TILE; }
    int ic = sc, iu = su, it = st;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, ic, o), b = __shfl_up_sync(0xffffffffu, iu, o), d = __shfl_up_sync(0xffffffffu, it, o);
      if (lane >= o) { ic += a; iu += b; it += d; }
    }
    int rc = ic - sc, ru = iu - su, rt = it - st;
    const int routed = __shfl_sync(0xffffffffu, ic, 31), U = __shfl_sync(0xffffffffu, iu, 31), NT = __shfl_sync(0xffffffffu, it, 31);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = lane * 8 + i;
      off[e] = rc, tb[e] = rt;
      if (rank == 0 && c[i] > 0 && ru < Umax) { T.experts[ru] = e; T.offsets[ru] = rc; }
      ru += c[i] > 0, rc += c[i], rt += (c[i] + TILE - 1) / TILE;
    }
    if (rank == 0) {
      for (int u = U + lane; u < Umax; u += 32) { T.experts[u] = -1; T.offsets[u + 1] = routed; }
      if (lane == 0) {
        if (U <= Umax) T.offsets[U] = routed;
        T.ntiles[0] = NT, T.ntiles[1] = U;
      }
    }
  }
  __syncthreads();
  if (tid < kPlanMaxE) {
    const int o = tb[tid] * TILE + mine;   // from here on: operand row (TILE per tile) of the first pair of expert e in warp w's run
#pragma unroll 8
    for (int w = 0; w < 32; ++w) wc[w][tid] += o;
  }
  __syncthreads();
  // ---- the row of every pair
#pragma unroll 1
  for (int s = p0; s < p1; s += 32 * kHeld) {
    if (!fits) {
#pragma unroll
      for (int k = 0; k < kHeld; ++k) held[k] = s + 32 * k + lane < p1 ? __ldcg(T.dst_row + s + 32 * k + lane) : -1;
    }
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
      const int p = s + 32 * k + lane;
      if (p < p1) T.dst_row[p] = held[k] < 0 ? -1 : wc[warp][held[k] >> 22] + (held[k] & ((1 << 22) - 1));
    }
  }
  // ---- tile tables: one warp of the cluster per expert
  for (int e = rank * 32 + warp; e < E; e += C * 32) {
    const int c = cnt[e], nt = (c + TILE - 1) / TILE;
    for (int j = lane; j < nt; j += 32) {
      const int t = tb[e] + j;
      T.tile_expert[t] = e, T.tile_first[t] = off[e] + j * TILE, T.tile_end[t] = off[e] + c;
    }
  }
  cluster_wait();
}

// The same plan worked out by every block of the kernel that would follow k_plan, for batches of few pairs: no launch of its own, and nothing
// travels but the ids. Blocks of 128 threads. Layer calls (W4A4) with the kernel and without: 24 tokens x 8 65.1 and 62.8 us, 128 x 8 on eight
// experts 30.2 and 27.7, 20 x 6 over 256 experts 47.8 and 43.6. Above, every block's own look at all ids costs more than it saves: 2400
// pairs 42.3 and 44.7, 4000 on eight experts 47.2 and 56.8.
constexpr int kBlockPlanPairs = 1024;
struct alignas(16) BlockPlan {
  uint16_t ids[kBlockPlanPairs];           // expert of every pair, 0xffff: empty slot or an id >= E
  int cnt[kPlanMaxE], off[kPlanMaxE], tb[kPlanMaxE];   // pairs of expert e, its first index in `pairs`, its first tile
  int NT;
  int found[2];                            // of block_plan_tile
};

// tables: this block also writes the tables that are not scattered (experts, offsets, ntiles, tile_*)
template <int TILE>
__device__ __forceinline__ void block_plan(const int* ids, int P, int E, int Umax, const PlanTables& T, bool tables, BlockPlan& B) {
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < kPlanMaxE; e += 128) B.cnt[e] = 0;
  __syncthreads();
#pragma unroll 1
  for (int p0 = 0; p0 < P; p0 += 1024) {
    int v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = p0 + k * 128 + tid < P ? __ldcg(ids + p0 + k * 128 + tid) : -1;   // in flight together
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool ok = v[k] >= 0 && v[k] < E;
      B.ids[p0 + k * 128 + tid] = ok ? (uint16_t)v[k] : (uint16_t)0xffff;
      if (ok) atomicAdd(&B.cnt[v[k]], 1);
    }
  }
  __syncthreads();
  if (tid < 32) {   // scans over the experts, eight per lane, as in k_plan
    int c[8], sc = 0, su = 0, st = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) { c[i] = B.cnt[lane * 8 + i]; sc += c[i]; su += c[i] > 0; st += (c[i] + TILE - 1) / TILE; }
    int ic = sc, iu = su, it = st;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, ic, o), b = __shfl_up_sync(0xffffffffu, iu, o), d = __shfl_up_sync(0xffffffffu, it, o);
      if (lane >= o) { ic += a; iu += b; it += d; }
    }
    int rc = ic - sc, ru = iu - su, rt = it - st;
    const int routed = __shfl_sync(0xffffffffu, ic, 31), U = __shfl_sync(0xffffffffu, iu, 31), NT = __shfl_sync(0xffffffffu, it, 31);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = lane * 8 + i;
      B.off[e] = rc, B.tb[e] = rt;
      if (tables && c[i] > 0 && ru < Umax) { T.experts[ru] = e; T.offsets[ru] = rc; }
      ru += c[i] > 0, rc += c[i], rt += (c[i] + TILE - 1) / TILE;
    }
    if (lane == 0) B.NT = NT;
    if (tables) {
      for (int u = U + lane; u < Umax; u += 32) { T.experts[u] = -1; T.offsets[u + 1] = routed; }
      if (lane == 0) {
        if (U <= Umax) T.offsets[U] = routed;
        T.ntiles[0] = NT, T.ntiles[1] = U;
      }
    }
  }
  __syncthreads();
  if (tables)
    for (int e = tid; e < E; e += 128) {
      const int c = B.cnt[e], nt = (c + TILE - 1) / TILE;
      for (int j = 0; j < nt; ++j) {
        const int t = B.tb[e] + j;
        T.tile_expert[t] = e, T.tile_first[t] = B.off[e] + j * TILE, T.tile_end[t] = B.off[e] + c;
      }
    }
}

// Operand row of pair p, -1 for an empty slot; first = tile_first of its tile. For a whole warp.
template <int TILE>
__device__ __forceinline__ int block_plan_row(const BlockPlan& B, int p, int* first) {
  const int e = B.ids[p], lane = threadIdx.x & 31;
  if (e == 0xffff) return -1;
  const uint32_t ee = (uint32_t)e | ((uint32_t)e << 16);
  int n = 0;   // pairs of the expert before p: eight ids a lane
  for (int q = lane * 8; q < p; q += 256) {
    const uint4 w = *reinterpret_cast<const uint4*>(B.ids + q);
    const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t eq = __vcmpeq2(x[i], ee);
      if (q + 2 * i >= p) eq = 0u;
      else if (q + 2 * i + 1 >= p) eq &= 0xffffu;
      n += __popc(eq) >> 4;
    }
  }
  n = __reduce_add_sync(0xffffffffu, n);
  *first = B.off[e] + n / TILE * TILE;
  return B.tb[e] * TILE + n;
}

// Expert of tile t and how many of its pairs lie in it or behind, for the whole block; t < NT.
template <int TILE>
__device__ __forceinline__ int2 block_plan_tile(BlockPlan& B, int t) {
  __syncthreads();
  for (int e = threadIdx.x; e < kPlanMaxE; e += 128) {
    const int j = t - B.tb[e];
    if (j >= 0 && j * TILE < B.cnt[e]) { B.found[0] = e; B.found[1] = B.cnt[e] - j * TILE; }
  }
  __syncthreads();
  return make_int2(B.found[0], B.found[1]);
}

// One cluster, as many CTAs as the pairs keep busy: 512 pairs a CTA (two steps of 32 for half of its warps) up to eight CTAs.
template <int TILE>
inline int launch_plan(const int* ids, int P, int E, int Umax, PlanTables T, cudaStream_t st) {
  const int C = P <= 1024 ? 1 : P <= 2048 ? 2 : P <= 4096 ? 4 : 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C), cfg.blockDim = dim3(1024), cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = 2;
  B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_plan<TILE>, ids, P, E, Umax, T));
  return B200MOE_OK;
}

}  // namespace b200
