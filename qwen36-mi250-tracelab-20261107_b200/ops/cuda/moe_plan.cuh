// The expert plan of the MoE block: (row, pair) -> expert table in, expert-sorted layout out (rows per expert,
// offsets, token-tile table, positions of the pairs), as one CTA, as the tail of the routing launch, or split into
// a grid-wide histogram + a scan by the last CTA + a grid-wide scatter. Used by elementwise.cu; kept in a header of
// its own so that the same source also compiles as host C++ for tests/emu (threads, barriers, shuffles and atomics
// then come from the shim).
#pragma once

#ifdef B200_EMU
#include "emu_shim.h"
#else
#include "common.cuh"
#endif
#include "moe_route.cuh"

namespace b200 {

// Rows per tile of an expert with c rows in t tiles. Tiles of 256 rows share an expert's rows evenly, in the steps of 32 that
// their MMAs take: 272 rows as 160 + 112 and not 256 + 16, whose second tile waits for its weights only (gate/up of 8192
// rows, about 256 per expert: 336 -> 324 us).
__device__ __forceinline__ int tile_rows(int c, int t, int bt) {
  return bt < 256 || t < 2 ? bt : ((c + t - 1) / t + 31) / 32 * 32;
}

// One CTA of 1024 threads turns the (row, pair) -> expert table into everything the grouped GEMMs need, without
// global atomics or a zeroed workspace: rows per expert (shared-memory histogram), exclusive offsets (experts laid
// out in id order, rows of one expert contiguous), the token-tile table (expert, row0, nrows) and its length, and
// the position of every pair in the expert-sorted order (perm / inv). The order inside an expert does not influence
// any output value: every sorted row is computed on its own.
template <int KEEP>
__device__ void plan_scatter(const int* idx, int n_pairs, int Et, int bt, int* offsets, int4* tiles, int* n_tiles,
                             int max_tiles, int* perm, int* inv, int* err, int P, int* src_rows,
                             const int* s_idx = nullptr) {
  // `s_idx`: the same table in shared memory, where the caller has it
  __shared__ int s_count[1024], s_off[1024], s_cur[1024];
  __shared__ int w_rows[32], w_tiles[32];
  const int e = threadIdx.x, lane = e & 31, w = e >> 5;
  s_count[e] = 0;
  s_cur[e] = 0;
  __syncthreads();
  const auto fetch = [&](int i) {
    return s_idx ? s_idx[i] : __ldcg(idx + i);  // through L2: other CTAs of the same launch may have written it
  };
  // A thread keeps its first KEEP pairs and the places that counting them gave them among their expert's, so that they need no
  // second fetch and no second counter (every row counts at the shared expert: its counter is what such a walk waits for). The
  // pairs behind those are counted first and take the first places by a second walk. Five are what 512 rows of nine pairs
  // need; with the few of up to 32 rows the empty turns cost the CTA 0.6 us of 6.5, which keeps one (block of 1 row 28.5 ->
  // 27.8 us, of 13 101.4 -> 100.8).
  if (n_pairs > KEEP * 1024) {
    for (int i = KEEP * 1024 + threadIdx.x; i < n_pairs; i += blockDim.x) {
      const int x = fetch(i);
      if (x >= 0 && x < Et) atomicAdd(&s_count[x], 1);
    }
    __syncthreads();
  }
  int mine[KEEP], place[KEEP];
#pragma unroll
  for (int u = 0; u < KEEP; ++u) {
    const int i = u * 1024 + threadIdx.x;
    mine[u] = i < n_pairs ? fetch(i) : -1;
  }
#pragma unroll
  for (int u = 0; u < KEEP; ++u) place[u] = mine[u] >= 0 && mine[u] < Et ? atomicAdd(&s_count[mine[u]], 1) : 0;
  __syncthreads();
  const int c = e < Et ? s_count[e] : 0;
  const int t = (c + bt - 1) / bt;
  int sc = c, stl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, sc, o), b2 = __shfl_up_sync(0xffffffffu, stl, o);
    if (lane >= o) { sc += a; stl += b2; }
  }
  if (lane == 31) { w_rows[w] = sc; w_tiles[w] = stl; }
  __syncthreads();
  if (w == 0) {
    int a = w_rows[lane], b2 = w_tiles[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b2, o);
      if (lane >= o) { a += x; b2 += y; }
    }
    w_rows[lane] = a; w_tiles[lane] = b2;
  }
  __syncthreads();
  const int row0 = sc - c + (w ? w_rows[w - 1] : 0);    // exclusive prefix
  const int tile0 = stl - t + (w ? w_tiles[w - 1] : 0);
  s_off[e] = row0;
  if (e < Et) {
    offsets[e] = row0;
    const int rows = tile_rows(c, t, bt);
    for (int i = 0, ti = tile0; i * rows < c && ti < max_tiles; ++i, ++ti)
      tiles[ti] = make_int4(e, row0 + i * rows, min(rows, c - i * rows), 0);
  }
  if (e == Et - 1) {
    offsets[Et] = row0 + c;
    const int total = tile0 + t;
    *n_tiles = total < max_tiles ? total : max_tiles;
  }
  __syncthreads();
  const auto put = [&](int i, int x, int at) {
    if (x < 0) { inv[i] = -1; return; }  // pair served by another rank
    if (x >= Et) { atomicCAS(err, 0, ERR_BAD_INDEX); inv[i] = -1; return; }
    const int pos = s_off[x] + at;
    perm[pos] = i;
    inv[i] = pos;
    if (src_rows) src_rows[pos] = i / P;  // the activation row behind sorted position pos (for a gathering GEMM)
  };
#pragma unroll
  for (int u = 0; u < KEEP; ++u) {
    const int i = u * 1024 + threadIdx.x;
    if (i < n_pairs) put(i, mine[u], place[u]);
  }
  for (int i = KEEP * 1024 + threadIdx.x; i < n_pairs; i += blockDim.x) {
    const int x = fetch(i);
    put(i, x, x >= 0 && x < Et ? atomicAdd(&s_cur[x], 1) : 0);
  }
}

__global__ void __launch_bounds__(1024)
moe_plan_kernel(const int* idx, int n_pairs, int Et, int bt, int* offsets, int4* tiles, int* n_tiles, int max_tiles,
                int* perm, int* inv, int* err, int P, int* src_rows) {
  pdl_wait();
  pdl_launch();
  plan_scatter<5>(idx, n_pairs, Et, bt, offsets, tiles, n_tiles, max_tiles, perm, inv, err, P, src_rows);
}

// Decode-size batches: routing of every row (one warp each, 32 warps) and the plan in ONE launch.
template <int PER_LANE>
__global__ void __launch_bounds__(1024)
moe_route_plan_kernel(const float* logits, int ldl, int T, int E, int top_k, int shared, float* wts, int* idx,
                      const int* expert_map, int Et, int bt, int* offsets, int4* tiles, int* n_tiles, int max_tiles,
                      int* perm, int* inv, int* err, int* src_rows) {
  pdl_wait();
  pdl_launch();
  const int P = top_k + (shared ? 1 : 0);
  const int lane = threadIdx.x & 31;
  // The plan reads the index table twice: from shared memory where it fits (it does up to 32 rows), which spares the small
  // step two trips to L2 (5.7 -> 4.6 us at one row, the reductions of route_row included).
  __shared__ int s_idx[32 * 33];
  const bool fits = T * P <= 32 * 33;
  int* dst = fits ? s_idx : idx;
  for (int r = threadIdx.x >> 5; r < T; r += 32)
    route_row<PER_LANE>(logits + static_cast<size_t>(r) * ldl, E, top_k, shared, wts + static_cast<size_t>(r) * P,
                        dst + static_cast<size_t>(r) * P, expert_map, nullptr, lane);
  __syncthreads();  // this CTA wrote the table: visible to all its threads after the barrier
  if (fits)
    for (int i = threadIdx.x; i < T * P; i += blockDim.x) idx[i] = s_idx[i];
  plan_scatter<1>(idx, T * P, Et, bt, offsets, tiles, n_tiles, max_tiles, perm, inv, err, P, src_rows, fits ? s_idx : nullptr);
}

// Any number of rows, still one launch: a grid of 1024-thread CTAs routes up to 32 rows each, shared evenly (a row is one warp's
// 500 instructions, and 32 of them on one SM wait for each other); the CTA that finishes last
// (a ticket counter in global memory, which it puts back to zero for the next launch) builds the plan from the whole
// index table. Everything the other CTAs wrote is visible to it: they fence before taking their ticket.
// `work` (optional): 2 * 1024 ints kept zero between launches (per-expert counts, per-expert cursors). With it the
// CTAs add their rows' expert counts to the global histogram and the last CTA only turns the counts into offsets and
// the tile table (a scan over the experts); the positions of the pairs are then handed out by a second, grid-wide
// launch (moe_scatter_kernel). Without it the last CTA does everything, which is right up to a few hundred rows: at
// 8192 rows the single CTA's histogram and scatter of 73,728 pairs took 87 us per layer.
template <int PER_LANE>
__global__ void __launch_bounds__(1024)
moe_route_plan_grid_kernel(const float* logits, int ldl, int T, int E, int top_k, int shared, float* wts, int* idx,
                           const int* expert_map, int Et, int bt, int* offsets, int4* tiles, int* n_tiles,
                           int max_tiles, int* perm, int* inv, int* err, int* src_rows, unsigned int* ticket, int* work) {
  pdl_wait();
  pdl_launch();
  __shared__ int s_last;
  __shared__ int s_hist[1024];
  const int P = top_k + (shared ? 1 : 0);
  const int lane = threadIdx.x & 31;
  const int rows = (T + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);  // at most 32
  const int row0 = blockIdx.x * rows, r = row0 + (threadIdx.x >> 5);
  if (work) s_hist[threadIdx.x] = 0;
  if (r < min(T, row0 + rows))
    route_row<PER_LANE>(logits + static_cast<size_t>(r) * ldl, E, top_k, shared, wts + static_cast<size_t>(r) * P,
                        idx + static_cast<size_t>(r) * P, expert_map, nullptr, lane);
  if (work) {
    __syncthreads();  // this CTA's 32 rows of idx are written (and visible to the CTA)
    const int n_here = max(0, min(rows, T - row0)) * P;
    for (int i = threadIdx.x; i < n_here; i += blockDim.x) {
      const int x = idx[static_cast<size_t>(row0) * P + i];
      if (x >= 0 && x < Et) atomicAdd(&s_hist[x], 1);
    }
    __syncthreads();
    if (threadIdx.x < Et && s_hist[threadIdx.x]) atomicAdd(&work[threadIdx.x], s_hist[threadIdx.x]);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int t = atomicAdd(ticket, 1u);
    s_last = t == gridDim.x - 1;
    if (s_last) *ticket = 0;  // every CTA has taken its ticket: ready for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (work == nullptr) {
    plan_scatter<5>(idx, T * P, Et, bt, offsets, tiles, n_tiles, max_tiles, perm, inv, err, P, src_rows);
    return;
  }
  // counts -> offsets and tile table (one thread per expert), counts and cursors back to zero
  __shared__ int w_rows[32], w_tiles[32];
  const int e = threadIdx.x, w = e >> 5;
  const int c = e < Et ? __ldcg(work + e) : 0;
  if (e < Et) { work[e] = 0; work[1024 + e] = 0; }
  const int t = (c + bt - 1) / bt;
  int sc = c, stl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, sc, o), b2 = __shfl_up_sync(0xffffffffu, stl, o);
    if (lane >= o) { sc += a; stl += b2; }
  }
  if (lane == 31) { w_rows[w] = sc; w_tiles[w] = stl; }
  __syncthreads();
  if (w == 0) {
    int a = w_rows[lane], b2 = w_tiles[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b2, o);
      if (lane >= o) { a += x; b2 += y; }
    }
    w_rows[lane] = a; w_tiles[lane] = b2;
  }
  __syncthreads();
  const int at = sc - c + (w ? w_rows[w - 1] : 0);
  const int tile0 = stl - t + (w ? w_tiles[w - 1] : 0);
  if (e < Et) {
    offsets[e] = at;
    const int step = tile_rows(c, t, bt);
    for (int i = 0, ti = tile0; i * step < c && ti < max_tiles; ++i, ++ti)
      tiles[ti] = make_int4(e, at + i * step, min(step, c - i * step), 0);
  }
  if (e == Et - 1) {
    offsets[Et] = at + c;
    const int total = tile0 + t;
    *n_tiles = total < max_tiles ? total : max_tiles;
  }
}

// Second half of the plan at prefill sizes: every pair takes a free position of its expert's run (the order inside an expert
// does not influence any output). A CTA counts the pairs of SCATTER_PAIRS in shared memory, takes that many places of each
// expert at once (a global cursor per expert, zero before the launch) and hands them out. One global atomic per pair made
// the launch wait for the shared expert's cursor, which every row takes a place of: 8192 rows 16.2 -> 4.9 us, 2048: 5.4 -> 4.1.
constexpr int SCATTER_PER = 4;  // pairs per thread
__global__ void __launch_bounds__(256)
moe_scatter_kernel(const int* idx, int n_pairs, int Et, const int* offsets, int* cursors, int* perm, int* inv, int* err, int P,
                   int* src_rows) {
  __shared__ int s_count[1024], s_base[1024];
  pdl_wait();
  pdl_launch();
  for (int first = blockIdx.x * blockDim.x * SCATTER_PER; first < n_pairs; first += gridDim.x * blockDim.x * SCATTER_PER) {
    for (int e = threadIdx.x; e < Et; e += blockDim.x) s_count[e] = 0;
    __syncthreads();
    int x[SCATTER_PER], place[SCATTER_PER];
#pragma unroll
    for (int u = 0; u < SCATTER_PER; ++u) {
      const int i = first + u * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
      x[u] = i < n_pairs ? idx[i] : -1;
    }
#pragma unroll
    for (int u = 0; u < SCATTER_PER; ++u) place[u] = x[u] >= 0 && x[u] < Et ? atomicAdd(&s_count[x[u]], 1) : 0;
    __syncthreads();
    for (int e = threadIdx.x; e < Et; e += blockDim.x)
      if (s_count[e]) s_base[e] = offsets[e] + atomicAdd(&cursors[e], s_count[e]);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < SCATTER_PER; ++u) {
      const int i = first + u * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
      if (i >= n_pairs) continue;
      if (x[u] < 0) { inv[i] = -1; continue; }  // pair served by another rank
      if (x[u] >= Et) { atomicCAS(err, 0, ERR_BAD_INDEX); inv[i] = -1; continue; }
      const int pos = s_base[x[u]] + place[u];
      perm[pos] = i;
      inv[i] = pos;
      if (src_rows) src_rows[pos] = i / P;
    }
    __syncthreads();  // the counters are cleared again
  }
}

}  // namespace b200
