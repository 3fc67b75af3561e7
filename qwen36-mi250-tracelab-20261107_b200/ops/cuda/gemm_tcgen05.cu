// Weight-stationary ("swap-AB") bf16 GEMM on the sm_100a tensor cores.
//
//   out[t, n] = sum_k X[t, k] * W[n, k]          X: [T, K] activations, W: [N, K] weights
//
// The MMA's M dimension (128 TMEM lanes) runs over *weight rows*, its N dimension over
// *token rows* (16..256 per tile). A decode step with a handful of rows and a prefill pass
// with thousands therefore use the same instruction shape along K; the accumulation order of
// one output element never depends on how many other rows share the launch, which is what
// keeps a request's greedy tokens identical whether it is served alone or in a batch (the
// reference gets the same property from fixed GEMV tiles, engine/fast/mfma.py:6-11, 60-71).
//
// Pipeline per CTA (192 threads): warp 0 = TMA producer, warp 1 = tcgen05.mma issuer and TMEM
// owner, warps 2..5 = epilogue (one TMEM lane quarter each); the 128-row gate/up tiles have a seventh warp that
// fetches half of the rows by index. Operand tiles are 64 bf16 wide
// (128 bytes, TMA 128B swizzle), STAGES deep, guarded by full/empty mbarriers; tcgen05.commit
// releases a stage when the MMAs that read it have finished. No load uses cluster multicast; the commits of the two-SM form
// (gemm_pair.cuh) arrive at both of its CTAs that way.
//
// Variants (template): plain store (bf16 or fp32), SiLU(gate)*up over two accumulators,
// per-tile argmax partials for the LM head, and a grouped mode where a device-side tile table
// names (expert, first row, row count) for each token tile of an expert-sorted activation
// buffer (replaces the reference's Triton GEMV / grouped GEMM family: engine/fast/mfma.py:90-179,
// engine/fast/moe_prefill.py:156-319, engine/fast/fused.py:581-692).
#include "comm.cuh"

namespace b200 {

constexpr int BM = 128;  // weight rows per tile (TMEM lanes)
constexpr int BK = 64;   // bf16 per operand row per stage (128 bytes)
constexpr int GATHER_BT_MAX = 128;  // widest token tile whose rows the grouped GEMM's producer warps can fetch by index
constexpr int UMMA_K = 16;
constexpr int VAR_BOX = 32;  // rows per activation load of a wide expert tile: a tile with 40 rows loads 64
constexpr int MAX_DEVICES = 64;  // per-device launch state (function attributes, SM counts)

enum Epilogue : int { EPI_BF16 = 0, EPI_F32 = 1, EPI_SILU_MUL = 2, EPI_ARGMAX = 3, EPI_ALLREDUCE = 4, EPI_SCATTER = 5, EPI_REDUCE_SCATTER = 6 };

struct GemmParams {
  int N;             // weight rows (per expert when grouped)
  int K;
  int T;             // activation rows (dense) or capacity of the sorted buffer (grouped)
  int ldo;           // output row stride in elements
  void* out;         // bf16 or fp32 [T, ldo]
  const int4* tiles; // grouped: (expert, row0, nrows, 0) per token tile
  const int* n_tiles;// grouped: number of valid entries in `tiles`
  int up_offset;     // EPI_SILU_MUL: row offset of the "up" half inside W
  float* part_max;   // EPI_ARGMAX: [n_tiles_n, T]
  int* part_idx;     // EPI_ARGMAX: [n_tiles_n, T]
  int* err;          // error word (0 = ok)
  const bf16* residual; // EPI_ALLREDUCE: optional [T, ldo] added after the cross-rank sum
  CommCtx comm;      // EPI_ALLREDUCE: the rank group's symmetric buffers
  int rows_per_rank; // EPI_REDUCE_SCATTER / gathered X: token rows owned by each rank (a multiple of the token tile)
  const uint32_t* x_flags;  // gathered X: per-owner arrival epochs of this rank's full activation buffer (or null)
  const uint32_t* x_epoch;  // gathered X: the epoch the current call waits for
  int splits;        // split-K: CTAs of one cluster share an output tile, each taking 1/splits of the k-blocks
  const int2* meta;  // EPI_SCATTER: (source rank, pair slot) of every sorted row
  bf16* pair_out[MAX_RANKS];  // EPI_SCATTER: every rank's pair-output buffer [pairs, ldo] as mapped here
  int y_rot;         // dense sequence-parallel GEMMs: token tile = (blockIdx.y + y_rot) % gridDim.y, so that each rank
                     // starts with the tiles whose data (or whose consumer) is furthest from being the bottleneck
  int grid_y;        // dense: number of token tiles (set by the launcher)
  const int* gather_rows;  // grouped, token tiles <= GATHER_BT_MAX rows: sorted position -> row of `gx`; the producer warp then
                     // fetches each activation row by index (16-byte async copies into the swizzled operand layout)
                     // instead of reading an expert-sorted copy through the tensor map
  const bf16* gx;    // gather source [rows, ldgx]
  int ldgx;
  int packed;        // W is stored tile by tile: [expert][weight tile][k-block][128 * A_TILES rows][64], each (tile,
                     // k-block) one contiguous 16 KB (32 KB with the up half) run, so a stage is one sequential DRAM read
  int w_tiles;       // packed: weight tiles per expert
  int x_rows;        // dense, not thin: rows per activation box (0: the token tile). With a single token tile it is the row
                     // count rounded up to 16: the MMA covers and shared memory takes no more columns than there are rows
  int pair_bt;       // gemm_pair_kernel, dense: token rows per tile
};

// RT: weight rows per tile. 128 fills the MMA's M; the thin forms (64, 32) exist for launches whose 128-row tiles would leave
// most SMs without work. Their MMA has 64 rows where the tile has no more: it reads half as much shared memory (27 cycles per
// instruction of 16 columns, not 42). An accumulator row depends on its own operand row only and is the same in both
// instructions; rows that a 32-row tile does not have are whatever shared memory holds behind it, and are never read back.
// A thin gate/up tile is one operand: RT gate rows and the RT up rows behind them, one MMA for both.
// KPS: k-blocks per pipeline stage. One trip through the pipeline (wait, expect, TMA, wait, MMAs, commit) costs a CTA about
// 0.2 us however little it moves, and at decode sizes a CTA's time is the sum of its trips; a stage of KPS k-blocks comes
// with one TMA instruction per operand. Thin tiles of tile-packed weights only.
template <int BT, int EPI, int RT = BM, int KPS = 1>
struct Cfg {
  static constexpr int A_TILES = (EPI == EPI_SILU_MUL) ? 2 : 1;
  static constexpr int A_BYTES = RT * BK * 2;
  static constexpr int B_BYTES = BT * BK * 2;
  static constexpr int STAGE_BYTES = KPS * (A_TILES * A_BYTES + B_BYTES);
  static constexpr int A_STEP = A_TILES * A_BYTES;  // bytes between the k-blocks of a stage
  static constexpr int B_OFF = KPS * A_TILES * A_BYTES;
  static constexpr bool THIN = RT < BM;
  static constexpr bool MERGED = THIN && EPI == EPI_SILU_MUL;  // gate and up rows in one accumulator
  static constexpr int A_ROWS = MERGED ? 2 * RT : RT;          // operand rows of an MMA
  static constexpr int MMA_M = A_ROWS <= 64 ? 64 : 128;        // accumulator row r: TMEM lane r, or 32 (r / 16) + r % 16 of 64
  // Wide expert tiles (prefill): the MMA's N follows the tile's row count (a 128-row tile with 40 rows costs 48 columns and
  // loads 64 rows), and two producer warps fetch the rows by index. Grouped launches only. What bounds the expert GEMMs is
  // shared memory: each k-block is written once and its weight half is read again for every MMA, so a wider tile moves
  // fewer bytes per product. Gate/up at 8192 rows of 9 pairs: 496 us with 64-row tiles, 365 with these (L2 prefetches of
  // the weights 4 to 16 k-blocks ahead made it 388 to 419). Plain weights only: packed ones take two SMs (gemm_pair.cuh).
  static constexpr bool VAR_N = BT == 128 && (EPI == EPI_SILU_MUL || EPI == EPI_BF16);
  static constexpr int GATHER_WARPS = (BT == 128 && EPI == EPI_SILU_MUL) ? 2 : 1;
  // Staged stores: 16 token rows at a time go through shared memory and leave as 16-byte pieces of 256-byte rows, instead of
  // 16 two-byte-per-lane stores per warp. Input projection and output projection of a pass, mean: 195 -> 186 us at 8192
  // rows, 57 -> 52 at 2048, 47 -> 42 at 1531 (one 256-byte bulk copy per row instead: no better, and 20 us slower in the
  // down projection).
  static constexpr bool STAGED = !THIN && BT >= 64 && (EPI == EPI_SILU_MUL || EPI == EPI_BF16);
  static constexpr int OUT_BUFS = STAGED ? 2 : 0;
  static constexpr int OUT_BYTES = OUT_BUFS * 16 * BM * 2;
  // small token tiles (decode) leave room for two CTAs per SM: one CTA's pipeline fill and epilogue
  // overlap the other's main loop, which matters when K is short (the MoE down projection has 8 k-blocks)
  // The fused gate/up GEMM at 16-row token tiles and plain weights (packed ones take thin tiles) runs three CTAs per SM with
  // two deep stages each: the same bytes in flight per SM, but a decode step's ~1300 tiles then fill 2.9 waves of 444 CTAs
  // instead of 4.4 waves of 296, and the partial last wave is what the weight-streaming time loses.
  // Thin tiles of four k-blocks per stage run alone on their SM, with all of its shared memory: more bytes on their way, and
  // one commit for two stages.
  static constexpr bool SOLO = THIN && KPS == 4;
  static constexpr int CTAS_PER_SM = SOLO ? 1 : THIN ? 2 : (BT <= 16 && EPI == EPI_SILU_MUL) ? 3 : BT <= 64 ? 2 : 1;
  static constexpr int BUDGET = SOLO ? 200 * 1024 : MERGED ? 108 * 1024 : THIN ? 96 * 1024 : CTAS_PER_SM == 3 ? 72 * 1024 : BT <= 64 ? 108 * 1024 : 200 * 1024;
  static constexpr int STAGES_RAW = BUDGET / STAGE_BYTES;
  // Stages that are released together, by one commit. A commit drains the tensor core: n MMAs and their commit take F + n e
  // cycles, with (F, e) = (281, 42) for 128 x 16, (332, 27) for 64 x 16, (192, 66) for 128 x 128; at 128 x 256 F is hidden.
  static constexpr int GROUP = SOLO && STAGES_RAW >= 4 ? 2 : 1;
  static constexpr int STAGES = (STAGES_RAW > 8 ? 8 : STAGES_RAW) / GROUP * GROUP;
  static constexpr int ACC_COLS = (MERGED ? 1 : A_TILES) * BT;  // one accumulator stage
  // two accumulator stages whenever they fit (512 columns per SM shared by the resident CTAs): the epilogue of
  // one tile then overlaps the main loop of the CTA's next tile
  static constexpr int ACC_STAGES = (2 * ACC_COLS * CTAS_PER_SM <= 512) ? 2 : 1;
  static constexpr int TMEM_COLS_RAW = ACC_COLS * ACC_STAGES;
  static constexpr int TMEM_COLS = TMEM_COLS_RAW <= 32 ? 32 : TMEM_COLS_RAW <= 64 ? 64 : TMEM_COLS_RAW <= 128 ? 128 : TMEM_COLS_RAW <= 256 ? 256 : 512;
  static constexpr int OVERREAD = (MMA_M - A_ROWS) * BK * 2;  // bytes behind the last stage that a thin tile's MMA may read
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + (OVERREAD > 256 ? OVERREAD : 256) /*barriers first*/ + OUT_BYTES;
};

// Whether `ok` holds in all 128 epilogue threads.
__device__ __forceinline__ bool epilogue_all(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.aligned.pred q, 2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"(static_cast<uint32_t>(ok)) : "memory");
  return r != 0;
}

// Largest of a warp's 32 weight rows (lanes; row n of this lane's column values v, left out where !n_ok) for each of 16 token
// columns, lowest row on ties. Lanes with bit 0 clear end with one column each, named by their bits 4..1 (argmax_column).
// Halves the columns a lane carries at every exchange instead of reducing each column over the whole warp (24 shuffles for 16
// columns instead of 160). This epilogue, not the weight stream, set the LM head's time: 321 -> 202 us for 256 rows x 248320 x
// 2048, 171 -> 154 us for 128.
__device__ __forceinline__ void argmax_columns(const float* v, int n, bool n_ok, int lane, float& best, int& at) {
  float m[16];
  int id[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) { m[j] = n_ok ? v[j] : -INFINITY; id[j] = n; }
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1) {
    const int o = 2 * w;
    const bool hi = lane & o;
#pragma unroll
    for (int j = 0; j < w; ++j) {
      const float sm = hi ? m[j] : m[j + w];
      const int si = hi ? id[j] : id[j + w];
      float km = hi ? m[j + w] : m[j];
      int ki = hi ? id[j + w] : id[j];
      const float om = __shfl_xor_sync(0xffffffffu, sm, o);
      const int oi = w == 8 ? (n ^ 16) : __shfl_xor_sync(0xffffffffu, si, o);
      if (om > km || (om == km && oi < ki)) { km = om; ki = oi; }
      m[j] = km; id[j] = ki;
    }
  }
  const float om = __shfl_xor_sync(0xffffffffu, m[0], 1);
  const int oi = __shfl_xor_sync(0xffffffffu, id[0], 1);
  if (om > m[0] || (om == m[0] && oi < id[0])) { m[0] = om; id[0] = oi; }
  best = m[0];
  at = id[0];
}
__device__ __forceinline__ int argmax_column(int lane) {
  return ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
}

template <int BT, int EPI, bool GROUPED, bool SPLIT = false, int RT = BM, int KPS = 1>
__global__ void __launch_bounds__(GROUPED ? 160 + 32 * Cfg<BT, EPI, RT, KPS>::GATHER_WARPS : 192, Cfg<BT, EPI, RT, KPS>::CTAS_PER_SM)
gemm_swapab_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, GemmParams p) {
  using C = Cfg<BT, EPI, RT, KPS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::STAGES * C::STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + C::STAGES;
  uint64_t* acc_full = bars + 2 * C::STAGES;   // [2]
  uint64_t* acc_empty = bars + 2 * C::STAGES + 2;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * C::STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* out_stage = smem + C::STAGES * C::STAGE_BYTES + 256;  // behind the barriers
  constexpr int RED = EPI == EPI_ARGMAX ? BT : 1;
  __shared__ float red_max[4][RED];
  __shared__ int red_idx[4][RED];
  __shared__ uint4 exchange[C::MERGED ? 128 : 1];

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // The grouped tile table is written by the kernel just before this one: wait for it before the first read, with the set-up
  // below behind it. 128-row gate/up tiles, whose launches fill the SMs with three CTAs each, wait ahead of the set-up (block of
  // 8 to 32 rows, plain weights, us, behind -> ahead: 87.2 -> 85.6, 116.4 -> 114.9, 159.5 -> 157.7, 198.3 -> 196.8; 128: 291.9
  // -> 289.5; thin tiles of one row 28.5 -> 29.0). Dense launches wait later (the producer streams the first weight stages
  // before it waits).
  constexpr bool WAIT_FIRST = SPLIT || (GROUPED && EPI == EPI_SILU_MUL && !C::THIN);
  if (WAIT_FIRST) pdl_wait();
  // Persistent tile loop: CTA b takes output tiles b, b + gridDim.x, ... (weight tile fastest, so CTAs that run
  // together share the activation tile). A split-K cluster takes the single tile its grid position names.
  const int tiles_n = (p.N + RT - 1) / RT;
  const int tile0 = SPLIT ? static_cast<int>(blockIdx.y) * tiles_n + static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x);
  const int tstep = SPLIT ? (1 << 30) : static_cast<int>(gridDim.x);
  constexpr int ACC = SPLIT ? 1 : C::ACC_STAGES;
  // the whole cluster leaves together, before any barrier or TMEM use
  if (SPLIT && tile0 >= tiles_n * (GROUPED ? *p.n_tiles : p.grid_y)) return;
  const int num_k_all = (p.K + BK * KPS - 1) / (BK * KPS);  // in stages
  // split-K: the cluster's CTAs (blockIdx.z = rank in the cluster) take consecutive runs of k-blocks; their fp32
  // partial tiles meet in the leader through distributed shared memory, added in rank order
  const int k_per = SPLIT ? (num_k_all + p.splits - 1) / p.splits : num_k_all;
  const int kb0 = SPLIT ? static_cast<int>(blockIdx.z) * k_per : 0;
  const int num_k = SPLIT ? max(0, min(num_k_all, kb0 + k_per) - kb0) : num_k_all;

  if (threadIdx.x == 0) {
    // a gathering producer: lane 0's expect_tx arrival for the weight tile plus one arrival per lane when that
    // lane's row copies have landed (all lanes of all gathering warps)
    const uint32_t full_count = (GROUPED && BT <= GATHER_BT_MAX && p.gather_rows != nullptr) ? 1 + 32 * C::GATHER_WARPS : 1;
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], full_count); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 4); }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (GROUPED) {
    if (!WAIT_FIRST) pdl_wait();
    if (!SPLIT && warp == 0) pdl_launch();
  }
  // The role's first table entry is read beside the entry count, not behind it (the table has room for the whole grid).
  int4 t_next = make_int4(0, 0, 0, 0);
  if (GROUPED) t_next = p.tiles[tile0 / tiles_n];
  const int tiles_y = GROUPED ? *p.n_tiles : p.grid_y;
  const int total = tiles_n * tiles_y;

  // geometry of output tile `tile`
  // (the table entry of the role's next tile is requested one tile ahead: its latency would otherwise open every tile)
  auto tile_geom = [&](int tile, int& n0, int& by, int& expert, int& row0, int& nrows) {
    const int nx = tile % tiles_n, byr = tile / tiles_n;
    n0 = nx * RT;
    by = (!GROUPED && p.y_rot) ? (byr + p.y_rot) % tiles_y : byr;
    expert = 0;
    if (GROUPED) {
      const int4 t = t_next;
      if (!SPLIT && total - tile > tstep) t_next = p.tiles[(tile + tstep) / tiles_n];
      expert = t.x; row0 = t.y; nrows = t.z;
    } else {
      row0 = by * BT;
      nrows = min(BT, p.T - row0);
    }
  };

  // weight rows [n0, n0 + RT) of pipeline step `kb` (and the matching up rows) into stage `st`
  auto load_weights = [&](uint8_t* st, uint64_t* bar, int n0, int expert, int kb) {
    if constexpr (C::THIN) {  // packed only: [expert, tile, k-block][rows of the tile][64], KPS k-blocks per box
      const int z = ((expert * p.w_tiles + n0 / BM) * num_k_all + kb) * KPS;
      if constexpr (C::MERGED) tma_load_4d(st, &tmW, bar, 0, n0 % BM, 0, z);  // [k-block][gate, up][rows][64]
      else tma_load_3d(st, &tmW, bar, 0, n0 % BM, z);
    } else if (p.packed) {
      tma_load_2d(st, &tmW, bar, 0, ((expert * p.w_tiles + n0 / BM) * num_k_all + kb) * (BM * C::A_TILES));
    } else if (GROUPED) {
      tma_load_3d(st, &tmW, bar, kb * BK, n0, expert);
      if (EPI == EPI_SILU_MUL) tma_load_3d(st + C::A_BYTES, &tmW, bar, kb * BK, p.up_offset + n0, expert);
    } else {
      tma_load_2d(st, &tmW, bar, kb * BK, n0);
      if (EPI == EPI_SILU_MUL) tma_load_2d(st + C::A_BYTES, &tmW, bar, kb * BK, p.up_offset + n0);
    }
  };

  // the stage of step `it` may be filled (a group's first stage stands for all of them)
  auto wait_free = [&](int it) {
    constexpr int NG = C::STAGES / C::GROUP;
    const int g = it / C::GROUP;
    return it % C::GROUP != 0 || mbar_wait(&empty[g % NG], ((g / NG) & 1) ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag);
  };

  constexpr int GW = GROUPED ? C::GATHER_WARPS : 1;
  if ((warp == 0 || warp >= 6) && GROUPED && BT <= GATHER_BT_MAX && p.gather_rows != nullptr) {
    // ---------------- gathering producer (all 32 lanes): weights by TMA from lane 0 of warp 0, activation rows by index
    // (with two gathering warps, each takes half of the tile's rows).
    // Chunk q = lane + 32 i of a k-block is bytes [16 (q & 7), +16) of tile row q >> 3; it lands where the 128-byte
    // swizzle of the K-major operand layout puts it: row r at (r >> 3) * 1024 + (r & 7) * 128, chunk j at
    // ((j ^ (r & 7)) * 16). Rows beyond the tile's row count are left as they are: an MMA column depends on its own
    // row only, and the epilogue never stores those columns.
    constexpr int PER_LANE = BT / 4 / GW > 0 ? BT / 4 / GW : 1;
    const int rbase = GW == 2 && warp >= 6 ? BT / 2 : 0;
    int it = 0;
    bool live = true;
    const int j = lane & 7;
    for (int tile = tile0; tile < total && live; tile += tstep) {
      int n0, by, expert, row0, nrows;
      tile_geom(tile, n0, by, expert, row0, nrows);
      const bf16* src[PER_LANE];
#pragma unroll
      for (int i = 0; i < PER_LANE; ++i) {
        const int r = rbase + (lane >> 3) + 4 * i;
        const int g = r < nrows ? p.gather_rows[row0 + r] : -1;
        src[i] = g >= 0 ? p.gx + static_cast<size_t>(g) * p.ldgx + j * 8 : nullptr;
      }
      for (int kb = 0; kb < num_k; ++kb, ++it) {
        const int s = it % C::STAGES;
        if (!wait_free(it)) { live = false; break; }
        uint8_t* st = smem + s * C::STAGE_BYTES;
        if (lane == 0 && (GW == 1 || warp == 0)) {
          mbar_expect_tx(&full[s], C::B_OFF);
          load_weights(st, &full[s], n0, expert, kb0 + kb);
        }
        const uint32_t xb = smem_u32(st + C::B_OFF);
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
          const int r = rbase + (lane >> 3) + 4 * i;
          if (src[i] != nullptr) {
            const uint32_t dst = xb + (r >> 3) * 1024 + (r & 7) * 128 + ((j ^ (r & 7)) << 4);
#pragma unroll
            for (int ks = 0; ks < KPS; ++ks)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + ks * C::B_BYTES),
                           "l"(src[i] + ((kb0 + kb) * KPS + ks) * BK) : "memory");
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s])) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // no copy of this lane may outlive the CTA's shared memory
  } else if (warp >= 6) {
    // the second gathering warp has nothing to do when the rows come through the tensor map
  } else if (warp == 0) {
    if (elect_one()) {
      int it = 0;  // k-blocks issued so far, over all tiles of this CTA
      const uint32_t x_stage = C::THIN || p.x_rows == 0 ? C::STAGE_BYTES : C::B_OFF + p.x_rows * (BK * 2);
      bool live = true;
      // Dense weights are written by nobody in the stream: fill the first stages of this CTA's first tile with weight
      // tiles before waiting for the previous kernel (whose output is X), so that their latency hides behind its tail.
      int pre = 0;
      if (!GROUPED && !SPLIT && tile0 < total) {
        int n0, by, expert, row0, nrows;
        tile_geom(tile0, n0, by, expert, row0, nrows);
        pre = num_k < C::STAGES ? num_k : C::STAGES;
        for (int kb = 0; kb < pre; ++kb) {
          uint8_t* st = smem + kb * C::STAGE_BYTES;
          mbar_expect_tx(&full[kb], x_stage);
          load_weights(st, &full[kb], n0, 0, kb);
        }
      }
      pdl_wait();
      if (!GROUPED) pdl_launch();
      for (int tile = tile0; tile < total && live; tile += tstep) {
      int n0, by, expert, row0, nrows;
      tile_geom(tile, n0, by, expert, row0, nrows);
      // all-gather -> GEMM: the activation rows of this tile were pushed here by their owner rank; wait for that
      // shard only, so tiles of shards that have already arrived run while the others are still in flight
      if (p.x_flags != nullptr && !wait_flag(p.x_flags + row0 / p.rows_per_rank, *p.x_epoch, p.err)) *abort_flag = 1;
      for (int kb = 0; kb < num_k; ++kb, ++it) {
        const int s = it % C::STAGES;
        uint8_t* st = smem + s * C::STAGE_BYTES;
        if (it >= pre) {
        if (!wait_free(it)) { live = false; break; }
        mbar_expect_tx(&full[s], !GROUPED ? x_stage : C::VAR_N ? C::B_OFF + (nrows + VAR_BOX - 1) / VAR_BOX * (VAR_BOX * BK * 2) : C::STAGE_BYTES);
        load_weights(st, &full[s], n0, expert, kb0 + kb);
        }
        if constexpr (GROUPED && C::VAR_N) {
          for (int r = 0; r < nrows; r += VAR_BOX)
            tma_load_2d(st + C::B_OFF + r * (BK * 2), &tmX, &full[s], (kb0 + kb) * BK, row0 + r);
        } else if constexpr (C::THIN) tma_load_3d(st + C::B_OFF, &tmX, &full[s], 0, row0, (kb0 + kb) * KPS);
        else tma_load_2d(st + C::B_OFF, &tmX, &full[s], (kb0 + kb) * BK, row0);
      }
      }
    }
    if (SPLIT) { __syncwarp(); cluster_sync(); }
  } else if (warp == 1) {
    // The warp runs this loop as a whole, which keeps descriptors in uniform registers, and one lane issues. In dense gate/up
    // launches, of two MMAs per step, that lane runs it alone but for 64-row tiles; us, warp -> lane (x 512 x 2048): 17 rows 17.2 ->
    // 16.3, 128: 25.2 -> 23.0, 2048: 26.2 -> 23.8 (64: 21.2 -> 21.9; grouped launches show no difference).
    constexpr bool LONE = EPI == EPI_SILU_MUL && !GROUPED && BT != 64;
    const uint32_t issue = elect_one();
    const auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
      return LONE ? mbar_wait(bar, parity, p.err, code, abort_flag) : mbar_wait_warp(bar, parity, p.err, code, abort_flag);
    };
    if (!LONE || issue) {
      uint32_t idesc = umma_idesc_bf16(C::MMA_M, !GROUPED && !C::THIN && p.x_rows > 0 ? p.x_rows : BT);
      bool ok = true;
      int it = 0, lt = 0;  // k-blocks and tiles consumed so far
      for (int tile = tile0; tile < total && ok; tile += tstep, ++lt) {
      if (GROUPED && C::VAR_N) {
        int n0, by, expert, row0, nrows;
        tile_geom(tile, n0, by, expert, row0, nrows);
        idesc = umma_idesc_bf16(BM, (nrows + 15) / 16 * 16);
      }
      const int acc = lt % ACC;
      const uint32_t tmem = tmem_base + acc * C::ACC_COLS;
      // the epilogue must have drained this accumulator stage (two tiles ago) before it is overwritten
      ok = wait(&acc_empty[acc], ((lt / ACC) & 1) ^ 1, ERR_WAIT_TMEM);
      if (ok) tc_fence_after();
      for (int kb = 0; kb < num_k && ok; ++kb, ++it) {
        const int s = it % C::STAGES;
        const uint32_t ph = (it / C::STAGES) & 1;
        ok = wait(&full[s], ph, ERR_WAIT_FULL);
        if (!ok) break;
        // rows that the gathering producer wrote through the generic proxy must be visible to the tensor core's reads
        if (GROUPED && BT <= GATHER_BT_MAX && p.gather_rows != nullptr) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + s * C::STAGE_BYTES);
        const uint32_t b_addr = a_addr + C::B_OFF;
#pragma unroll
        for (int k = 0; k < KPS * BK / UMMA_K; ++k) {
          const uint32_t koff = (k % (BK / UMMA_K)) * UMMA_K * 2;  // bytes inside the 128-byte swizzled row
          const uint32_t aoff = k / (BK / UMMA_K) * C::A_STEP + koff;
          const uint64_t db = umma_smem_desc(b_addr + k / (BK / UMMA_K) * C::B_BYTES + koff);
          umma_bf16_if(LONE ? 1u : issue, tmem, umma_smem_desc(a_addr + aoff), db, idesc, (kb | k) != 0);
          if (EPI == EPI_SILU_MUL && !C::MERGED)
            umma_bf16_if(LONE ? 1u : issue, tmem + BT, umma_smem_desc(a_addr + C::A_BYTES + aoff), db, idesc, (kb | k) != 0);
        }
        // the group's stages are reusable once these MMAs have read them
        if (it % C::GROUP == C::GROUP - 1) umma_commit_if(LONE ? 1u : issue, &empty[it / C::GROUP % (C::STAGES / C::GROUP)]);
      }
      umma_commit_if(LONE ? 1u : issue, &acc_full[acc]);  // always arrive so that the epilogue is released
      }
    }
    if (SPLIT) { __syncwarp(); cluster_sync(); }
  } else {
    // ---------------- epilogue: warp q owns TMEM lanes [32q, 32q+32)
    pdl_wait();  // first global write of the CTA comes from here
    const int q = warp & 3;
    int lt = 0;
    int out_buf = 0;  // staging buffer of the next 16 rows
    const bool staged = C::STAGED && p.ldo % 8 == 0 && p.N % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
    for (int tile = tile0; tile < total; tile += tstep, ++lt) {
    int n0, by, expert, row0, nrows;
    tile_geom(tile, n0, by, expert, row0, nrows);
    (void)expert;
    const int nx = n0 / RT;
    const int acc = lt % ACC;
    const uint32_t tmem = tmem_base + acc * C::ACC_COLS;
    bool ok = mbar_wait(&acc_full[acc], (lt / ACC) & 1, p.err, ERR_WAIT_TMEM, abort_flag) && !*abort_flag;
    // batches that hold barriers: all four warps take them, or none
    if (C::MERGED || (C::STAGED && staged)) ok = epilogue_all(ok);
    tc_fence_after();
    const int arow = C::MMA_M == 64 ? q * 16 + lane : q * 32 + lane;  // accumulator row of this thread
    const int n = n0 + (C::MERGED ? arow % RT : arow);
    const bool n_ok = n < p.N && (C::MMA_M == 128 || lane < 16) && arow < C::A_ROWS;
    if (EPI == EPI_ALLREDUCE) {
      // Fused GEMM -> one-shot all-reduce: this tile's fp32 partial goes straight from TMEM into every
      // rank's receive slot over NVLink; when all R partials of the tile have arrived they are added in
      // rank order (+ residual) and stored as bf16. No partial ever touches this rank's output buffer.
      const CommCtx& cc = p.comm;
      const int blk = by * tiles_n + nx;
      __shared__ uint32_t s_epoch;
      __shared__ int s_peer_ok;
      const int et = threadIdx.x - 64;  // 0..127 among the epilogue threads
      if (et == 0) { s_epoch = cc.epoch[blk] + 1; cc.epoch[blk] = s_epoch; s_peer_ok = 1; }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const uint32_t e = s_epoch;
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < nrows; c += 16) {
          float v[16];
          tmem_ld16(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, v);  // warp-collective: never predicated
          if (n_ok) {
            for (int r = 0; r < cc.world; ++r) {
              float* dst = comm_slot(cc, r, e, cc.rank);
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (c + j < nrows) dst[static_cast<size_t>(row0 + c + j) * p.ldo + n] = v[j];
            }
          }
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (et < cc.world) {
        __threadfence_system();
        st_release_sys(cc.flags[et] + static_cast<size_t>(cc.rank) * cc.max_blocks + blk, e);
        if (!wait_flag(cc.flags[cc.rank] + static_cast<size_t>(et) * cc.max_blocks + blk, e, cc.err)) s_peer_ok = 0;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ok && n_ok && s_peer_ok) {
        for (int t = 0; t < nrows; ++t) {
          const size_t o = static_cast<size_t>(row0 + t) * p.ldo + n;
          float acc = comm_slot(cc, cc.rank, e, 0)[o];
          for (int r = 1; r < cc.world; ++r) acc += comm_slot(cc, cc.rank, e, r)[o];
          if (p.residual) acc = __bfloat162float(__float2bfloat16(acc)) + __bfloat162float(p.residual[o]);
          reinterpret_cast<bf16*>(p.out)[o] = __float2bfloat16(acc);
        }
      }
    } else if (EPI == EPI_REDUCE_SCATTER) {
      // Fused GEMM -> reduce-scatter: the tile's token rows belong to one owner rank. Every rank stores its fp32
      // partial straight from TMEM into the owner's receive slot (a peer store over NVLink unless it is the
      // owner) and releases the tile's arrival flag there. Nothing waits here: the owner adds the R partials in
      // rank order inside the following norm kernel (allreduce.cu, reduce_norm_allgather_kernel), at full occupancy.
      const CommCtx& cc = p.comm;
      const int blk = by * tiles_n + nx;
      const int owner = row0 / p.rows_per_rank;
      const int lrow0 = row0 - owner * p.rows_per_rank;
      __shared__ uint32_t s_epoch_rs;
      const int et = threadIdx.x - 64;
      if (et == 0) { s_epoch_rs = cc.epoch[blk] + 1; cc.epoch[blk] = s_epoch_rs; }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const uint32_t e = s_epoch_rs;
      if (ok) {
        float* dst = comm_slot(cc, owner, e, cc.rank);
#pragma unroll 1
        for (int c = 0; c < nrows; c += 16) {
          float v[16];
          tmem_ld16(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, v);  // warp-collective: never predicated
          if (n_ok) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (c + j < nrows) dst[static_cast<size_t>(lrow0 + c + j) * p.ldo + n] = v[j];
          }
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (et == 0) {
        __threadfence_system();
        st_release_sys(cc.flags[owner] + static_cast<size_t>(cc.rank) * cc.max_blocks + blk, e);
      }
    } else
    if (SPLIT && blockIdx.z != 0) {
      // split-K follower: park the partial tile in shared memory (the pipeline stages are idle now) as
      // red[column][weight row]; a CTA without k-blocks contributes zeros
      float* red = reinterpret_cast<float*>(smem);
#pragma unroll 1
      for (int c = 0; c < nrows; c += 16) {
        float v[16];
        if (num_k > 0 && ok) tmem_ld16(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, v);
        else { for (int j = 0; j < 16; ++j) v[j] = 0.f; }
#pragma unroll
        for (int j = 0; j < 16; ++j) red[(c + j) * BM + q * 32 + lane] = v[j];
        if (EPI == EPI_SILU_MUL) {
          if (num_k > 0 && ok) tmem_ld16(tmem + (static_cast<uint32_t>(q * 32) << 16) + BT + c, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) red[(BT + c + j) * BM + q * 32 + lane] = v[j];
        }
      }
      cluster_sync();  // first cluster barrier (every thread of the cluster takes part exactly once)
    } else {
    if (SPLIT) cluster_sync();  // first cluster barrier: the followers' partial tiles are in place
    if (ok && q * (C::MMA_M / 4) < C::A_ROWS) {
      const uint32_t red_local = smem_u32(smem);
#pragma unroll 1
      for (int c = 0; c < BT; c += 16) {
        if (c >= nrows) break;  // warp-uniform
        float v[16];
        tmem_ld16(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, v);
        if (SPLIT) {
          for (int r = 1; r < p.splits; ++r) {
            const uint32_t remote = dsmem_addr(red_local, r);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += ld_dsmem_f32(remote + ((c + j) * BM + q * 32 + lane) * 4);
          }
        }
        if constexpr (C::MERGED) {
          // the threads of an output's gate and up row swap half of their columns, rounded to bf16 as the unfused sequence
          // of ops rounds them, and finish eight each
          const bool up = q >= 2;
          const int tid = q * 32 + lane;
          uint4 mine, theirs;
          bf16* me = reinterpret_cast<bf16*>(&mine);
          const bf16* te = reinterpret_cast<const bf16*>(&theirs);
#pragma unroll
          for (int j = 0; j < 8; ++j) me[j] = __float2bfloat16(up ? v[j] : v[8 + j]);
          exchange[tid] = mine;
          asm volatile("bar.sync 2, 128;" ::: "memory");
          theirs = exchange[tid ^ 64];
          asm volatile("bar.sync 2, 128;" ::: "memory");
          const int c0 = c + (up ? 8 : 0);
          if (n_ok) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float own = __bfloat162float(__float2bfloat16(up ? v[8 + j] : v[j])), other = __bfloat162float(te[j]);
              const float gate = up ? other : own, lin = up ? own : other;
              if (c0 + j < nrows)
                reinterpret_cast<bf16*>(p.out)[static_cast<size_t>(row0 + c0 + j) * p.ldo + n] =
                    __float2bfloat16(__bfloat162float(__float2bfloat16(silu_f(gate))) * lin);
            }
          }
          continue;
        }
        if (EPI == EPI_SILU_MUL) {
          float u[16];
          tmem_ld16(tmem + (static_cast<uint32_t>(q * 32) << 16) + BT + c, u);
          if (SPLIT) {
            for (int r = 1; r < p.splits; ++r) {
              const uint32_t remote = dsmem_addr(red_local, r);
#pragma unroll
              for (int j = 0; j < 16; ++j) u[j] += ld_dsmem_f32(remote + ((BT + c + j) * BM + q * 32 + lane) * 4);
            }
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            // round gate and up to bf16 first, as the unfused sequence of ops does
            const float g = __bfloat162float(__float2bfloat16(v[j]));
            const float uu = __bfloat162float(__float2bfloat16(u[j]));
            v[j] = __bfloat162float(__float2bfloat16(silu_f(g))) * uu;
          }
        }
        if (EPI == EPI_ARGMAX) {
          float best;
          int at;
          argmax_columns(v, n, n_ok, lane, best, at);
          if ((lane & 1) == 0) {
            const int col = c + argmax_column(lane);
            red_max[q][col] = best;
            red_idx[q][col] = at;
          }
        } else if (EPI == EPI_SCATTER) {
          // expert-parallel combine: each output row goes straight to the rank that owns the token,
          // into the slot of its (token, pair) - a peer store over NVLink when that rank is not this one
          if (n_ok) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (c + j < nrows) {
                const int2 m = p.meta[row0 + c + j];
                p.pair_out[m.x][static_cast<size_t>(m.y) * p.ldo + n] = __float2bfloat16(v[j]);
              }
            }
          }
        } else if (C::STAGED && staged) {
          // [16 rows][128 weight rows] bf16, two buffers: a lane writes its column, and behind the barrier the 128 threads
          // send the rows. A thread's reads of a buffer precede its next barrier, behind which the buffer is written again.
          bf16* ob = reinterpret_cast<bf16*>(out_stage) + out_buf * (16 * BM);
          out_buf ^= 1;
#pragma unroll
          for (int j = 0; j < 16; ++j) ob[j * BM + q * 32 + lane] = __float2bfloat16(v[j]);
          asm volatile("bar.sync 2, 128;" ::: "memory");
          const int col = (lane & 15) * 8;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = i * 8 + q * 2 + (lane >> 4);
            const uint4 o = *reinterpret_cast<const uint4*>(ob + r * BM + col);
            if (c + r < nrows && n0 + col < p.N)
              *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(p.out) + static_cast<size_t>(row0 + c + r) * p.ldo + n0 + col) = o;
          }
        } else if (n_ok) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (c + j < nrows) {
              const size_t o = static_cast<size_t>(row0 + c + j) * p.ldo + n;
              if (EPI == EPI_F32) reinterpret_cast<float*>(p.out)[o] = v[j];
              else reinterpret_cast<bf16*>(p.out)[o] = __float2bfloat16(v[j]);
            }
          }
        }
      }
    }
    }
    if (EPI == EPI_ARGMAX) {
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the four epilogue warps only
      const int t = (warp - 2) * 32 + lane;
      for (int c = t; c < BT; c += 128) {
        if (c < nrows && ok) {
          float m = red_max[0][c]; int idx = red_idx[0][c];
#pragma unroll
          for (int w = 1; w < 4; ++w) {
            const float om = red_max[w][c]; const int oi = red_idx[w][c];
            if (om > m || (om == m && oi < idx)) { m = om; idx = oi; }
          }
          const size_t o = static_cast<size_t>(nx) * p.T + row0 + c;
          p.part_max[o] = m; p.part_idx[o] = idx;
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");  // red_max / red_idx are reused by the next tile
    }
    // this accumulator stage may be overwritten: every tcgen05.ld of the warp has completed (wait::ld)
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&acc_empty[acc]);
    if (!ok) break;
    }
  }
  if (SPLIT) cluster_sync();  // second cluster barrier: the leader has read every partial tile
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, C::TMEM_COLS); }
}

// Reduce the LM-head partials of each row over the vocabulary tiles, first maximum wins. Bound by the latency of a thread's
// loads: while there are no more rows than SMs a row gets 1024 threads (two loads each at 1940 tiles, not eight): 6.4 -> 4.6 us
// at one to twelve rows, 8.0 -> 6.9 at 128.
__global__ void argmax_finish_kernel(const float* part_max, const int* part_idx, int n_tiles, int T, int64_t* out,
                                     float* out_val) {
  pdl_wait();
  pdl_launch();
  const int t = blockIdx.x;
  float m = -INFINITY; int idx = 0x7fffffff;
#pragma unroll 2
  for (int i = threadIdx.x; i < n_tiles; i += blockDim.x) {
    const float om = part_max[static_cast<size_t>(i) * T + t]; const int oi = part_idx[static_cast<size_t>(i) * T + t];
    if (om > m || (om == m && oi < idx)) { m = om; idx = oi; }
  }
  __shared__ float sm[32]; __shared__ int si[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, o); const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (om > m || (om == m && oi < idx)) { m = om; idx = oi; }
  }
  if ((threadIdx.x & 31) == 0) { sm[threadIdx.x >> 5] = m; si[threadIdx.x >> 5] = idx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w)
      if (sm[w] > m || (sm[w] == m && si[w] < idx)) { m = sm[w]; idx = si[w]; }
    out[t] = idx;
    if (out_val) out_val[t] = m;
  }
}

}  // namespace b200
#include "gemm_pair.cuh"
namespace b200 {

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess) fn = reinterpret_cast<EncodeFn>(ptr);
  }
  return fn;
}

// bf16 tensor [d2, d1, d0] (d0 contiguous), box {BK, box1, 1}, 128-byte swizzle, zero fill.
static int make_map(CUtensorMap* m, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t ld1, uint64_t ld2,
                    uint32_t box1) {
  EncodeFn fn = encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {ld1 * 2, ld2 * 2};
  cuuint32_t box[3] = {BK, box1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const int rank = d2 > 0 ? 3 : 2;
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// Tile-packed weights: a 2-D view [tiles * box_rows, 64] whose boxes of `box_rows` rows are contiguous runs.
static int make_map_packed(CUtensorMap* m, const void* base, uint64_t total_rows, uint32_t box_rows) {
  EncodeFn fn = encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[2] = {BK, total_rows};
  cuuint64_t strides[1] = {BK * 2};
  cuuint32_t box[2] = {BK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// Maps of the thin forms: `kps` k-blocks of `rows` rows per box. Packed weights: [tile, k-block][tile rows][64]; activations:
// the k-blocks of a row are 128 bytes apart.
static int make_map_kblocks(CUtensorMap* m, const void* base, uint64_t rows, uint64_t row_bytes, uint64_t blocks,
                            uint64_t block_bytes, uint32_t box_rows, uint32_t kps) {
  EncodeFn fn = encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[3] = {BK, rows, blocks};
  cuuint64_t strides[2] = {row_bytes, block_bytes};
  cuuint32_t box[3] = {BK, box_rows, kps};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// The same for thin gate/up tiles: [tile, k-block][gate, up][BM rows][64], `rows` rows of either half and `kps` k-blocks per box.
static int make_map_gate_up(CUtensorMap* m, const void* base, uint64_t blocks, uint32_t rows, uint32_t kps) {
  EncodeFn fn = encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[4] = {BK, BM, 2, blocks};
  cuuint64_t strides[3] = {BK * 2, BM * BK * 2, 2 * BM * BK * 2};
  cuuint32_t box[4] = {BK, rows, 2, kps};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// Weight map of a launch: `packed` selects the tile-packed layout (N padded to a multiple of 128 per expert, K a
// multiple of 64; with the SiLU-mul epilogue the gate and up tiles of a k-block are stored back to back).
static int weight_map(CUtensorMap* m, const void* W, int E, int N, int w_rows, int K, int ldw, bool silu, int packed,
                      GemmParams* p) {
  if (!packed) return E > 0 ? make_map(m, W, K, w_rows, E, K, static_cast<uint64_t>(w_rows) * K, BM)
                            : make_map(m, W, K, w_rows, 0, ldw, 0, BM);
  if (K % BK) return -7;
  const uint64_t tiles = (N + BM - 1) / BM, nk = K / BK, a = silu ? 2 : 1;
  p->packed = 1;
  p->w_tiles = static_cast<int>(tiles);
  return make_map_packed(m, W, static_cast<uint64_t>(E > 0 ? E : 1) * tiles * nk * BM * a, static_cast<uint32_t>(BM * a));
}

template <int BT, int EPI, bool GROUPED>
static int launch_split(const CUtensorMap& tw, const CUtensorMap& tx, const GemmParams& p, int grid_y, cudaStream_t st) {
  using C = Cfg<BT, EPI>;
  auto kern = gemm_swapab_kernel<BT, EPI, GROUPED, true>;
  static bool configured[MAX_DEVICES] = {};  // a function attribute is set per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return -3;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess) return -3;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + BM - 1) / BM, grid_y, p.splits);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = p.splits;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  GemmParams q = p;
  q.grid_y = grid_y;
  return cudaLaunchKernelEx(&cfg, kern, tw, tx, q) == cudaSuccess ? 0 : -4;
}

template <int BT, int EPI, bool GROUPED, int RT = BM, int KPS = 1>
static int launch(const CUtensorMap& tw, const CUtensorMap& tx, const GemmParams& p, int grid_y, cudaStream_t st) {
  using C = Cfg<BT, EPI, RT, KPS>;
  if constexpr (!C::THIN && (EPI == EPI_BF16 || EPI == EPI_F32 || EPI == EPI_SILU_MUL)) {
    if (p.splits > 1) return launch_split<BT, EPI, GROUPED>(tw, tx, p, grid_y, st);
  }
  auto kern = gemm_swapab_kernel<BT, EPI, GROUPED, false, RT, KPS>;
  // per device: the shared-memory attribute is set on the device that is current, and the persistent grid is sized
  // from that device's SM count (a process may drive several GPUs)
  static bool configured[MAX_DEVICES] = {};
  static int resident_of[MAX_DEVICES] = {};  // CTAs the device holds at once: the persistent grid is never larger
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return -3;
  if (!configured[dev]) {
    int sms = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess) return -3;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -3;
    resident_of[dev] = sms * C::CTAS_PER_SM;
    configured[dev] = true;
  }
  const int resident = resident_of[dev];
  GemmParams q = p;
  q.grid_y = grid_y;
  const long long tiles = static_cast<long long>((p.N + RT - 1) / RT) * grid_y;
  constexpr int threads = GROUPED ? 160 + 32 * C::GATHER_WARPS : 192;
  return launch_pdl(kern, dim3(static_cast<unsigned>(tiles < resident ? tiles : resident)), dim3(threads), C::SMEM, st, tw,
                    tx, q) == cudaSuccess ? 0 : -4;
}

template <int EPI, bool GROUPED>
static int dispatch_bt(int bt, const CUtensorMap& tw, const CUtensorMap& tx, const GemmParams& p, int grid_y, cudaStream_t st) {
  switch (bt) {
    case 16: return launch<16, EPI, GROUPED>(tw, tx, p, grid_y, st);
    case 32: return launch<32, EPI, GROUPED>(tw, tx, p, grid_y, st);
    case 64: return launch<64, EPI, GROUPED>(tw, tx, p, grid_y, st);
    case 128: return launch<128, EPI, GROUPED>(tw, tx, p, grid_y, st);
    case 256:
      if (EPI != EPI_SILU_MUL) return launch<(EPI != EPI_SILU_MUL ? 256 : 128), EPI, GROUPED>(tw, tx, p, grid_y, st);
      return -5;  // the gate/up epilogue has no 256-row form
    default: return -5;
  }
}

static int sm_count() {  // of the current device; 148 on a B200
  static int of[MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return 148;
  if (of[dev] == 0 && cudaDeviceGetAttribute(&of[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return of[dev];
}

struct DenseForm {
  int bt, rt, kps;  // token rows per tile, weight rows per tile, k-blocks per stage
};

// The form of a dense bf16 / fp32 GEMM with one SM per tile. It never changes a row's bits (every element sees the same k order
// in the same products), so it may follow the number of rows. Measured in chains of launches on weights that are not in L2, us,
// 128-row tiles with one k-block per stage -> chosen form; 12352 x 2048 is a GDN layer's input projection, 9216 x 2048 an
// attention layer's, 2048 x 4096 the output projection, 257 x 2048 the router (in a decode step):
//   up to 16 rows     12352: 13.0 -> 12.0   9216: 11.6 -> 7.4   2048: 15.4 -> 7.9   257: 8.5 -> 4.9
//   61 rows           2048: 14.7 -> 11.5   257: 8.4 -> 5.0
//   128 rows          2048: 15.0 -> 10.3   257: 8.4 -> 5.3
//   256 rows          2048: 16.1 -> 13.0   257: 8.4 -> 5.3
static DenseForm dense_form(int T, int N, int K, bool packed) {
  const int sms = sm_count();
  const auto tiles = [&](int rt, int bt) { return static_cast<long long>((N + rt - 1) / rt) * ((T + bt - 1) / bt); };
  const bool by2 = packed && K % (2 * BK) == 0, by4 = packed && K % (4 * BK) == 0;
  if (T <= 16) {
    // one token tile: the weights are streamed once whatever the tile, so the thinnest tile whose CTAs have an SM each wins
    // (9216 rows as 288 CTAs of 32 rows, two per SM: 8.4 us, as 144 of 64: 7.4), then the thinnest whose CTAs, two per SM, are
    // all resident; beyond that the second wave costs more (386 CTAs of 32 rows: 14.2 us for the 12352 rows)
    if (by4 && tiles(32, 16) <= sms) return {16, 32, 4};
    if (by4 && tiles(64, 16) <= sms) return {16, 64, 4};
    if (by2 && tiles(64, 16) <= 2 * sms) return {16, 64, 2};
    return {16, BM, 1};
  }
  if (T <= 256 && N <= 32 * BM) {
    // few weight tiles: 16-row token tiles put 8x more CTAs on the K loop. Several token tiles re-read the weights, so
    // thin tiles pay only while the CTAs have an SM each, with a little room (144 CTAs already share some). Output projection
    // of 128 rows in a step 13.1 us with two 32-row tiles' stages per SM, 11 with all of an SM's shared memory; 256 rows 16 as
    // 256 CTAs of 16 x 128, 14 as 128 of 64 x 64
    const int lim = sms * 7 / 8;
    if (by4 && tiles(32, 16) <= lim) return {16, 32, 4};
    if (by4 && tiles(64, 16) <= lim) return {16, 64, 4};
    if (by4 && tiles(64, 32) <= lim) return {32, 64, 4};
    if (by4 && tiles(64, 64) <= lim) return {64, 64, 4};
    // an odd number of 128-element k-steps, us, 128-row tiles -> these: 257 x 1920 7.5 -> 6.3, 512 x 4224 at 48 rows 13.9 -> 11.1, 2048
    // x 1152 at 48 5.8 -> 4.9, at 100, as 32 x 64, 6.1 -> 5.8 (x 896 5.1 -> 5.2, x 384 3.6 -> 4.1)
    if (by2 && tiles(64, 16) <= lim) return {16, 64, 2};
    if (by2 && K >= 16 * BK && tiles(64, 32) <= lim) return {32, 64, 2};
    return {16, BM, 1};
  }
  if (T > 256) {
    // few weight tiles and many rows (the router): the narrowest token tile whose CTAs are resident together, as long as the
    // K loop of a CTA and not the rows it reads sets the time. Router, 257 x 2048, us, 256-row tiles -> these: 300 rows
    // 16.4 -> 7.6, 1531: 16.6 -> 8.8 (16 rows); 2048: 16.6 -> 9.6 (64; 16: 14.1); 4096: 17.0 -> 10.9 (128); 8192: 17.8
    if (tiles(BM, 16) <= 2 * sms) return {16, BM, 1};
    if (tiles(BM, 64) <= sms) return {64, BM, 1};
    if (tiles(BM, 128) <= sms) return {128, BM, 1};
  }
  return {T <= 32 ? 32 : T <= 64 ? 64 : T <= 128 ? 128 : 256, BM, 1};
}

constexpr int PAIR_FORM = -256;  // token tile of up to 256 rows on two SMs, in the `bt` argument of the launchers
constexpr int PAIR_FORM_128 = -128;  // of up to 128 rows

// Two SMs per tile (gemm_pair.cuh). A cluster's CTAs sit on one SM each; the persistent grid is one cluster per pair of SMs.
template <int EPI, bool GROUPED, int PBT>
static int launch_pair(const CUtensorMap& tw, const CUtensorMap& tx, GemmParams p, int grid_y, cudaStream_t st) {
  auto kern = gemm_pair_kernel<EPI, GROUPED, PBT>;
  static bool configured[MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return -3;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<PBT>::SMEM) != cudaSuccess) return -3;
    configured[dev] = true;
  }
  p.grid_y = grid_y;
  const int rows = EPI == EPI_SILU_MUL ? BM : 2 * BM;
  const long long tiles = static_cast<long long>((p.N + rows - 1) / rows) * grid_y, pairs = sm_count() / 2;
  return launch_clusters(2, kern, dim3(2 * static_cast<unsigned>(tiles < pairs ? tiles : pairs)), dim3(pair_threads(EPI)), PairCfg<PBT>::SMEM,
                         st, tw, tx, p) == cudaSuccess ? 0 : -4;
}

// What the pair form asks of a launch: an epilogue that it has (gate/up grouped only), whole k-blocks, and bf16 output rows that
// leave in 16-byte pieces.
static bool pair_takes(const GemmParams& p, int epi, bool grouped) {
  if (p.K % BK) return false;
  if (epi == EPI_ARGMAX || epi == EPI_F32) return !grouped;
  if (epi != EPI_BF16 && !(epi == EPI_SILU_MUL && grouped)) return false;
  return p.N % 8 == 0 && p.ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
}

// Token rows per tile of a dense launch: the fewest cycles over the waves of the persistent grid. A k-block of bt rows takes an
// SM 2 bt cycles of MMA, and its 16 KB of weights and 64 bt bytes of rows 256 + bt cycles out of L2.
static int pair_rows(int T, int N) {
  const long long n = (N + 2 * BM - 1) / (2 * BM), pairs = sm_count() / 2;
  int best = PAIR_BT;
  long long least = -1;
  for (int bt = PAIR_BT; bt >= PAIR_N_STEP; bt -= PAIR_N_STEP) {
    const long long waves = (n * ((T + bt - 1) / bt) + pairs - 1) / pairs, cost = waves * (2 * BM + bt);
    if (least < 0 || cost < least) { least = cost; best = bt; }
  }
  return best;
}

// Whether up to 128 rows have too few k-blocks for two SMs per tile: nothing but the launch's ends is left then, and one SM per tile
// ends sooner where the pairs are mostly busy. Up to nine k-blocks where the rows are cut into several tiles (bf16, x 384, 512, us,
// pair -> one SM: 9216 at 48 rows 5.3 -> 4.4, 6.1 -> 5.1, at 100 5.7 -> 5.0, 6.5 -> 5.8; at 640 6.5 -> 6.1, at 768 6.9 -> 6.6), up to
// six where they are one tile (16384 x 256 at 48 rows 4.9 -> 3.9, x 384 5.8 -> 5.1; 12352 x 384 5.0 -> 4.7, x 512 5.6 -> 5.8). fp32
// rows, whose stores one SM has twice as many of, up to 48 rows (9216 x 384 at 48 rows 5.4 -> 4.8, at 100 5.9 -> 6.0). While the
// tiles leave half of the pairs idle, or a fifth from 65 rows on, two SMs are the better form (4104 x 384 at 48 rows 3.8 and 4.1, 5120
// x 384 at 128 rows 4.7 and 5.2).
static bool pair_too_short(int T, int N, int K, int epi) {
  const int bt = pair_rows(T, N), cut = (T + bt - 1) / bt;
  if ((N + 2 * BM - 1) / (2 * BM) * cut <= (T <= 64 ? sm_count() / 4 : sm_count() * 2 / 5)) return false;
  return cut > 1 ? T <= (epi == EPI_BF16 ? 128 : 48) && K <= 9 * BK : T <= (epi == EPI_BF16 ? 64 : 48) && K <= 6 * BK;
}

// Whether a dense launch is better off with two SMs per tile, us, best other form -> pair, weights not in L2 (about 10 us of
// each is the measurement's own):
//   rows    129           256           257           512           1024          2048          8192
//   12352   26.7 -> 22.5  26.6 -> 24.6  34.8 -> 29.4  40.9 -> 32.8  53.3 -> 47.1  88.1 -> 75.8  277 -> 253
//   9216    24.6 -> 21.3  26.7 -> 23.6  27.6 -> 23.6  27.5 -> 25.3  41.0 -> 36.9  63.5 -> 57.3  203 -> 186
//   2048    20.5 -> 22.5  23.5 -> 22.6  35.8 -> 22.6  35.5 -> 23.3  36.9 -> 24.6  36.9 -> 32.8  113 -> 86
// (12352 and 9216 x 2048, 2048 x 4096). A single pair of weight tiles would leave half of one idle below 256 columns.
// Many weight tiles and 17 to 128 rows, in chains of norm and projection, 64- or 128-row tiles of one SM -> pair: 12352 x 2048 at
// 24 rows 13.0 -> 13.0, at 64 15.7 -> 13.4, at 128 15.0 -> 14.4; 9216 x 2048 at 24 rows 11.4 -> 11.6, at 64 14.6 -> 12.9, at 128
// 15.1 -> 13.2.
// The LM head (argmax or fp32 logits of 248320 x 2048) is bound by its weights up to 128 rows and by shared memory beyond:
// picks of 160 rows 192 -> 172 us, of 256 226 -> 206; logits of 160 rows 221 -> 199, of 256 275 -> 240. fp32 rows of fewer
// weight tiles than SMs are better off from 17 on, x 2048: 16384 at 48 rows 16.1 -> 14.5, at 128 16.3 -> 15.4; 18944 at 17 rows
// 16.9 -> 15.4, at 64 18.7 -> 16.3 (31104 at 64 rows 24.6 -> 24.9; 62080 at 17 41.7 -> 45.0).
static bool pair_pays(int T, int N, int K, int epi) {
  if (T <= 128 && pair_too_short(T, N, K, epi)) return false;
  if (epi == EPI_ARGMAX || epi == EPI_F32)
    return N > 32 * BM && (T > 128 || (epi == EPI_F32 && T > 16 && N <= BM * sm_count()));
  return N >= 2 * BM && (T > 256 || (T > 16 && N > 32 * BM));
}

// Dense GEMM with two SMs per tile.
template <int EPI>
static int launch_pair_dense(const void* X, const void* W, GemmParams p, int ldx, int ldw, int packed, cudaStream_t st) {
  CUtensorMap tw, tx;
  p.pair_bt = pair_rows(p.T, p.N);
  if (weight_map(&tw, W, 0, p.N, p.N, p.K, ldw, false, packed, &p)) return -1;
  if (make_map(&tx, X, p.K, p.T, 0, ldx, 0, p.pair_bt / 2)) return -1;
  const int gy = (p.T + p.pair_bt - 1) / p.pair_bt;
  return p.pair_bt <= 128 ? launch_pair<EPI, false, 128>(tw, tx, p, gy, st) : launch_pair<EPI, false, PAIR_BT>(tw, tx, p, gy, st);
}

// Grouped GEMMs with two SMs per tile of up to PBT rows: gate/up with rows by index, or a bf16 projection of sorted rows.
// Tile-packed weights only.
template <int PBT>
static int launch_pair_grouped(const void* X, const void* W, GemmParams p, int E, int w_rows, int epi, const int* gather_rows,
                               int ldx, int max_tiles, cudaStream_t st) {
  CUtensorMap tw, tx;
  const bool silu = epi == EPI_SILU_MUL;
  if (weight_map(&tw, W, E, p.N, w_rows, p.K, p.K, silu, 1, &p)) return -1;
  if (!silu) {
    if (make_map(&tx, X, p.K, p.T, 0, p.K, 0, VAR_BOX)) return -1;
    return launch_pair<EPI_BF16, true, PBT>(tw, tx, p, max_tiles, st);
  }
  // a CTA's half of a k-block of a tile: 64 gate rows, then 64 up rows
  const uint64_t nk = p.K / BK;
  if (make_map_packed(&tw, W, static_cast<uint64_t>(E) * p.w_tiles * nk * BM * 2, BM / 2)) return -1;
  p.gather_rows = gather_rows;
  p.gx = static_cast<const bf16*>(X);
  p.ldgx = ldx;
  if (make_map(&tx, X, p.K, 1, 0, ldx, 0, 1)) return -1;  // never read through, but a valid map
  return launch_pair<EPI_SILU_MUL, true, PBT>(tw, tx, p, max_tiles, st);
}

// Launch of a thin dense form; -5 where there is no such form.
template <int EPI>
static int launch_thin_dense(const DenseForm& f, const void* X, const void* W, GemmParams p, int ldx, cudaStream_t st) {
  CUtensorMap tw, tx;
  const uint64_t nk = p.K / BK;
  p.packed = 1;
  p.w_tiles = (p.N + BM - 1) / BM;
  if (make_map_kblocks(&tw, W, BM, BK * 2, p.w_tiles * nk, BM * BK * 2, f.rt, f.kps)) return -1;
  if (make_map_kblocks(&tx, X, p.T, static_cast<uint64_t>(ldx) * 2, nk, BK * 2, f.bt, f.kps)) return -1;
  const int gy = (p.T + f.bt - 1) / f.bt;
  if (f.bt == 16 && f.rt == 32 && f.kps == 4) return launch<16, EPI, false, 32, 4>(tw, tx, p, gy, st);
  if (f.bt == 16 && f.rt == 64 && f.kps == 4) return launch<16, EPI, false, 64, 4>(tw, tx, p, gy, st);
  if (f.bt == 16 && f.rt == 64 && f.kps == 2) return launch<16, EPI, false, 64, 2>(tw, tx, p, gy, st);
  if (f.bt == 32 && f.rt == 64 && f.kps == 4) return launch<32, EPI, false, 64, 4>(tw, tx, p, gy, st);
  if (f.bt == 32 && f.rt == 64 && f.kps == 2) return launch<32, EPI, false, 64, 2>(tw, tx, p, gy, st);
  if (f.bt == 64 && f.rt == 64 && f.kps == 4) return launch<64, EPI, false, 64, 4>(tw, tx, p, gy, st);
  return -5;
}

// Gate/up GEMM of the experts with token tiles of 16 or 32 rows and tile-packed weights: tiles of 64 gate and 64 up rows, or of
// 32 and 32 while that leaves at most one CTA per SM (16-row token tiles, at most one per pair). A tile is one operand and not
// two of 128 rows, and twice as many tiles spread more evenly over the SMs. This GEMM, us, 128-row tiles -> these: 1 row of 9
// pairs 14.7 -> 9.2, 5 rows 40.5 -> 34.8, 13: 75.3 -> 71.7, 40: 140 -> 132, 128: 176.6 -> 170.2, 256: 179.5 -> 179; 32-row
// token tiles, 700 rows: 183 -> 180, 1024: 209 -> 191. (Tiles of 32 and 32 for all: 13 rows 73.7, 128: 175; 64-row token tiles
// are as good with 128 rows: 1300 rows 186 and 190.) The down projection has 16 weight tiles per expert and CTAs enough at
// one row. Two k-blocks per stage where K has no multiple of four (block of 1 row, 33 experts of 256 x 1152: 128-row tiles 27.5 us,
// these 21 to 22). Returns 1 when the plain form is to run.
static int launch_thin_grouped(const void* X, const void* W, GemmParams p, int E, const int* gather_rows, int ldx,
                               int max_tiles, int bt, cudaStream_t st) {
  const long long tiles = static_cast<long long>((p.N + BM - 1) / BM) * p.T;  // p.T: pairs
  const int rt = bt == 16 && 4 * tiles <= sm_count() ? 32 : 64, kps = rt == 32 && p.K % (4 * BK) == 0 ? 4 : 2;
  if (p.K % (kps * BK) || p.N % BM) return 1;
  CUtensorMap tw, tx;
  const uint64_t nk = p.K / BK;
  p.packed = 1;
  p.w_tiles = p.N / BM;
  if (make_map_gate_up(&tw, W, static_cast<uint64_t>(E) * p.w_tiles * nk, rt, kps)) return -1;
  if (gather_rows != nullptr) {
    p.gather_rows = gather_rows;
    p.gx = static_cast<const bf16*>(X);
    p.ldgx = ldx;
  }
  // with row indices the producer never reads through this map, but it has to be a valid one
  if (make_map_kblocks(&tx, X, gather_rows ? bt : p.T, static_cast<uint64_t>(gather_rows ? ldx : p.K) * 2, nk, BK * 2, bt, kps)) return -1;
  if (bt == 32) return launch<32, EPI_SILU_MUL, true, 64, 2>(tw, tx, p, max_tiles, st);
  if (rt == 32 && kps == 4) return launch<16, EPI_SILU_MUL, true, 32, 4>(tw, tx, p, max_tiles, st);
  if (rt == 32) return launch<16, EPI_SILU_MUL, true, 32, 2>(tw, tx, p, max_tiles, st);
  return launch<16, EPI_SILU_MUL, true, 64, 2>(tw, tx, p, max_tiles, st);
}

}  // namespace b200

using namespace b200;

// Token-tile width for a dense GEMM over T rows: a function of T only through the tile
// count, never through the per-element arithmetic.
extern "C" int b200_pick_bt(int T) {
  if (T <= 16) return 16;
  if (T <= 32) return 32;
  if (T <= 64) return 64;
  if (T <= 128) return 128;
  return 256;
}

// Dense: out[T, N] = X[T, K] W[N, K]^T. bt <= 0: the launcher picks the form, otherwise the token tile is `bt` rows; PAIR_FORM
// asks for two SMs per tile.
// epi: 0 bf16, 1 fp32, 2 silu(gate)*up (N = rows of each half, W has 2N rows with the up half at row `up_offset`),
// 3 argmax partials (part_max/part_idx sized [ceil(N/128), T]).
extern "C" int b200_gemm_dense(const void* X, const void* W, void* out, int T, int N, int K, int ldx, int ldw, int ldo,
                               int epi, int up_offset, int bt, float* part_max, int* part_idx, int* err,
                               int splits, int packed, cudaStream_t st) {
  if (T <= 0) return 0;
  if (splits < 1 || splits > 8 || splits > (K + BK - 1) / BK) splits = 1;
  const int w_rows = (epi == EPI_SILU_MUL) ? up_offset + N : N;
  GemmParams p{N, K, T, ldo, out, nullptr, nullptr, up_offset, part_max, part_idx, err, nullptr, CommCtx{}, 0, nullptr, nullptr, splits, nullptr, {}};
  const bool pair_ok = splits == 1 && pair_takes(p, epi, false);
  if (bt == PAIR_FORM && !pair_ok) return -7;
  if (bt == PAIR_FORM || (bt <= 0 && pair_ok && pair_pays(T, N, K, epi))) {
    switch (epi) {
      case EPI_BF16: return launch_pair_dense<EPI_BF16>(X, W, p, ldx, ldw, packed, st);
      case EPI_F32: return launch_pair_dense<EPI_F32>(X, W, p, ldx, ldw, packed, st);
      case EPI_ARGMAX: return launch_pair_dense<EPI_ARGMAX>(X, W, p, ldx, ldw, packed, st);
    }
    return -7;
  }
  if (bt <= 0 && (epi == EPI_BF16 || epi == EPI_F32)) {
    const DenseForm f = dense_form(T, N, K, packed && splits == 1);
    if (f.rt < BM)
      return epi == EPI_F32 ? launch_thin_dense<EPI_F32>(f, X, W, p, ldx, st) : launch_thin_dense<EPI_BF16>(f, X, W, p, ldx, st);
    bt = f.bt;
  }
  if (bt <= 0) bt = b200_pick_bt(T);
  if (epi == EPI_SILU_MUL && bt > 128) bt = 128;
  CUtensorMap tw, tx;
  if (weight_map(&tw, W, 0, N, w_rows, K, ldw, epi == EPI_SILU_MUL, packed, &p)) return -1;
  // a single token tile takes no more columns than there are rows (LM head of 160 rows in this form 198 -> 177 us)
  const int gy = (T + bt - 1) / bt;
  if (gy == 1) p.x_rows = (T + 15) / 16 * 16;
  if (make_map(&tx, X, K, T, 0, ldx, 0, gy == 1 ? p.x_rows : bt)) return -1;
  switch (epi) {
    case EPI_BF16: return dispatch_bt<EPI_BF16, false>(bt, tw, tx, p, gy, st);
    case EPI_F32: return dispatch_bt<EPI_F32, false>(bt, tw, tx, p, gy, st);
    case EPI_SILU_MUL: return dispatch_bt<EPI_SILU_MUL, false>(bt, tw, tx, p, gy, st);
    case EPI_ARGMAX: return dispatch_bt<EPI_ARGMAX, false>(bt, tw, tx, p, gy, st);
  }
  return -6;
}

// Grouped: X is the expert-sorted activation buffer [cap, K]; tile i covers rows
// [tiles[i].y, +tiles[i].z) of expert tiles[i].x; W is [E, rows, K]. `max_tiles` bounds the grid.
extern "C" int b200_gemm_grouped(const void* X, const void* W, void* out, int cap, int E, int N, int w_rows, int K,
                                 int ldo, int epi, int up_offset, int bt, const void* tiles, const int* n_tiles,
                                 int max_tiles, int* err, int splits, int packed, const int* gather_rows, int ldx,
                                 cudaStream_t st) {
  // gather_rows != null (token tiles of at most GATHER_BT_MAX rows): X is [any rows, ldx] and sorted position i reads row
  // gather_rows[i] of it; otherwise X is the expert-sorted buffer [cap, K] itself.
  if (max_tiles <= 0) return 0;
  if (bt == PAIR_FORM || bt == PAIR_FORM_128) {
    GemmParams p{N, K, cap, ldo, out, reinterpret_cast<const int4*>(tiles), n_tiles, up_offset, nullptr, nullptr, err, nullptr, CommCtx{}, 0, nullptr, nullptr, 1, nullptr, {}};
    if (!packed || splits > 1 || !pair_takes(p, epi, true) || N % (epi == EPI_SILU_MUL ? BM : 2 * BM) ||
        (epi == EPI_SILU_MUL) != (gather_rows != nullptr)) return -7;
    return bt == PAIR_FORM ? launch_pair_grouped<PAIR_BT>(X, W, p, E, w_rows, epi, gather_rows, ldx, max_tiles, st)
                           : launch_pair_grouped<128>(X, W, p, E, w_rows, epi, gather_rows, ldx, max_tiles, st);
  }
  if (gather_rows != nullptr && (bt > GATHER_BT_MAX || splits > 1 || ldx % 8)) return -7;
  if (splits < 1 || splits > 8 || splits > (K + BK - 1) / BK) splits = 1;
  CUtensorMap tw, tx;
  GemmParams p{N, K, cap, ldo, out, reinterpret_cast<const int4*>(tiles), n_tiles, up_offset, nullptr, nullptr, err, nullptr, CommCtx{}, 0, nullptr, nullptr, splits, nullptr, {}};
  if (packed && splits == 1 && (bt == 16 || bt == 32) && epi == EPI_SILU_MUL) {
    const int rc = launch_thin_grouped(X, W, p, E, gather_rows, ldx, max_tiles, bt, st);
    if (rc <= 0) return rc;
  }
  if (weight_map(&tw, W, E, N, w_rows, K, K, epi == EPI_SILU_MUL, packed, &p)) return -1;
  if (gather_rows != nullptr) {
    p.gather_rows = gather_rows;
    p.gx = static_cast<const bf16*>(X);
    p.ldgx = ldx;
    if (make_map(&tx, X, K, bt, 0, ldx, 0, bt)) return -1;  // unused by the gathering producer, but a valid map
  } else if (make_map(&tx, X, K, cap, 0, K, 0, bt == 128 ? VAR_BOX : bt)) return -1;  // 128: Cfg::VAR_N
  switch (epi) {
    case EPI_BF16: return dispatch_bt<EPI_BF16, true>(bt, tw, tx, p, max_tiles, st);
    case EPI_SILU_MUL: return dispatch_bt<EPI_SILU_MUL, true>(bt, tw, tx, p, max_tiles, st);
  }
  return -6;
}

// Tensor-parallel output projection: out[T, N] = bf16(residual + sum over ranks of X_r[T, K_r] W_r[N, K_r]^T).
// Every rank calls this with its K-shard; the all-reduce happens inside the GEMM epilogue over peer memory.
// Needs T * N <= ctx->slot_elems and ceil(N/128) * ceil(T/bt) <= ctx->max_blocks.
extern "C" int b200_gemm_allreduce(const CommCtx* ctx, const void* X, const void* W, const void* residual, void* out,
                                   int T, int N, int K, int ldx, int ldw, int bt, cudaStream_t st) {
  if (T <= 0) return 0;
  if (bt <= 0) bt = b200_pick_bt(T);
  const int gy = (T + bt - 1) / bt;
  if (static_cast<unsigned long long>(T) * N > ctx->slot_elems || ((N + BM - 1) / BM) * gy > ctx->max_blocks) return -7;
  CUtensorMap tw, tx;
  if (make_map(&tw, W, K, N, 0, ldw, 0, BM)) return -1;
  if (make_map(&tx, X, K, T, 0, ldx, 0, bt)) return -1;
  GemmParams p{N, K, T, N, out, nullptr, nullptr, 0, nullptr, nullptr, ctx->err, static_cast<const bf16*>(residual), *ctx, 0, nullptr, nullptr, 1, nullptr, {}};
  return dispatch_bt<EPI_ALLREDUCE, false>(bt, tw, tx, p, gy, st);
}

// Expert-parallel down projection: grouped GEMM whose epilogue scatters every output row to the owner of its
// token (`meta[row] = (rank, pair slot)`, `pair_out[rank]` = that rank's [pairs, N] buffer as mapped in this process).
extern "C" int b200_gemm_grouped_scatter(const void* X, const void* W, int cap, int E, int N, int K, int bt,
                                         const void* tiles, const int* n_tiles, int max_tiles, const void* meta,
                                         void* const* pair_out, int world, int* err, int packed, cudaStream_t st) {
  if (max_tiles <= 0) return 0;
  CUtensorMap tw, tx;
  GemmParams p{N, K, cap, N, nullptr, reinterpret_cast<const int4*>(tiles), n_tiles, 0, nullptr, nullptr, err, nullptr,
               CommCtx{}, 0, nullptr, nullptr, 1, static_cast<const int2*>(meta), {}};
  if (weight_map(&tw, W, E, N, N, K, K, false, packed, &p)) return -1;
  if (make_map(&tx, X, K, cap, 0, K, 0, bt)) return -1;
  for (int r = 0; r < world && r < MAX_RANKS; ++r) p.pair_out[r] = static_cast<bf16*>(pair_out[r]);
  return dispatch_bt<EPI_SCATTER, true>(bt, tw, tx, p, max_tiles, st);
}

// Tensor-parallel output projection with a reduce-scatter epilogue: every rank calls it with its K-shard of X and
// W [N, K]; afterwards the fp32 partials of rank r's rows [r * T / R, (r + 1) * T / R) sit in rank r's receive
// slots, one per source rank, with one arrival flag per (source, tile). b200_reduce_norm_allgather consumes them.
// T must be a multiple of world * bt. Needs (T / R) * N <= ctx->slot_elems and the tile count <= ctx->max_blocks.
extern "C" int b200_gemm_reduce_scatter(const CommCtx* ctx, const void* X, const void* W, int T, int N, int K, int ldx,
                                        int ldw, int bt, cudaStream_t st) {
  if (T <= 0) return 0;
  if (bt <= 0) bt = b200_pick_bt(T / ctx->world);
  if (T % (ctx->world * bt)) return -7;
  const int rpr = T / ctx->world, gy = T / bt;
  if (static_cast<unsigned long long>(rpr) * N > ctx->slot_elems || ((N + BM - 1) / BM) * gy > ctx->max_blocks) return -7;
  CUtensorMap tw, tx;
  if (make_map(&tw, W, K, N, 0, ldw, 0, BM)) return -1;
  if (make_map(&tx, X, K, T, 0, ldx, 0, bt)) return -1;
  GemmParams p{N, K, T, N, nullptr, nullptr, nullptr, 0, nullptr, nullptr, ctx->err, nullptr, *ctx,
               rpr, nullptr, nullptr, 1, nullptr, {}};
  // each rank runs the tiles of the next rank first and its own last: partials reach their owners early, and an
  // owner's waits fall at the end of its grid, on tiles every peer has already pushed
  p.y_rot = ((ctx->rank + 1) % ctx->world) * (rpr / bt);
  return dispatch_bt<EPI_REDUCE_SCATTER, false>(bt, tw, tx, p, gy, st);
}

// All-gather -> GEMM: X [T, K] is this rank's full activation buffer into which every owner rank pushes its row
// shard (allreduce.cu: norm_allgather); a tile starts as soon as its owner's shard has arrived (x_flags[owner] >=
// *x_epoch). out[T, N] = X W^T, bf16 or fp32. `y_rot` = rank * (rows_per_rank / bt) makes each rank start with its
// own shard, which is already there.
extern "C" int b200_gemm_gathered(const void* X, const void* W, void* out, int T, int N, int K, int ldx, int ldw,
                                  int out_f32, int bt, int rows_per_rank, int y_rot, const uint32_t* x_flags,
                                  const uint32_t* x_epoch, int* err, cudaStream_t st) {
  if (T <= 0) return 0;
  if (bt <= 0) bt = b200_pick_bt(rows_per_rank);
  if (rows_per_rank % bt) return -7;
  CUtensorMap tw, tx;
  if (make_map(&tw, W, K, N, 0, ldw, 0, BM)) return -1;
  if (make_map(&tx, X, K, T, 0, ldx, 0, bt)) return -1;
  GemmParams p{N, K, T, N, out, nullptr, nullptr, 0, nullptr, nullptr, err, nullptr, CommCtx{}, rows_per_rank, x_flags,
               x_epoch, 1, nullptr, {}};
  p.y_rot = y_rot;
  const int gy = (T + bt - 1) / bt;
  return out_f32 ? dispatch_bt<EPI_F32, false>(bt, tw, tx, p, gy, st) : dispatch_bt<EPI_BF16, false>(bt, tw, tx, p, gy, st);
}

extern "C" int b200_argmax_finish(const float* part_max, const int* part_idx, int n_tiles, int T, int64_t* out,
                                  float* out_val, cudaStream_t st) {
  if (T <= 0) return 0;
  const int threads = T <= sm_count() && n_tiles > 512 ? 1024 : 256;
  return launch_pdl(argmax_finish_kernel, dim3(T), dim3(threads), 0, st, part_max, part_idx, n_tiles, T, out, out_val) ==
                 cudaSuccess ? 0 : -4;
}

// ------------------------------------------------------------------ allocation-free greedy head
// See b200serve_noalloc.h. The per-tile (max, index) partials of the LM-head argmax live in a
// fixed device array instead of caller-provided workspace.
#include <stdio.h>

#include "b200serve_noalloc.h"

namespace {
constexpr size_t NOALLOC_PART_ELEMS = static_cast<size_t>(B200_NOALLOC_MAX_ROWS) * B200_NOALLOC_MAX_TILES;
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_PART_ELEMS * (sizeof(float) + sizeof(int))];
constexpr int NOALLOC_MAX_DEVICES = MAX_DEVICES;
void* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {nullptr};
}  // namespace

extern "C" int b200_lm_head_argmax_noalloc(const void* X, const void* W, int64_t* out_idx, float* out_val, int T, int V,
                                           int K, int ldx, int ldw, int* err, cudaStream_t st) {
  if (T <= 0) return 0;
  const int n_tiles = (V + BM - 1) / BM;
  if (T > B200_NOALLOC_MAX_ROWS || n_tiles > B200_NOALLOC_MAX_TILES) {
    fprintf(stderr,
            "b200_lm_head_argmax_noalloc: %d rows x %d vocabulary entries exceed the built-in scratch "
            "(at most %d rows and %d entries)\n",
            T, V, B200_NOALLOC_MAX_ROWS, B200_NOALLOC_MAX_TILES * BM);
    return B200_NOALLOC_TOO_LARGE;
  }
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return B200_NOALLOC_BAD_DEVICE;
  if (g_noalloc_ptr[dev] == nullptr) {
    // The array's name is only a host-side handle; the device address of this device's copy has to be
    // asked for, once, with the device current. Not a stream operation: do the first call outside capture.
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr) return B200_NOALLOC_NO_SYMBOL;
    g_noalloc_ptr[dev] = p;
  }
  float* part_max = static_cast<float*>(g_noalloc_ptr[dev]);
  int* part_idx = reinterpret_cast<int*>(part_max + NOALLOC_PART_ELEMS);
  const int bt = b200_pick_bt(T);
  CUtensorMap tw, tx;
  if (make_map(&tw, W, K, V, 0, ldw, 0, BM)) return -1;
  if (make_map(&tx, X, K, T, 0, ldx, 0, bt)) return -1;
  GemmParams p{V, K, T, 0, nullptr, nullptr, nullptr, 0, part_max, part_idx, err, nullptr, CommCtx{}, 0, nullptr, nullptr, 1, nullptr, {}};
  const int rc = dispatch_bt<EPI_ARGMAX, false>(bt, tw, tx, p, (T + bt - 1) / bt, st);
  if (rc) return rc;
  argmax_finish_kernel<<<T, 256, 0, st>>>(part_max, part_idx, n_tiles, T, out_idx, out_val);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
