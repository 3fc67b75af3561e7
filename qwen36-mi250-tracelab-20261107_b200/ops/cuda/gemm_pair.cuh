// The same weight-stationary GEMM as gemm_tcgen05.cu with two SMs on one output tile (tcgen05 cta_group::2), for launches
// with enough token rows. Included by gemm_tcgen05.cu, whose parameters, epilogue names and tensor maps it uses.
//
// A cluster of two CTAs owns a tile of 256 accumulator rows x up to 256 token rows: each CTA holds 128 accumulator rows (all
// token columns of them, in its own TMEM), loads the 128 weight rows that belong to them and HALF of the token rows; the MMA
// that the first CTA issues for both reads the other half out of its peer's shared memory.
//
// Why: on one SM a 128 x 256 tile is bound by shared memory, not by the tensor cores. Per k-block it writes 48 KB and reads
// 48 KB for 512 cycles of MMA (the SM moves 128 bytes a cycle), the 128 x 128 gate + up pair of an expert tile 48 and 64 KB.
// Here a k-block writes 32 KB and reads 32 KB per SM for the same 512 cycles, and a third fewer bytes come out of L2.
#pragma once

namespace b200 {

constexpr int PAIR_BT = 256;      // most token rows of a tile
constexpr int PAIR_N_STEP = 32;   // the MMA's column count is a multiple of this when it has 256 rows
constexpr int PAIR_A_BYTES = BM * BK * 2;
constexpr int PAIR_GROUPS = 2;    // epilogue warpgroups: they take alternate batches of 16 token columns
constexpr int PAIR_GATHER_WARP = 2 + 4 * PAIR_GROUPS;  // the row-fetching warps: warp 0 and three behind the epilogue's
constexpr int PAIR_GATHER_WARPS = 4;
constexpr int pair_threads(int epi) { return 32 * (epi == EPI_SILU_MUL ? PAIR_GATHER_WARP + PAIR_GATHER_WARPS - 1 : PAIR_GATHER_WARP); }
constexpr int PAIR_OUT_BYTES = 2 * 16 * BM * 2;  // per group: two staging buffers (SiLU: the exchange and one buffer)

// PBT: most token rows of a tile, 256 or 128. Tiles of up to 128 rows leave room for eight stages instead of six, which is 128 KB
// of weights on their way to an SM and not 96: expert block of 64 rows per expert, gate/up 202 -> 193 us, down 99 -> 96.
template <int PBT>
struct PairCfg {
  static constexpr int B_BYTES = PBT / 2 * BK * 2;
  static constexpr int STAGE_BYTES = PAIR_A_BYTES + B_BYTES;
  static constexpr int STAGES = PBT == 256 ? 6 : 8;
  static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + 256 + PAIR_GROUPS * PAIR_OUT_BYTES;
};

// Whether `ok` holds in all 128 threads of epilogue group `id - 2`.
__device__ __forceinline__ bool group_all(bool ok, int id) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.aligned.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"(static_cast<uint32_t>(ok)), "r"(id) : "memory");
  return r != 0;
}
__device__ __forceinline__ void group_sync(int id) { asm volatile("barrier.cta.sync.aligned %0, 128;" ::"r"(id) : "memory"); }

// EPI_BF16 (dense, or grouped with rows that are sorted already), EPI_F32 or EPI_ARGMAX (dense) or EPI_SILU_MUL (grouped, rows fetched by index,
// tile-packed weights). In a SiLU tile a CTA's 128 accumulator rows are 64 gate rows and the 64 up rows
// that go with them.
template <int EPI, bool GROUPED, int PBT>
__global__ void __launch_bounds__(pair_threads(EPI), 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, GemmParams p) {
  constexpr bool SILU = EPI == EPI_SILU_MUL;
  constexpr int PAIR_ROWS = SILU ? BM : 2 * BM;  // output columns of a tile
  constexpr int CTA_ROWS = PAIR_ROWS / 2;
  constexpr int STAGES = PairCfg<PBT>::STAGES, STAGE_BYTES = PairCfg<PBT>::STAGE_BYTES;
  constexpr int LANE_ROWS = PBT / 8;  // of a CTA's half of the rows, fetched by a group of eight lanes
  static_assert(EPI == EPI_BF16 || (!GROUPED && (EPI == EPI_F32 || EPI == EPI_ARGMAX)) || (SILU && GROUPED), "epilogues of the pair form");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full = bars;                         // used in the first CTA: both CTAs' loads are counted there
  uint64_t* empty = bars + STAGES;          // one in each CTA, the MMAs' commits arrive at both
  uint64_t* acc_full = bars + 2 * STAGES;   // [2], both CTAs
  uint64_t* acc_empty = acc_full + 2;            // [2], used in the first CTA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* out_stage = smem + STAGES * STAGE_BYTES + 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int tiles_n = (p.N + PAIR_ROWS - 1) / PAIR_ROWS;
  const int tile0 = static_cast<int>(blockIdx.x >> 1), tstep = static_cast<int>(gridDim.x >> 1);
  const int bt = p.pair_bt;
  const int num_k = p.K / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], SILU ? 3 : 1);  // the announcement of bytes, and of each CTA's rows
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 2 * 4 * PAIR_GROUPS); }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // both CTAs' barriers are ready before anything arrives at them from the other side
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (GROUPED) {  // the tile table was written by the kernel just before this one
    pdl_wait();
    if (warp == 0) pdl_launch();
  }
  int4 t_next = make_int4(0, 0, 0, 0);
  if (GROUPED) t_next = p.tiles[tile0 / tiles_n];
  const int total = tiles_n * (GROUPED ? *p.n_tiles : p.grid_y);

  // tile -> weight tile, expert, first token row, token rows; the next table entry is requested one tile ahead
  auto tile_geom = [&](int tile, int& nx, int& expert, int& row0, int& nrows) {
    nx = tile % tiles_n;
    expert = 0;
    if (GROUPED) {
      const int4 t = t_next;
      if (total - tile > tstep) t_next = p.tiles[(tile + tstep) / tiles_n];
      expert = t.x; row0 = t.y; nrows = t.z;
    } else {
      row0 = tile / tiles_n * bt;
      nrows = min(bt, p.T - row0);
    }
  };
  auto columns = [](int nrows) { return (nrows + PAIR_N_STEP - 1) / PAIR_N_STEP * PAIR_N_STEP; };
  // this CTA's weight rows of k-block kb; its bytes count at the first CTA's barrier `bar`
  auto load_weights = [&](uint8_t* st, uint32_t bar, int nx, int expert, int kb) {
    if (SILU) {  // packed: 128 gate rows, then 128 up rows of a k-block
      const int y = ((expert * p.w_tiles + nx) * num_k + kb) * (2 * BM) + static_cast<int>(rank) * CTA_ROWS;
      tma_load_2d_pair(st, &tmW, bar, 0, y);
      tma_load_2d_pair(st + PAIR_A_BYTES / 2, &tmW, bar, 0, y + BM);
    } else {  // (a last tile without a second half: a row behind the map's end, which loads zeros)
      const int wt = 2 * nx + static_cast<int>(rank);
      if (p.packed) tma_load_2d_pair(st, &tmW, bar, 0, ((expert * p.w_tiles + wt) * num_k + kb) * BM);
      else tma_load_2d_pair(st, &tmW, bar, kb * BK, wt * BM);
    }
  };

  if (SILU && (warp == 0 || warp >= PAIR_GATHER_WARP)) {
    // ---------------- row-fetching producers: warp w of PAIR_GATHER_WARPS fills every PAIR_GATHER_WARPS-th stage, the weights
    // by TMA, this CTA's half of the token rows by index as 16-byte asynchronous copies into the swizzled operand layout (as
    // in gemm_swapab_kernel), and announces the rows when they have landed.
    // The announcement is a release for the cluster (the first CTA issues the MMA that reads the second one's rows, and acquires
    // at that scope), of shared memory only, which is all that the copies wrote and costs nothing that shows: passes of 8 x 1024
    // and 2048 rows 6.21 and 2.59 ms with and without it. A release of everything waits for the SM's other traffic: 6.38 ->
    // 6.78 and 2.67 -> 2.80, and 7.88 and 3.92 where one thread of the second CTA passes its warps' announcements on. A whole
    // stage per warp, so that one lane announces it. (Four-row TMA gathers take 70 cycles each: 1.26 us for the 32 of a stage.)
    const int gw = warp == 0 ? 0 : warp - PAIR_GATHER_WARP + 1, j = lane & 7;
    int first = gw;  // the warp's first k-block of the tile
    int it = gw;     // stages of this warp and all others before it
    bool live = true;
    for (int tile = tile0; tile < total && live; tile += tstep) {
      int nx, expert, row0, nrows;
      tile_geom(tile, nx, expert, row0, nrows);
      const int cols = columns(nrows), half = cols / 2, t0 = static_cast<int>(rank) * half;
      int g[LANE_ROWS];
#pragma unroll
      for (int i = 0; i < LANE_ROWS; ++i) {  // (columns behind the last row keep what they hold: nobody reads their results)
        const int r = (lane >> 3) + 4 * i;
        g[i] = r < half && t0 + r < nrows ? p.gather_rows[row0 + t0 + r] : -1;
      }
      int kb = first;
      for (; kb < num_k; kb += PAIR_GATHER_WARPS, it += PAIR_GATHER_WARPS) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!mbar_wait<true>(&empty[s], ph ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag)) { live = false; break; }
        uint8_t* st = smem + s * STAGE_BYTES;
        const uint32_t bar = dsmem_addr(smem_u32(&full[s]), 0);
        if (lane == 0) {
          if (rank == 0) mbar_expect_tx(&full[s], 2 * PAIR_A_BYTES);
          load_weights(st, bar, nx, expert, kb);
        }
        const uint32_t xb = smem_u32(st + PAIR_A_BYTES);
        const bf16* gx = p.gx + kb * BK + j * 8;
#pragma unroll
        for (int i = 0; i < LANE_ROWS; ++i) {
          const int r = (lane >> 3) + 4 * i;
          if (g[i] >= 0)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                         ::"r"(xb + (r >> 3) * 1024 + (r & 7) * 128 + ((j ^ (r & 7)) << 4)), "l"(gx + static_cast<size_t>(g[i]) * p.ldgx)
                         : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");  // (also: no copy of this lane may outlive the CTA's shared memory)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // for the tensor core's reads
        __syncwarp();
        if (lane == 0) mbar_arrive_release_shared(bar);
      }
      first = kb - num_k;
    }
  } else if (warp == 0) {
    // ---------------- producer, one in each CTA
    if (elect_one()) {
      int it = 0, pre = 0;
      bool live = true;
      const uint32_t dense_bytes = 2 * PAIR_A_BYTES + bt * (BK * 2);  // (rows behind the last one load zeros)
      // dense weights are written by nobody in the stream: the first stages of the first tile are requested before the wait
      if (!GROUPED && tile0 < total) {
        int nx, expert, row0, nrows;
        tile_geom(tile0, nx, expert, row0, nrows);
        pre = num_k < STAGES ? num_k : STAGES;
        for (int kb = 0; kb < pre; ++kb) {
          if (rank == 0) mbar_expect_tx(&full[kb], dense_bytes);
          load_weights(smem + kb * STAGE_BYTES, dsmem_addr(smem_u32(&full[kb]), 0), nx, 0, kb);
        }
      }
      pdl_wait();
      if (!GROUPED) pdl_launch();
      for (int tile = tile0; tile < total && live; tile += tstep) {
        int nx, expert, row0, nrows;
        tile_geom(tile, nx, expert, row0, nrows);
        const int half = columns(nrows) / 2;
        // grouped: boxes of VAR_BOX rows, as many as cover the half
        const int boxes = (half + VAR_BOX - 1) / VAR_BOX;
        for (int kb = 0; kb < num_k; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          uint8_t* st = smem + s * STAGE_BYTES;
          const uint32_t bar = dsmem_addr(smem_u32(&full[s]), 0);
          if (it >= pre) {
            if (!mbar_wait<true>(&empty[s], ph ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag)) { live = false; break; }
            if (rank == 0) mbar_expect_tx(&full[s], GROUPED ? 2 * (PAIR_A_BYTES + boxes * (VAR_BOX * BK * 2)) : dense_bytes);
            load_weights(st, bar, nx, expert, kb);
          }
          const int x0 = row0 + static_cast<int>(rank) * half;
          if (GROUPED) {
            for (int b = 0; b < boxes; ++b)
              tma_load_2d_pair(st + PAIR_A_BYTES + b * (VAR_BOX * BK * 2), &tmX, bar, kb * BK, x0 + b * VAR_BOX);
          } else {
            tma_load_2d_pair(st + PAIR_A_BYTES, &tmX, bar, kb * BK, x0);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: the first CTA's, for both
    if (rank == 0 && elect_one()) {
      bool ok = true;
      int it = 0, lt = 0;
      for (int tile = tile0; tile < total && ok; tile += tstep, ++lt) {
        int nx, expert, row0, nrows;
        tile_geom(tile, nx, expert, row0, nrows);
        const uint32_t idesc = umma_idesc_bf16(2 * BM, columns(nrows));
        const int acc = lt & 1;
        const uint32_t tmem = tmem_base + acc * PAIR_BT;
        ok = mbar_wait<true>(&acc_empty[acc], ((lt >> 1) & 1) ^ 1, p.err, ERR_WAIT_TMEM, abort_flag);
        if (ok) tc_fence_after();
        for (int kb = 0; kb < num_k && ok; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait<true>(&full[s], (it / STAGES) & 1, p.err, ERR_WAIT_FULL, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_pair(tmem, umma_smem_desc(a_addr + k * UMMA_K * 2), umma_smem_desc(a_addr + PAIR_A_BYTES + k * UMMA_K * 2),
                           idesc, (kb | k) != 0);
          umma_commit_pair(&empty[s]);
        }
        umma_commit_pair(&acc_full[acc]);  // always arrive so that the epilogues are released
      }
    }
  } else {
    // ---------------- epilogue of this CTA's accumulator rows: warp quarter q owns TMEM lanes [32 q, 32 q + 32)
    pdl_wait();
    const int q = warp & 3, group = (warp - 2) >> 2, bar_id = 2 + group;
    const int tid = q * 32 + lane;
    uint8_t* stage = out_stage + group * PAIR_OUT_BYTES;
    int lt = 0, out_buf = 0;
    for (int tile = tile0; tile < total; tile += tstep, ++lt) {
      int nx, expert, row0, nrows;
      tile_geom(tile, nx, expert, row0, nrows);
      (void)expert;
      const int acc = lt & 1;
      const uint32_t tmem = tmem_base + acc * PAIR_BT + (static_cast<uint32_t>(q * 32) << 16);
      const int n0 = nx * PAIR_ROWS + static_cast<int>(rank) * CTA_ROWS;
      // the batches below hold barriers: all four warps of the group take them, or none
      const bool ok = group_all(mbar_wait<true>(&acc_full[acc], (lt >> 1) & 1, p.err, ERR_WAIT_TMEM, abort_flag) && !*abort_flag, bar_id);
      tc_fence_after();
      if (ok) {
#pragma unroll 1
        for (int c = 16 * group; c < nrows; c += 16 * PAIR_GROUPS) {
          float v[16];
          tmem_ld16(tmem + c, v);
          if (SILU) {
            // lanes 0-63 hold gate rows, 64-127 the up rows of the same outputs: the two threads of an output swap half of
            // their columns (rounded to bf16, as the unfused sequence of ops rounds them) and finish eight each
            const bool up = q >= 2;
            uint4 mine, theirs;
            bf16* me = reinterpret_cast<bf16*>(&mine);
            const bf16* te = reinterpret_cast<const bf16*>(&theirs);
#pragma unroll
            for (int j = 0; j < 8; ++j) me[j] = __float2bfloat16(up ? v[j] : v[8 + j]);
            reinterpret_cast<uint4*>(stage)[tid] = mine;
            group_sync(bar_id);
            theirs = reinterpret_cast<const uint4*>(stage)[tid ^ 64];
            bf16* ob = reinterpret_cast<bf16*>(stage + 128 * 16) + (up ? 8 * CTA_ROWS : 0) + (tid & 63);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float own = __bfloat162float(__float2bfloat16(up ? v[8 + j] : v[j])), other = __bfloat162float(te[j]);
              const float gate = up ? other : own, lin = up ? own : other;
              ob[j * CTA_ROWS] = __float2bfloat16(__bfloat162float(__float2bfloat16(silu_f(gate))) * lin);
            }
            group_sync(bar_id);
            const int r = tid >> 3, col = (tid & 7) * 8;
            const uint4 o = *reinterpret_cast<const uint4*>(stage + 128 * 16 + (r * CTA_ROWS + col) * 2);
            if (c + r < nrows && n0 + col < p.N)
              *reinterpret_cast<uint4*>(static_cast<bf16*>(p.out) + static_cast<size_t>(row0 + c + r) * p.ldo + n0 + col) = o;
          } else if (EPI == EPI_F32) {
            if (n0 + tid < p.N) {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (c + j < nrows) static_cast<float*>(p.out)[static_cast<size_t>(row0 + c + j) * p.ldo + n0 + tid] = v[j];
            }
          } else if (EPI == EPI_ARGMAX) {
            // the warps' picks of 16 columns meet in one of two buffers (as below: read ahead of the reader's next barrier)
            float2* red = reinterpret_cast<float2*>(stage) + out_buf * (4 * 16);
            out_buf ^= 1;
            float best;
            int at;
            argmax_columns(v, n0 + tid, n0 + tid < p.N, lane, best, at);
            if ((lane & 1) == 0) red[q * 16 + argmax_column(lane)] = make_float2(best, __int_as_float(at));
            group_sync(bar_id);
            const int wt = 2 * nx + static_cast<int>(rank);
            if (tid < 16 && c + tid < nrows && wt * BM < p.N) {
              float2 m = red[tid];
#pragma unroll
              for (int w = 1; w < 4; ++w) {
                const float2 o = red[w * 16 + tid];
                if (o.x > m.x || (o.x == m.x && __float_as_int(o.y) < __float_as_int(m.y))) m = o;
              }
              const size_t o = static_cast<size_t>(wt) * p.T + row0 + c + tid;
              p.part_max[o] = m.x;
              p.part_idx[o] = __float_as_int(m.y);
            }
          } else {
            // [16 rows][128 weight rows] bf16, two buffers: a thread's reads of one precede its next barrier, behind which
            // it is written again
            bf16* ob = reinterpret_cast<bf16*>(stage) + out_buf * (16 * BM);
            out_buf ^= 1;
#pragma unroll
            for (int j = 0; j < 16; ++j) ob[j * BM + tid] = __float2bfloat16(v[j]);
            group_sync(bar_id);
            const int col = (lane & 15) * 8;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int r = i * 8 + q * 2 + (lane >> 4);
              const uint4 o = *reinterpret_cast<const uint4*>(ob + r * BM + col);
              if (c + r < nrows && n0 + col < p.N)
                *reinterpret_cast<uint4*>(static_cast<bf16*>(p.out) + static_cast<size_t>(row0 + c + r) * p.ldo + n0 + col) = o;
            }
          }
        }
      }
      // every tcgen05.ld of the warp has completed: the next but one tile may overwrite this accumulator
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(dsmem_addr(smem_u32(&acc_empty[acc]), 0));
      if (!ok) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the peer's shared memory and barriers are in use until both are done
  if (warp == 1) { tc_fence_after(); tmem_dealloc_pair(tmem_base, 512); }
}

}  // namespace b200
