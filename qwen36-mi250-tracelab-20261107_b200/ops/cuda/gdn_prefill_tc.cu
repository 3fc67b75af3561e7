// Gated DeltaNet chunked prefill on the sm_100a tensor cores (head dims 128 x 128, 64-row chunks).
//
// Two kernels replace the fp32 CUDA-core WY transform and state pass of gdn_prefill.cu for the full-size model:
//
//  gdn_wy_tc   : one CTA per (pair of chunks, value head); thread i owns token row i of the 128 rows = TMEM lane i.
//                TMA brings the raw q / k / v rows of both chunks into 128B-swizzled tiles. tcgen05.mma forms the
//                128 x 128 Gram matrices K K^T and Q K^T (only the two 64 x 64 diagonal blocks are used), threads
//                turn them into A = (k beta) k^T decay (strictly lower) and the causal scores, each thread then
//                solves its own column of T = (I + A)^-1 by forward substitution, and a second pair of MMAs with
//                the block-diagonal T diag(beta) forms w = T (k beta e^g) and u = T (v beta). Everything the state
//                pass needs is written as bf16: w, u, q e^g, k e^{g_last - g}, scores, and g_last in fp32
//                (reference: engine/fast/gdn_chunk.py:203-471).
//  gdn_scan_tc : one CTA per (sequence, value head), chunks in order. The transposed fp32 state S^T [dv, dk] lives
//                in TMEM for the whole sequence, with a bf16 copy in shared memory as the MMA operand. Per chunk:
//                v_new^T = u^T - S^T w^T and o^T = S^T (q e^g)^T (tcgen05, N = 64 tokens), v_new goes to shared memory
//                as bf16, then S^T = S^T e^{g_last} + v_new^T (k e^{g_last-g}) and o^T += v_new^T scores^T
//                (reference: engine/fast/gdn_chunk.py:494-628). A TMA producer warp runs two chunks ahead, four warps
//                store o while the next chunk is under way.
//
// Operands are rounded to bf16 where the reference's chunk kernels round them too (w, u, the decayed q / k, the
// state as an MMA operand); accumulation and the resident state are fp32. Padding rows of a partial chunk have
// beta = 0 and g = 0, which makes them identity rows of T and keeps them out of the state.
#include "common.cuh"

namespace b200 {

struct ChunkInfoTc {  // same layout as gdn_prefill.cu's ChunkInfo
  int seg, row0, nrows, first;
};

// Workspace (bytes) for NCH = chunks * heads: A-region [NCH * 256 rows][128] bf16 (w | u | qg | kg, 64 rows each),
// then the scores [NCH * 64 rows][64] bf16, then g_last fp32 [NCH].
__host__ __device__ inline size_t tc_region_b(size_t nch) { return nch * 65536; }
__host__ __device__ inline size_t tc_region_g(size_t nch) { return nch * 65536 + nch * 8192; }

// byte offset of the 16-byte chunk `c16` (0..7) of row `row` inside a 128B-swizzled tile atom
__device__ __forceinline__ uint32_t swz(uint32_t row, uint32_t c16) { return row * 128 + ((c16 ^ (row & 7)) << 4); }

struct WyParams {
  const bf16* mixed;
  int ld, b_off, a_off;
  const ChunkInfoTc* chunks;
  int n_chunks;
  const float* A_log;
  const float* dt_bias;
  uint8_t* work;
  int HK, HV;
  int* err;
};

constexpr int WY_SMEM = 3 * 32768 + 1024 /*align*/ + 5120 /*small arrays + barriers*/;

// In-kernel phase clocks: thread 0 of CTA (0, 0) stamps clock64() at the phase boundaries of the WY kernel; the host
// reads the last launch's stamps with b200_gdn_wy_phase_clocks (the reference's HIP kernel has the same kind of
// phase clocks behind its PROF template argument, engine/fast/hip/gdn_chain.hip:163-165, 367-385).
__device__ long long g_wy_clocks[12];
#define WY_STAMP(k) do { if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) g_wy_clocks[k] = clock64(); } while (0)

// Bound by shared memory: the substitution's reads of A (16 bytes for two lanes' four products each) and two CTAs per SM.
// 230 -> 198 us at 8192 rows x 32 heads, 64 -> 54 at 2048, since the columns of T live in registers (the v rows then load at
// the start and not behind the substitution) and w and u leave by TMA.
// 256 threads. Row phases: thread (i = tid & 127, half = tid >> 7) works on token row i = TMEM lane i and on one
// 64-column half of it. Substitution phase: thread (col = tid >> 1, part = tid & 1) owns column col of T together with
// its neighbour lane; the pair splits every dot product and meets in one shuffle.
__global__ void __launch_bounds__(256, 2)
gdn_wy_tc_kernel(const __grid_constant__ CUtensorMap tmConv, const __grid_constant__ CUtensorMap tmA, WyParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;            // raw q, later the fp32 A blocks, the bf16 block-diagonal T diag(beta), at last w
  uint8_t* sK = smem + 32768;    // raw k, later k e^g / |k|, at last u
  uint8_t* sV = smem + 65536;    // raw v
  float* sG = reinterpret_cast<float*>(smem + 98304);  // [128] cumulative log decay
  float* sRk = sG + 128;                               // [128] 1 / |k|
  float* sBeta = sRk + 128;                            // [128]
  float* sPart = sBeta + 128;                          // [2][128][2] partial squared norms of the two row halves
  float* sFq = sPart + 512;                            // [128] row factors of the decayed q copy
  float* sFk = sFq + 128;                              // [128] row factors of the decayed k copy
  float* sTot = sFk + 128;                             // [4] warp totals of the scan
  uint64_t* bars = reinterpret_cast<uint64_t*>(sTot + 8);
  uint64_t* tma_bar = bars;
  uint64_t* mma_bar = bars + 1;
  uint64_t* v_bar = bars + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i = tid & 127, half = tid >> 7;
  const int c = i >> 6, r = i & 63;  // chunk of the pair, row inside it
  const int h = blockIdx.y, hk = h / (p.HV / p.HK);
  const int key_dim = p.HK * 128;
  const int chunk_idx = 2 * blockIdx.x + c;
  const bool present = chunk_idx < p.n_chunks;

  if (tid == 0) {
    mbar_init(tma_bar, 1);
    mbar_init(mma_bar, 1);
    mbar_init(v_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmConv);
    tma_prefetch_desc(&tmA);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  pdl_wait();
  pdl_launch();
  const ChunkInfoTc ci = p.chunks[present ? chunk_idx : 2 * blockIdx.x];
  const bool valid = present && r < ci.nrows;

  if (tid == 0) {
    // q and k rows of both chunks (a missing second chunk re-reads the first: finite data, never written out), then v
    mbar_expect_tx(tma_bar, 2 * 32768);
    mbar_expect_tx(v_bar, 32768);
    for (int cc = 0; cc < 2; ++cc) {
      const int idx = 2 * blockIdx.x + cc;
      const int row0 = p.chunks[idx < p.n_chunks ? idx : 2 * blockIdx.x].row0;
      for (int a = 0; a < 2; ++a) {
        tma_load_2d(sQ + a * 16384 + cc * 8192, &tmConv, tma_bar, hk * 128 + a * 64, row0);
        tma_load_2d(sK + a * 16384 + cc * 8192, &tmConv, tma_bar, key_dim + hk * 128 + a * 64, row0);
      }
      for (int a = 0; a < 2; ++a)
        tma_load_2d(sV + a * 16384 + cc * 8192, &tmConv, v_bar, 2 * key_dim + h * 128 + a * 64, row0);
    }
  }
  WY_STAMP(0);
  // gates and their inclusive scan inside each chunk (two warps per chunk; both halves compute the same values)
  float g = 0.f, beta = 0.f;
  if (valid) {
    const size_t row = static_cast<size_t>(ci.row0 + r);
    g = -__expf(p.A_log[h]) * softplus_f(__bfloat162float(p.mixed[row * p.ld + p.a_off + h]) + p.dt_bias[h]);
    beta = sigmoid_f(__bfloat162float(p.mixed[row * p.ld + p.b_off + h]));
  }
  float gs = g;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float x = __shfl_up_sync(0xffffffffu, gs, o);
    if (lane >= o) gs += x;
  }
  if (half == 0 && lane == 31) sTot[warp] = gs;
  __syncthreads();
  if (warp & 1) gs += sTot[(warp & 3) - 1];
  if (half == 0) { sG[i] = gs; sBeta[i] = beta; }
  __syncthreads();
  const float glast = sG[c * 64 + 63];

  WY_STAMP(1);  // gates done
  bool ok = mbar_wait(tma_bar, 0, p.err, ERR_WAIT_FULL, abort_flag);
  tc_fence_after();
  __syncthreads();
  if (tid == 0 && ok) {
    constexpr uint32_t idesc = umma_idesc_bf16(128, 128);
    const uint32_t qa = smem_u32(sQ), ka = smem_u32(sK);
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const uint32_t off = (kk >> 2) * 16384 + (kk & 3) * 32;
      umma_bf16(tmem, umma_smem_desc(ka + off), umma_smem_desc(ka + off), idesc, kk != 0);          // K K^T
    }
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const uint32_t off = (kk >> 2) * 16384 + (kk & 3) * 32;
      umma_bf16(tmem + 128, umma_smem_desc(qa + off), umma_smem_desc(ka + off), idesc, kk != 0);    // Q K^T
    }
    umma_commit(mma_bar);
  }
  WY_STAMP(2);  // q / k tiles arrived, Gram MMAs issued
  // squared norms: each half sums its 64 columns of the q and k rows
  const uint32_t tile_row = i;  // row inside each 128-row atom
  {
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int c16 = 0; c16 < 8; ++c16) {
      const uint4 qv = *reinterpret_cast<const uint4*>(sQ + half * 16384 + swz(tile_row, c16));
      const uint4 kv = *reinterpret_cast<const uint4*>(sK + half * 16384 + swz(tile_row, c16));
      const bf16* qe = reinterpret_cast<const bf16*>(&qv);
      const bf16* ke = reinterpret_cast<const bf16*>(&kv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x = __bfloat162float(qe[j]), y = __bfloat162float(ke[j]);
        sq += x * x;
        sk += y * y;
      }
    }
    sPart[(half * 128 + i) * 2] = sq;
    sPart[(half * 128 + i) * 2 + 1] = sk;
  }
  __syncthreads();
  const float rq = rsqrtf(sPart[i * 2] + sPart[(128 + i) * 2] + 1e-6f) * 0.08838834764831845f;  // 1 / |q| / sqrt(128)
  const float rk = rsqrtf(sPart[i * 2 + 1] + sPart[(128 + i) * 2 + 1] + 1e-6f);
  if (half == 0) {
    sRk[i] = rk;
    sFq[i] = rq * __expf(gs);
    sFk[i] = rk * __expf(glast - gs);
  }
  const size_t ch = static_cast<size_t>(present ? chunk_idx : 0) * p.HV + h;
  if (present && r == 63 && half == 0)
    *reinterpret_cast<float*>(p.work + tc_region_g(static_cast<size_t>(p.n_chunks) * p.HV) + ch * 4) = glast;
  __syncthreads();
  // the decayed copies the state pass consumes, q e^g / |q| / sqrt(dk) and k e^{g_last - g} / |k|: warp w copies rows
  // [16 w, 16 w + 16); 16 lanes cover the 256 bytes of one row, so every store instruction writes two whole rows
#pragma unroll 2
  for (int it = 0; it < 8; ++it) {
    const int row = warp * 16 + it * 2 + (lane >> 4), chunk = lane & 15;
    const int cpr = row >> 6, rrow = row & 63;
    const int cidx = 2 * blockIdx.x + cpr;
    const uint32_t off = (chunk >> 3) * 16384 + swz(row, chunk & 7);
    const uint4 qv = *reinterpret_cast<const uint4*>(sQ + off);
    const uint4 kv = *reinterpret_cast<const uint4*>(sK + off);
    const float fq = sFq[row], fk = sFk[row];
    const bf16* qe = reinterpret_cast<const bf16*>(&qv);
    const bf16* ke = reinterpret_cast<const bf16*>(&kv);
    uint4 qo, ko;
    bf16* qoe = reinterpret_cast<bf16*>(&qo);
    bf16* koe = reinterpret_cast<bf16*>(&ko);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      qoe[j] = __float2bfloat16(__bfloat162float(qe[j]) * fq);
      koe[j] = __float2bfloat16(__bfloat162float(ke[j]) * fk);
    }
    if (cidx < p.n_chunks) {
      bf16* base = reinterpret_cast<bf16*>(p.work) + (static_cast<size_t>(cidx) * p.HV + h) * 256 * 128;
      reinterpret_cast<uint4*>(base + (128 + rrow) * 128)[chunk] = qo;
      reinterpret_cast<uint4*>(base + (192 + rrow) * 128)[chunk] = ko;
    }
  }
  WY_STAMP(3);  // norms + decayed copies written
  __syncthreads();  // sRk complete; every thread is done with the raw q tile
  ok = mbar_wait(mma_bar, 0, p.err, ERR_WAIT_TMEM, abort_flag) && !*abort_flag;
  tc_fence_after();

  WY_STAMP(4);  // Gram matrices in TMEM
  // A = (k beta) k^T decay, strictly lower, fp32 into the q region: element (r, j) of chunk c at
  // c * 16384 + r * 256 + (((j >> 2) + r) & 15) * 16 + (j & 3) * 4 bytes (row-rotated float4 groups).
  // Each half builds 32 of the row's 64 columns.
  float* sA = reinterpret_cast<float*>(sQ + c * 16384);
  bf16* regB = reinterpret_cast<bf16*>(p.work + tc_region_b(static_cast<size_t>(p.n_chunks) * p.HV)) + ch * 64 * 64;
#pragma unroll
  for (int jj0 = 0; jj0 < 32; jj0 += 16) {
    const int j0 = half * 32 + jj0;
    float kk[16], qk[16];
    tmem_ld16(tmem + lane_base + c * 64 + j0, kk);
    tmem_ld16(tmem + lane_base + 128 + c * 64 + j0, qk);
    uint4 so[2];
    bf16* soe = reinterpret_cast<bf16*>(so);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int jj = j0 + j;
      const float dec = jj <= r ? __expf(gs - sG[c * 64 + jj]) * sRk[c * 64 + jj] : 0.f;
      kk[j] = jj < r ? kk[j] * rk * beta * dec : 0.f;
      soe[j] = __float2bfloat16(qk[j] * rq * dec);
    }
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4)
      *reinterpret_cast<float4*>(sA + r * 64 + ((((j0 >> 2) + q4 + r) & 15) << 2)) =
          make_float4(kk[4 * q4], kk[4 * q4 + 1], kk[4 * q4 + 2], kk[4 * q4 + 3]);
    if (present) {
      reinterpret_cast<uint4*>(regB + r * 64 + j0)[0] = so[0];
      reinterpret_cast<uint4*>(regB + r * 64 + j0)[1] = so[1];
    }
  }
  // k <- k e^g / |k| in place (the first pair of MMAs has finished reading it); beta is folded into T below
  {
    const float fk = rk * __expf(gs);
#pragma unroll
    for (int c16 = 0; c16 < 8; ++c16) {
      uint4* kp = reinterpret_cast<uint4*>(sK + half * 16384 + swz(tile_row, c16));
      uint4 kv = *kp;
      bf16* ke = reinterpret_cast<bf16*>(&kv);
#pragma unroll
      for (int j = 0; j < 8; ++j) ke[j] = __float2bfloat16(__bfloat162float(ke[j]) * fk);
      *kp = kv;
    }
  }
  __syncthreads();
  WY_STAMP(5);  // A built, k scaled
  // T = (I + A)^-1 by forward substitution. Lanes (2m, 2m + 1) of a warp own column col = tid >> 1 of T, each the groups of
  // four entries of its own parity, in registers; the pair splits every dot product that way and adds the halves with
  // one shuffle. The reads of A are the same two addresses across the warp.
  {
    const int col = tid >> 1, part = tid & 1;
    const int cc = col >> 6, rr = col & 63;
    const float* sAc = reinterpret_cast<const float*>(sQ + cc * 16384);
    // Blocked by 16 rows: for block b, first the panel acc[i] = sum over earlier blocks' entries j of A[16 b + i][j] T[j],
    // then the 16 x 16 triangle with the block's own entries. Blocks that lie entirely above every diagonal of the warp's
    // columns are zero and skipped, as are zero groups.
    const int lo = (warp & 3) * 16;  // smallest column of this warp inside its chunk
    float tc[8][4];                  // entries 4 (2 gi + part) + x of the column
#pragma unroll
    for (int blk = 0; blk < 4; ++blk) {
      if (16 * blk + 15 < lo) {  // warp-uniform
#pragma unroll
        for (int x = 0; x < 4; ++x) tc[2 * blk][x] = tc[2 * blk + 1][x] = 0.f;
        continue;
      }
      float t[16], acc[16];
#pragma unroll
      for (int ii = 0; ii < 16; ++ii) acc[ii] = 0.f;
#pragma unroll
      for (int gi = 0; gi < 2 * blk; ++gi) {
        if (8 * gi + 7 < lo) continue;  // warp-uniform
        const int j4 = 2 * gi + part;
#pragma unroll
        for (int ii = 0; ii < 16; ++ii) {
          const int row = 16 * blk + ii;
          const float4 a4 = *reinterpret_cast<const float4*>(sAc + row * 64 + (((j4 + row) & 15) << 2));
          acc[ii] += (a4.x * tc[gi][0] + a4.y * tc[gi][1]) + (a4.z * tc[gi][2] + a4.w * tc[gi][3]);
        }
      }
#pragma unroll
      for (int ii = 0; ii < 16; ++ii) acc[ii] += __shfl_xor_sync(0xffffffffu, acc[ii], 1);
      // the block's own triangle: both lanes of the pair compute it (entries in registers, static indices)
#pragma unroll
      for (int ii = 0; ii < 16; ++ii) {
        const int row = 16 * blk + ii;
        float a = acc[ii];
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          if (4 * q4 < ii) {
            const float4 a4 = *reinterpret_cast<const float4*>(sAc + row * 64 + (((4 * blk + q4 + row) & 15) << 2));
            if (4 * q4 + 0 < ii) a += a4.x * t[4 * q4 + 0];
            if (4 * q4 + 1 < ii) a += a4.y * t[4 * q4 + 1];
            if (4 * q4 + 2 < ii) a += a4.z * t[4 * q4 + 2];
            if (4 * q4 + 3 < ii) a += a4.w * t[4 * q4 + 3];
          }
        }
        t[ii] = row > rr ? -a : (row == rr ? 1.f : 0.f);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        tc[2 * blk][x] = part ? t[4 + x] : t[x];
        tc[2 * blk + 1][x] = part ? t[12 + x] : t[8 + x];
      }
    }
    WY_STAMP(6);  // substitution done (this warp)
    __syncthreads();  // every thread has finished reading A: the region becomes the bf16 operand tile
    // T diag(beta), block-diagonal, as a K-major A operand: row (cc * 64 + ii), K index (cc * 64 + rr) -> atom cc
    uint8_t* tile = sQ + cc * 16384;
    const float bcol = sBeta[col];
#pragma unroll
    for (int gi = 0; gi < 8; ++gi)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int ii = 4 * (2 * gi + part) + x;
        *reinterpret_cast<bf16*>(tile + swz(cc * 64 + ii, rr >> 3) + (rr & 7) * 2) = __float2bfloat16(tc[gi][x] * bcol);
      }
  }
  {  // the other atom's rows of this chunk are zero: w = (T diag(beta)) (k e^g), u = (T diag(beta)) v
    uint8_t* other = sQ + (1 - c) * 16384;
#pragma unroll
    for (int c16 = 0; c16 < 4; ++c16) *reinterpret_cast<uint4*>(other + swz(tile_row, half * 4 + c16)) = make_uint4(0, 0, 0, 0);
  }
  WY_STAMP(7);  // T tile written
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && ok) {
    tc_fence_after();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 128) | (1u << 16);  // B operand MN-major: [token][feature]
    const uint32_t ta = smem_u32(sQ), ka = smem_u32(sK), va = smem_u32(sV);
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const uint32_t aoff = (kk >> 2) * 16384 + (kk & 3) * 32;
      umma_bf16(tmem, umma_smem_desc(ta + aoff), umma_smem_desc_mn(ka + kk * 2048, 16384), idesc, kk != 0);        // w
    }
    if (!mbar_wait(v_bar, 0, p.err, ERR_WAIT_FULL, abort_flag)) ok = false;
    tc_fence_after();
    if (ok) {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const uint32_t aoff = (kk >> 2) * 16384 + (kk & 3) * 32;
        umma_bf16(tmem + 128, umma_smem_desc(ta + aoff), umma_smem_desc_mn(va + kk * 2048, 16384), idesc, kk != 0);  // u
      }
    }
    umma_commit(mma_bar);
  }
  WY_STAMP(8);  // second pair of MMAs issued
  ok = mbar_wait(mma_bar, 1, p.err, ERR_WAIT_TMEM, abort_flag) && !*abort_flag;
  tc_fence_after();
  WY_STAMP(9);  // w / u in TMEM
  // w and u as bf16 into the tiles that the MMAs have read, and from there by TMA to rows [0, 64) and [64, 128) of the
  // chunk's A-region (a workspace of whole chunks: there are no ragged edges). Stored by the threads, each its own row, the
  // 16-byte pieces of 32 rows made 32 lines of every instruction.
#pragma unroll 1
  for (int which = 0; which < 2; ++which) {
    uint8_t* dst = (which ? sK : sQ) + half * 16384;
#pragma unroll
    for (int c0 = 0; c0 < 64; c0 += 16) {
      float v[16];
      tmem_ld16(tmem + lane_base + which * 128 + half * 64 + c0, v);  // warp-collective: never predicated
      uint4 o[2];
      bf16* oe = reinterpret_cast<bf16*>(o);
#pragma unroll
      for (int j = 0; j < 16; ++j) oe[j] = __float2bfloat16(v[j]);
      *reinterpret_cast<uint4*>(dst + swz(tile_row, c0 >> 3)) = o[0];
      *reinterpret_cast<uint4*>(dst + swz(tile_row, (c0 >> 3) + 1)) = o[1];
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  if (tid == 0) {
    for (int cc = 0; cc < 2 && ok; ++cc) {
      const int idx = 2 * blockIdx.x + cc;
      if (idx >= p.n_chunks) break;
      for (int which = 0; which < 2; ++which)
        for (int a = 0; a < 2; ++a)
          tma_store_2d(&tmA, (which ? sK : sQ) + a * 16384 + cc * 8192, a * 64, (idx * p.HV + h) * 256 + which * 64);
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  WY_STAMP(10);  // w / u written
  tc_fence_before();
  __syncthreads();
  if (warp == 0) { tc_fence_after(); tmem_dealloc(tmem, 256); }
}

}  // namespace b200

namespace b200 {

// ------------------------------------------------------------------ state pass
struct ScanParams {
  const ChunkInfoTc* chunks;
  const int2* seg_chunks;  // (first chunk, number of chunks) per sequence
  const int* slots;
  float* rec_state;        // [slots, HV, 128 (dk), 128 (dv)] fp32
  const float* glast;      // [n_chunks * HV]
  bf16* o_out;             // [T, HV * 128]
  int HV;
  int* err;
};

constexpr int SC_STAGE = 4 * 16384 + 8192;  // w | u | qg | kg | scores
constexpr int SC_SMEM = 32768 + 16384 + 2 * SC_STAGE + 16384 + 1024 /*align*/ + 256 /*barriers*/;

// The chunks of a sequence are a serial chain, and with few sequences nothing else hides it: 148 -> 74 us for one
// span of 2048 tokens x 32 heads (32 chunks, 8500 -> 3100 cycles each), 168 -> 89 us for 8 x 1024 (256 CTAs, 148 SMs).
// What is kept out of the chain: the next chunk's u rows are read while the state MMAs run; the scaling by the next chunk's
// decay rides on the pass that refreshes the bf16 copy of the state; two threads share a TMEM lane, each with half of the
// columns; the state MMAs go before the rest of o's; and four warps of their own take o (two accumulators in turn) out of
// TMEM, transpose it through shared memory and store 16-byte pieces (the chain's threads spent 2950 of 6000 cycles a chunk on
// two-byte stores; the gated norm in these warps as well made them the bottleneck, 6700 cycles).
__global__ void __launch_bounds__(448, 1)
gdn_scan_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, ScanParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sS = smem;                 // bf16 S^T [128 dv][128 dk], two K atoms
  uint8_t* sVN = smem + 32768;        // bf16 v_new^T [128 dv][64 tokens]
  uint8_t* stages = smem + 49152;
  uint8_t* sO = stages + 2 * SC_STAGE;  // bf16 o [64 tokens][128 dv]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 16384);
  uint64_t* full = bars;              // [3][2]: w and qg | u | kg and scores
  uint64_t* empty = bars + 6;         // [3][2]
  uint64_t* vn_done = bars + 12;      // MMA -> threads: S^T w^T is in TMEM
  uint64_t* vn_ready = bars + 13;     // threads -> MMA: bf16 v_new in shared memory
  uint64_t* s_done = bars + 14;       // MMA -> threads: state updated, its bf16 copy no longer read
  uint64_t* s_ready = bars + 15;      // threads -> MMA: bf16 state copy refreshed, state scaled for the next chunk
  uint64_t* o_done = bars + 16;       // [2] MMA -> output threads: o of an even / odd chunk is complete
  uint64_t* o_free = bars + 18;       // [2] output threads -> MMA: it has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seg = blockIdx.x, h = blockIdx.y;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 6; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], s == 2 || s == 3 ? 256 : 1); }
    mbar_init(vn_done, 1);
    mbar_init(vn_ready, 256);
    mbar_init(s_done, 1);
    mbar_init(s_ready, 256);
    mbar_init(&o_done[0], 1);
    mbar_init(&o_done[1], 1);
    mbar_init(&o_free[0], 128);
    mbar_init(&o_free[1], 128);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_launch();
  const int2 sc = p.seg_chunks[seg];
  const int nc = sc.y;
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_S = tmem, tmem_VN = tmem + 128, tmem_O = tmem + 192;  // o of chunk i at tmem_O + (i & 1) * 64

  if (warp == 0) {
    if (elect_one()) {
      for (int i = 0; i < nc; ++i) {
        // Three groups of operands with barriers of their own, so that each is asked for again as soon as it has been
        // used, up to two chunks before its next use: one chunk's time does not cover the way from memory.
        const int s = i & 1;
        const uint32_t ph = ((i >> 1) & 1) ^ 1;
        uint8_t* st = stages + s * SC_STAGE;
        const int ch = (sc.x + i) * p.HV + h;
        auto load = [&](int part, uint64_t* bar) {
          for (int a = 0; a < 2; ++a) tma_load_2d(st + part * 16384 + a * 8192, &tmA, bar, a * 64, ch * 256 + part * 64);
        };
        if (!mbar_wait(&empty[s], ph, p.err, ERR_WAIT_EMPTY, abort_flag)) break;
        mbar_expect_tx(&full[s], 32768);
        load(0, &full[s]);
        load(2, &full[s]);
        if (!mbar_wait(&empty[2 + s], ph, p.err, ERR_WAIT_EMPTY, abort_flag)) break;
        mbar_expect_tx(&full[2 + s], 16384);
        load(1, &full[2 + s]);
        if (!mbar_wait(&empty[4 + s], ph, p.err, ERR_WAIT_EMPTY, abort_flag)) break;
        mbar_expect_tx(&full[4 + s], 16384 + 8192);
        load(3, &full[4 + s]);
        tma_load_2d(st + 65536, &tmB, &full[4 + s], 0, ch * 64);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc64 = umma_idesc_bf16(128, 64);
      constexpr uint32_t idesc_kg = umma_idesc_bf16(128, 128) | (1u << 16);  // B MN-major: [token][dk]
      const uint32_t sa = smem_u32(sS), vna = smem_u32(sVN);
      for (int i = 0; i < nc; ++i) {
        const int s = i & 1;
        const uint32_t st = smem_u32(stages + s * SC_STAGE), o = tmem_O + (i & 1) * 64;
        if (!mbar_wait(&full[s], (i >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag)) break;
        if (!mbar_wait(s_ready, i & 1, p.err, ERR_WAIT_FULL, abort_flag)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {  // v_new^T partial: S^T w^T, contraction over dk
          const uint32_t aoff = (kk >> 2) * 16384 + (kk & 3) * 32, boff = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_bf16(tmem_VN, umma_smem_desc(sa + aoff), umma_smem_desc(st + boff), idesc64, kk != 0);
        }
        umma_commit(vn_done);
        if (!mbar_wait(&o_free[s], ((i >> 1) & 1) ^ 1, p.err, ERR_WAIT_TMEM, abort_flag)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {  // o^T = S^T (q e^g)^T
          const uint32_t aoff = (kk >> 2) * 16384 + (kk & 3) * 32, boff = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_bf16(o, umma_smem_desc(sa + aoff), umma_smem_desc(st + 32768 + boff), idesc64, kk != 0);
        }
        umma_commit(&empty[s]);
        if (!mbar_wait(&full[4 + s], (i >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag)) break;
        if (!mbar_wait(vn_ready, i & 1, p.err, ERR_WAIT_FULL, abort_flag)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)    // S^T += v_new^T (k e^{g_last - g}), contraction over the chunk's tokens
          umma_bf16(tmem_S, umma_smem_desc(vna + kk * 32), umma_smem_desc_mn(st + 49152 + kk * 2048, 8192), idesc_kg, 1);
        umma_commit(s_done);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)    // o^T += v_new^T scores^T
          umma_bf16(o, umma_smem_desc(vna + kk * 32), umma_smem_desc(st + 65536 + kk * 32), idesc64, 1);
        umma_commit(&empty[4 + s]);
        umma_commit(&o_done[s]);
      }
    }
  } else if (warp >= 10) {
    // ---------------- output: thread dv reads TMEM lane dv; then 16 lanes share a token's 128 values, 16 bytes each
    const int q = warp & 3, dv = q * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    const int col = (lane & 15) * 8, t_own = (warp - 10) * 2 + (lane >> 4);  // tokens t_own + 8 j
    bf16* so = reinterpret_cast<bf16*>(sO);
    bool ok = true;
    for (int i = 0; i < nc; ++i) {
      const ChunkInfoTc ci = p.chunks[sc.x + i];
      ok = mbar_wait(&o_done[i & 1], (i >> 1) & 1, p.err, ERR_WAIT_TMEM, abort_flag) && ok;
      tc_fence_after();
#pragma unroll
      for (int t0 = 0; t0 < 64; t0 += 16) {
        float v[16];
        tmem_ld16(tmem_O + (i & 1) * 64 + lane_base + t0, v);  // warp-collective: never predicated
#pragma unroll
        for (int j = 0; j < 16; ++j) so[(t0 + j) * 128 + dv] = __float2bfloat16(v[j]);
      }
      tc_fence_before();
      mbar_arrive(&o_free[i & 1]);
      asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int t = t_own + 8 * j;
        const uint4 o = *reinterpret_cast<const uint4*>(so + t * 128 + col);
        if (ok && t < ci.nrows)
          *reinterpret_cast<uint4*>(p.o_out + (static_cast<size_t>(ci.row0 + t) * p.HV + h) * 128 + col) = o;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the tile has been read
    }
  } else {
    // ---------------- thread (dv, hf) works on TMEM lane dv, one row of S^T and v_new^T, and on half hf of the columns
    const int q = warp & 3, hf = warp >= 6 ? 1 : 0;
    const int dv = q * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    float* Sg = p.rec_state + (static_cast<size_t>(p.slots[seg]) * p.HV + h) * 128 * 128;
    const float* glast = p.glast + static_cast<size_t>(sc.x) * p.HV + h;
    uint8_t* s_copy = sS + hf * 16384;
    const uint32_t s_row = tmem_S + lane_base + hf * 64;
    // 16 state columns: the bf16 operand copy, and the state scaled by the next chunk's decay back into TMEM
    auto keep = [&](int k0, float* v, float scale) {
      uint4 o[2];
      bf16* oe = reinterpret_cast<bf16*>(o);
#pragma unroll
      for (int j = 0; j < 16; ++j) { oe[j] = __float2bfloat16(v[j]); v[j] *= scale; }
      tmem_st16(s_row + k0, v);
      *reinterpret_cast<uint4*>(s_copy + swz(dv, k0 >> 3)) = o[0];
      *reinterpret_cast<uint4*>(s_copy + swz(dv, (k0 >> 3) + 1)) = o[1];
    };
    float g_next = nc > 0 ? glast[0] : 0.f;
    {
      const float eg = __expf(g_next);
#pragma unroll
      for (int k0 = 0; k0 < 64; k0 += 16) {  // initial state: S[k][dv] -> TMEM row dv and the bf16 copy
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = Sg[static_cast<size_t>(hf * 64 + k0 + j) * 128 + dv];
        keep(k0, v, eg);
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    mbar_arrive(s_ready);
    bool ok = true;
    bf16 u[32];
    auto read_u = [&](int i) {  // chunk i's u rows: 32 tokens of this thread's dv
      const int s = i & 1;
      if (!mbar_wait(&full[2 + s], (i >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag)) return false;
      const uint8_t* su = stages + s * SC_STAGE + 16384 + (dv >> 6) * 8192 + (dv & 7) * 2;
#pragma unroll
      for (int j = 0; j < 32; ++j) u[j] = *reinterpret_cast<const bf16*>(su + swz(hf * 32 + j, (dv & 63) >> 3));
      mbar_arrive(&empty[2 + s]);
      return true;
    };
    if (nc > 0) ok = read_u(0);
    for (int i = 0; i < nc && ok; ++i) {
      const bool last = i + 1 == nc;
      g_next = last ? 0.f : glast[static_cast<size_t>(i + 1) * p.HV];
      ok = mbar_wait(vn_done, i & 1, p.err, ERR_WAIT_TMEM, abort_flag);
      if (!ok) break;
      tc_fence_after();
      // v_new^T[dv][t] = u[t][dv] - (S^T w^T)[dv][t], as bf16 into the K-major operand tile (row dv, 64 tokens)
#pragma unroll
      for (int t0 = 0; t0 < 32; t0 += 16) {
        float v[16];
        tmem_ld16(tmem_VN + lane_base + hf * 32 + t0, v);
        uint4 o[2];
        bf16* oe = reinterpret_cast<bf16*>(o);
#pragma unroll
        for (int j = 0; j < 16; ++j) oe[j] = __float2bfloat16(__bfloat162float(u[t0 + j]) - v[j]);
        const uint32_t c16 = (hf * 32 + t0) >> 3;
        *reinterpret_cast<uint4*>(sVN + swz(dv, c16)) = o[0];
        *reinterpret_cast<uint4*>(sVN + swz(dv, c16 + 1)) = o[1];
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      mbar_arrive(vn_ready);
      const float eg = __expf(g_next);
      if (!last) ok = read_u(i + 1);
      ok = ok && mbar_wait(s_done, i & 1, p.err, ERR_WAIT_TMEM, abort_flag);
      if (!ok) break;
      tc_fence_after();
      if (last) {
#pragma unroll
        for (int k0 = 0; k0 < 64; k0 += 16) {
          float v[16];
          tmem_ld16(s_row + k0, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) Sg[static_cast<size_t>(hf * 64 + k0 + j) * 128 + dv] = v[j];
        }
      } else {
#pragma unroll
        for (int k0 = 0; k0 < 64; k0 += 16) {
          float v[16];
          tmem_ld16(s_row + k0, v);
          keep(k0, v, eg);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        mbar_arrive(s_ready);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

}  // namespace b200

using namespace b200;

namespace {
typedef CUresult (*TcEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
TcEncodeFn tc_encode_fn() {
  static TcEncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess)
      fn = reinterpret_cast<TcEncodeFn>(ptr);
  }
  return fn;
}
// bf16 [rows, cols] row-major with row stride `ld` elements; box 64 columns x 64 rows, 128-byte swizzle, zero fill
int tc_map_2d(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t ld) {
  TcEncodeFn fn = tc_encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {64, 64};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}
}  // namespace

// Phase clocks of CTA (0, 0) of the last WY launch on the current device: 11 clock64() stamps (see WY_STAMP).
extern "C" int b200_gdn_wy_phase_clocks(long long* out11) {
  return cudaMemcpyFromSymbol(out11, g_wy_clocks, 11 * sizeof(long long)) == cudaSuccess ? 0 : -1;
}

// Workspace bytes per (chunk, head) of the tensor-core path (fits inside the fp32 path's workspace).
extern "C" int b200_gdn_prefill_tc_work_bytes() { return 65536 + 8192 + 4; }

// Tensor-core WY transform + state pass for DK = DV = 128. Arguments as b200_gdn_prefill's second half: conv_out
// [T, C] bf16 holds the convolved q | k | v, `work` holds at least n_chunks * HV * b200_gdn_prefill_tc_work_bytes()
// bytes (256-byte aligned), o_tmp receives the un-normalised outputs [T, HV * 128].
extern "C" int b200_gdn_prefill_tc(const void* mixed, int ld, const void* conv_out, const void* chunks, int n_chunks,
                                   const void* seg_chunks, int n_seg, const int* slots, float* rec_state,
                                   const float* A_log, const float* dt_bias, void* work, void* o_tmp, int T, int HK,
                                   int HV, int* err, cudaStream_t st) {
  if (n_chunks <= 0) return 0;
  const int key_dim = HK * 128, value_dim = HV * 128, C = 2 * key_dim + value_dim;
  const size_t nch = static_cast<size_t>(n_chunks) * HV;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gdn_wy_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WY_SMEM) != cudaSuccess) return -3;
    if (cudaFuncSetAttribute(gdn_scan_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SC_SMEM) != cudaSuccess) return -3;
    configured = true;
  }
  CUtensorMap tc, ta, tb;
  if (tc_map_2d(&tc, conv_out, C, T, C)) return -1;
  if (tc_map_2d(&ta, work, 128, nch * 256, 128)) return -1;
  if (tc_map_2d(&tb, static_cast<uint8_t*>(work) + tc_region_b(nch), 64, nch * 64, 64)) return -1;
  WyParams wp{static_cast<const bf16*>(mixed), ld, C + value_dim, C + value_dim + HV,
              static_cast<const ChunkInfoTc*>(chunks), n_chunks, A_log, dt_bias, static_cast<uint8_t*>(work), HK, HV, err};
  if (launch_pdl(gdn_wy_tc_kernel, dim3((n_chunks + 1) / 2, HV), dim3(256), WY_SMEM, st, tc, ta, wp) != cudaSuccess) return -4;
  ScanParams sp{static_cast<const ChunkInfoTc*>(chunks), static_cast<const int2*>(seg_chunks), slots, rec_state,
                reinterpret_cast<const float*>(static_cast<uint8_t*>(work) + tc_region_g(nch)),
                static_cast<bf16*>(o_tmp), HV, err};
  return launch_pdl(gdn_scan_tc_kernel, dim3(n_seg, HV), dim3(448), SC_SMEM, st, ta, tb, sp) == cudaSuccess ? 0 : -4;
}
