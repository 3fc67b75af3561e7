// Causal gated flash attention for prefill spans over the paged KV cache, on tcgen05.
//
// One CTA per (query tile, kv head). A tile is 128 MMA rows = (128 / GROUP) consecutive query
// positions x the GROUP query heads that share the kv head, so every K/V page fetched by TMA is
// used by all heads of the group (reference: engine/fast/flash_prefill.py:97-186 tiles
// M = BLOCK_R x GROUP rows the same way on MFMA). Per 64-key page:
//
//   S[128 x 64]  = Q[128 x D] K[64 x D]^T      tcgen05.mma, both operands K-major, S in TMEM
//   softmax      : warps 0..3 take the even pages, warps 4..7 the odd ones, each thread one whole row (TMEM lane), so a
//                  page's maximum, exponentials and sum need no other thread. What two pages share is the running row
//                  maximum, which the thread of page i hands to the thread of page i + 1 as soon as it has seen its
//                  scores: the exponentials of two pages run at the same time. P = exp2(S - m) goes to shared memory
//                  as bf16 in the swizzled K-major layout the next MMA reads; the O accumulator in TMEM is rescaled only
//                  when a row maximum grew by more than 2^8 (exact: the final division uses the same m)
//   O[128 x D]  += P[128 x 64] V[64 x D]       V is read straight from its page layout as an
//                                              MN-major B operand (no transpose)
//
// Warp 8 issues the MMAs (Q K^T two pages ahead of P V), warps 9 and 10 drive TMA (Q once; K and V pages in rings of their own: a
// K page is free when its scores are there, a V page after its P V). The epilogue divides by the row sum, multiplies by
// sigmoid(gate) and stores bf16. Bound: shared memory, which per page and SM takes 64 KB of K and V in and gives the MMAs
// 96 KB (Q K^T: N = 64, 48 cycles an MMA) and 48 KB (P V). With one thread for all loads and MMAs, which also read the page
// table between a free stage and its load, and one page in the softmax at a time, a page took 3400 cycles; it takes about
// 1800 now: 4 x 2048 rows behind 6.5k to 28.7k tokens 3.70 -> 1.94 ms (1.23 PFLOP/s at 30k), 8 x 1024 rows 249 -> 206 us.
// The exponentials keep results below 2^-126, which count where the value beside them is large; the unit's flushing form
// would save nothing. Passes of one position per sequence take flash_decode.cu.
// Chunked prefill: queries sit at positions pos0.. of their sequence, keys are 0..pos.
// All waits are bounded (common.cuh). No cluster multicast.
#include "common.cuh"

namespace b200 {

constexpr int FP_PAGE = 64;

struct FlashParams {
  const int4* tiles;      // (segment, first local position, segment start row, segment length)
  const int* seg_pos0;    // position of each segment's first row
  const int64_t* positions;  // instead of seg_pos0: position of every row (decode passes have these; a conversion kernel in
                             // front cost a step about 2 us per attention layer)
  const int* tables;      // [segments, max_pages]
  int max_pages;
  int num_pages;
  const bf16* gate;       // [T, n_q * D]
  bf16* out;              // [T, n_q * D]
  int n_q, n_kv;
  float scale_log2;       // D^-0.5 * log2(e)
  int* err;
  int split_pages;        // > 0: blockIdx.z handles pages [z*split, (z+1)*split) and writes partials
  float* part_acc;        // [T, n_q, gridDim.z, D] unnormalised partial outputs
  float* part_ml;         // [T, n_q, gridDim.z, 2] (row maximum in natural-log units, row sum)
};

template <int D>
struct FlashCfg {
  static constexpr int DB = D / 64;             // 64-element (128-byte) blocks along the head dim
  static constexpr int Q_BLOCK = 128 * 128;     // bytes between the 64-element blocks of the Q tile
  static constexpr int Q_BYTES = DB * Q_BLOCK;
  static constexpr int KV_BYTES = DB * FP_PAGE * 128;  // one of K or V, one stage
  static constexpr int P_BYTES = 128 * 128;     // one probability tile; two are kept
  static constexpr int ST = 2;                  // K/V stages
  // dynamic shared memory is declared 1024-byte aligned (checked at run time), so no alignment slack is budgeted:
  // with D = 256 the tiles, the barriers and 512 bytes of static arrays fill the 227 KB of an SM
  static constexpr int SMEM = Q_BYTES + 2 * ST * KV_BYTES + 2 * P_BYTES + 256;
  static constexpr int ROW_WARPS = 4;           // softmax warps per page
  static constexpr int TMEM_COLS = (128 + D) <= 256 ? 256 : 512;  // two score tiles of 64 columns + the output
};

template <int D, int GROUP>
__global__ void __launch_bounds__(352, 1)
flash_prefill_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, FlashParams p) {
  using C = FlashCfg<D>;
  constexpr int DB = C::DB;
  constexpr int ST = C::ST;
  constexpr int R = 128 / GROUP;  // query positions per tile
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {  // the swizzled tiles need this alignment; leave with a status rather than compute garbage
    if (threadIdx.x == 0) atomicCAS(p.err, 0, ERR_BAD_INDEX);
    return;
  }
  uint8_t* sQ = smem;
  uint8_t* sP = sQ + C::Q_BYTES;               // [2][128 x 128 B]: page i uses tile i & 1
  uint8_t* sK = sP + 2 * C::P_BYTES;           // [ST stages][DB][64 x 128 B]
  uint8_t* sV = sK + ST * C::KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + ST * C::KV_BYTES);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;                 // [ST]
  uint64_t* v_full = bars + 4;                 // [ST]
  uint64_t* k_empty = bars + 7;                // [ST]: Q K^T of the page in that stage has finished
  uint64_t* v_empty = bars + 10;               // [ST]: P V of the page in that stage has finished
  uint64_t* s_full = bars + 13;                // [2]: one per score tile
  uint64_t* p_full = bars + 15;                // [2]: one per probability tile
  uint64_t* pv_done = bars + 17;               // [2]: P V of an even / odd page has finished
  uint64_t* acc_done = bars + 19;
  uint64_t* x_bar = bars + 20;                 // exchange point of the softmax threads (bounded wait, unlike bar.sync)
  uint64_t* m_bar = bars + 21;                 // [2][4]: the row maxima up to an even / odd page, one per warp of rows
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 29);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  pdl_wait();  // the tile table, positions and Q / K / V all come from kernels earlier in the stream
  const int4 tile = p.tiles[blockIdx.x];
  const int seg = tile.x, p0 = tile.y, seg_row0 = tile.z, seg_len = tile.w;
  const int kh = blockIdx.y;
  const int pos0 = p.positions ? static_cast<int>(p.positions[seg_row0]) : p.seg_pos0[seg];
  const int n_pos = min(R, seg_len - p0);
  if (n_pos <= 0) return;  // filler entry: a captured prefill pass keeps its tile table at a fixed length
  const int np_all = (pos0 + p0 + n_pos - 1) / FP_PAGE + 1;  // pages that hold visible keys
  // split mode: a fixed number of consecutive pages per CTA, so the partition of a sequence's context
  // depends on its own length only, never on what else is in the batch
  const int first = p.split_pages > 0 ? static_cast<int>(blockIdx.z) * p.split_pages : 0;
  const int np = p.split_pages > 0 ? max(0, min(np_all, first + p.split_pages) - first) : np_all;
  if (np == 0) {  // nothing for this split: publish an empty partial and leave before any barrier / TMEM use
    const int r = threadIdx.x;
    if (r < 128 && r / GROUP < n_pos) {
      const size_t row = static_cast<size_t>(seg_row0 + p0 + r / GROUP);
      float* pm = p.part_ml + ((row * p.n_q + kh * GROUP + r % GROUP) * gridDim.z + blockIdx.z) * 2;
      pm[0] = -INFINITY; pm[1] = 0.f;
    }
    return;
  }

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < ST; ++s) { mbar_init(&k_full[s], 1); mbar_init(&v_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 32 * C::ROW_WARPS); mbar_init(&pv_done[s], 1); }
    for (int w = 0; w < 8; ++w) mbar_init(&m_bar[w], 1);
    mbar_init(acc_done, 1);
    mbar_init(x_bar, 64 * C::ROW_WARPS);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKV);
  }
  if (warp == 8) { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch();  // this CTA holds its TMEM columns: the next kernel's CTAs may queue behind it
  const uint32_t tmem_S = tmem, tmem_O = tmem + 128;  // score tile of page i at tmem_S + (i & 1) * 64

  if (warp >= 9) {
    // warp 9 brings Q and the K pages, warp 10 the V pages: K runs a page ahead of what frees V, and one thread for both
    // would hold each back behind the other. The next page number is read before the wait for a free stage.
    if (elect_one()) {
      const int which = warp - 9;
      uint64_t* full = which ? v_full : k_full;
      uint64_t* empty = which ? v_empty : k_empty;
      uint8_t* stages = which ? sV : sK;
      const int* table = p.tables + static_cast<size_t>(seg) * p.max_pages + first;
      if (which == 0) {
        mbar_expect_tx(q_full, C::Q_BYTES);
        for (int a = 0; a < DB; ++a) tma_load_4d(sQ + a * C::Q_BLOCK, &tmQ, q_full, a * 64, 0, kh, seg_row0 + p0);
      }
      int next = table[0];
      for (int i = 0; i < np; ++i) {
        const int s = i % ST;
        int page = next;
        if (i + 1 < np) next = table[i + 1];
        if (page < 0 || page >= p.num_pages) { atomicCAS(p.err, 0, ERR_BAD_INDEX); page = 0; }
        if (!mbar_wait(&empty[s], ((i / ST) & 1) ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag)) break;
        mbar_expect_tx(&full[s], C::KV_BYTES);
        const int row = ((page * 2 + which) * p.n_kv + kh) * FP_PAGE;
        for (int a = 0; a < DB; ++a) tma_load_2d(stages + s * C::KV_BYTES + a * FP_PAGE * 128, &tmKV, &full[s], a * 64, row);
      }
    }
  } else if (warp == 8) {
    if (elect_one()) {
      constexpr uint32_t idesc_qk = umma_idesc_bf16(128, 64);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(128, D) | (1u << 16);  // B operand MN-major
      const uint32_t qa = smem_u32(sQ);
      auto issue_qk = [&](int i) {
        const int s = i % ST;
        if (!mbar_wait(&k_full[s], (i / ST) & 1, p.err, ERR_WAIT_FULL, abort_flag)) return false;
        tc_fence_after();
        const uint32_t ka = smem_u32(sK + s * C::KV_BYTES);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t blk = kk >> 2, koff = (kk & 3) * 32;
          umma_bf16(tmem_S + (i & 1) * 64, umma_smem_desc(qa + blk * C::Q_BLOCK + koff),
                    umma_smem_desc(ka + blk * FP_PAGE * 128 + koff), idesc_qk, kk != 0);
        }
        umma_commit(&s_full[i & 1]);
        umma_commit(&k_empty[s]);
        return true;
      };
      bool ok = mbar_wait(q_full, 0, p.err, ERR_WAIT_FULL, abort_flag);
      ok = ok && issue_qk(0) && (np < 2 || issue_qk(1));
      for (int i = 0; i < np && ok; ++i) {
        // the probabilities of page i are written, so its score tile has been read: Q K^T of page i + 2 goes first, the
        // threads that just finished page i wait for it
        ok = mbar_wait(&p_full[i & 1], (i >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag);
        if (ok && i + 2 < np) ok = issue_qk(i + 2);
        const int s = i % ST;
        ok = ok && mbar_wait(&v_full[s], (i / ST) & 1, p.err, ERR_WAIT_FULL, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t pa = smem_u32(sP + (i & 1) * C::P_BYTES), va = smem_u32(sV + s * C::KV_BYTES);
#pragma unroll
        for (int kk = 0; kk < FP_PAGE / 16; ++kk)
          umma_bf16(tmem_O, umma_smem_desc(pa + kk * 32), umma_smem_desc_mn(va + kk * 2048, FP_PAGE * 128), idesc_pv,
                    (i | kk) != 0);
        umma_commit(&pv_done[i & 1]);
        umma_commit(&v_empty[s]);
      }
      umma_commit(acc_done);
    }
  } else if ((warp & 3) < C::ROW_WARPS) {
    // ---------------- softmax + epilogue: thread (r = tid & 127, hf = tid >> 7) owns row r = one (position, head) on the
    // pages i with i & 1 == hf, and the half hf of the output columns at the end.
    __shared__ float s_m[128];  // the running row maximum, in the hands of the page that is to see its scores next
    const int r = threadIdx.x & 127, hf = threadIdx.x >> 7, rw = warp & 3;
    const uint32_t lane_base = static_cast<uint32_t>(rw * 32) << 16;
    const int lp = r / GROUP, head = r % GROUP;
    const int qpos = pos0 + p0 + lp;
    const bool row_valid = lp < n_pos;
    constexpr int DH = D / 2;
    float m_loc = -INFINITY, l = 0.f;  // the maximum and the sum of this thread's own pages, at that maximum
    bool ok = true;
    for (int i = hf; i < np && ok; i += 2) {
      const uint32_t ph = (i >> 1) & 1;
      ok = mbar_wait(&s_full[hf], ph, p.err, ERR_WAIT_TMEM, abort_flag);
      if (!ok) break;
      tc_fence_after();
      float sc[64];
      tmem_ld64(tmem_S + hf * 64 + lane_base, sc);
      const int kbase = (first + i) * FP_PAGE;
      if (kbase + FP_PAGE - 1 > pos0 + p0) {  // only pages that end behind the tile's first query hide keys
#pragma unroll
        for (int j = 0; j < 64; ++j) sc[j] = kbase + j <= qpos ? sc[j] : -INFINITY;
      }
      float mx4[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
      for (int j = 4; j < 64; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], sc[j]);
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
      float m_prev = -INFINITY;
      if (i > 0) {
        ok = mbar_wait(&m_bar[(hf ^ 1) * 4 + rw], ((i - 1) >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag);
        if (!ok) break;
        m_prev = s_m[r];
      }
      const bool need = mx > m_prev + 8.0f;
      const float m = need ? mx : m_prev;
      s_m[r] = m;
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(&m_bar[hf * 4 + rw]);
      // The output tile may only be rescaled once P V of page i - 1 has finished; P V of this page and the later ones wait
      // for this page's probabilities.
      if (__any_sync(0xffffffffu, need) && i > 0) {  // warp-uniform: TMEM loads/stores are warp-collective
        ok = mbar_wait(&pv_done[hf ^ 1], ((i - 1) >> 1) & 1, p.err, ERR_WAIT_EMPTY, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const float factor = need ? exp2f(m_prev - m) : 1.0f;
#pragma unroll 1
        for (int c = 0; c < D; c += 16) {
          float o[16];
          tmem_ld16(tmem_O + lane_base + c, o);
#pragma unroll
          for (int j = 0; j < 16; ++j) o[j] *= factor;
          tmem_st16(tmem_O + lane_base + c, o);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      if (m != m_loc) { l *= exp2f(m_loc - m); m_loc = m; }  // exp2(-inf) = 0 on this thread's first page
      if (i >= 2) {  // this page's probability tile was last read by P V of page i - 2
        ok = mbar_wait(&pv_done[hf], ph ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag);
        if (!ok) break;
      }
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint8_t* prow = sP + hf * C::P_BYTES + r * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint4 packed;
        __nv_bfloat162* pe = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float a = exp2f(fmaf(sc[c * 8 + 2 * j], p.scale_log2, -m)), b2 = exp2f(fmaf(sc[c * 8 + 2 * j + 1], p.scale_log2, -m));
          sum[(2 * j) & 3] += a;
          sum[(2 * j + 1) & 3] += b2;
          pe[j] = __floats2bfloat162_rn(a, b2);
        }
        *reinterpret_cast<uint4*>(prow + ((c ^ (r & 7)) * 16)) = packed;  // 128-byte swizzle of the K-major tile
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      mbar_arrive(&p_full[hf]);
    }
    ok = ok && mbar_wait(acc_done, 0, p.err, ERR_WAIT_TMEM, abort_flag) && !*abort_flag;
    tc_fence_after();
    float m_used = m_loc;
    if (ok) {  // the probability tiles are free now: even and odd pages put their sums together, even + odd
      float* ex = reinterpret_cast<float*>(sP);
      constexpr int STRIDE = 32 * C::ROW_WARPS;
      ex[(hf * STRIDE + r) * 2] = l;
      ex[(hf * STRIDE + r) * 2 + 1] = m_loc;
      mbar_arrive(x_bar);
      ok = mbar_wait(x_bar, 0, p.err, ERR_WAIT_FULL, abort_flag);
      const float l0 = ex[r * 2], m0 = ex[r * 2 + 1], l1 = ex[(STRIDE + r) * 2], m1 = ex[(STRIDE + r) * 2 + 1];
      m_used = fmaxf(m0, m1);  // a running maximum never falls: the larger one is the last page's
      l = l0 * exp2f(m0 - m_used) + l1 * exp2f(m1 - m_used);
    }
    if (ok && p.split_pages > 0) {
      const size_t row = static_cast<size_t>(seg_row0 + p0 + lp);
      const size_t slot = (row * p.n_q + kh * GROUP + head) * gridDim.z + blockIdx.z;
#pragma unroll 1
      for (int c = hf * DH; c < hf * DH + DH; c += 16) {
        float o[16];
        tmem_ld16(tmem_O + lane_base + c, o);  // warp-collective: never predicated
        if (row_valid) {
          float4* dst = reinterpret_cast<float4*>(p.part_acc + slot * D + c);
#pragma unroll
          for (int j = 0; j < 4; ++j) dst[j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        }
      }
      if (row_valid && hf == 0) {
        p.part_ml[slot * 2] = m_used * 0.6931471805599453f;  // log2 units -> natural log, as the combine expects
        p.part_ml[slot * 2 + 1] = l;
      }
    } else
    if (ok) {
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      const size_t row = static_cast<size_t>(seg_row0 + p0 + lp);
      const size_t base = row * (static_cast<size_t>(p.n_q) * D) + static_cast<size_t>(kh * GROUP + head) * D;
#pragma unroll 1
      for (int c = hf * DH; c < hf * DH + DH; c += 16) {
        float o[16];
        tmem_ld16(tmem_O + lane_base + c, o);  // warp-collective: never predicated
        if (row_valid) {
          uint4 g0 = *reinterpret_cast<const uint4*>(p.gate + base + c), g1 = *reinterpret_cast<const uint4*>(p.gate + base + c + 8);
          const bf16* ge0 = reinterpret_cast<const bf16*>(&g0);
          const bf16* ge1 = reinterpret_cast<const bf16*>(&g1);
          uint4 o0, o1;
          bf16* oe0 = reinterpret_cast<bf16*>(&o0);
          bf16* oe1 = reinterpret_cast<bf16*>(&o1);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            oe0[j] = __float2bfloat16(__bfloat162float(__float2bfloat16(o[j] * inv)) * sigmoid_f(__bfloat162float(ge0[j])));
            oe1[j] = __float2bfloat16(__bfloat162float(__float2bfloat16(o[8 + j] * inv)) * sigmoid_f(__bfloat162float(ge1[j])));
          }
          *reinterpret_cast<uint4*>(p.out + base + c) = o0;
          *reinterpret_cast<uint4*>(p.out + base + c + 8) = o1;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
}

}  // namespace b200

using namespace b200;

namespace {
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn fp_encode_fn() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess) fn = reinterpret_cast<EncodeFn>(ptr);
  }
  return fn;
}
int fp_make_map(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
                const cuuint32_t* box) {
  EncodeFn fn = fp_encode_fn();
  if (!fn) return -1;
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides_bytes, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

template <int D, int GROUP>
int fp_launch(const CUtensorMap& tq, const CUtensorMap& tkv, const FlashParams& p, int n_tiles, int gz, cudaStream_t st) {
  auto kern = flash_prefill_kernel<D, GROUP>;
  static bool configured[64] = {};  // a function attribute is set per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FlashCfg<D>::SMEM) != cudaSuccess) return -3;
    configured[dev] = true;
  }
  return launch_pdl(kern, dim3(n_tiles, p.n_kv, gz), dim3(352), FlashCfg<D>::SMEM, st, tq, tkv, p) == cudaSuccess ? 0 : -4;
}
}  // namespace

// q: [T, n_q, D] bf16 (already normed and rotated), gate/out: [T, n_q * D], kv: one layer of the paged pool
// [num_pages, 2, n_kv, 64, D]; tiles: int4 (segment, first local position, segment start row, segment length) with
// 128 / (n_q / n_kv) positions per tile; seg_pos0 (or `positions`, one per row) and tables per segment. The span's K/V must already be in the pages.
extern "C" int b200_flash_prefill(const void* q, const void* gate, const void* kv, void* out, const void* tiles,
                                  int n_tiles, const int* seg_pos0, const int64_t* positions, const int* tables, int max_pages, int num_pages,
                                  int T, int n_q, int n_kv, int D, int split_pages, int n_splits, float* part_acc,
                                  float* part_ml, int* err, cudaStream_t st) {
  if (n_tiles <= 0) return 0;
  const int group = n_q / n_kv;
  if (group * n_kv != n_q || (D != 64 && D != 128 && D != 256) || 128 % group) return -7;
  CUtensorMap tq, tkv;
  {
    cuuint64_t dims[4] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(group), static_cast<cuuint64_t>(n_kv),
                          static_cast<cuuint64_t>(T)};
    cuuint64_t strides[3] = {static_cast<cuuint64_t>(D) * 2, static_cast<cuuint64_t>(group) * D * 2,
                             static_cast<cuuint64_t>(n_q) * D * 2};
    cuuint32_t box[4] = {64, static_cast<cuuint32_t>(group), 1, static_cast<cuuint32_t>(128 / group)};
    if (fp_make_map(&tq, q, 4, dims, strides, box)) return -1;
  }
  {
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(num_pages) * 2 * n_kv * FP_PAGE};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(D) * 2};
    cuuint32_t box[2] = {64, FP_PAGE};
    if (fp_make_map(&tkv, kv, 2, dims, strides, box)) return -1;
  }
  FlashParams p{static_cast<const int4*>(tiles), seg_pos0, positions, tables, max_pages, num_pages, static_cast<const bf16*>(gate),
                static_cast<bf16*>(out), n_q, n_kv, 1.4426950408889634f / sqrtf(static_cast<float>(D)), err,
                split_pages, part_acc, part_ml};
  const int gz = split_pages > 0 ? n_splits : 1;
#define FP_GROUPS(DD)                                                         \
  switch (group) {                                                            \
    case 1: return fp_launch<DD, 1>(tq, tkv, p, n_tiles, gz, st);          \
    case 2: return fp_launch<DD, 2>(tq, tkv, p, n_tiles, gz, st);          \
    case 4: return fp_launch<DD, 4>(tq, tkv, p, n_tiles, gz, st);          \
    case 8: return fp_launch<DD, 8>(tq, tkv, p, n_tiles, gz, st);          \
    default: return -7;                                                       \
  }
  if (D == 256) { FP_GROUPS(256) }
  if (D == 128) { FP_GROUPS(128) }
  FP_GROUPS(64)
#undef FP_GROUPS
}
