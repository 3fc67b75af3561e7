// Attention of one query position per sequence over the paged cache (decode steps, links of a draft chain), with the same
// arithmetic, and the same bits, as the split form of flash_prefill.cu: a context is cut into runs of `split_pages` pages, each
// run leaves an unnormalised fp32 partial, its row maxima and row sums, and attn_combine adds them.
//
// One persistent CTA per SM walks the runs that hold keys. Why: a run of eight pages takes about 12 us of memory time, and a CTA of
// its own adds the table look-ups, barrier set-up, TMEM allocation, first page and last store, in which nothing is on its
// way; and a grid that covers the page table's width (a captured step's grid cannot follow the contexts) starts a CTA with
// 200 KB of shared memory for every run that holds none. Here the next run's Q, K and V are asked for while the last one
// is being finished. Runs of full length come first, so that what is left for the end is short. Against a CTA per run, kernel
// time in a step: four sequences of 50,000 to 90,000 tokens 122 -> 99 us (84 at the bytes), 256 of about 2,300 247 -> 222 (176),
// 128 of 1,088 75 -> 71 (44).
//
// Q K^T, softmax and P V as in flash_prefill.cu: MMAs of 64 rows, of which the GROUP query heads of a KV head are real (Q and P
// keep one 8-row swizzle atom per 128-byte block, the MMA reads its other rows from what follows, into accumulator rows
// that nobody reads); two softmax warps take alternate pages; K, V and MMAs have warps of their own. All waits are bounded.
#include "common.cuh"

namespace b200 {

constexpr int FD_PAGE = 64;
constexpr int FD_MAX_SEQS = 1024;  // of one launch

struct FlashDecodeParams {
  const int64_t* positions;  // [B] position of each sequence's row
  const int* tables;         // [B] rows of `width` pages, max_pages apart
  int B, max_pages, width, num_pages, n_q, n_kv, n_splits, split_pages;
  float scale_log2;          // D^-0.5 * log2(e)
  float* part_acc;           // [B, n_q, n_splits, D]
  float* part_ml;            // [B, n_q, n_splits, 2]
  int* err;
};

template <int D>
struct FlashDecodeCfg {
  static constexpr int DB = D / 64;                     // 64-element (128-byte) blocks along the head dim
  static constexpr int Q_BYTES = DB * 1024;             // two of them: of the run in the MMAs and of the next one
  static constexpr int KV_BYTES = DB * FD_PAGE * 128;   // one of K or V, one stage
  static constexpr int ST = 3;                          // K / V stages
  static constexpr int P_BYTES = 1024;                  // one probability tile, two are kept
  static constexpr int TABLE_BYTES = (3 * FD_MAX_SEQS + 4) * 4;
  static constexpr int SMEM = 2 * Q_BYTES + 2 * P_BYTES + 2 * ST * KV_BYTES + 256 + TABLE_BYTES;
  static constexpr int TMEM_COLS = (128 + D) <= 256 ? 256 : 512;  // two score tiles of 64 columns + the output
};

// Sequence whose runs [first[b], first[b + 1]) hold run x.
__device__ __forceinline__ int find_seq(const int* first, int B, int x) {
  int lo = 0, hi = B;  // first[lo] <= x < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

template <int D, int GROUP>
__global__ void __launch_bounds__(352, 1)
flash_decode_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, FlashDecodeParams p) {
  using C = FlashDecodeCfg<D>;
  constexpr int DB = C::DB, ST = C::ST;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {  // the swizzled tiles need this alignment; leave with a status rather than compute garbage
    if (threadIdx.x == 0) atomicCAS(p.err, 0, ERR_BAD_INDEX);
    return;
  }
  uint8_t* sQ = smem;                        // [2]
  uint8_t* sP = sQ + 2 * C::Q_BYTES;         // [2]: page g uses tile g & 1
  uint8_t* sK = sP + 2 * C::P_BYTES;         // [ST][DB][64 x 128 B]
  uint8_t* sV = sK + ST * C::KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + ST * C::KV_BYTES);
  uint64_t* q_full = bars;                   // [2]
  uint64_t* q_empty = bars + 2;              // [2]
  uint64_t* k_full = bars + 4;               // [ST]
  uint64_t* v_full = bars + 7;
  uint64_t* k_empty = bars + 10;
  uint64_t* v_empty = bars + 13;
  uint64_t* s_full = bars + 16;              // [2]: one per score tile
  uint64_t* p_full = bars + 18;              // [2]: one per probability tile
  uint64_t* pv_done = bars + 20;             // [2]
  uint64_t* m_bar = bars + 22;               // [2]: the row maxima up to an even / odd page
  uint64_t* acc_done = bars + 24;            // a run's output is complete
  uint64_t* o_free = bars + 25;              // ... and has been read
  uint64_t* x_bar = bars + 26;               // the two softmax warps meet at the end of a run
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* s_np = reinterpret_cast<int*>(sV + ST * C::KV_BYTES + 256);  // [B] pages that hold visible keys
  int* s_full_runs = s_np + FD_MAX_SEQS;     // [B + 1] full runs of the sequences before
  int* s_rest_runs = s_full_runs + FD_MAX_SEQS + 1;  // [B + 1] shorter last runs of the sequences before
  __shared__ float s_m[32];                  // the running row maximum, in the hands of the page that is to see its scores next
  __shared__ float s_ex[2][64][2];           // sums and maxima of a run's even and odd pages

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 32);
      mbar_init(&pv_done[s], 1); mbar_init(&m_bar[s], 1);
    }
    for (int s = 0; s < ST; ++s) { mbar_init(&k_full[s], 1); mbar_init(&v_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_empty[s], 1); }
    mbar_init(acc_done, 1);
    mbar_init(o_free, 64);
    mbar_init(x_bar, 64);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKV);
  }
  if (warp == 8) { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
  pdl_wait();  // positions and Q / K / V come from kernels earlier in the stream
  for (int b = threadIdx.x; b < p.B; b += blockDim.x)
    s_np[b] = max(0, min(static_cast<int>(p.positions[b]) / FD_PAGE + 1, min(p.width, p.n_splits * p.split_pages)));
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch();  // this CTA holds its TMEM columns
  const uint32_t tmem_S = tmem, tmem_O = tmem + 128;  // score tile of page g at tmem_S + (g & 1) * 64
  if (warp == 0) {  // exclusive sums over the sequences, a lane a stretch of them
    const int per = (p.B + 31) / 32, b0 = min(p.B, lane * per), b1 = min(p.B, b0 + per);
    int full = 0, rest = 0;
    for (int b = b0; b < b1; ++b) { full += s_np[b] / p.split_pages; rest += s_np[b] % p.split_pages != 0; }
    int f = full, r = rest;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int uf = __shfl_up_sync(0xffffffffu, f, o), ur = __shfl_up_sync(0xffffffffu, r, o);
      if (lane >= o) { f += uf; r += ur; }
    }
    f -= full;
    r -= rest;
    for (int b = b0; b < b1; ++b) {
      s_full_runs[b] = f;
      s_rest_runs[b] = r;
      f += s_np[b] / p.split_pages;
      r += s_np[b] % p.split_pages != 0;
    }
    if (lane == 31) { s_full_runs[p.B] = f; s_rest_runs[p.B] = r; }
  }
  __syncthreads();
  const int n_full = s_full_runs[p.B] * p.n_kv, total = n_full + s_rest_runs[p.B] * p.n_kv;
  // run id -> sequence, KV head, split, pages
  auto run_of = [&](int id, int& b, int& kh, int& z, int& np) {
    const bool full = id < n_full;
    const int x = full ? id : id - n_full;
    kh = x % p.n_kv;
    b = find_seq(full ? s_full_runs : s_rest_runs, p.B, x / p.n_kv);
    z = full ? x / p.n_kv - s_full_runs[b] : s_np[b] / p.split_pages;
    np = full ? p.split_pages : s_np[b] % p.split_pages;
  };

  // In all roles: t counts the CTA's runs, g the pages of the runs before.
  if (warp >= 9) {
    // warp 9 brings Q and the K pages, warp 10 the V pages
    if (elect_one()) {
      const int which = warp - 9;
      uint64_t* full = which ? v_full : k_full;
      uint64_t* empty = which ? v_empty : k_empty;
      uint8_t* stages = which ? sV : sK;
      bool ok = true;
      int t = 0, g = 0;
      for (int id = blockIdx.x; id < total && ok; id += gridDim.x, ++t) {
        int b, kh, z, np;
        run_of(id, b, kh, z, np);
        const int* table = p.tables + static_cast<size_t>(b) * p.max_pages + z * p.split_pages;
        int next = table[0];
        if (which == 0) {
          const int s = t & 1;
          ok = mbar_wait(&q_empty[s], ((t >> 1) & 1) ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&q_full[s], DB * GROUP * 128);  // GROUP rows of 128 bytes per block
          for (int a = 0; a < DB; ++a) tma_load_4d(sQ + s * C::Q_BYTES + a * 1024, &tmQ, &q_full[s], a * 64, 0, kh, b);
        }
        for (int i = 0; i < np; ++i, ++g) {
          const int s = g % ST;
          int page = next;
          if (i + 1 < np) next = table[i + 1];
          if (page < 0 || page >= p.num_pages) { atomicCAS(p.err, 0, ERR_BAD_INDEX); page = 0; }
          ok = mbar_wait(&empty[s], ((g / ST) & 1) ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&full[s], C::KV_BYTES);
          const int row = ((page * 2 + which) * p.n_kv + kh) * FD_PAGE;
          for (int a = 0; a < DB; ++a) tma_load_2d(stages + s * C::KV_BYTES + a * FD_PAGE * 128, &tmKV, &full[s], a * 64, row);
        }
      }
    }
  } else if (warp == 8) {
    if (elect_one()) {
      constexpr uint32_t idesc_qk = umma_idesc_bf16(64, 64);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(64, D) | (1u << 16);  // B operand MN-major
      // Q K^T runs two pages ahead of P V, into the next run where this one ends
      int qid = blockIdx.x, qt = 0, qi = 0, qg = 0, qnp = 0;
      if (qid < total) { int b, kh, z; run_of(qid, b, kh, z, qnp); }
      auto issue_qk = [&]() {
        if (qid >= total) return true;
        if (qi == 0 && !mbar_wait(&q_full[qt & 1], (qt >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag)) return false;
        const int s = qg % ST;
        if (!mbar_wait(&k_full[s], (qg / ST) & 1, p.err, ERR_WAIT_FULL, abort_flag)) return false;
        tc_fence_after();
        const uint32_t qa = smem_u32(sQ + (qt & 1) * C::Q_BYTES), ka = smem_u32(sK + s * C::KV_BYTES);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t blk = kk >> 2, koff = (kk & 3) * 32;
          umma_bf16(tmem_S + (qg & 1) * 64, umma_smem_desc(qa + blk * 1024 + koff), umma_smem_desc(ka + blk * FD_PAGE * 128 + koff),
                    idesc_qk, kk != 0);
        }
        umma_commit(&s_full[qg & 1]);
        umma_commit(&k_empty[s]);
        ++qg;
        if (++qi == qnp) {
          umma_commit(&q_empty[qt & 1]);
          qi = 0;
          ++qt;
          qid += gridDim.x;
          if (qid < total) { int b, kh, z; run_of(qid, b, kh, z, qnp); }
        }
        return true;
      };
      bool ok = issue_qk() && issue_qk();
      int t = 0, g = 0;
      for (int id = blockIdx.x; id < total && ok; id += gridDim.x, ++t) {
        int b, kh, z, np;
        run_of(id, b, kh, z, np);
        for (int i = 0; i < np && ok; ++i, ++g) {
          // the probabilities of page g are written, so its score tile has been read: Q K^T of page g + 2 goes first
          ok = mbar_wait(&p_full[g & 1], (g >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag) && issue_qk();
          if (ok && i == 0 && t > 0) ok = mbar_wait(o_free, (t - 1) & 1, p.err, ERR_WAIT_TMEM, abort_flag);
          const int s = g % ST;
          ok = ok && mbar_wait(&v_full[s], (g / ST) & 1, p.err, ERR_WAIT_FULL, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t pa = smem_u32(sP + (g & 1) * C::P_BYTES), va = smem_u32(sV + s * C::KV_BYTES);
#pragma unroll
          for (int kk = 0; kk < FD_PAGE / 16; ++kk)
            umma_bf16(tmem_O, umma_smem_desc(pa + kk * 32), umma_smem_desc_mn(va + kk * 2048, FD_PAGE * 128), idesc_pv, (i | kk) != 0);
          umma_commit(&pv_done[g & 1]);
          umma_commit(&v_empty[s]);
        }
        if (ok) umma_commit(acc_done);
      }
    }
  } else if ((warp & 3) == 0) {
    // ---------------- softmax: warp hf * 4 takes the CTA's pages g with g & 1 == hf, and half hf of the output's columns at a
    // run's end; lane r owns row r = one query head
    const int r = lane, hf = warp >> 2;
    const bool row_valid = r < GROUP;
    constexpr int DH = D / 2;
    bool ok = true;
    int t = 0, g = 0;
    for (int id = blockIdx.x; id < total && ok; id += gridDim.x, ++t) {
      int b, kh, z, np;
      run_of(id, b, kh, z, np);
      const int qpos = static_cast<int>(p.positions[b]);
      const int mine = hf ^ (g & 1);  // this warp's pages of the run: the even or the odd ones
      float m_loc = -INFINITY, l = 0.f;  // the maximum and the sum of this thread's own pages, at that maximum
      for (int i = mine; i < np; i += 2) {
        const int gp = g + i;
        ok = mbar_wait(&s_full[hf], (gp >> 1) & 1, p.err, ERR_WAIT_TMEM, abort_flag);
        if (!ok) break;
        tc_fence_after();
        float sc[64];
        tmem_ld64(tmem_S + hf * 64, sc);
        const int kbase = (z * p.split_pages + i) * FD_PAGE;
        // rows past the real ones hold whatever the MMA read behind the Q atom; masked, so that they never ask for a rescale
#pragma unroll
        for (int j = 0; j < 64; ++j) sc[j] = (kbase + j <= qpos && row_valid) ? sc[j] : -INFINITY;
        float mx4[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
        for (int j = 4; j < 64; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], sc[j]);
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
        float m_prev = -INFINITY;
        if (i > 0) {
          ok = mbar_wait(&m_bar[hf ^ 1], ((gp - 1) >> 1) & 1, p.err, ERR_WAIT_FULL, abort_flag);
          if (!ok) break;
          m_prev = s_m[r];
        }
        const bool need = mx > m_prev + 8.0f;
        const float m = need ? mx : m_prev;
        s_m[r] = m;
        __syncwarp();
        if (lane == 0) mbar_arrive(&m_bar[hf]);
        // The output tile may only be rescaled once P V of the page before has finished; P V of this page and the later ones
        // wait for this page's probabilities.
        if (__any_sync(0xffffffffu, need) && i > 0) {
          ok = mbar_wait(&pv_done[hf ^ 1], ((gp - 1) >> 1) & 1, p.err, ERR_WAIT_EMPTY, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const float factor = need ? exp2f(m_prev - m) : 1.0f;
#pragma unroll 1
          for (int c = 0; c < D; c += 16) {
            float o[16];
            tmem_ld16(tmem_O + c, o);
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] *= factor;
            tmem_st16(tmem_O + c, o);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        if (m != m_loc) { l *= exp2f(m_loc - m); m_loc = m; }  // exp2(-inf) = 0 on this thread's first page
        if (gp >= 2) {  // this page's probability tile was last read by P V of page gp - 2
          ok = mbar_wait(&pv_done[hf], ((gp >> 1) & 1) ^ 1, p.err, ERR_WAIT_EMPTY, abort_flag);
          if (!ok) break;
        }
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        uint8_t* prow = sP + hf * C::P_BYTES + r * 128;
        if (r < 8)  // the tile holds one 8-row atom; the other rows' scores are not kept
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
      ok = ok && mbar_wait(acc_done, t & 1, p.err, ERR_WAIT_TMEM, abort_flag) && !*abort_flag;
      if (!ok) break;
      tc_fence_after();
      // even and odd pages put their sums together, even + odd. Nobody starts the next run before both have come here.
      float(*ex)[2] = s_ex[t & 1];
      ex[mine * 32 + r][0] = l;
      ex[mine * 32 + r][1] = m_loc;
      mbar_arrive(x_bar);
      ok = mbar_wait(x_bar, t & 1, p.err, ERR_WAIT_FULL, abort_flag);
      const float l0 = ex[r][0], m0 = ex[r][1], l1 = ex[32 + r][0], m1 = ex[32 + r][1];
      const float m_used = fmaxf(m0, m1);  // a running maximum never falls: the larger one is the last page's
      l = l0 * exp2f(m0 - m_used) + l1 * exp2f(m1 - m_used);
      const size_t slot = (static_cast<size_t>(b) * p.n_q + kh * GROUP + (row_valid ? r : 0)) * p.n_splits + z;
      __syncwarp();
#pragma unroll 1
      for (int c = hf * DH; c < hf * DH + DH; c += 16) {
        float o[16];
        tmem_ld16(tmem_O + c, o);  // warp-collective: never predicated
        if (ok && row_valid) {
          float4* dst = reinterpret_cast<float4*>(p.part_acc + slot * D + c);
#pragma unroll
          for (int j = 0; j < 4; ++j) dst[j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        }
      }
      tc_fence_before();
      mbar_arrive(o_free);
      if (ok && row_valid && hf == 0) {
        p.part_ml[slot * 2] = m_used * 0.6931471805599453f;  // log2 units -> natural log, as the combine expects
        p.part_ml[slot * 2 + 1] = l;
      }
      g += np;
    }
  } else {
    // ---------------- the other warps: partials of the runs that hold no key are marked empty
    const int w = (warp < 4 ? warp - 1 : warp - 2), tid = (blockIdx.x * 6 + w) * 32 + lane, step = gridDim.x * 6 * 32;
    const int per = p.n_q * p.n_splits;
    for (int i = tid; i < p.B * per; i += step) {
      const int b = i / per, z = i % p.n_splits;
      if (z * p.split_pages >= s_np[b]) reinterpret_cast<float2*>(p.part_ml)[i] = make_float2(-INFINITY, 0.f);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
}

}  // namespace b200

using namespace b200;

namespace {
typedef CUresult (*FdEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                               CUtensorMapFloatOOBfill);
int fd_make_map(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
                const cuuint32_t* box) {
  static FdEncodeFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || !ptr) return -1;
    fn = reinterpret_cast<FdEncodeFn>(ptr);
  }
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides_bytes, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}

template <int D, int GROUP>
int fd_launch(const CUtensorMap& tq, const CUtensorMap& tkv, const FlashDecodeParams& p, cudaStream_t st) {
  auto kern = flash_decode_kernel<D, GROUP>;
  static int sms_of[64] = {};  // per device, with the function attribute set
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -3;
  if (sms_of[dev] == 0) {
    int sms = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FlashDecodeCfg<D>::SMEM) != cudaSuccess) return -3;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -3;
    sms_of[dev] = sms;
  }
  const long long runs = static_cast<long long>(p.B) * p.n_kv * p.n_splits;
  const int grid = static_cast<int>(runs < sms_of[dev] ? runs : sms_of[dev]);
  return launch_pdl(kern, dim3(grid), dim3(352), FlashDecodeCfg<D>::SMEM, st, tq, tkv, p) == cudaSuccess ? 0 : -4;
}
}  // namespace

// q: [B, n_q, D] bf16 (normed and rotated), one row per sequence; kv: one layer of the paged pool [num_pages, 2, n_kv, 64, D] that
// holds the rows' own K / V already; positions [B], tables [B] rows of `width` pages, max_pages apart (any distance, 0 too).
// n_splits runs of split_pages pages cover a row. part_ml is written for all of [B, n_q, n_splits], part_acc only where a run
// holds keys: the combine passes over the others.
extern "C" int b200_flash_decode(const void* q, const void* kv, const int64_t* positions, const int* tables, int max_pages,
                                 int width, int num_pages, int B, int n_q, int n_kv, int D, int split_pages, int n_splits, float* part_acc,
                                 float* part_ml, int* err, cudaStream_t st) {
  const int group = n_kv > 0 ? n_q / n_kv : 0;
  if (group * n_kv != n_q || (D != 64 && D != 128 && D != 256) || split_pages <= 0 || n_splits <= 0) return -7;
  CUtensorMap tkv;
  {
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(num_pages) * 2 * n_kv * FD_PAGE};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(D) * 2};
    cuuint32_t box[2] = {64, FD_PAGE};
    if (fd_make_map(&tkv, kv, 2, dims, strides, box)) return -1;
  }
  for (int b0 = 0; b0 < B; b0 += FD_MAX_SEQS) {
    const int n = B - b0 < FD_MAX_SEQS ? B - b0 : FD_MAX_SEQS;
    const size_t heads = static_cast<size_t>(b0) * n_q;
    CUtensorMap tq;
    cuuint64_t dims[4] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(group), static_cast<cuuint64_t>(n_kv),
                          static_cast<cuuint64_t>(n)};
    cuuint64_t strides[3] = {static_cast<cuuint64_t>(D) * 2, static_cast<cuuint64_t>(group) * D * 2,
                             static_cast<cuuint64_t>(n_q) * D * 2};
    cuuint32_t box[4] = {64, static_cast<cuuint32_t>(group), 1, 1};
    if (fd_make_map(&tq, static_cast<const bf16*>(q) + heads * D, 4, dims, strides, box)) return -1;
    const FlashDecodeParams p{positions + b0, tables + static_cast<size_t>(b0) * max_pages, n, max_pages, width, num_pages, n_q, n_kv,
                              n_splits, split_pages, 1.4426950408889634f / sqrtf(static_cast<float>(D)),
                              part_acc + heads * n_splits * D, part_ml + heads * n_splits * 2, err};
    int rc = -7;
#define FD_GROUPS(DD)                                        \
  switch (group) {                                           \
    case 1: rc = fd_launch<DD, 1>(tq, tkv, p, st); break;    \
    case 2: rc = fd_launch<DD, 2>(tq, tkv, p, st); break;    \
    case 4: rc = fd_launch<DD, 4>(tq, tkv, p, st); break;    \
    case 8: rc = fd_launch<DD, 8>(tq, tkv, p, st); break;    \
  }
    if (D == 256) { FD_GROUPS(256) } else if (D == 128) { FD_GROUPS(128) } else { FD_GROUPS(64) }
#undef FD_GROUPS
    if (rc) return rc;
  }
  return 0;
}
