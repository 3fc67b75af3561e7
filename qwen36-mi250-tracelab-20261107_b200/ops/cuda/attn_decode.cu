// Gated full-attention decode path over the paged KV pool.
//
//  attn_prep:    split the merged q|gate|k|v projection row, zero-centred RMSNorm of q and k per
//                head, partial RoPE on the first `rot` dims, write k and v into the sequence's page
//                (reference: engine/fast/fused.py:476-528).
//  paged_attn:   flash-decoding of G query rows per sequence against its pages. One CTA per
//                (sequence, kv head, lane z of Z); warp w serves query head w of the GQA group.
//                CTA z walks pages z, z+Z, z+2Z, ... with one running online softmax, so the
//                reduction order of a sequence depends only on its own length, never on the batch
//                (reference: engine/fast/kernels.py:377-443 splits the context the same way).
//  attn_combine: merge the Z partials in an order that the splits with keys fix (up to 16 of them one after the other,
//                more as sixteen running sums), multiply by sigmoid(gate), store bf16
//                (reference: engine/fast/fused.py:530-551).
//
// KV layout: kv[page][2][n_kv][PAGE][D] bf16; page tables int32 [B, max_pages]; page 0 is scratch.
#include "common.cuh"

namespace b200 {

constexpr int PAGE = 64;

// PER consecutive bf16 (PER = 1, 2, 4 or 8) as floats with one vector load.
template <int PER>
__device__ __forceinline__ void load_bf16_vec(const bf16* p, float* out) {
  if constexpr (PER == 8) {
    uint4 raw = *reinterpret_cast<const uint4*>(p);
    const bf16* e = reinterpret_cast<const bf16*>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = __bfloat162float(e[i]);
  } else if constexpr (PER == 4) {
    uint2 raw = *reinterpret_cast<const uint2*>(p);
    const bf16* e = reinterpret_cast<const bf16*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = __bfloat162float(e[i]);
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i) out[i] = __bfloat162float(p[i]);
  }
}

// PER consecutive floats rounded to bf16 with one vector store; copy_bf16_vec moves PER bf16 as they are.
template <int PER>
__device__ __forceinline__ void store_bf16_vec(bf16* p, const float* v) {
  bf16 e[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) e[i] = __float2bfloat16(v[i]);
  if constexpr (PER == 8) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(e);
  else if constexpr (PER == 4) *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(e);
  else {
#pragma unroll
    for (int i = 0; i < PER; ++i) p[i] = e[i];
  }
}
template <int PER>
__device__ __forceinline__ void copy_bf16_vec(bf16* dst, const bf16* src) {
  if constexpr (PER == 8) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
  else if constexpr (PER == 4) *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(src);
  else {
#pragma unroll
    for (int i = 0; i < PER; ++i) dst[i] = src[i];
  }
}

// One CTA per row, one warp per head (query heads, then key, then value heads; a warp takes several when there are more than
// PREP_WARPS). The row's rotary factors are evaluated once per CTA, one frequency per thread, while the heads' vectors
// are on their way: a power and a sine per head and frequency bounded the kernel before (121 us at 8192 rows of 20
// heads, 302 MB; 94 us now, 23 instead of 30 us at 2048). A lane owns D / 32 consecutive dims, one vector load / store per tensor.
constexpr int PREP_WARPS = 20;
template <int D>
__global__ void __launch_bounds__(32 * PREP_WARPS)
attn_prep_kernel(const bf16* qkv, int ld, const int64_t* positions, const int* tables, int max_pages,
                 const int* seq_of_row, const bf16* q_norm, const bf16* k_norm, bf16* q_out,
                 bf16* gate_out, bf16* kv, int n_q, int n_kv, int rot, float theta, float eps,
                 int num_pages, int* err) {
  constexpr int PER = D / 32;
  __shared__ float s_cos[D / 2], s_sin[D / 2];
  __shared__ __align__(16) bf16 s_rot[PREP_WARPS][D];  // a head's normed vector: the rotary partner is another lane's
  pdl_wait();
  pdl_launch();
  const int row = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int heads = n_q + 2 * n_kv, half = rot / 2, d0 = lane * PER;
  const bf16* base = qkv + static_cast<size_t>(row) * ld;
  const auto source = [&](int head) {
    return head < n_q ? base + head * 2 * D : base + n_q * 2 * D + (head - n_q) * D;  // keys, then values
  };
  float v[PER];
  if (warp < heads) load_bf16_vec<PER>(source(warp) + d0, v);
  const int64_t pos = positions[row];
  for (int f = threadIdx.x; f < rot - half; f += blockDim.x) {
    const float inv_freq = powf(theta, -2.0f * f / rot);
    float sn, c;
    sincosf(static_cast<float>(pos) * inv_freq, &sn, &c);
    s_cos[f] = __bfloat162float(__float2bfloat16(c));
    s_sin[f] = __bfloat162float(__float2bfloat16(sn));
  }
  __syncthreads();
  for (int head = warp; head < heads; head += warps) {
    const bf16* src = source(head);
    if (head != warp) load_bf16_vec<PER>(src + d0, v);
    if (head < n_q + n_kv) {
      const bf16* nw = head < n_q ? q_norm : k_norm;
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i) ss += v[i] * v[i];
      ss = warp_sum(ss);
      const float inv = rsqrtf(ss / D + eps);
      float g[PER];
      load_bf16_vec<PER>(nw + d0, g);
#pragma unroll
      for (int i = 0; i < PER; ++i) v[i] = __bfloat162float(__float2bfloat16(v[i] * inv * (1.0f + g[i])));
      // partial RoPE, half-split pairing: (d, d + rot/2) for d < rot/2
      bf16* t = s_rot[warp];
      __syncwarp();  // the previous head of this warp has been read
      if (d0 < rot) store_bf16_vec<PER>(t + d0, v);  // already rounded: exact
      __syncwarp();
      if (d0 < rot) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int d = d0 + i;
          if (d >= rot) break;
          const int f = d < half ? d : d - half;
          const float other = d < half ? -__bfloat162float(t[d + half]) : __bfloat162float(t[d - half]);
          v[i] = __bfloat162float(__float2bfloat16(v[i] * s_cos[f])) + __bfloat162float(__float2bfloat16(other * s_sin[f]));
        }
      }
    }
    if (head < n_q) {
      store_bf16_vec<PER>(q_out + (static_cast<size_t>(row) * n_q + head) * D + d0, v);
      copy_bf16_vec<PER>(gate_out + (static_cast<size_t>(row) * n_q + head) * D + d0, src + D + d0);
    } else {
      const int seq = seq_of_row[row];
      const int page = tables[static_cast<size_t>(seq) * max_pages + pos / PAGE];
      if (page < 0 || page >= num_pages) { if (lane == 0) atomicCAS(err, 0, ERR_BAD_INDEX); continue; }
      const int which = head < n_q + n_kv ? 0 : 1;
      const int kh = which ? head - n_q - n_kv : head - n_q;
      bf16* dst = kv + ((((static_cast<size_t>(page) * 2 + which) * n_kv + kh) * PAGE) + pos % PAGE) * D;
      store_bf16_vec<PER>(dst + d0, v);
    }
  }
}

// Partials: part_acc [B*G, n_q, Z, D] fp32, part_ml [B*G, n_q, Z, 2] (running max, running sum).
//
// One CTA per (sequence, kv head, lane z); warp w serves query head w of the GQA group. A page's
// K and V tiles (64 tokens x D) are staged in shared memory once with coalesced 16-byte loads
// and shared by all heads of the group, so HBM sees every KV byte once per layer. K rows are
// padded by 16 bytes: lane t reads row t, and the pad spreads rows over the banks. Scores: lane
// owns tokens `lane` and `lane + 32`; softmax statistics by warp reductions once per page;
// P.V: lane owns D/32 consecutive output dims.
template <int D>
struct AttnSmem {
  static constexpr int KSTRIDE = D + 8;  // bf16 elements per padded K row
  static constexpr size_t bytes(int group) {
    return static_cast<size_t>(PAGE) * KSTRIDE * 2 + static_cast<size_t>(PAGE) * D * 2 +
           static_cast<size_t>(group) * D * 4 + static_cast<size_t>(group) * PAGE * 4;
  }
};

template <int D, int GROUP>
__global__ void __launch_bounds__(32 * GROUP)
paged_attn_kernel(const bf16* q, const bf16* kv, const int* tables, int max_pages, const int64_t* positions,
                  float* part_acc, float* part_ml, int n_q, int n_kv, int G, int Z, float scale, int num_pages) {
  constexpr int KS = AttnSmem<D>::KSTRIDE;
  constexpr int PER = D / 32;
  constexpr int NT = 32 * GROUP;
  constexpr int CHUNKS = D / 8;  // 16-byte chunks per row
  extern __shared__ __align__(16) uint8_t smem_attn[];
  bf16* sK = reinterpret_cast<bf16*>(smem_attn);
  bf16* sV = sK + PAGE * KS;
  float* sQ = reinterpret_cast<float*>(sV + PAGE * D);
  float* sP = sQ + GROUP * D;
  const int b = blockIdx.x, kh = blockIdx.y, z = blockIdx.z;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qh = kh * GROUP + w;
  for (int g = 0; g < G; ++g) {
    const int row = b * G + g;
    const int len = static_cast<int>(positions[row]) + 1;  // keys 0..pos inclusive
    {
      const bf16* qp = q + (static_cast<size_t>(row) * n_q + qh) * D;
#pragma unroll
      for (int i = 0; i < PER; ++i) sQ[w * D + lane + 32 * i] = __bfloat162float(qp[lane + 32 * i]) * scale;
    }
    float m = -INFINITY, l = 0.f;
    float acc[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) acc[i] = 0.f;
    const int n_pages = (len + PAGE - 1) / PAGE;
    for (int pg = z; pg < n_pages; pg += Z) {
      int page = tables[static_cast<size_t>(b) * max_pages + pg];
      if (page < 0 || page >= num_pages) page = 0;
      const bf16* kp = kv + ((static_cast<size_t>(page) * 2 + 0) * n_kv + kh) * PAGE * D;
      const bf16* vp = kv + ((static_cast<size_t>(page) * 2 + 1) * n_kv + kh) * PAGE * D;
      const int n_tok = min(PAGE, len - pg * PAGE);
      __syncthreads();  // previous page (and the q of a previous row) fully consumed
      for (int c = threadIdx.x; c < n_tok * CHUNKS; c += NT) {
        const int t = c / CHUNKS, j = c % CHUNKS;
        *reinterpret_cast<uint4*>(sK + t * KS + j * 8) = *reinterpret_cast<const uint4*>(kp + static_cast<size_t>(t) * D + j * 8);
        *reinterpret_cast<uint4*>(sV + t * D + j * 8) = *reinterpret_cast<const uint4*>(vp + static_cast<size_t>(t) * D + j * 8);
      }
      __syncthreads();
      // scores of this head against tokens lane and lane + 32
      float s0 = 0.f, s1 = 0.f;
      const bool v0 = lane < n_tok, v1 = lane + 32 < n_tok;
      const bf16* k0 = sK + lane * KS;
      const bf16* k1 = sK + (lane + 32) * KS;
      const float* qv = sQ + w * D;
#pragma unroll 4
      for (int j = 0; j < CHUNKS; ++j) {
        const float4 qa = *reinterpret_cast<const float4*>(qv + j * 8);
        const float4 qb = *reinterpret_cast<const float4*>(qv + j * 8 + 4);
        if (v0) {
          uint4 raw = *reinterpret_cast<const uint4*>(k0 + j * 8);
          const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&raw);
          const float2 a = __bfloat1622float2(e[0]), bb = __bfloat1622float2(e[1]), c2 = __bfloat1622float2(e[2]), d2 = __bfloat1622float2(e[3]);
          s0 += qa.x * a.x + qa.y * a.y + qa.z * bb.x + qa.w * bb.y + qb.x * c2.x + qb.y * c2.y + qb.z * d2.x + qb.w * d2.y;
        }
        if (v1) {
          uint4 raw = *reinterpret_cast<const uint4*>(k1 + j * 8);
          const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&raw);
          const float2 a = __bfloat1622float2(e[0]), bb = __bfloat1622float2(e[1]), c2 = __bfloat1622float2(e[2]), d2 = __bfloat1622float2(e[3]);
          s1 += qa.x * a.x + qa.y * a.y + qa.z * bb.x + qa.w * bb.y + qb.x * c2.x + qb.y * c2.y + qb.z * d2.x + qb.w * d2.y;
        }
      }
      if (!v0) s0 = -INFINITY;
      if (!v1) s1 = -INFINITY;
      const float mn = fmaxf(m, warp_max(fmaxf(s0, s1)));
      const float corr = __expf(m - mn);
      const float p0 = v0 ? __expf(s0 - mn) : 0.f, p1 = v1 ? __expf(s1 - mn) : 0.f;
      sP[w * PAGE + lane] = p0;
      sP[w * PAGE + lane + 32] = p1;
      l = l * corr + warp_sum(p0 + p1);
      m = mn;
#pragma unroll
      for (int i = 0; i < PER; ++i) acc[i] *= corr;
      __syncwarp();
      const float* pw = sP + w * PAGE;
      for (int t = 0; t < n_tok; ++t) {
        const float pt = pw[t];
        float ve[PER];
        load_bf16_vec<PER>(sV + t * D + lane * PER, ve);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] += pt * ve[i];
      }
      __syncwarp();
    }
    float* pa = part_acc + ((static_cast<size_t>(row) * n_q + qh) * Z + z) * D + lane * PER;
#pragma unroll
    for (int i = 0; i < PER; ++i) pa[i] = acc[i];
    if (lane == 0) {
      float* pm = part_ml + ((static_cast<size_t>(row) * n_q + qh) * Z + z) * 2;
      pm[0] = m; pm[1] = l;
    }
    __syncthreads();  // sQ is rewritten for the next row
  }
}

constexpr int COMBINE_GROUPS = 16;
__device__ __forceinline__ bf16 gated(float o, bf16 gate) {
  return __float2bfloat16(__bfloat162float(__float2bfloat16(o)) * sigmoid_f(__bfloat162float(gate)));
}

// Merge the Z partials of one (row, head). Up to COMBINE_GROUPS splits are added in order, each sum one chain of fused
// multiply-adds (a product that is rounded before it is added costs the sum bits where partials cancel). Of more splits,
// partial z goes to running sum z % COMBINE_GROUPS, and the sums are added in order at the end. Which of the two, and the
// order, depends on the splits that hold keys only, never on the table width behind them or on the launch. A thread owns
// four columns and GPT of the sums, so GPT partial rows are in flight at once (one thread per column walking all
// partials was bound by their latency: 58 us for four sequences of 50-90k tokens in a 512-partial table, 7.4 us now).
template <int D, int GPT>
__global__ void __launch_bounds__(D / 4 * COMBINE_GROUPS / GPT)
attn_combine_kernel(const float* part_acc, const float* part_ml, const bf16* gate, bf16* out, int n_q, int Z) {
  constexpr int QUADS = D / 4, THREADS = QUADS * COMBINE_GROUPS / GPT, WARPS = THREADS / 32;
  __shared__ float s_max[WARPS], s_l[COMBINE_GROUPS], s_f[COMBINE_GROUPS];
  __shared__ int s_last[WARPS];
  __shared__ __align__(16) float s_acc[COMBINE_GROUPS][D];
  const int row = blockIdx.x, qh = blockIdx.y;
  const size_t head = static_cast<size_t>(row) * n_q + qh;
  const int quad = threadIdx.x % QUADS, g0 = threadIdx.x / QUADS * GPT;
  pdl_wait();
  pdl_launch();
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + head * Z;
  float m = -INFINITY;
  int last = 0;  // one past the last partial that holds a key
  for (int z = threadIdx.x; z < Z; z += THREADS) {
    const float mz = ml[z].x;
    m = fmaxf(m, mz);
    if (mz != -INFINITY) last = z + 1;
  }
  m = warp_max(m);
  last = __reduce_max_sync(0xffffffffu, last);
  if ((threadIdx.x & 31) == 0) { s_max[threadIdx.x >> 5] = m; s_last[threadIdx.x >> 5] = last; }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < WARPS; ++w) { m = fmaxf(m, s_max[w]); last = max(last, s_last[w]); }
  const bool few = last <= COMBINE_GROUPS;
  const float4* pa = reinterpret_cast<const float4*>(part_acc + head * Z * D) + quad;
  float l[GPT], f[GPT];  // f, few: the factor of the sum's one partial, applied when it is added
  float4 acc[GPT];
#pragma unroll
  for (int u = 0; u < GPT; ++u) { l[u] = f[u] = 0.f; acc[u] = make_float4(0.f, 0.f, 0.f, 0.f); }
#pragma unroll 2
  for (int z0 = g0; z0 < last; z0 += COMBINE_GROUPS) {
    float2 pm[GPT];
    float4 v[GPT];
#pragma unroll
    for (int u = 0; u < GPT; ++u) {
      pm[u] = z0 + u < last ? ml[z0 + u] : make_float2(-INFINITY, 0.f);
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (pm[u].x != -INFINITY) v[u] = pa[static_cast<size_t>(z0 + u) * QUADS];  // an empty partial is never written
    }
#pragma unroll
    for (int u = 0; u < GPT; ++u) {
      if (pm[u].x == -INFINITY) continue;
      f[u] = __expf(pm[u].x - m);
      const float sc = few ? 1.f : f[u];
      l[u] += pm[u].y * sc;
      acc[u].x += v[u].x * sc; acc[u].y += v[u].y * sc; acc[u].z += v[u].z * sc; acc[u].w += v[u].w * sc;
    }
  }
#pragma unroll
  for (int u = 0; u < GPT; ++u) {
    *reinterpret_cast<float4*>(&s_acc[g0 + u][quad * 4]) = acc[u];
    if (quad == 0) { s_l[g0 + u] = l[u]; s_f[g0 + u] = f[u]; }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < D; d += THREADS) {
    float ls = 0.f, o = 0.f;
    if (few) {
#pragma unroll
      for (int g = 0; g < COMBINE_GROUPS; ++g) { ls = fmaf(s_l[g], s_f[g], ls); o = fmaf(s_acc[g][d], s_f[g], o); }
    } else {
#pragma unroll
      for (int g = 0; g < COMBINE_GROUPS; ++g) { ls += s_l[g]; o += s_acc[g][d]; }
    }
    out[head * D + d] = gated(o / ls, gate[head * D + d]);
  }
}

// At most COMBINE_GROUPS partials: neither an exchange between threads nor a barrier. D / 4 threads per (row, head).
template <int D>
__global__ void __launch_bounds__(256)
attn_combine_few_kernel(const float* part_acc, const float* part_ml, const bf16* gate, bf16* out, int heads, int Z) {
  constexpr int QUADS = D / 4, BATCH = 4;
  const int quad = threadIdx.x % QUADS;
  const size_t head = static_cast<size_t>(blockIdx.x) * (256 / QUADS) + threadIdx.x / QUADS;
  pdl_wait();
  pdl_launch();
  if (head >= heads) return;
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + head * Z;
  const float4* pa = reinterpret_cast<const float4*>(part_acc + head * Z * D) + quad;
  const uint2 graw = reinterpret_cast<const uint2*>(gate + head * D)[quad];
  float2 pm[COMBINE_GROUPS];
  float m = -INFINITY;
#pragma unroll
  for (int z = 0; z < COMBINE_GROUPS; ++z) pm[z] = z < Z ? ml[z] : make_float2(-INFINITY, 0.f);
#pragma unroll
  for (int z = 0; z < COMBINE_GROUPS; ++z) m = fmaxf(m, pm[z].x);
  float ls = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int z0 = 0; z0 < COMBINE_GROUPS; z0 += BATCH) {
    float4 v[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
      if (pm[z0 + u].x != -INFINITY) v[u] = pa[static_cast<size_t>(z0 + u) * QUADS];  // an empty partial is never written
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      if (pm[z0 + u].x == -INFINITY) continue;
      const float sc = __expf(pm[z0 + u].x - m);
      ls = fmaf(pm[z0 + u].y, sc, ls);
      o[0] = fmaf(v[u].x, sc, o[0]);
      o[1] = fmaf(v[u].y, sc, o[1]);
      o[2] = fmaf(v[u].z, sc, o[2]);
      o[3] = fmaf(v[u].w, sc, o[3]);
    }
  }
  const bf16* ge = reinterpret_cast<const bf16*>(&graw);
  uint2 raw;
  bf16* oe = reinterpret_cast<bf16*>(&raw);
#pragma unroll
  for (int j = 0; j < 4; ++j) oe[j] = gated(o[j] / ls, ge[j]);
  reinterpret_cast<uint2*>(out + head * D)[quad] = raw;
}

// Up to 16 partials (contexts up to 8192 tokens, or short tables): no exchange between threads (128 rows of 8 partials:
// 4.3 us, 11.7 us with the exchange; 256 rows 12.9 -> 8.7 us). Below 64 partials (512 pages of table) four sums per thread
// fill a CTA of 256 threads (D = 256) and rows and heads fill the GPU; beyond, few sequences share the GPU and one sum per thread keeps
// four times as many rows in flight per CTA.
template <int D>
static cudaError_t launch_combine(const float* part_acc, const float* part_ml, const bf16* gate, bf16* out, int rows,
                                  int n_q, int Z, cudaStream_t st) {
  constexpr int T4 = D / 4 * COMBINE_GROUPS / 4;
  const dim3 grid(rows, n_q);
  const auto at = [](const void* p, int bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; };
  if (!at(part_acc, 16) || !at(part_ml, 8)) return cudaErrorInvalidValue;
  // (the gate may be a view that starts at any element: the other kernels read it and write `out` element by element)
  if (Z <= COMBINE_GROUPS && at(gate, 8) && at(out, 8)) {
    const int per = 256 / (D / 4), heads = rows * n_q;
    return launch_pdl(attn_combine_few_kernel<D>, dim3((heads + per - 1) / per), dim3(256), 0, st, part_acc, part_ml, gate,
                      out, heads, Z);
  }
  if (Z < 64) return launch_pdl(attn_combine_kernel<D, 4>, grid, dim3(T4), 0, st, part_acc, part_ml, gate, out, n_q, Z);
  return launch_pdl(attn_combine_kernel<D, 1>, grid, dim3(T4 * 4), 0, st, part_acc, part_ml, gate, out, n_q, Z);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_attn_prep(const void* qkv, int ld, const int64_t* positions, const int* tables, int max_pages,
                              const int* seq_of_row, const void* q_norm, const void* k_norm, void* q_out, void* gate_out,
                              void* kv, int rows, int n_q, int n_kv, int D, int rot, float theta, float eps,
                              int num_pages, int* err, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (rot > D) return -7;
  const int heads = n_q + 2 * n_kv;
  const dim3 grid(rows), block(32 * (heads < PREP_WARPS ? heads : PREP_WARPS));
#define PREP(DD)                                                                                                      \
  launch_pdl(attn_prep_kernel<DD>, grid, block, 0, st, static_cast<const bf16*>(qkv), ld, positions, tables,    \
             max_pages, seq_of_row, static_cast<const bf16*>(q_norm), static_cast<const bf16*>(k_norm),              \
             static_cast<bf16*>(q_out), static_cast<bf16*>(gate_out), static_cast<bf16*>(kv), n_q, n_kv, rot, theta, \
             eps, num_pages, err)
  if (D == 256) PREP(256);
  else if (D == 128) PREP(128);
  else if (D == 64) PREP(64);
  else if (D == 32) PREP(32);
  else return -7;
#undef PREP
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

extern "C" int b200_paged_attn(const void* q, const void* gate, const void* kv, const int* tables, int max_pages,
                               const int64_t* positions, float* part_acc, float* part_ml, void* out, int B, int G,
                               int n_q, int n_kv, int D, int Z, int num_pages, cudaStream_t st) {
  if (B <= 0) return 0;
  const int group = n_q / n_kv;
  const float scale = 1.0f / sqrtf(static_cast<float>(D));
  dim3 grid(B, n_kv, Z);
#define ATT(DD, GG)                                                                                                  \
  do {                                                                                                                \
    auto kern = paged_attn_kernel<DD, GG>;                                                                           \
    const size_t smem = AttnSmem<DD>::bytes(GG);                                                                     \
    static bool configured = false;                                                                                  \
    if (!configured) {                                                                                               \
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess) return -3; \
      configured = true;                                                                                             \
    }                                                                                                                \
    kern<<<grid, 32 * GG, smem, st>>>(static_cast<const bf16*>(q), static_cast<const bf16*>(kv), tables, max_pages, \
                                      positions, part_acc, part_ml, n_q, n_kv, G, Z, scale, num_pages);              \
  } while (0)
#define ATT_GROUPS(DD)                         \
  if (group == 8) ATT(DD, 8);                  \
  else if (group == 4) ATT(DD, 4);             \
  else if (group == 2) ATT(DD, 2);             \
  else if (group == 1) ATT(DD, 1);             \
  else return -7
  if (D == 256) { ATT_GROUPS(256); }
  else if (D == 128) { ATT_GROUPS(128); }
  else if (D == 64) { ATT_GROUPS(64); }
  else if (D == 32) { ATT_GROUPS(32); }
  else return -7;
#undef ATT_GROUPS
#undef ATT
  const bf16* g = static_cast<const bf16*>(gate);
  bf16* o = static_cast<bf16*>(out);
  cudaError_t rc = cudaGetLastError();
  if (rc != cudaSuccess) return -4;
  if (D == 256) rc = launch_combine<256>(part_acc, part_ml, g, o, B * G, n_q, Z, st);
  else if (D == 128) rc = launch_combine<128>(part_acc, part_ml, g, o, B * G, n_q, Z, st);
  else if (D == 64) rc = launch_combine<64>(part_acc, part_ml, g, o, B * G, n_q, Z, st);
  else rc = launch_combine<32>(part_acc, part_ml, g, o, B * G, n_q, Z, st);
  return rc == cudaSuccess ? 0 : -4;
}

// Merge split partials [rows, n_q, Z, D] / [rows, n_q, Z, 2] (the order: attn_combine_kernel), apply sigmoid(gate), store bf16.
extern "C" int b200_attn_combine(const float* part_acc, const float* part_ml, const void* gate, void* out, int rows,
                                 int n_q, int D, int Z, cudaStream_t st) {
  if (rows <= 0) return 0;
  const bf16* g = static_cast<const bf16*>(gate);
  bf16* o = static_cast<bf16*>(out);
  cudaError_t rc;
  if (D == 256) rc = launch_combine<256>(part_acc, part_ml, g, o, rows, n_q, Z, st);
  else if (D == 128) rc = launch_combine<128>(part_acc, part_ml, g, o, rows, n_q, Z, st);
  else if (D == 64) rc = launch_combine<64>(part_acc, part_ml, g, o, rows, n_q, Z, st);
  else return -7;
  return rc == cudaSuccess ? 0 : -4;
}
