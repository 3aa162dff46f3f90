// Grouped-query decode attention over the KV cache (the decode branch of
// attention, examples/llm/qwen3.py:322-327): scores q.k over the head dim from
// K [B, KV, S, D], an f32 softmax over positions, p.v over positions from
// V [B, KV, D, S] (both caches are read along their minor axis, the layout the
// reference chose, qwen3.py:279-291).
//
// Split over positions: a CTA owns 64 cache slots of one (batch, KV head) and
// all G query heads that share it, and writes an unnormalised partial
// (sum p v, running max, sum p) to scratch; a second kernel merges the
// partials.  All K and V bytes of a CTA are requested up front (one DRAM
// latency per CTA).  Both products run on mma.sync with the query heads as the 8-wide operand and the cache bytes, as
// loaded, as the 16-row one (positions for q.k, head dimensions for p.v): multiply-adds on the FMA pipes, with a shared
// load for every eight of them, kept an SM busy twice as long as its share of the KV bytes takes.  The f32 probabilities
// go in as three bf16 terms, which hold all of their 24 bits, and every MMA of a leading term starts from zero, its sum being added in
// f32: along a chain of accumulators the tensor core drops low bits (merged partials, D 128, position 777, against float64: FMA chains
// 1.9e-7, accumulator chains 3.4e-7, as here 1.5e-7; no difference in time).  Decoder step (6 layers) at batch 32, position 2048:
// 1636 -> 1264 us; batch 8, position 777: 661 -> 611; batch 1, position 2048: 380 -> 361.  (Longer runs of chunks per CTA,
// prefetched, were slower than a CTA per chunk: 1697 -> 1754 us at batch 32.)  In the fused form the kernel also does what precedes
// attention in the layer (qwen3.py:366-369): per-head RMSNorm and rotate-half
// RoPE of q from the fused qkv row, and - in the CTA whose slots contain the
// new position - of k, plus the cache writes of k and v.  That CTA takes the
// new key/value from shared memory, so nothing is read back after being written.
#include <mutex>

#include "common.cuh"

using namespace b200;

namespace {

constexpr int kChunk = 64;     // cache positions per CTA
constexpr int kThreads = 128;

struct AttnArgs {
  const __nv_bfloat16* q;        // [B, H, D], already normalised + rotated (plain form)
  const __nv_bfloat16* qkv;      // [B, (H + 2 KV) D] (fused form), else null
  const __nv_bfloat16* q_norm;
  const __nv_bfloat16* k_norm;
  const float* inv_freq;         // [D / 2] or null (computed in the kernel)
  __nv_bfloat16* k_cache;        // [B, KV, S, D]
  __nv_bfloat16* v_cache;        // [B, KV, D, S]
  __nv_bfloat16* out;            // [B, H, D]
  const int32_t* pos;
  float* scratch;                // [B, KV, splits, G, D + 2]
  int heads, kv_heads;
  int64_t max_len;
  int splits;
  int vec_v;                     // V rows allow 16-byte loads (max_len % 8 == 0, base aligned)
  float scale, theta, eps;
  int* status;                   // device status word
};

// RMSNorm + RoPE of one head by one warp; the results (bf16-rounded, as the
// reference rounds after rms_norm and after rope) go to dst1[i], dst2[i] for
// i < D/2 (first and second half of the head).
template <int D>
__device__ __forceinline__ void norm_rope_head(const __nv_bfloat16* src, const __nv_bfloat16* w, int pos,
                                               const AttnArgs& a, int lane, __nv_bfloat16* dst1, __nv_bfloat16* dst2) {
  constexpr int PAIRS = D / 64;
  float x1[PAIRS], x2[PAIRS];
  float ss = 0.0f;
#pragma unroll
  for (int p = 0; p < PAIRS; ++p) {
    const int i = lane + 32 * p;
    x1[p] = __bfloat162float(src[i]);
    x2[p] = __bfloat162float(src[i + D / 2]);
    ss = fmaf(x1[p], x1[p], ss);
    ss = fmaf(x2[p], x2[p], ss);
  }
  ss = warp_sum(ss);
  const float r = 1.0f / sqrtf(ss / static_cast<float>(D) + a.eps);
#pragma unroll
  for (int p = 0; p < PAIRS; ++p) {
    const int i = lane + 32 * p;
    const float n1 = bf16_round((x1[p] * r) * __bfloat162float(w[i]));
    const float n2 = bf16_round((x2[p] * r) * __bfloat162float(w[i + D / 2]));
    const float inv_freq = a.inv_freq != nullptr
                               ? a.inv_freq[i]
                               : static_cast<float>(1.0 / pow(static_cast<double>(a.theta), static_cast<double>(2 * i) / D));
    float sn, cs;
    sincosf(static_cast<float>(pos) * inv_freq, &sn, &cs);
    dst1[i] = __float2bfloat16_rn(n1 * cs - n2 * sn);
    dst2[i] = __float2bfloat16_rn(n2 * cs + n1 * sn);
  }
}

// The three bf16 terms of eight f32 values, as the operand pairs of two MMAs (pairs of neighbours in a word).
__device__ __forceinline__ void split3(const float (&p)[8], uint32_t (&t)[3][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a = p[2 * j], b = p[2 * j + 1];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      t[k][j] = pack_bf16(a, b);
      a -= bf16_lo(t[k][j]);
      b -= bf16_hi(t[k][j]);
    }
  }
}

template <int D, int G>
__global__ void __launch_bounds__(kThreads, 4) attn_partial_kernel(const AttnArgs a) {
  // A lane (g = lane / 4, t = lane % 4) holds eight consecutive inputs 8 t .. of every 32 of its rows g and g + 8 and of
  // its column g: the order of k inside an MMA does not matter as long as both operands share it.
  constexpr int KB = D / 32;         // blocks of 32 head dimensions (q.k)
  constexpr int VB = kChunk / 32;    // blocks of 32 positions (p.v)
  constexpr int DT = D / 64;         // 16-row tiles of head dimensions per warp (p.v)
  constexpr int QP = D + 32;         // pitch: rows 64 bytes apart modulo 128
  __shared__ __align__(16) __nv_bfloat16 qs[G][QP];
  __shared__ __align__(16) float sc[G][kChunk + 8];
  __shared__ float red[2][G][kThreads / 32];
  __shared__ __align__(16) __nv_bfloat16 knew[D];
  __shared__ __nv_bfloat16 vnew[D];
  // Fused form: the position and the cache slots of earlier steps (all below *pos) do not
  // come from the kernel before this one, so they are requested before waiting for it.
  // Plain form: slot *pos itself is read, and the kernel before this one (the cache write
  // of b200_qk_norm_rope_cache) may still be storing it, so the wait comes first.
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int split = blockIdx.x, kv = blockIdx.y, b = blockIdx.z;
  const bool fused = a.qkv != nullptr;
  if (!fused) pdl_wait();
  const int pos = *a.pos;
  if (pos < 0 || pos >= a.max_len) {         // nothing may be written outside the cache
    pdl_wait();
    if (tid == 0) report_status(a.status, B200_INVALID_ARGUMENT, 500);
    return;
  }
  const int n_valid = pos + 1;
  const int n_old = fused ? pos : pos + 1;   // slots whose K/V are already in the cache
  const int s0 = split * kChunk;
  if (s0 >= n_valid) {                       // the merge only reads splits below n_valid
    pdl_wait();
    return;
  }
  const int cnt = min(kChunk, n_valid - s0);
  const bool owner = fused && pos >= s0 && pos < s0 + kChunk;
  const int64_t bkv = static_cast<int64_t>(b) * a.kv_heads + kv;

  // ---- request every K and V byte of this CTA now ------------------------------------
  const int g = lane >> 2, t = lane & 3;
  const int p0 = warp * 16 + g;              // positions p0 and p0 + 8 of the chunk
  uint4 kreg[2][KB];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool have = s0 + p0 + 8 * h < n_old;
    const uint4* krow = reinterpret_cast<const uint4*>(a.k_cache + (bkv * a.max_len + s0 + p0 + 8 * h) * D + 8 * t);
#pragma unroll
    for (int v = 0; v < KB; ++v) kreg[h][v] = have ? krow[4 * v] : make_uint4(0, 0, 0, 0);
  }
  const int d0 = warp * 16 * DT + g;         // head dimensions d0 + 16 i and d0 + 16 i + 8
  uint4 vreg[DT][2][VB];
#pragma unroll
  for (int i = 0; i < DT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const __nv_bfloat16* vrow = a.v_cache + (bkv * D + d0 + 16 * i + 8 * h) * a.max_len + s0;
#pragma unroll
      for (int v = 0; v < VB; ++v) {
        const int o = 32 * v + 8 * t;
        if (a.vec_v) {
          vreg[i][h][v] = s0 + o < n_old ? *reinterpret_cast<const uint4*>(vrow + o) : make_uint4(0, 0, 0, 0);
        } else {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint16_t* q = reinterpret_cast<const uint16_t*>(vrow + o + 2 * e);
            w[e] = (s0 + o + 2 * e < n_old ? q[0] : 0u) | (s0 + o + 2 * e + 1 < n_old ? static_cast<uint32_t>(q[1]) << 16 : 0u);
          }
          vreg[i][h][v] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }

  // ---- queries (and, in the owning CTA, the new key and value) -----------------------
  pdl_wait();   // q (or the fused qkv row) is the previous kernel's output
  if (fused) {
    const int total_heads = a.heads + 2 * a.kv_heads;
    const __nv_bfloat16* row = a.qkv + static_cast<int64_t>(b) * total_heads * D;
    for (int gq = warp; gq < G; gq += kThreads / 32)
      norm_rope_head<D>(row + static_cast<int64_t>(kv * G + gq) * D, a.q_norm, pos, a, lane, qs[gq], qs[gq] + D / 2);
    if (owner) {
      if (warp == (G % 4)) {
        norm_rope_head<D>(row + static_cast<int64_t>(a.heads + kv) * D, a.k_norm, pos, a, lane, knew, knew + D / 2);
        __syncwarp();
        __nv_bfloat16* kdst = a.k_cache + (bkv * a.max_len + pos) * D;
        for (int i = lane; i < D; i += 32) kdst[i] = knew[i];
      } else if (warp == ((G + 1) % 4)) {
        const __nv_bfloat16* vsrc = row + static_cast<int64_t>(a.heads + a.kv_heads + kv) * D;
        __nv_bfloat16* vdst = a.v_cache + bkv * D * a.max_len + pos;
        for (int d = lane; d < D; d += 32) {
          const __nv_bfloat16 v = vsrc[d];
          vnew[d] = v;
          vdst[static_cast<int64_t>(d) * a.max_len] = v;
        }
      }
    }
  } else {
    for (int i = tid; i < G * D; i += kThreads) {
      const int gq = i / D, d = i % D;
      qs[gq][d] = a.q[(static_cast<int64_t>(b) * a.heads + kv * G + gq) * D + d];
    }
  }
  __syncthreads();

  // ---- scores: rows = positions, columns = heads; c[2 h + j] is position p0 + 8 h, head 2 t + j
  if (owner) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (s0 + p0 + 8 * h == pos) {
#pragma unroll
        for (int v = 0; v < KB; ++v) kreg[h][v] = *reinterpret_cast<const uint4*>(knew + 32 * v + 8 * t);
      }
  }
  float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int v = 0; v < KB; ++v) {
    const uint4 q = g < G ? *reinterpret_cast<const uint4*>(&qs[g < G ? g : 0][32 * v + 8 * t]) : make_uint4(0, 0, 0, 0);
    float d[2][4];
    mma_bf16_16816_z(d[0], kreg[0][v].x, kreg[1][v].x, kreg[0][v].y, kreg[1][v].y, q.x, q.y);
    mma_bf16_16816_z(d[1], kreg[0][v].z, kreg[1][v].z, kreg[0][v].w, kreg[1][v].w, q.z, q.w);
#pragma unroll
    for (int e = 0; e < 4; ++e) c[e] += d[0][e] + d[1][e];
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    c[j] = p0 < cnt ? c[j] * a.scale : -INFINITY;
    c[2 + j] = p0 + 8 < cnt ? c[2 + j] * a.scale : -INFINITY;
    float m = fmaxf(c[j], c[2 + j]);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (g == 0 && 2 * t + j < G) red[0][2 * t + j][warp] = m;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int head = 2 * t + j;
    float l = 0.0f;
    if (head < G) {
      const float m = fmaxf(fmaxf(red[0][head][0], red[0][head][1]), fmaxf(red[0][head][2], red[0][head][3]));
      const float e0 = p0 < cnt ? expf(c[j] - m) : 0.0f, e1 = p0 + 8 < cnt ? expf(c[2 + j] - m) : 0.0f;
      sc[head][p0] = e0;
      sc[head][p0 + 8] = e1;
      l = e0 + e1;
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (g == 0 && head < G) red[1][head][warp] = l;
  }
  __syncthreads();

  // ---- p . v: rows = head dimensions, columns = heads
  if (s0 + kChunk > n_old) {   // only the chunk that holds the newest position has slots that are not in the cache (yet)
#pragma unroll
    for (int i = 0; i < DT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t fresh = owner ? __bfloat16_as_ushort(vnew[d0 + 16 * i + 8 * h]) : 0u;
#pragma unroll
        for (int v = 0; v < VB; ++v) {
          uint32_t w[4] = {vreg[i][h][v].x, vreg[i][h][v].y, vreg[i][h][v].z, vreg[i][h][v].w};
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int slot = s0 + 32 * v + 8 * t + e;
            if (slot >= n_old) {
              const uint32_t x = owner && slot == pos ? fresh : 0u;
              w[e / 2] = (e & 1) ? (w[e / 2] & 0xffffu) | (x << 16) : (w[e / 2] & 0xffff0000u) | x;
            }
          }
          vreg[i][h][v] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
  }
  float o[DT][4];
#pragma unroll
  for (int i = 0; i < DT; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
#pragma unroll
  for (int v = 0; v < VB; ++v) {
    float pr[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) pr[e] = 0.0f;
    if (g < G) {
      const float4 x = *reinterpret_cast<const float4*>(&sc[g < G ? g : 0][32 * v + 8 * t]), y = *reinterpret_cast<const float4*>(&sc[g < G ? g : 0][32 * v + 8 * t + 4]);
      pr[0] = x.x, pr[1] = x.y, pr[2] = x.z, pr[3] = x.w, pr[4] = y.x, pr[5] = y.y, pr[6] = y.z, pr[7] = y.w;
    }
    uint32_t term[3][4];
    split3(pr, term);
#pragma unroll
    for (int i = 0; i < DT; ++i) {
      float d[2][4], small[4];
      mma_bf16_16816_z(small, vreg[i][0][v].x, vreg[i][1][v].x, vreg[i][0][v].y, vreg[i][1][v].y, term[2][0], term[2][1]);
      mma_bf16_16816(small, vreg[i][0][v].z, vreg[i][1][v].z, vreg[i][0][v].w, vreg[i][1][v].w, term[2][2], term[2][3]);
      mma_bf16_16816(small, vreg[i][0][v].x, vreg[i][1][v].x, vreg[i][0][v].y, vreg[i][1][v].y, term[1][0], term[1][1]);
      mma_bf16_16816(small, vreg[i][0][v].z, vreg[i][1][v].z, vreg[i][0][v].w, vreg[i][1][v].w, term[1][2], term[1][3]);
      mma_bf16_16816_z(d[0], vreg[i][0][v].x, vreg[i][1][v].x, vreg[i][0][v].y, vreg[i][1][v].y, term[0][0], term[0][1]);
      mma_bf16_16816_z(d[1], vreg[i][0][v].z, vreg[i][1][v].z, vreg[i][0][v].w, vreg[i][1][v].w, term[0][2], term[0][3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][e] += (small[e] + d[0][e]) + d[1][e];
    }
  }
  // An infinite value meets the zero terms of its probability as NaN: such sums are formed again, term by term.
#pragma unroll
  for (int i = 0; i < DT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int head = 2 * t + (e & 1), d = d0 + 16 * i + 8 * (e >> 1);
      if (o[i][e] == o[i][e] || head >= G) continue;
      const __nv_bfloat16* vrow = a.v_cache + (bkv * D + d) * a.max_len + s0;
      float sum = 0.0f;
#pragma unroll 1
      for (int s = 0; s < cnt; ++s) sum = fmaf(sc[head][s], __bfloat162float(s0 + s < n_old ? vrow[s] : vnew[d]), sum);
      o[i][e] = sum;
    }
  float* part = a.scratch + (bkv * a.splits + split) * G * (D + 2);
#pragma unroll
  for (int i = 0; i < DT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int head = 2 * t + (e & 1);
      if (head < G) part[head * (D + 2) + d0 + 16 * i + 8 * (e >> 1)] = o[i][e];
    }
  if (tid < G) {
    part[tid * (D + 2) + D] = fmaxf(fmaxf(red[0][tid][0], red[0][tid][1]), fmaxf(red[0][tid][2], red[0][tid][3]));
    part[tid * (D + 2) + D + 1] = (red[1][tid][0] + red[1][tid][1]) + (red[1][tid][2] + red[1][tid][3]);
  }
}

// Merges the partials of one (batch, query head): out = sum_s e^{m_s - M} o_s / sum_s e^{m_s - M} l_s.
template <int D, int G>
__global__ void __launch_bounds__(kThreads) attn_combine_kernel(const AttnArgs a) {
  extern __shared__ float wsm[];   // [2][splits]: weights e^{m_s - M}, then the partial sums l_s
  __shared__ float red[kThreads / 32];
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.x, b = blockIdx.y;
  const int kv = h / G, gq = h % G;
  if (*a.pos < 0 || *a.pos >= a.max_len) return;
  const int n_valid = *a.pos + 1;
  const int nsplit = (n_valid + kChunk - 1) / kChunk;
  const float* base = a.scratch + (static_cast<int64_t>(b) * a.kv_heads + kv) * a.splits * G * (D + 2) + gq * (D + 2);
  const int64_t stride = static_cast<int64_t>(G) * (D + 2);
  // Everything this thread needs from the partials is requested at once (one trip to L2):
  // its output dimension of the first kPre splits, and the (max, sum) pair of split `tid`.
  constexpr int kPre = 40;
  const int d0 = tid < D ? tid : 0;
  float o[kPre];
#pragma unroll
  for (int s = 0; s < kPre; ++s) o[s] = s < nsplit ? base[s * stride + d0] : 0.0f;
  float m = -INFINITY;
  for (int s = tid; s < nsplit; s += kThreads) {
    const float2 ml = *reinterpret_cast<const float2*>(&base[s * stride + D]);
    wsm[s] = ml.x;
    wsm[a.splits + s] = ml.y;
    m = fmaxf(m, ml.x);
  }
  m = warp_max(m);
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  __syncthreads();
  float den = 0.0f;
  for (int s = tid; s < nsplit; s += kThreads) {
    const float w = expf(wsm[s] - m);
    wsm[s] = w;
    den = fmaf(w, wsm[a.splits + s], den);
  }
  den = warp_sum(den);
  if (lane == 0) red[warp] = den;
  __syncthreads();
  den = (red[0] + red[1]) + (red[2] + red[3]);
  for (int d = tid; d < D; d += kThreads) {
    float num = 0.0f;
    if (d == d0) {
#pragma unroll
      for (int s = 0; s < kPre; ++s)
        if (s < nsplit) num = fmaf(wsm[s], o[s], num);
    } else {
      for (int s = 0; s < min(nsplit, kPre); ++s) num = fmaf(wsm[s], base[s * stride + d], num);
    }
#pragma unroll 8
    for (int s = kPre; s < nsplit; ++s) num = fmaf(wsm[s], base[s * stride + d], num);
    a.out[(static_cast<int64_t>(b) * a.heads + h) * D + d] = __float2bfloat16_rn(num / den);
  }
}

template <int D>
b200_status LaunchAttn(b200_context* ctx, cudaStream_t stream, const AttnArgs& a, int group, int64_t batch) {
  LaunchCfg lc;
  lc.stream = stream;
  lc.pdl = true;
  lc.block = dim3(kThreads);
  lc.grid = dim3(a.splits, a.kv_heads, static_cast<unsigned>(batch));
  cudaError_t e;
  switch (group) {
    case 1: e = Launch(lc, attn_partial_kernel<D, 1>, a); break;
    case 2: e = Launch(lc, attn_partial_kernel<D, 2>, a); break;
    case 4: e = Launch(lc, attn_partial_kernel<D, 4>, a); break;
    case 8: e = Launch(lc, attn_partial_kernel<D, 8>, a); break;
    default: return Fail(B200_UNIMPLEMENTED, "attention: %d query heads per KV head (1, 2, 4 or 8)", group);
  }
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "attention launch: %s", cudaGetErrorString(e)));
  lc.grid = dim3(a.heads, static_cast<unsigned>(batch));
  lc.smem = static_cast<size_t>(2 * a.splits) * sizeof(float);
  switch (group) {
    case 1: e = Launch(lc, attn_combine_kernel<D, 1>, a); break;
    case 2: e = Launch(lc, attn_combine_kernel<D, 2>, a); break;
    case 4: e = Launch(lc, attn_combine_kernel<D, 4>, a); break;
    default: e = Launch(lc, attn_combine_kernel<D, 8>, a); break;
  }
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "attention merge launch: %s", cudaGetErrorString(e)));
  return EndLaunch(ctx, "b200_attention", 2);
}

b200_status Run(b200_context* ctx, cudaStream_t stream, AttnArgs a, const char* who, int64_t batch, int head_dim) {
  b200_status s = BeginLaunch(ctx);
  if (s != B200_OK) return s;
  if (batch < 0 || a.heads <= 0 || a.kv_heads <= 0 || a.max_len <= 0 || a.heads % a.kv_heads != 0)
    return Fail(B200_INVALID_ARGUMENT, "%s: bad sizes", who);
  if (head_dim != 64 && head_dim != 128) return Fail(B200_UNIMPLEMENTED, "%s: head_dim %d (64 or 128)", who, head_dim);
  if (batch > 65535 || a.kv_heads > 65535) return Fail(B200_UNIMPLEMENTED, "%s: batch or head count too large", who);
  if (a.max_len > (1 << 20)) return Fail(B200_UNIMPLEMENTED, "%s: max_len above 2^20", who);
  if (batch == 0) return B200_OK;
  if (!a.k_cache || !a.v_cache || !a.out || !a.pos || !a.scratch || (!a.q && !a.qkv))
    return Fail(B200_INVALID_ARGUMENT, "%s: null buffer", who);
  if (a.qkv && (!a.q_norm || !a.k_norm)) return Fail(B200_INVALID_ARGUMENT, "%s: null norm gain", who);
  if (!Aligned(a.k_cache, 16) || !Aligned(a.v_cache, 2))
    return Fail(B200_INVALID_ARGUMENT, "%s: the K cache must be 16-byte aligned", who);
  a.splits = static_cast<int>((a.max_len + kChunk - 1) / kChunk);
  a.vec_v = Aligned(a.v_cache, 16) && a.max_len % 8 == 0;
  a.scale = 1.0f / sqrtf(static_cast<float>(head_dim));
  a.status = ctx->dev_status;
  return head_dim == 128 ? LaunchAttn<128>(ctx, stream, a, a.heads / a.kv_heads, batch)
                         : LaunchAttn<64>(ctx, stream, a, a.heads / a.kv_heads, batch);
}

// ---- scratch that nobody has to allocate ------------------------------------------------
// Some hosts of this library may not allocate device memory when they call it: code that
// runs inside a stream capture, or a runtime whose allocator owns every byte of the device
// and forbids cudaMalloc from plugins.  For them the split-attention partials can live in
// this fixed array instead of a caller-provided buffer.  Every GPU that loads the library
// carries it until the process exits.
constexpr size_t kStaticScratchFloats = size_t(2) << 20;   // 8 MiB
static __device__ __align__(256) float g_attn_scratch[kStaticScratchFloats];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
float* g_scratch_ptr[kMaxDevices] = {};   // device address of g_attn_scratch, per device ordinal

// In host code `g_attn_scratch` is only a handle for the symbol, not a device address, so
// the address is asked for once per device (with that device current) and cached.
b200_status StaticScratch(b200_context* ctx, float** out) {
  if (ctx->device < 0 || ctx->device >= kMaxDevices)
    return Fail(B200_UNIMPLEMENTED, "b200_attention_decode_static: device ordinal %d beyond %d", ctx->device, kMaxDevices);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (g_scratch_ptr[ctx->device] == nullptr) {
    float* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_attn_scratch);
    if (e != cudaSuccess || p == nullptr)
      return Stick(ctx, Fail(B200_INTERNAL, "cudaGetSymbolAddress(static attention scratch): %s", cudaGetErrorString(e)));
    g_scratch_ptr[ctx->device] = p;
  }
  *out = g_scratch_ptr[ctx->device];
  return B200_OK;
}

}  // namespace

namespace b200 {
// Called by b200_context_create: the address of the built-in scratch is looked up while the
// context is made, so that b200_attention_decode_static itself never calls into the runtime
// for it (it may run inside a stream capture).
b200_status AttnStaticScratchInit(b200_context* ctx) {
  if (ctx->device < 0 || ctx->device >= kMaxDevices) return B200_OK;   // (the static entry point refuses such a device itself)
  float* p = nullptr;
  return StaticScratch(ctx, &p);
}
}  // namespace b200

extern "C" {

size_t b200_attention_scratch_bytes(int64_t batch, int heads, int head_dim, int64_t max_len) {
  const int64_t splits = (max_len + kChunk - 1) / kChunk;
  return static_cast<size_t>(batch) * heads * splits * (head_dim + 2) * sizeof(float);
}

b200_status b200_attention_decode(b200_context* ctx, b200_stream stream, const void* q, const void* k_cache,
                                  const void* v_cache, void* out, const int32_t* pos, void* scratch, int64_t batch,
                                  int heads, int kv_heads, int head_dim, int64_t max_len) {
  AttnArgs a = {};
  a.q = static_cast<const __nv_bfloat16*>(q);
  a.k_cache = static_cast<__nv_bfloat16*>(const_cast<void*>(k_cache));
  a.v_cache = static_cast<__nv_bfloat16*>(const_cast<void*>(v_cache));
  a.out = static_cast<__nv_bfloat16*>(out);
  a.pos = pos;
  a.scratch = static_cast<float*>(scratch);
  a.heads = heads;
  a.kv_heads = kv_heads;
  a.max_len = max_len;
  return Run(ctx, stream, a, "b200_attention_decode", batch, head_dim);
}

b200_status b200_attention_step(b200_context* ctx, b200_stream stream, const void* qkv, const void* q_norm,
                                const void* k_norm, const float* inv_freq_or_null, void* k_cache, void* v_cache,
                                void* out, const int32_t* pos, void* scratch, int64_t batch, int heads,
                                int kv_heads, int head_dim, int64_t max_len, float theta, float eps) {
  AttnArgs a = {};
  a.qkv = static_cast<const __nv_bfloat16*>(qkv);
  a.q_norm = static_cast<const __nv_bfloat16*>(q_norm);
  a.k_norm = static_cast<const __nv_bfloat16*>(k_norm);
  a.inv_freq = inv_freq_or_null;
  a.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  a.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  a.out = static_cast<__nv_bfloat16*>(out);
  a.pos = pos;
  a.scratch = static_cast<float*>(scratch);
  a.heads = heads;
  a.kv_heads = kv_heads;
  a.max_len = max_len;
  a.theta = theta;
  a.eps = eps;
  return Run(ctx, stream, a, "b200_attention_step", batch, head_dim);
}

b200_status b200_attention_decode_static(b200_context* ctx, b200_stream stream, const void* q, const void* k_cache,
                                         const void* v_cache, void* out, const int32_t* pos, int64_t batch,
                                         int heads, int kv_heads, int head_dim, int64_t max_len) {
  b200_status s = BeginLaunch(ctx);   // makes the context's device current
  if (s != B200_OK) return s;
  if (batch < 0 || heads <= 0 || max_len <= 0 || (head_dim != 64 && head_dim != 128))
    return Fail(B200_INVALID_ARGUMENT, "b200_attention_decode_static: bad sizes");
  const size_t need = b200_attention_scratch_bytes(batch, heads, head_dim, max_len);
  if (need > kStaticScratchFloats * sizeof(float))
    return Fail(B200_RESOURCE_EXHAUSTED,
                "b200_attention_decode_static: batch %lld x heads %d x max_len %lld needs %zu bytes of scratch; the "
                "built-in scratch holds %zu (use b200_attention_decode with a caller buffer)",
                static_cast<long long>(batch), heads, static_cast<long long>(max_len), need,
                kStaticScratchFloats * sizeof(float));
  float* scratch = nullptr;
  s = StaticScratch(ctx, &scratch);
  if (s != B200_OK) return s;
  AttnArgs a = {};
  a.q = static_cast<const __nv_bfloat16*>(q);
  a.k_cache = static_cast<__nv_bfloat16*>(const_cast<void*>(k_cache));
  a.v_cache = static_cast<__nv_bfloat16*>(const_cast<void*>(v_cache));
  a.out = static_cast<__nv_bfloat16*>(out);
  a.pos = pos;
  a.scratch = scratch;   // every partial the merge reads is written earlier in the same call: nothing to clear
  a.heads = heads;
  a.kv_heads = kv_heads;
  a.max_len = max_len;
  return Run(ctx, stream, a, "b200_attention_decode_static", batch, head_dim);
}

}  // extern "C"
