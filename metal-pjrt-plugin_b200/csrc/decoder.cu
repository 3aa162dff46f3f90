// One decode step of the Qwen3-shaped int4 decoder
// (examples/llm/qwen3.py:334-390 with T = 1).  Two implementations:
//   * a fixed sequence of this library's kernels on one stream, captured once
//     per batch size into a CUDA graph (the launches carry programmatic-
//     dependent-launch edges, so each projection's weight stream starts while
//     the kernel before it drains): the default;
//   * one persistent kernel for the whole step (decode_stream.cu), on request
//     (B200_DECODER_STREAM=1), where the shapes and the batch allow it.
//
// With a tensor-parallel group the projections are sharded Megatron-style:
// qkv and gate_up by output rows (heads / intermediate columns stay local, as
// do the per-head norms, RoPE, the KV-cache shard and attention), o and down
// by input columns, followed by an f32 all-reduce of the [B, hidden] partial
// sums; the LM head by vocabulary rows, followed by an all-gather of logits.
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <list>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "decode_stream.cuh"
#include "qmm_mid.cuh"

using namespace b200;

namespace {

bool EnvFlag(const char* name) {
  // Same grammar as the reference's EnvFlag (metal_pjrt/runtime/env.cc:17-22):
  // unset, empty, 0, false, no, off (any case) are false; anything else is true.
  const char* v = std::getenv(name);
  if (v == nullptr) return false;
  std::string s(v);
  size_t b = s.find_first_not_of(" \t\n\r"), e = s.find_last_not_of(" \t\n\r");
  s = b == std::string::npos ? "" : s.substr(b, e - b + 1);
  for (char& c : s) c = static_cast<char>(std::tolower(static_cast<unsigned char>(c)));
  return !(s.empty() || s == "0" || s == "false" || s == "no" || s == "off");
}

// x = bf16(x + bf16(y)); h = rms_norm(x) * gain.  One CTA per row.  Used after
// the all-reduce of a K-sharded projection (y holds the f32 sum over ranks).
__global__ void residual_rmsnorm_kernel(__nv_bfloat16* x, const float* y, const __nv_bfloat16* gain,
                                        __nv_bfloat16* h, int n, float eps) {
  extern __shared__ float row[];
  __shared__ float scratch[32];
  pdl_wait();
  pdl_launch_dependents();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * n;
  float ss = 0.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float v = bf16_round(__bfloat162float(x[base + i]) + bf16_round(y[base + i]));
    row[i] = v;
    x[base + i] = __float2bfloat16_rn(v);
    ss = fmaf(v, v, ss);
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = ss;
  __syncthreads();
  float t = (threadIdx.x & 31) < (blockDim.x >> 5) ? scratch[threadIdx.x & 31] : 0.0f;
  t = warp_sum(t);
  const float r = 1.0f / sqrtf(t / static_cast<float>(n) + eps);
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    h[base + i] = __float2bfloat16_rn((row[i] * r) * __bfloat162float(gain[i]));
}

// bf16 -> f32, eight elements per thread (count a multiple of 8, 16-byte aligned buffers).
__global__ void widen_bf16_kernel(const __nv_bfloat16* in, float* out, int64_t count) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
  if (i >= count) return;
  const uint4 raw = *reinterpret_cast<const uint4*>(in + i);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  float4 lo = make_float4(bf16_lo(w[0]), bf16_hi(w[0]), bf16_lo(w[1]), bf16_hi(w[1]));
  float4 hi = make_float4(bf16_lo(w[2]), bf16_hi(w[2]), bf16_lo(w[3]), bf16_hi(w[3]));
  *reinterpret_cast<float4*>(out + i) = lo;
  *reinterpret_cast<float4*>(out + i + 4) = hi;
}

}  // namespace

struct b200_decoder {
  b200_context* ctx = nullptr;
  b200_decoder_config cfg = {};
  std::vector<b200_decoder_layer> layers;
  const void* embed = nullptr;
  const void* final_norm = nullptr;
  const void* lm_head = nullptr;
  b200_tp* tp = nullptr;
  // activations (device, sized for max_batch)
  __nv_bfloat16 *x = nullptr, *h = nullptr, *qkv = nullptr, *attn = nullptr, *gu = nullptr;
  __nv_bfloat16* x2 = nullptr;   // second residual buffer of the push exchange (one CTA writes the new rows while all read the old)
  float *y32 = nullptr, *attn_scratch = nullptr, *logits_local = nullptr, *inv_freq = nullptr;
  __nv_bfloat16* logits_bf16 = nullptr;   // LM head output of the tensor-core route (batches above 8)
  // sums of the slices of K of any one projection (batches above 8).  Memory of the pool instead would be an allocation node
  // between every two kernels of the captured step: a graph that a caller's own capture cannot take in, without
  // the edges that let a projection request its weights early.
  float* slices = nullptr;
  size_t slices_floats = 0;
  bool use_graph = true;
  cudaStream_t capture_stream = nullptr;  // graphs are captured here (the caller's stream may be the legacy one)
  // Captured steps, keyed by (batch, logits pointer) and most recently used first.  Tokens and
  // the position are copied into decoder-owned buffers before every replay, so only the
  // output pointer is baked into a graph; at most kMaxGraphs are kept (the oldest is destroyed).
  static constexpr size_t kMaxGraphs = 8;
  std::list<std::pair<std::pair<int, const void*>, cudaGraphExec_t>> graphs;
  int64_t graphs_built = 0;
  int32_t* tokens_buf = nullptr;   // int32 [max_batch]
  int32_t* pos_buf = nullptr;      // int32 [1]
  std::map<int, int64_t> launches;
  std::mutex mu;                   // steps may come from several host threads
  DecodeStream* stream_path = nullptr;   // the single-kernel step, or null
  // gate_up with its rows rearranged (8 gate rows, then the 8 up rows of the same outputs, per 16): with it the
  // projection's epilogue forms silu(gate) * up itself, so the 148 CTAs of the down projection no longer each
  // recompute all of it while staging their input.  One copy per layer, made at creation; empty: not in use.
  std::vector<b200_qweight> gate_up_pair;
  std::vector<void*> pair_storage;
};

namespace {

// A step's first kernel (the embedding) waits for everything before the step, and no kernel of a step writes a weight.
QmmCaller CallerOf(const b200_decoder* d, const QmmTp* tp) {
  QmmCaller c;
  c.tp = tp;
  c.weights_settled = true;
  c.scratch = d->slices;
  c.scratch_floats = d->slices_floats;
  return c;
}

b200_status Qmm(b200_decoder* d, cudaStream_t stream, const b200_qweight& w, const void* x, void* out, int batch,
                int64_t N, int64_t K, int epilogue, const void* residual, int prologue = B200_QMM_PRO_NONE,
                const void* gain = nullptr, const QmmTp* tp = nullptr) {
  b200_qmm_params p = {};
  p.prologue = prologue;
  p.prologue_gain = gain;
  p.eps = d->cfg.rms_eps;
  p.bits = 4;
  p.group = 64;
  p.nibble_order = 0;
  p.epilogue = epilogue;
  p.x = x;
  p.q = w.q;
  p.scale = w.scale;
  p.bias = w.bias;
  p.residual = residual;
  p.out = out;
  p.M = batch;
  p.N = N;
  p.K = K;
  return QmmRunEx(d->ctx, stream, &p, CallerOf(d, tp));
}

b200_status ResidualNorm(b200_decoder* d, cudaStream_t stream, const void* gain, int batch) {
  b200_status s = BeginLaunch(d->ctx);
  if (s != B200_OK) return s;
  LaunchCfg lc;
  lc.stream = stream;
  lc.pdl = true;
  lc.grid = dim3(batch);
  lc.block = dim3(256);
  lc.smem = static_cast<size_t>(d->cfg.hidden) * 4;
  cudaError_t e = Launch(lc, residual_rmsnorm_kernel, d->x, static_cast<const float*>(d->y32),
                         static_cast<const __nv_bfloat16*>(gain), d->h, static_cast<int>(d->cfg.hidden),
                         d->cfg.rms_eps);
  if (e != cudaSuccess) return Stick(d->ctx, Fail(B200_INTERNAL, "residual_rmsnorm launch: %s", cudaGetErrorString(e)));
  return EndLaunch(d->ctx, "residual_rmsnorm");
}

#define B200_TRY(expr)                 \
  do {                                 \
    b200_status _s = (expr);           \
    if (_s != B200_OK) return _s;      \
  } while (0)

b200_status Enqueue(b200_decoder* d, cudaStream_t stream, const int32_t* tokens, const int32_t* pos, float* logits,
                    int batch) {
  const b200_decoder_config& c = d->cfg;
  b200_context* ctx = d->ctx;
  const int64_t E = c.hidden, HD = static_cast<int64_t>(c.heads) * c.head_dim;
  const int64_t QKV = static_cast<int64_t>(c.heads + 2 * c.kv_heads) * c.head_dim;
  // (A group of ONE rank takes the sharded path too: the whole exchange, lines and two-level sum
  // included, then runs on a single GPU, which is how a one-GPU test or profile reaches that code.)
  const bool tp = d->tp != nullptr;
  const bool peer = tp && d->tp->peer && static_cast<int64_t>(batch) * E <= d->tp->cap;

  // Push exchange (up to 8 rows, peers connected): the o / down projections store their f32
  // partial sums into every rank's exchange block from their epilogue, and the projection
  // after them sums the ranks' sub-slots from its own memory, adds the residual and
  // applies the RMSNorm while it stages its input: no kernel of its own for the exchange.
  QmmTp link;
  // (Up to 4 rows by default.  Measured on 2 GPUs, ms per step, push against the separate exchange kernel:
  // batch 1 2.03 against 2.63, batch 4 2.81 against 2.84, batch 8 3.89 against 3.50: the staging of the
  // consuming projection re-reads the whole summed row in every CTA, which grows with the rows.
  // B200_TP_PUSH_ROWS overrides the limit, B200_TP_PULL=1 switches the push off.)
  static const int push_rows = [] {
    const char* v = std::getenv("B200_TP_PUSH_ROWS");
    return v != nullptr ? std::atoi(v) : 4;
  }();
  const bool push = peer && batch <= std::min(push_rows, 8) && !EnvFlag("B200_TP_PULL") && TpPushLink(d->tp, &link);
  // Up to 8 rows the RMSNorm in front of a projection is fused into its input
  // staging (h is never written); beyond that it is its own kernel.
  const bool fuse_norm = batch <= 8 && (!tp || push);
  __nv_bfloat16* xb[2] = {d->x, d->x2};
  int xp = 0;   // which of the two holds the current residual rows (push exchange)
  QmmTp from_peers = link, to_peers = link;   // the projection that reads the summed rows / the one that pushes and sums
  to_peers.push = true;
  B200_TRY(b200_embed(ctx, stream, d->embed, tokens, d->x, batch, E,
                      static_cast<int64_t>(c.vocab) * (d->tp != nullptr ? d->tp->world : 1)));
  if (!fuse_norm)
    B200_TRY(b200_rownorm(ctx, stream, 0, d->x, d->layers[0].attn_norm, nullptr, d->h, batch, E, B200_BF16, c.rms_eps));
  for (int li = 0; li < c.layers; ++li) {
    const b200_decoder_layer& L = d->layers[li];
    if (push) {
      if (li == 0) {
        B200_TRY(Qmm(d, stream, L.qkv, xb[xp], d->qkv, batch, QKV, E, B200_QMM_OUT_BF16, nullptr, B200_QMM_PRO_RMSNORM,
                     L.attn_norm));
      } else {   // the down projection of the layer before pushed its partial sums and published the new residual rows
        B200_TRY(Qmm(d, stream, L.qkv, xb[xp], d->qkv, batch, QKV, E, B200_QMM_OUT_BF16, nullptr, B200_QMM_PRO_RMSNORM,
                     L.attn_norm, &from_peers));
      }
      B200_TRY(b200_attention_step(ctx, stream, d->qkv, L.q_norm, L.k_norm, d->inv_freq, L.k_cache, L.v_cache, d->attn,
                                   pos, d->attn_scratch, batch, c.heads, c.kv_heads, c.head_dim, c.max_len,
                                   c.rope_theta, c.rms_eps));
      to_peers.x_old = xb[xp];
      to_peers.x_out = xb[xp ^ 1];
      B200_TRY(Qmm(d, stream, L.o, d->attn, link.dst[link.rank], batch, E, HD, B200_QMM_OUT_F32_RAW, nullptr,
                   B200_QMM_PRO_NONE, nullptr, &to_peers));
      xp ^= 1;
      const bool pair = !d->gate_up_pair.empty();
      B200_TRY(Qmm(d, stream, pair ? d->gate_up_pair[li] : L.gate_up, xb[xp], d->gu, batch, 2 * static_cast<int64_t>(c.inter), E,
                   pair ? B200_QMM_OUT_SILU_PAIR : B200_QMM_OUT_BF16, nullptr, B200_QMM_PRO_RMSNORM, L.mlp_norm, &from_peers));
      to_peers.x_old = xb[xp];
      to_peers.x_out = xb[xp ^ 1];
      B200_TRY(Qmm(d, stream, L.down, d->gu, link.dst[link.rank], batch, E, c.inter, B200_QMM_OUT_F32_RAW, nullptr,
                   pair ? B200_QMM_PRO_NONE : B200_QMM_PRO_SILU_MUL, nullptr, &to_peers));
      xp ^= 1;
      continue;
    }
    if (fuse_norm)
      B200_TRY(Qmm(d, stream, L.qkv, d->x, d->qkv, batch, QKV, E, B200_QMM_OUT_BF16, nullptr, B200_QMM_PRO_RMSNORM,
                   L.attn_norm));
    else
      B200_TRY(Qmm(d, stream, L.qkv, d->h, d->qkv, batch, QKV, E, B200_QMM_OUT_BF16, nullptr));
    B200_TRY(b200_attention_step(ctx, stream, d->qkv, L.q_norm, L.k_norm, d->inv_freq, L.k_cache, L.v_cache, d->attn,
                                 pos, d->attn_scratch, batch, c.heads, c.kv_heads, c.head_dim, c.max_len,
                                 c.rope_theta, c.rms_eps));
    if (tp && peer) {
      // slot 0: the sum over ranks, the residual add and the next RMSNorm are one kernel over peer memory
      B200_TRY(Qmm(d, stream, L.o, d->attn, TpPeerPartial(d->tp, 0), batch, E, HD, B200_QMM_OUT_F32_RAW, nullptr));
      B200_TRY(TpSumResidualNorm(d->tp, stream, 0, d->x, L.mlp_norm, d->h, batch, E, c.rms_eps));
    } else if (tp) {
      B200_TRY(Qmm(d, stream, L.o, d->attn, d->y32, batch, E, HD, B200_QMM_OUT_F32_RAW, nullptr));
      B200_TRY(TpAllReduce(d->tp, stream, d->y32, static_cast<int64_t>(batch) * E, B200_F32));
      B200_TRY(ResidualNorm(d, stream, L.mlp_norm, batch));
    } else {
      B200_TRY(Qmm(d, stream, L.o, d->attn, d->x, batch, E, HD, B200_QMM_ADD_RESIDUAL, d->x));
      if (!fuse_norm)
        B200_TRY(b200_rownorm(ctx, stream, 0, d->x, L.mlp_norm, nullptr, d->h, batch, E, B200_BF16, c.rms_eps));
    }
    const bool pair = fuse_norm && !tp && !d->gate_up_pair.empty();   // (the push flow above has its own use of it)
    if (pair)
      B200_TRY(Qmm(d, stream, d->gate_up_pair[li], d->x, d->gu, batch, 2 * static_cast<int64_t>(c.inter), E,
                   B200_QMM_OUT_SILU_PAIR, nullptr, B200_QMM_PRO_RMSNORM, L.mlp_norm));
    else if (fuse_norm)
      B200_TRY(Qmm(d, stream, L.gate_up, d->x, d->gu, batch, 2 * static_cast<int64_t>(c.inter), E, B200_QMM_OUT_BF16,
                   nullptr, B200_QMM_PRO_RMSNORM, L.mlp_norm));
    else
      B200_TRY(Qmm(d, stream, L.gate_up, d->h, d->gu, batch, 2 * static_cast<int64_t>(c.inter), E, B200_QMM_OUT_BF16,
                   nullptr));
    const void* next_norm = li + 1 < c.layers ? d->layers[li + 1].attn_norm : d->final_norm;
    // silu(gate) * up is fused into the staging of the down projection's input
    if (tp && peer) {
      B200_TRY(Qmm(d, stream, L.down, d->gu, TpPeerPartial(d->tp, 1), batch, E, c.inter, B200_QMM_OUT_F32_RAW, nullptr,
                   B200_QMM_PRO_SILU_MUL));
      B200_TRY(TpSumResidualNorm(d->tp, stream, 1, d->x, next_norm, d->h, batch, E, c.rms_eps));
    } else if (tp) {
      B200_TRY(Qmm(d, stream, L.down, d->gu, d->y32, batch, E, c.inter, B200_QMM_OUT_F32_RAW, nullptr,
                   B200_QMM_PRO_SILU_MUL));
      B200_TRY(TpAllReduce(d->tp, stream, d->y32, static_cast<int64_t>(batch) * E, B200_F32));
      B200_TRY(ResidualNorm(d, stream, next_norm, batch));
    } else {
      B200_TRY(Qmm(d, stream, L.down, d->gu, d->x, batch, E, c.inter, B200_QMM_ADD_RESIDUAL, d->x,
                   pair ? B200_QMM_PRO_NONE : B200_QMM_PRO_SILU_MUL));
      if (!fuse_norm)
        B200_TRY(b200_rownorm(ctx, stream, 0, d->x, next_norm, nullptr, d->h, batch, E, B200_BF16, c.rms_eps));
    }
  }
  // LM head: bf16 rows, logits are the bf16-rounded products widened to f32 (qwen3.py:389-390)
  float* head_out = tp ? d->logits_local : logits;
  const int64_t head_count = static_cast<int64_t>(batch) * c.vocab;
  if (batch > 8 && d->logits_bf16 != nullptr && head_count % 8 == 0 && Aligned(head_out, 16)) {
    // above 8 rows x no longer fits beside a streaming CTA's ring without splitting K; the
    // tensor-core GEMM (x . W^T, bf16 out) plus a widening pass is several times faster
    b200_gemm_params g = {};
    g.m = batch;
    g.n = c.vocab;
    g.k = E;
    g.batch = 1;
    g.alpha = 1.0;
    g.a.ptr = d->h;
    g.a.ld = E;
    g.a.dtype = B200_BF16;
    g.b.ptr = const_cast<void*>(d->lm_head);
    g.b.ld = E;
    g.b.dtype = B200_BF16;
    g.b.transpose = 1;
    g.c.ptr = d->logits_bf16;
    g.c.ld = c.vocab;
    g.c.dtype = B200_BF16;
    b200_epilogue epi = {};
    B200_TRY(b200_gemm(ctx, stream, &g, &epi));
    B200_TRY(BeginLaunch(ctx));
    LaunchCfg lc;
    lc.stream = stream;
    lc.pdl = true;
    lc.block = dim3(256);
    lc.grid = dim3(static_cast<unsigned>(CeilDiv(head_count / 8, 256)));
    cudaError_t e = Launch(lc, widen_bf16_kernel, static_cast<const __nv_bfloat16*>(d->logits_bf16), head_out, head_count);
    if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "widen launch: %s", cudaGetErrorString(e)));
    B200_TRY(EndLaunch(ctx, "widen"));
  } else {
    b200_qmm_params p = {};
    p.bits = 16;
    p.epilogue = B200_QMM_OUT_F32;
    p.x = push ? xb[xp] : (fuse_norm ? d->x : d->h);
    if (fuse_norm) {
      p.prologue = B200_QMM_PRO_RMSNORM;
      p.prologue_gain = d->final_norm;
      p.eps = c.rms_eps;
    }
    p.q = d->lm_head;
    p.out = head_out;
    p.M = batch;
    p.N = c.vocab;
    p.K = E;
    B200_TRY(QmmRunEx(ctx, stream, &p, CallerOf(d, push ? &from_peers : nullptr)));
  }
  if (tp) B200_TRY(TpAllGather(d->tp, stream, d->logits_local, logits, static_cast<int64_t>(batch) * c.vocab, B200_F32));
  return B200_OK;
}

template <typename T>
cudaError_t Alloc(T** p, size_t count) { return cudaMalloc(reinterpret_cast<void**>(p), count * sizeof(T)); }

}  // namespace

extern "C" {

b200_status b200_decoder_create(b200_context* ctx, const b200_decoder_config* cfg, const b200_decoder_layer* layers,
                                const void* embed, const void* final_norm, const void* lm_head, b200_tp* tp,
                                b200_decoder** out) {
  if (out == nullptr) return Fail(B200_INVALID_ARGUMENT, "b200_decoder_create: null out");
  *out = nullptr;
  b200_status s = BeginLaunch(ctx);
  if (s != B200_OK) return s;
  if (cfg == nullptr || layers == nullptr || embed == nullptr || final_norm == nullptr || lm_head == nullptr)
    return Fail(B200_INVALID_ARGUMENT, "b200_decoder_create: null argument");
  const b200_decoder_config& c = *cfg;
  if (c.layers <= 0 || c.hidden <= 0 || c.heads <= 0 || c.kv_heads <= 0 || c.inter <= 0 || c.vocab <= 0 ||
      c.max_len <= 0 || c.max_batch <= 0)
    return Fail(B200_INVALID_ARGUMENT, "b200_decoder_create: non-positive size");
  if (c.max_batch > 32) return Fail(B200_UNIMPLEMENTED, "b200_decoder_create: max_batch %d (the decode path takes up to 32)", c.max_batch);
  if (c.head_dim != 64 && c.head_dim != 128) return Fail(B200_UNIMPLEMENTED, "b200_decoder_create: head_dim %d", c.head_dim);
  if (c.heads % c.kv_heads != 0) return Fail(B200_INVALID_ARGUMENT, "b200_decoder_create: heads not a multiple of kv_heads");
  if (c.hidden % 64 != 0 || c.inter % 64 != 0 || (c.heads * c.head_dim) % 64 != 0)
    return Fail(B200_UNIMPLEMENTED, "b200_decoder_create: hidden, inter and heads*head_dim must be multiples of 64");
  b200_decoder* d = new b200_decoder();
  d->ctx = ctx;
  d->cfg = c;
  d->layers.assign(layers, layers + c.layers);
  d->embed = embed;
  d->final_norm = final_norm;
  d->lm_head = lm_head;
  d->tp = tp;
  d->use_graph = !EnvFlag("B200_DECODER_NO_GRAPH");
  const size_t B = c.max_batch;
  const size_t qkv = static_cast<size_t>(c.heads + 2 * c.kv_heads) * c.head_dim;
  cudaError_t e = Alloc(&d->x, B * c.hidden);
  if (e == cudaSuccess) e = Alloc(&d->x2, B * c.hidden);
  if (e == cudaSuccess) e = Alloc(&d->h, B * c.hidden);
  if (e == cudaSuccess) e = Alloc(&d->qkv, B * qkv);
  if (e == cudaSuccess) e = Alloc(&d->attn, B * c.heads * c.head_dim);
  if (e == cudaSuccess) e = Alloc(&d->gu, B * 2 * c.inter);
  if (e == cudaSuccess) e = Alloc(&d->y32, B * c.hidden);
  if (e == cudaSuccess)
    e = cudaMalloc(reinterpret_cast<void**>(&d->attn_scratch),
                   b200_attention_scratch_bytes(c.max_batch, c.heads, c.head_dim, c.max_len));
  if (e == cudaSuccess && tp != nullptr) e = Alloc(&d->logits_local, B * c.vocab);
  if (e == cudaSuccess && c.max_batch > 8) e = Alloc(&d->logits_bf16, B * c.vocab);
  if (c.max_batch > 8) {
    const int64_t shapes[4][2] = {{static_cast<int64_t>(qkv), c.hidden}, {c.hidden, static_cast<int64_t>(c.heads) * c.head_dim},
                                  {2 * static_cast<int64_t>(c.inter), c.hidden}, {c.hidden, c.inter}};
    for (int m : {9, c.max_batch})   // (a plan depends on the rows only through up to 16 or more)
      for (const auto& nk : shapes) d->slices_floats = std::max(d->slices_floats, QmmMidScratchFloats(ctx, 4, 64, m, nk[0], nk[1]));
    d->slices_floats = std::max<size_t>(d->slices_floats, 1);
    if (e == cudaSuccess) e = Alloc(&d->slices, d->slices_floats);
  }
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&d->capture_stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = Alloc(&d->inv_freq, static_cast<size_t>(c.head_dim / 2));
  if (e == cudaSuccess) e = Alloc(&d->tokens_buf, B);
  if (e == cudaSuccess) e = Alloc(&d->pos_buf, 1);
  if (e == cudaSuccess) {
    std::vector<float> f(c.head_dim / 2);
    for (int i = 0; i < c.head_dim / 2; ++i)
      f[i] = static_cast<float>(1.0 / pow(static_cast<double>(c.rope_theta), static_cast<double>(2 * i) / c.head_dim));
    e = cudaMemcpy(d->inv_freq, f.data(), f.size() * sizeof(float), cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) {
    s = Fail(B200_RESOURCE_EXHAUSTED, "b200_decoder_create: %s", cudaGetErrorString(e));
    b200_decoder_destroy(d);
    return s;
  }
  // gate_up in the order its silu(gate) * up epilogue takes (up to 8 rows per step; plans without a K split)
  if (!EnvFlag("B200_DECODER_NO_SILU_PAIR") && c.inter % 8 == 0 && c.hidden % 64 == 0) {
    bool ok = true;
    for (int m = 1; m <= std::min(c.max_batch, 8) && ok; ++m) {
      b200_qmm_params pp = {};
      pp.bits = 4;
      pp.group = 64;
      pp.epilogue = B200_QMM_OUT_BF16;
      pp.prologue = B200_QMM_PRO_RMSNORM;
      pp.M = m;
      pp.N = 2 * static_cast<int64_t>(c.inter);
      pp.K = c.hidden;
      pp.x = pp.q = pp.scale = pp.bias = pp.prologue_gain = d->x;   // (placeholders: the plan looks at alignment only)
      pp.out = d->x;
      int rows = 0, split = 0, blocks = 0;
      ok = b200_qmm_plan(&pp, &rows, &split, &blocks) == B200_OK && split == 1 && blocks == 1;
    }
    const int64_t rows = 2 * static_cast<int64_t>(c.inter), qb = c.hidden / 2, sb = c.hidden / 64 * 2;
    for (int li = 0; ok && li < c.layers; ++li) {
      void *q = nullptr, *sc = nullptr, *bi = nullptr;
      cudaError_t ce = cudaMalloc(&q, rows * qb);
      if (ce == cudaSuccess) d->pair_storage.push_back(q);
      if (ce == cudaSuccess) ce = cudaMalloc(&sc, rows * sb);
      if (ce == cudaSuccess) d->pair_storage.push_back(sc);
      if (ce == cudaSuccess) ce = cudaMalloc(&bi, rows * sb);
      if (ce == cudaSuccess) d->pair_storage.push_back(bi);
      if (ce != cudaSuccess) {
        (void)cudaGetLastError();
        b200_decoder_destroy(d);
        return Fail(B200_RESOURCE_EXHAUSTED, "b200_decoder_create: copy of gate_up for layer %d: %s", li, cudaGetErrorString(ce));
      }
      const b200_qweight& w = d->layers[li].gate_up;
      s = b200_interleave_gate_up(ctx, nullptr, w.q, q, c.inter, qb);
      if (s == B200_OK) s = b200_interleave_gate_up(ctx, nullptr, w.scale, sc, c.inter, sb);
      if (s == B200_OK) s = b200_interleave_gate_up(ctx, nullptr, w.bias, bi, c.inter, sb);
      if (s != B200_OK) {
        b200_decoder_destroy(d);
        return s;
      }
      b200_qweight pw = {q, sc, bi};
      d->gate_up_pair.push_back(pw);
    }
    if (ok && cudaStreamSynchronize(nullptr) != cudaSuccess) {
      b200_decoder_destroy(d);
      return Stick(ctx, Fail(B200_INTERNAL, "b200_decoder_create: rearranging gate_up failed"));
    }
  }
  // B200_DECODER_STREAM=1 selects the single persistent kernel where it applies.  It is not the
  // default: measured on the Qwen3-8B shape it takes 2.5 ms per step at batch 1 against 2.2 ms
  // for the captured kernel-per-operator graph (its grid barriers and input staging cost what
  // the launches they replace cost, and its attention stage is slower), and it falls further
  // behind with more rows.
  if (EnvFlag("B200_DECODER_STREAM")) {
    s = DecodeStreamCreate(ctx, c, d->layers, embed, final_norm, lm_head,
                           static_cast<int64_t>(c.vocab) * (tp != nullptr ? tp->world : 1), tp, &d->stream_path);
    if (s != B200_OK) {
      b200_decoder_destroy(d);
      return s;
    }
  }
  *out = d;
  return B200_OK;
}

void b200_decoder_destroy(b200_decoder* d) {
  if (d == nullptr) return;
  cudaSetDevice(d->ctx->device);
  DecodeStreamDestroy(d->stream_path);
  for (auto& kv : d->graphs) cudaGraphExecDestroy(kv.second);
  if (d->capture_stream != nullptr) cudaStreamDestroy(d->capture_stream);
  for (void* p : {static_cast<void*>(d->x), static_cast<void*>(d->h), static_cast<void*>(d->qkv),
                  static_cast<void*>(d->attn), static_cast<void*>(d->gu),
                  static_cast<void*>(d->y32), static_cast<void*>(d->attn_scratch),
                  static_cast<void*>(d->logits_local), static_cast<void*>(d->inv_freq),
                  static_cast<void*>(d->logits_bf16), static_cast<void*>(d->x2), static_cast<void*>(d->tokens_buf),
                  static_cast<void*>(d->pos_buf), static_cast<void*>(d->slices)})
    if (p != nullptr) cudaFree(p);
  for (void* p : d->pair_storage) cudaFree(p);
  delete d;
}

b200_status b200_decoder_step(b200_decoder* d, b200_stream stream, const int32_t* tokens, const int32_t* pos,
                              float* logits, int batch) {
  if (d == nullptr) return Fail(B200_INVALID_ARGUMENT, "b200_decoder_step: null decoder");
  b200_status s = BeginLaunch(d->ctx);
  if (s != B200_OK) return s;
  if (batch < 0 || batch > d->cfg.max_batch)
    return Fail(B200_INVALID_ARGUMENT, "b200_decoder_step: batch %d outside [0, %d]", batch, d->cfg.max_batch);
  if (batch == 0) return B200_OK;
  if (tokens == nullptr || pos == nullptr || logits == nullptr)
    return Fail(B200_INVALID_ARGUMENT, "b200_decoder_step: null buffer");
  std::lock_guard<std::mutex> lock(d->mu);
  if (DecodeStreamSupports(d->stream_path, batch)) {
    d->launches[batch] = 1;
    return DecodeStreamStep(d->stream_path, stream, tokens, pos, logits, nullptr, batch);
  }
  if (!d->use_graph) {
    const int64_t before = d->ctx->launches.load();
    s = Enqueue(d, stream, tokens, pos, logits, batch);
    d->launches[batch] = d->ctx->launches.load() - before;
    return s;
  }
  // The graph reads tokens and the position from the decoder's own buffers, so a caller may
  // pass fresh tensors every step without a new capture.
  cudaError_t e = cudaMemcpyAsync(d->tokens_buf, tokens, static_cast<size_t>(batch) * sizeof(int32_t),
                                  cudaMemcpyDeviceToDevice, stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d->pos_buf, pos, sizeof(int32_t), cudaMemcpyDeviceToDevice, stream);
  if (e != cudaSuccess) return Stick(d->ctx, Fail(B200_INTERNAL, "staging tokens: %s", cudaGetErrorString(e)));
  const auto key = std::make_pair(batch, static_cast<const void*>(logits));
  auto it = d->graphs.begin();
  while (it != d->graphs.end() && it->first != key) ++it;
  if (it == d->graphs.end()) {
    cudaStream_t cs = d->capture_stream;
    e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return Stick(d->ctx, Fail(B200_INTERNAL, "cudaStreamBeginCapture: %s", cudaGetErrorString(e)));
    const int64_t before = d->ctx->launches.load();
    s = Enqueue(d, cs, d->tokens_buf, d->pos_buf, logits, batch);
    const int64_t count = d->ctx->launches.load() - before;
    cudaGraph_t graph = nullptr;
    e = cudaStreamEndCapture(cs, &graph);
    if (s != B200_OK) {
      if (graph != nullptr) cudaGraphDestroy(graph);
      return s;
    }
    if (e != cudaSuccess) return Stick(d->ctx, Fail(B200_INTERNAL, "cudaStreamEndCapture: %s", cudaGetErrorString(e)));
    cudaGraphExec_t exec = nullptr;
    e = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return Stick(d->ctx, Fail(B200_INTERNAL, "cudaGraphInstantiate: %s", cudaGetErrorString(e)));
    d->ctx->launches.fetch_sub(count);  // capture enqueued nothing; replays are counted below
    d->launches[batch] = count;
    ++d->graphs_built;
    if (d->graphs.size() >= b200_decoder::kMaxGraphs) {
      // The oldest graph may still be running on the caller's stream: wait before destroying it.
      // This only happens to callers that rotate through more than kMaxGraphs output buffers.
      cudaStreamSynchronize(stream);
      cudaGraphExecDestroy(d->graphs.back().second);
      d->graphs.pop_back();
    }
    d->graphs.emplace_front(key, exec);
    it = d->graphs.begin();
  } else if (it != d->graphs.begin()) {
    d->graphs.splice(d->graphs.begin(), d->graphs, it);   // most recently used first
    it = d->graphs.begin();
  }
  e = cudaGraphLaunch(it->second, stream);
  if (e != cudaSuccess) return Stick(d->ctx, Fail(B200_INTERNAL, "cudaGraphLaunch: %s", cudaGetErrorString(e)));
  d->ctx->launches.fetch_add(d->launches[batch]);
  return B200_OK;
}

b200_status b200_decoder_trace(b200_decoder* d, int enable) {
  if (d == nullptr) return Fail(B200_INVALID_ARGUMENT, "b200_decoder_trace: null decoder");
  std::lock_guard<std::mutex> lock(d->mu);
  return DecodeStreamTrace(d->stream_path, enable != 0);
}

b200_status b200_decoder_trace_read(b200_decoder* d, uint64_t* out, int64_t capacity, int32_t* ctas, int32_t* stages,
                                    int32_t* stage_types) {
  if (d == nullptr) return Fail(B200_INVALID_ARGUMENT, "b200_decoder_trace_read: null decoder");
  std::lock_guard<std::mutex> lock(d->mu);
  return DecodeStreamTraceRead(d->stream_path, reinterpret_cast<unsigned long long*>(out), capacity, ctas, stages, stage_types);
}

int64_t b200_decoder_graphs_built(b200_decoder* d) {
  if (d == nullptr) return 0;
  std::lock_guard<std::mutex> lock(d->mu);
  return d->graphs_built;
}

int64_t b200_decoder_launches_per_step(b200_decoder* d, int batch) {
  if (d == nullptr) return 0;
  auto it = d->launches.find(batch);
  return it == d->launches.end() ? 0 : it->second;
}

}  // extern "C"
