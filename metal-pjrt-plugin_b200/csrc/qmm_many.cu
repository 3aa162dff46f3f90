// Weight-only quantised matmul for MORE than 32 rows of x (prefill-sized batches; ≙ the reference beyond ROWS_MAX:
// dequantize(w, dtype), then x @ w.T, examples/llm/qwen3.py:199-230).  Two ways:
//   * the tensor-core GEMM takes the weights as they are and widens them to bf16 on their way into its ring
//     (gemm_tcgen05.cu): no bf16 copy exists, but every row of 128 x tiles widens them again;
//   * the weights are dequantised panel by panel into bf16 scratch and each panel goes through the general GEMM
//     (PanelsAreFaster says when, and rows of x that TMA cannot read).  A panel is at most 96 MB (or 256 rows), so that it stays in
//     the 126 MB L2: 32 MB panels gave GEMMs of less than a wave of tiles (int4 512 x 12288 -> 4096: 147 us, now 88).  The scratch
//     is stream-ordered memory of the context's pool: calls on several streams each have their own, and a graph owns its.
#include <algorithm>

#include "common.cuh"
#include "qmm_many.cuh"

using namespace b200;

namespace {

constexpr int64_t kPanelBytes = 96ll << 20;

// Sequential int4 in groups of 64: one thread per 8 inputs (one word), 16-byte stores.
__global__ void dequant_int4_seq_kernel(const uint32_t* q, const __nv_bfloat16* scale, const __nv_bfloat16* bias, uint4* out,
                                        int64_t words, int words_per_row) {
  pdl_wait();   // the GEMM of the panel before still reads the workspace
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < words;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t n = i / words_per_row;
    const int w = static_cast<int>(i % words_per_row);
    const uint32_t v = __ldg(q + i);
    const int64_t g = n * (words_per_row / 8) + w / 8;
    const float s = __bfloat162float(scale[g]), b = __bfloat162float(bias[g]);
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      // w = q*s + b in f32 with one rounding per operation, then one rounding to bf16 (b200_dequantize's values)
      const float lo = __fadd_rn(__fmul_rn(static_cast<float>((v >> (8 * j)) & 15u), s), b);
      const float hi = __fadd_rn(__fmul_rn(static_cast<float>((v >> (8 * j + 4)) & 15u), s), b);
      o[j] = pack_bf16(lo, hi);
    }
    out[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// The product by panels of `panel` weight rows (the residual rows are in `out` already).
b200_status RunPanels(b200_context* ctx, cudaStream_t stream, const b200_qmm_params* p, int64_t panel, void* ws) {
  const int64_t M = p->M, N = p->N, K = p->K;
  const int64_t ldx = p->ldx ? p->ldx : K, ldo = p->ldo ? p->ldo : N;
  const bool f32_out = p->epilogue == B200_QMM_OUT_F32_RAW;
  const size_t esz = f32_out ? 4 : 2;
  const int64_t row_bytes = p->bits == 4 ? K / 2 : (p->bits == 8 ? K : 2 * K);
  const int64_t spr = p->bits == 16 ? 0 : K / p->group;
  for (int64_t r0 = 0; r0 < N; r0 += panel) {
    const int64_t rows = std::min(panel, N - r0);
    const uint8_t* qp = static_cast<const uint8_t*>(p->q) + r0 * row_bytes;
    const void* wmat = qp;
    if (p->bits != 16) {
      const __nv_bfloat16* sp = static_cast<const __nv_bfloat16*>(p->scale) + r0 * spr;
      const __nv_bfloat16* bp = p->bits == 4 ? static_cast<const __nv_bfloat16*>(p->bias) + r0 * spr : nullptr;
      if (p->bits == 4 && p->nibble_order == 0 && Aligned(ws, 16)) {
        b200_status s = BeginLaunch(ctx);
        if (s != B200_OK) return s;
        const int64_t words = rows * (K / 8);
        LaunchCfg lc;
        lc.grid = dim3(static_cast<unsigned>(std::min<int64_t>(CeilDiv(words, 256), ctx->sm_count * 16)));
        lc.block = dim3(256);
        lc.stream = stream;
        lc.pdl = true;
        cudaError_t e = Launch(lc, dequant_int4_seq_kernel, reinterpret_cast<const uint32_t*>(qp), sp, bp,
                               static_cast<uint4*>(ws), words, static_cast<int>(K / 8));
        if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_qmm: dequantise launch: %s", cudaGetErrorString(e)));
        s = EndLaunch(ctx, "b200_qmm (dequantise)");
        if (s != B200_OK) return s;
      } else {
        b200_status s = b200_dequantize(ctx, stream, p->bits, p->group, p->nibble_order, qp, sp, bp, ws, rows, K, B200_BF16);
        if (s != B200_OK) return s;
      }
      wmat = ws;
    }
    // out[:, r0 : r0 + rows] = x . W_panel^T
    b200_gemm_params g = {};
    g.m = M;
    g.n = rows;
    g.k = K;
    g.batch = 1;
    g.alpha = 1.0;
    g.beta = p->epilogue == B200_QMM_ADD_RESIDUAL ? 1.0 : 0.0;
    g.a.ptr = const_cast<void*>(p->x);
    g.a.ld = ldx;
    g.a.dtype = B200_BF16;
    g.b.ptr = const_cast<void*>(wmat);
    g.b.ld = K;
    g.b.dtype = B200_BF16;
    g.b.transpose = 1;
    g.c.ptr = static_cast<uint8_t*>(p->out) + static_cast<size_t>(r0) * esz;
    g.c.ld = ldo;
    g.c.dtype = f32_out ? B200_F32 : B200_BF16;
    b200_epilogue epi = {};
    b200_status s = b200_gemm(ctx, stream, &g, &epi);
    if (s != B200_OK) return s;
  }
  return B200_OK;
}

}  // namespace

namespace b200 {

// gemm_tcgen05.cu
bool QuantisedGemmSupports(const b200_qmm_params* p);
bool PanelsAreFaster(const b200_context* ctx, const b200_qmm_params* p, int64_t panel);
b200_status RunQuantisedGemm(b200_context* ctx, cudaStream_t stream, const b200_qmm_params* p);

b200_status QmmManyRows(b200_context* ctx, cudaStream_t stream, const b200_qmm_params* p) {
  if (p->prologue != B200_QMM_PRO_NONE)
    return Fail(B200_UNIMPLEMENTED, "b200_qmm: the fused input transforms take up to 32 rows (8 for RMSNorm); M = %lld",
                static_cast<long long>(p->M));
  if (p->epilogue == B200_QMM_OUT_F32)
    return Fail(B200_UNIMPLEMENTED, "b200_qmm: above 32 rows the output is bf16, bf16 + residual, or raw f32");
  const int64_t M = p->M, N = p->N, K = p->K;
  const int64_t ldo = p->ldo ? p->ldo : N;
  // bf16 weights need no scratch: one GEMM over the whole matrix
  int64_t panel = N;
  if (p->bits != 16) {
    // panels of equal height: a short last one is less than a wave of tiles
    const int64_t most = std::max<int64_t>(256, kPanelBytes / (2 * K) / 256 * 256);
    panel = std::min(CeilDiv(CeilDiv(N, CeilDiv(N, most)), 256) * 256, N);
  }
  const bool direct_ok = QuantisedGemmSupports(p);
  bool direct = direct_ok && !PanelsAreFaster(ctx, p, panel);
  void* ws = nullptr;
  if (p->bits != 16 && !direct) {
    const size_t need = static_cast<size_t>(panel) * K * 2;
    const cudaError_t e = cudaMallocFromPoolAsync(&ws, need, ctx->pool, stream);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      ws = nullptr;
      if (!direct_ok)
        return Fail(B200_RESOURCE_EXHAUSTED, "b200_qmm: %zu bytes of scratch for dequantised weights: %s", need, cudaGetErrorString(e));
      direct = true;
    }
  }
  b200_status s = B200_OK;
  if (p->epilogue == B200_QMM_ADD_RESIDUAL && p->residual != p->out) {
    const cudaError_t e = cudaMemcpy2DAsync(p->out, ldo * 2, p->residual, ldo * 2, N * 2, M, cudaMemcpyDeviceToDevice, stream);
    if (e != cudaSuccess) s = Stick(ctx, Fail(B200_INTERNAL, "b200_qmm: residual copy: %s", cudaGetErrorString(e)));
  }
  if (s == B200_OK) s = direct ? RunQuantisedGemm(ctx, stream, p) : RunPanels(ctx, stream, p, panel, ws);
  if (ws != nullptr) cudaFreeAsync(ws, stream);
  return s;
}

}  // namespace b200
