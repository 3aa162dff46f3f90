// Dense GEMM with the fused epilogue: validation, routing and the SIMT tile
// kernel.  Semantics kept from the reference: GemmParams / SteelEpilogue
// (metal_pjrt/blas/mps_gemm.h:23-53, steel_gemm.h:38-46), the acceptance rules
// of SteelGemmSupports / RunSteelGemm (steel_gemm.cc:140-196), and the
// per-element epilogue of kernels/steel_gemm.metal:217-225:
//     v = alpha*acc (+ beta*D) (+ bias[col]);  aux = T(v);  D = T(act(v)).
// Routing replaces ChooseGemv / ChooseSteelTile (gemv.cc:68-108,
// steel_gemm.cc:115-138) with three B200 kernels:
//   tcgen05  - TMA-fed tensor-core tiles with TMEM accumulators (gemm_tcgen05.cu),
//              for 16-bit operands whose layout the TMA descriptors accept;
//   few-row  - the bandwidth-bound streaming kernel (qmm.cu, 16-bit weights), for
//              x . W^T with up to 32 rows on either side; preferred up to 8 rows, above
//              that the tensor-core route (which splits K across a cluster) is faster;
//              (operands whose rows are not 16-byte aligned are copied into aligned rows first,
//              where the product is large enough to pay for the copy);
//   SIMT     - the general tile kernel below: every dtype, transpose, stride,
//              batch and beta; true f32 arithmetic for f32 operands (tensor
//              cores have no f32 multiply, and the f32 block must hold rtol 1e-5).
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"

namespace cg = cooperative_groups;
using namespace b200;

namespace b200 {
b200_status RunFewRowNT(b200_context* ctx, cudaStream_t stream, const void* mat, const void* vecs, void* out,
                        int64_t R, int64_t V, int64_t K, int64_t ld_vec, int64_t out_row_stride,
                        int64_t out_vec_stride, float alpha, int act, const void* bias, int bias_by_vec,
                        void* aux, int out_f32);
// gemm_tcgen05.cu
bool Tcgen05Supports(const b200_gemm_params* p, const b200_epilogue* epi);
bool TmaReadable(const b200_operand& x, int64_t batch);
b200_status RunTcgen05(b200_context* ctx, cudaStream_t stream, const b200_gemm_params* p, const b200_epilogue* epi);
}  // namespace b200

namespace {

constexpr size_t kSmemPerSm = 228 * 1024;   // 1 KB of it is taken by each CTA beside what it asks for
constexpr int64_t kMaxInt = INT32_MAX;
constexpr int64_t kMaxLd = INT32_MAX / 256;  // steel_gemm.cc:153

struct SimtArgs {
  const void* a;
  const void* b;
  void* d;
  const void* bias;
  void* aux;
  int m, n, k;
  int64_t lda, ldb, ldd;
  int64_t sa, sb, sd;  // batch strides
  int ta, tb;
  float alpha, beta;
  int act;
  int split;           // CTAs of a cluster along K
};

__device__ __forceinline__ void add_pair(float2& d, const float2& a) {
  asm("{\n\t.reg .b64 x, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 z, {%0, %1};\n\tadd.rn.f32x2 z, z, x;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "+f"(d.x), "+f"(d.y)
      : "f"(a.x), "f"(a.y));
}
// d += {a, a} * {b0, b1}: two IEEE multiply-adds per lane in one instruction, so that the FMA pipes are kept busy
// with half of the issue slots and the rest go to loads.
__device__ __forceinline__ void fma_pair(float2& d, float a, const float2& b) {
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b64 z, {%0, %1};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "+f"(d.x), "+f"(d.y)
      : "f"(a), "f"(b.x), "f"(b.y));
}

// One shape of the tile kernel: a BM x BN tile by KG groups of threads, TM x TN values a thread; a group takes its own
// part of every BK-deep step.
template <int BM_, int BN_, int TM_, int TN_, int KG_, int BK_, int RESIDENT_>
struct Tile {
  static constexpr int kResident = RESIDENT_;   // CTAs per SM that registers are kept for
  static constexpr bool kDirect = KG_ == 1 && BM_ == 64;   // results go from registers to memory; no split of K
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, KG = KG_, BK = BK_;
  static constexpr int kGroup = (BM / TM) * (BN / TN);
  static constexpr int kThreads = kGroup * KG;
  static constexpr int kPitchA = BM + 4, kPitchB = BN + 4;   // floats; keeps 16-byte reads aligned
  static constexpr int kBuffer = BK * (kPitchA + kPitchB);   // floats of one of the two steps held
  static constexpr size_t kSmem = sizeof(float) * (kDirect || 2 * kBuffer > KG * BM * BN ? 2 * kBuffer : KG * BM * BN);
  static constexpr int kLoadsA = BM * BK / kThreads, kLoadsB = BN * BK / kThreads;
  static_assert(BM * BK % kThreads == 0 && BN * BK % kThreads == 0 && kThreads % BK == 0 && kThreads % BM == 0 && kThreads % BN == 0, "");
};
// Large products: 8 x 8 values a thread (a step of k costs 4 shared loads of 16 bytes for 32 paired multiply-adds).
using Large = Tile<128, 128, 8, 8, 1, 16, 2>;
// Products whose 128 x 128 tiles leave SMs idle: two groups of four warps on a 64 x 64 tile.
using Medium = Tile<64, 64, 4, 8, 2, 32, 1>;
// Few rows: eight groups of two warps, each with its own part of k.
using Few = Tile<16, 64, 4, 4, 8, 64, 1>;
// Many tiles of a short K: what a tile costs beside its multiply-adds (the first loads, the last step, the stores) is hidden by
// other CTAs of the same SM, not by more work per thread.  Sums of 32 values are added up, as finely as the medium tile's two groups
// have it.
using Short = Tile<64, 64, 4, 4, 1, 16, 4>;

// One thread's share of a step of an operand: `kLoads` values, along the operand's contiguous dimension first.
// OUTER: rows of op(A) or columns of op(B); BYK: k is the contiguous dimension.
template <typename TIn, int OUTER, int BK, int THREADS, int LOADS>
struct Loader {
  const TIn* p;
  int64_t step, next;   // elements between a thread's values, between steps of k
  unsigned inside;      // bit i: value i lies inside the matrix's outer dimension
  int kk, kk_step;
  __device__ __forceinline__ Loader(const TIn* base, int64_t ld, bool by_k, int outer0, int outer_size, int k0, int tid) {
    const int o = by_k ? tid / BK : tid % OUTER;
    const int o_step = by_k ? THREADS / BK : 0;
    kk = by_k ? tid % BK : tid / OUTER;
    kk_step = by_k ? 0 : THREADS / OUTER;
    p = base + (by_k ? static_cast<int64_t>(outer0 + o) * ld + k0 + kk : static_cast<int64_t>(k0 + kk) * ld + outer0 + o);
    step = (by_k ? o_step : kk_step) * ld;
    next = by_k ? BK : BK * ld;
    inside = 0;
#pragma unroll
    for (int i = 0; i < LOADS; ++i) inside |= (outer0 + o + i * o_step < outer_size ? 1u : 0u) << i;
  }
  __device__ __forceinline__ void load(int k_left, float (&v)[LOADS]) {   // k_left: values of k from this step on
#pragma unroll
    for (int i = 0; i < LOADS; ++i)
      v[i] = ((inside >> i) & 1u) != 0 && kk + i * kk_step < k_left ? load_as_f32<TIn>(p + i * step) : 0.0f;
    p += next;
  }
};

// What bounds it: the FMA pipes.  Steps are double buffered (registers, then shared memory), the values of a thread lie
// in runs of four along both dimensions, and finished tiles go through shared memory so that rows are stored whole.
// split > 1: the CTAs of a cluster (along x) take parts of K and add their tiles through distributed shared memory.
// Sums run in the order of k within a group; groups and CTAs are added in order.
// f32 512 x 1024 x 1024: 81 us with 4 x 4 values a thread and unpaired multiply-adds -> 45; 2048 x 2048 x 1024 runs at
// 35 TFLOP/s.
template <typename TIn, typename TOut, typename T>
__global__ void __launch_bounds__(T::kThreads, T::kResident) gemm_simt_kernel(const SimtArgs p) {
  constexpr int BM = T::BM, BN = T::BN, TM = T::TM, TN = T::TN, BK = T::BK;
  extern __shared__ __align__(16) float smem_f[];
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x;
  const int group = tid / T::kGroup, gt = tid % T::kGroup;
  const int tx = gt % (BN / TN), ty = gt / (BN / TN);
  const int rank = static_cast<int>(blockIdx.x) % p.split;
  const int m0 = blockIdx.y * BM, n0 = static_cast<int>(blockIdx.x) / p.split * BN;
  const int64_t batch = blockIdx.z;
  const TIn* A = static_cast<const TIn*>(p.a) + batch * p.sa;
  const TIn* B = static_cast<const TIn*>(p.b) + batch * p.sb;
  const int steps = (p.k + BK - 1) / BK;
  const int s0 = static_cast<int>(static_cast<int64_t>(rank) * steps / p.split), s1 = static_cast<int>(static_cast<int64_t>(rank + 1) * steps / p.split);

  Loader<TIn, BM, BK, T::kThreads, T::kLoadsA> la(A, p.lda, p.ta == 0, m0, p.m, s0 * BK, tid);
  Loader<TIn, BN, BK, T::kThreads, T::kLoadsB> lb(B, p.ldb, p.tb != 0, n0, p.n, s0 * BK, tid);
  float va[T::kLoadsA], vb[T::kLoadsB];
  auto put = [&](float* buf) {
#pragma unroll
    for (int i = 0; i < T::kLoadsA; ++i)
      buf[p.ta == 0 ? la.kk * T::kPitchA + tid / BK + i * (T::kThreads / BK)
                    : (la.kk + i * (T::kThreads / BM)) * T::kPitchA + tid % BM] = va[i];
    float* bb = buf + BK * T::kPitchA;
#pragma unroll
    for (int i = 0; i < T::kLoadsB; ++i)
      bb[p.tb != 0 ? lb.kk * T::kPitchB + tid / BK + i * (T::kThreads / BK)
                   : (lb.kk + i * (T::kThreads / BN)) * T::kPitchB + tid % BN] = vb[i];
  };
  float2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.0f, 0.0f);

  float2 sums[T::kDirect ? TM : 1][TN / 2];   // finished sums of 32 values of k
  if constexpr (T::kDirect) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) sums[i][j] = make_float2(0.0f, 0.0f);
  }

  if (s0 < s1) {
    la.load(p.k - s0 * BK, va);
    lb.load(p.k - s0 * BK, vb);
    put(smem_f);
  }
  __syncthreads();
  for (int s = s0; s < s1; ++s) {
    const float* buf = smem_f + ((s - s0) & 1) * T::kBuffer;
    if (s + 1 < s1) {
      la.load(p.k - (s + 1) * BK, va);
      lb.load(p.k - (s + 1) * BK, vb);
    }
    const float* pa = buf + group * (BK / T::KG) * T::kPitchA + ty * 4;
    const float* pb = buf + BK * T::kPitchA + group * (BK / T::KG) * T::kPitchB + tx * 4;
#pragma unroll
    for (int kk = 0; kk < BK / T::KG; ++kk) {
      float4 av[TM / 4], bv[TN / 4];
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) av[i] = *reinterpret_cast<const float4*>(pa + kk * T::kPitchA + i * (BM / (TM / 4)));
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) bv[j] = *reinterpret_cast<const float4*>(pb + kk * T::kPitchB + j * (BN / (TN / 4)));
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) {
        const float a4[4] = {av[i].x, av[i].y, av[i].z, av[i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int j = 0; j < TN / 4; ++j) {
            fma_pair(acc[4 * i + e][2 * j], a4[e], make_float2(bv[j].x, bv[j].y));
            fma_pair(acc[4 * i + e][2 * j + 1], a4[e], make_float2(bv[j].z, bv[j].w));
          }
      }
    }
    if constexpr (T::kDirect) {
      if ((s & 1) != 0 || s + 1 == s1) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) {
            add_pair(sums[i][j], acc[i][j]);
            acc[i][j] = make_float2(0.0f, 0.0f);
          }
      }
    }
    if (s + 1 < s1) put(smem_f + ((s + 1 - s0) & 1) * T::kBuffer);   // (last read in the step before: the barrier below)
    __syncthreads();
  }

  TOut* D = static_cast<TOut*>(p.d) + batch * p.sd;
  TOut* AUX = p.aux ? static_cast<TOut*>(p.aux) + batch * p.sd : nullptr;
  auto finish = [&](int gi, int gj, float sum) {
    const int64_t o = static_cast<int64_t>(gi) * p.ldd + gj;
    float v = p.alpha * sum;
    if (p.beta != 0.0f) v += p.beta * load_as_f32<TOut>(D + o);
    if (p.bias != nullptr) v += load_as_f32<TOut>(static_cast<const TOut*>(p.bias) + gj);
    if (AUX != nullptr) AUX[o] = store_from_f32<TOut>(v);
    D[o] = store_from_f32<TOut>(apply_act(p.act, v));
  };
  if constexpr (T::kDirect) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gi = m0 + ty * 4 + i;
      if (gi >= p.m) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (n0 + tx * 4 + j < p.n) finish(gi, n0 + tx * 4 + j, (j & 1) ? sums[i][j / 2].y : sums[i][j / 2].x);
    }
    return;
  }
  // ---- the groups' tiles -> shared memory [group][BM][BN]
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = (i / 4) * (BM / (TM / 4)) + ty * 4 + i % 4;
#pragma unroll
    for (int j = 0; j < TN / 4; ++j)
      *reinterpret_cast<float4*>(smem_f + (group * BM + r) * BN + j * (BN / (TN / 4)) + tx * 4) =
          make_float4(acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y);
  }
  cg::cluster_group cl = cg::this_cluster();
  if (p.split > 1) cl.sync();
  else __syncthreads();
  for (int e = rank * T::kThreads + tid; e < BM * BN; e += p.split * T::kThreads) {
    const int gi = m0 + e / BN, gj = n0 + e % BN;
    if (gi >= p.m || gj >= p.n) continue;
    float sum = 0.0f;
    for (int r = 0; r < p.split; ++r) {
      const float* t = p.split > 1 ? cl.map_shared_rank(smem_f, r) : smem_f;
#pragma unroll
      for (int g = 0; g < T::KG; ++g) sum += t[g * BM * BN + e];
    }
    finish(gi, gj, sum);
  }
  if (p.split > 1) cl.sync();   // the peers may still be reading this CTA's tile
}

template <typename TIn, typename TOut, typename T>
cudaError_t LaunchTile(const SimtArgs& a, int64_t batch, cudaStream_t stream, size_t smem = T::kSmem) {
  auto kernel = gemm_simt_kernel<TIn, TOut, T>;
  smem = std::max(smem, T::kSmem);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  LaunchCfg lc;
  lc.grid = dim3(static_cast<unsigned>(CeilDiv(a.n, T::BN) * a.split), static_cast<unsigned>(CeilDiv(a.m, T::BM)),
                 static_cast<unsigned>(batch));
  lc.block = dim3(T::kThreads);
  lc.smem = smem;
  lc.stream = stream;
  lc.pdl = true;
  lc.cluster_x = a.split;
  return Launch(lc, kernel, a);
}

// The tile by its time, in microseconds fitted to 148 SMs (f32, 16 sets of sizes, K from 16 to 4096): the busiest SM takes `n` tiles,
// each a fixed part and a part per value of k; short tiles run up to four at a time.  Where few tiles leave SMs
// idle, a cluster splits K.  Measured with the short tile and with the best of the others (us): 32 x 777 x 777 x 128 202 / 253, 32 x 512 x
// 512 x 64 49 / 71, 512 x 64 x 64 x 64 17 / 30, 100000 x 8 x 64 39 / 81; and where it loses: 1024 x 1024 x 1024 92 / 89 (medium), 4096 x 4096 x
// 512 540 / 432 (large), 300 x 200 x 256 19 / 7 (few).
template <typename TIn, typename TOut>
cudaError_t LaunchSimt(SimtArgs a, int64_t batch, int sm_count, cudaStream_t stream) {
  auto tiles = [&](int bm, int bn) { return CeilDiv(a.m, bm) * CeilDiv(a.n, bn) * batch; };
  auto split = [&](int64_t count) {
    int s = 1;
    while (s < 8 && count * s * 2 <= sm_count && a.k / (2 * s) >= 256) s *= 2;
    return s;
  };
  auto turns = [&](int bm, int bn) { return static_cast<double>(CeilDiv(tiles(bm, bn), sm_count)); };
  const int s_few = split(tiles(16, 64)), s_medium = split(tiles(64, 64));
  const double k = a.k, n_large = turns(128, 128), n_64 = turns(64, 64);
  // (of clusters of eight, of which a GPC takes whole ones only, about twelve are resident at once)
  auto waves = [&](int s, int64_t count) { return s == 8 && count > 12 ? 2.0 : 1.0; };
  const double few = CeilDiv(a.m, 16) > 65535 ? 1e30 : turns(16, 64) * (0.016 * k / s_few + 1.8) * waves(s_few, tiles(16, 64)) + (s_few > 1 ? 3.0 : 1.5);
  const double medium = n_64 * (0.0385 * k / s_medium + 4.5) * waves(s_medium, tiles(64, 64)) + (s_medium > 1 ? 3.0 : 1.5);
  const double large = n_large == 1 ? 0.1225 * k + 20.0 : n_large * (0.1 * k + 11.3) + 2.0;
  const double short_k = n_64 == 1 ? 0.055 * k + 5.5 : (n_64 == 2 ? 0.085 * k + 5.5 : (n_64 == 3 ? 0.118 * k + 6.5 : n_64 * (0.037 * k + 1.05) + 2.0));
  const double best = std::min({few, medium, large, short_k});
  a.split = 1;
  if (best == short_k) {
    // Up to four tiles per SM: shared memory for just that many, or some SMs get four and others one.
    const size_t share = n_64 <= 4 ? kSmemPerSm / static_cast<size_t>(n_64) - 1024 : 0;
    return LaunchTile<TIn, TOut, Short>(a, batch, stream, share);
  }
  if (best == large) return LaunchTile<TIn, TOut, Large>(a, batch, stream);
  if (best == medium) {
    a.split = s_medium;
    return LaunchTile<TIn, TOut, Medium>(a, batch, stream);
  }
  a.split = s_few;
  return LaunchTile<TIn, TOut, Few>(a, batch, stream);
}

// Copies rows of `cols` 16-bit elements that start anywhere into rows of `dst_words` 32-bit words.  Bound by memory:
// a warp moves 128 contiguous bytes; a row that starts on an odd element is put together from the two words around
// each pair (the second comes from L1).
__global__ void __launch_bounds__(256) align_rows_kernel(const uint16_t* src, uint32_t* dst, int64_t rows_per_batch, int64_t rows,
                                                         int cols, int64_t ld, int64_t batch_stride, int dst_words) {
  pdl_wait();
  pdl_launch_dependents();
  const int words = (cols + 1) / 2;
  for (int64_t r = blockIdx.y * static_cast<int64_t>(blockDim.y) + threadIdx.y; r < rows; r += static_cast<int64_t>(gridDim.y) * blockDim.y) {
    const uint16_t* s = src + (r / rows_per_batch) * batch_stride + (r % rows_per_batch) * ld;
    uint32_t* d = dst + r * dst_words;
    const bool odd = (reinterpret_cast<uintptr_t>(s) & 2) != 0;
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x) {
      uint32_t v;
      if (2 * w + 1 >= cols) v = __ldg(s + 2 * w);
      else if (!odd) v = __ldg(reinterpret_cast<const uint32_t*>(s) + w);
      else v = __byte_perm(__ldg(reinterpret_cast<const uint32_t*>(s - 1) + w), __ldg(reinterpret_cast<const uint32_t*>(s - 1) + w + 1), 0x5432);
      d[w] = v;
    }
  }
}

b200_status AlignRows(b200_context* ctx, cudaStream_t stream, const b200_operand& x, int64_t rows, int64_t cols, int64_t batches,
                      void* dst, int64_t dst_ld) {
  b200_status s = BeginLaunch(ctx);
  if (s != B200_OK) return s;
  const int words = static_cast<int>(CeilDiv(cols, 2));
  const int tx = words >= 128 ? 128 : 32, ty = 256 / tx;
  LaunchCfg lc;
  lc.block = dim3(tx, ty);
  const int64_t all = rows * batches, gx = std::min<int64_t>(CeilDiv(words, 4 * tx), 64);
  lc.grid = dim3(static_cast<unsigned>(std::max<int64_t>(gx, 1)), static_cast<unsigned>(std::min<int64_t>(CeilDiv(all, ty), std::max<int64_t>(1, ctx->sm_count * 16 / std::max<int64_t>(gx, 1)))));
  lc.stream = stream;
  lc.pdl = true;
  cudaError_t e = Launch(lc, align_rows_kernel, static_cast<const uint16_t*>(x.ptr), static_cast<uint32_t*>(dst), rows, all,
                         static_cast<int>(cols), x.ld, batches > 1 ? x.batch_stride : 0, static_cast<int>(dst_ld / 2));
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_gemm: row alignment launch: %s", cudaGetErrorString(e)));
  return EndLaunch(ctx, "b200_gemm (row alignment)");
}

// The same product with every operand that TMA cannot read copied into aligned rows.  The copy lives in
// stream-ordered memory of the context's pool (safe for any streams and threads).
b200_status RunTcgen05Aligned(b200_context* ctx, cudaStream_t stream, const b200_gemm_params* p, const b200_epilogue* epi) {
  b200_gemm_params q = *p;
  void* scratch[2] = {nullptr, nullptr};
  b200_status s = B200_OK;
  for (int i = 0; i < 2 && s == B200_OK; ++i) {
    b200_operand& x = i == 0 ? q.a : q.b;
    if (TmaReadable(x, p->batch)) continue;
    const bool rows_are_k = i == 0 ? x.transpose != 0 : x.transpose == 0;
    const int64_t outer = i == 0 ? p->m : p->n, rows = rows_are_k ? p->k : outer, cols = rows_are_k ? outer : p->k;
    const int64_t ld = CeilDiv(cols, 8) * 8, batches = p->batch > 1 && x.batch_stride != 0 ? p->batch : 1;
    cudaError_t e = cudaMallocFromPoolAsync(&scratch[i], static_cast<size_t>(rows) * ld * batches * 2, ctx->pool, stream);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      scratch[i] = nullptr;
      s = Fail(B200_RESOURCE_EXHAUSTED, "b200_gemm: memory for an aligned copy of an operand: %s", cudaGetErrorString(e));
      break;
    }
    s = AlignRows(ctx, stream, x, rows, cols, batches, scratch[i], ld);
    x.ptr = scratch[i];
    x.ld = ld;
    x.batch_stride = batches > 1 ? rows * ld : 0;
  }
  if (s == B200_OK) s = RunTcgen05(ctx, stream, &q, epi);
  for (void* d : scratch)
    if (d != nullptr) cudaFreeAsync(d, stream);
  return s;
}

// f32 results show the low bits that the tensor core's accumulator drops (bf16 operands, k = 1625, against float64: 1.6e-6, the SIMT
// kernel 3.4e-7), results of 16 bits do not.  One aligned product takes the tensor core for either; batches and copied operands,
// where the SIMT kernel is the alternative in earnest, only for 16-bit results (or where the caller asks for that route).
bool KeepsPrecision(const b200_gemm_params* p) { return p->c.dtype != B200_F32; }

// Worth an aligned copy: the SIMT kernel runs at about 20 TFLOP/s, the copies cost a few microseconds each.
bool WorthAligning(const b200_gemm_params* p, const b200_epilogue* epi) {
  if (!KeepsPrecision(p)) return false;
  b200_gemm_params q = *p;
  for (b200_operand* x : {&q.a, &q.b})
    if (!TmaReadable(*x, p->batch)) x->ptr = nullptr, x->ld = 8, x->batch_stride = 0;
  return Tcgen05Supports(&q, epi) && static_cast<double>(p->m) * p->n * p->k * p->batch >= 67108864.0;
}

b200_status Validate(const b200_gemm_params* p, const b200_epilogue* epi) {
  if (p == nullptr) return Fail(B200_INVALID_ARGUMENT, "b200_gemm: null params");
  if (epi != nullptr && (epi->act < 0 || epi->act > 3))
    return Fail(B200_INVALID_ARGUMENT, "b200_gemm: unknown activation %d", epi->act);
  for (const b200_operand* x : {&p->a, &p->b, &p->c})
    if (x->dtype != B200_F32 && x->dtype != B200_F16 && x->dtype != B200_BF16)
      return Fail(B200_INVALID_ARGUMENT, "b200_gemm: unknown dtype %d", x->dtype);
  if (p->a.dtype != p->b.dtype) return Fail(B200_INVALID_ARGUMENT, "b200_gemm: A and B dtypes differ");
  if (p->c.dtype != p->a.dtype && p->c.dtype != B200_F32)
    return Fail(B200_INVALID_ARGUMENT, "b200_gemm: unsupported output dtype");
  if (p->c.transpose) return Fail(B200_INVALID_ARGUMENT, "b200_gemm: transposed C");
  if (p->m < 0 || p->n < 0 || p->k < 0 || p->batch < 0) return Fail(B200_INVALID_ARGUMENT, "b200_gemm: negative size");
  if (p->m > kMaxInt || p->n > kMaxInt || p->k > kMaxInt)
    return Fail(B200_INVALID_ARGUMENT, "b200_gemm: dimension exceeds int32");
  for (const b200_operand* x : {&p->a, &p->b, &p->c}) {
    if (x->ld < 0 || x->ld > kMaxLd) return Fail(B200_INVALID_ARGUMENT, "b200_gemm: leading dimension too large");
    if (x->batch_stride < 0) return Fail(B200_INVALID_ARGUMENT, "b200_gemm: negative batch stride");
  }
  if (p->batch > kMaxInt) return Fail(B200_INVALID_ARGUMENT, "b200_gemm: batch too large");
  if (p->batch > 65535) return Fail(B200_UNIMPLEMENTED, "b200_gemm: more than 65535 batches");
  const int64_t a_cols = p->a.transpose ? p->m : p->k;
  const int64_t b_cols = p->b.transpose ? p->k : p->n;
  if ((p->k > 0 && ((p->m > 0 && p->a.ld < a_cols) || (p->n > 0 && p->b.ld < b_cols))) ||
      (p->m > 0 && p->c.ld < p->n))
    return Fail(B200_INVALID_ARGUMENT, "b200_gemm: leading dimension smaller than row length");
  if (p->m == 0 || p->n == 0 || p->batch == 0) return B200_OK;
  if (p->c.ptr == nullptr || (p->k > 0 && (p->a.ptr == nullptr || p->b.ptr == nullptr)))
    return Fail(B200_INVALID_ARGUMENT, "b200_gemm: null buffer");
  return B200_OK;
}

bool FewRowSupports(const b200_gemm_params* p, bool* vectors_are_b) {
  // x . W^T with K contiguous on both sides (the reference's gemv layout,
  // gemv.cc:71-75), widened from 2..8 to 1..32 vectors.
  if (p->a.dtype != B200_BF16 || p->a.transpose || !p->b.transpose) return false;
  if (p->c.dtype != B200_BF16 && p->c.dtype != B200_F32) return false;
  if (p->batch != 1 || p->beta != 0.0) return false;
  const bool vb = p->n < p->m;
  const int64_t vecs = vb ? p->n : p->m;
  if (vecs < 1 || vecs > 32 || p->k < 512 || p->k % 64 != 0) return false;
  const b200_operand& mat = vb ? p->a : p->b;
  if (mat.ld != p->k || !Aligned(mat.ptr, 16)) return false;
  if (vectors_are_b) *vectors_are_b = vb;
  return true;
}

int Route(const b200_gemm_params* p, const b200_epilogue* epi, int forced) {
  if (p->m == 0 || p->n == 0 || p->batch == 0) return B200_ROUTE_NONE;
  if (forced == B200_ROUTE_SIMT) return B200_ROUTE_SIMT;
  const bool few = FewRowSupports(p, nullptr);
  const bool tc = Tcgen05Supports(p, epi);
  if (forced == B200_ROUTE_FEWROW && few) return B200_ROUTE_FEWROW;
  if (forced == B200_ROUTE_TCGEN05 && tc) return B200_ROUTE_TCGEN05;
  // measured on 4096 x 4096 weights: 9 vs 13 us at 1 row, 12 vs 14 at 8, 20 vs 13 at 16, 33 vs 16 at 32
  if (few && (std::min(p->m, p->n) <= 8 || !tc)) return B200_ROUTE_FEWROW;
  if ((tc && (p->batch == 1 || KeepsPrecision(p))) || WorthAligning(p, epi)) return B200_ROUTE_TCGEN05;
  return B200_ROUTE_SIMT;
}

}  // namespace

extern "C" {

b200_status b200_gemm_validate(const b200_gemm_params* p, const b200_epilogue* epi) { return Validate(p, epi); }

int b200_gemm_route(const b200_gemm_params* p, const b200_epilogue* epi) {
  if (Validate(p, epi) != B200_OK) return -1;
  return Route(p, epi, 0);
}

uint64_t b200_gemm_work(const b200_gemm_params* p) {
  if (p == nullptr) return 0;
  const uint64_t b = static_cast<uint64_t>(p->batch > 0 ? p->batch : 0);
  const uint64_t m = p->m, n = p->n, k = p->k;
  const uint64_t flops = 2 * b * m * n * k;
  const uint64_t bytes = b * (DtypeSize(p->a.dtype) * (m * k + k * n) + DtypeSize(p->c.dtype) * m * n);
  return flops > 64 * bytes ? flops : 64 * bytes;
}

b200_status b200_gemm(b200_context* ctx, b200_stream stream, const b200_gemm_params* p, const b200_epilogue* epi) {
  b200_status s = BeginLaunch(ctx);
  if (s != B200_OK) return s;
  s = Validate(p, epi);
  if (s != B200_OK) return s;
  const b200_epilogue none = {0, nullptr, nullptr};
  if (epi == nullptr) epi = &none;
  const int route = Route(p, epi, ctx->force_route.load());
  if (route == B200_ROUTE_NONE) return B200_OK;
  if (route == B200_ROUTE_TCGEN05) {
    if (Tcgen05Supports(p, epi)) return RunTcgen05(ctx, stream, p, epi);
    s = RunTcgen05Aligned(ctx, stream, p, epi);
    if (s != B200_RESOURCE_EXHAUSTED) return s;   // without memory for the copies: the SIMT kernel
  }
  if (route == B200_ROUTE_FEWROW) {
    bool vb = false;
    FewRowSupports(p, &vb);
    const b200_operand& mat = vb ? p->a : p->b;
    const b200_operand& vec = vb ? p->b : p->a;
    const int64_t rows = vb ? p->m : p->n, vecs = vb ? p->n : p->m;
    // D[i, j] at i*ldc + j: the vectors index i (m small) or j (n small).
    const int64_t out_vec_stride = vb ? 1 : p->c.ld;
    const int64_t out_row_stride = vb ? p->c.ld : 1;
    return RunFewRowNT(ctx, stream, mat.ptr, vec.ptr, p->c.ptr, rows, vecs, p->k, vec.ld, out_row_stride,
                       out_vec_stride, static_cast<float>(p->alpha), epi->act, epi->bias, vb ? 1 : 0, epi->aux,
                       p->c.dtype == B200_F32);
  }
  SimtArgs a;
  a.a = p->a.ptr;
  a.b = p->b.ptr;
  a.d = p->c.ptr;
  a.bias = epi->bias;
  a.aux = epi->aux;
  a.m = static_cast<int>(p->m);
  a.n = static_cast<int>(p->n);
  a.k = static_cast<int>(p->k);
  a.lda = p->a.ld;
  a.ldb = p->b.ld;
  a.ldd = p->c.ld;
  const bool batched = p->batch > 1;
  a.sa = batched ? p->a.batch_stride : 0;
  a.sb = batched ? p->b.batch_stride : 0;
  a.sd = batched ? p->c.batch_stride : 0;
  a.ta = p->a.transpose;
  a.tb = p->b.transpose;
  a.alpha = static_cast<float>(p->alpha);
  a.beta = static_cast<float>(p->beta);
  a.act = epi->act;
  if (CeilDiv(p->m, 64) > 65535) return Fail(B200_UNIMPLEMENTED, "b200_gemm: m too large for the SIMT kernel grid");
  cudaError_t e;
  const int in = p->a.dtype, out = p->c.dtype;
  if (in == B200_F32) e = LaunchSimt<float, float>(a, p->batch, ctx->sm_count, stream);
  else if (in == B200_F16 && out == B200_F16) e = LaunchSimt<__half, __half>(a, p->batch, ctx->sm_count, stream);
  else if (in == B200_F16) e = LaunchSimt<__half, float>(a, p->batch, ctx->sm_count, stream);
  else if (out == B200_BF16) e = LaunchSimt<__nv_bfloat16, __nv_bfloat16>(a, p->batch, ctx->sm_count, stream);
  else e = LaunchSimt<__nv_bfloat16, float>(a, p->batch, ctx->sm_count, stream);
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_gemm launch: %s", cudaGetErrorString(e)));
  return EndLaunch(ctx, "b200_gemm");
}

}  // extern "C"
