// Dense 16-bit GEMM on the 5th-generation tensor cores:
//   D[b] = act(alpha * op(A[b]) op(B[b]) + beta * D[b] + bias[col]),  aux = pre-activation,
// the semantics of the reference's steel GEMM (metal_pjrt/blas/steel_gemm.cc:163-255,
// kernels/steel_gemm.metal:217-225) with f32 accumulation and one rounding.
//
// Structure (one persistent CTA per SM, 320 threads):
//   warp 0    TMA producer: per K step one 128 x 64 tile of op(A) and one 64-deep tile
//             of op(B), as 128-byte-swizzled boxes of cp.async.bulk.tensor (no cluster
//             multicast), into a shared-memory ring of up to 24 stages guarded by mbarriers;
//   warp 1    allocates tensor memory and issues tcgen05.mma (kind::f16, K = 16) from
//             shared-memory descriptors; tcgen05.commit releases ring slots and signals a
//             finished accumulator;
//   warps 2-9 epilogue: tcgen05.ld of their 32 accumulator lanes, the fused epilogue in
//             f32, one rounding, rows gathered in shared memory and stored 128 bytes at a time.
// Two accumulators (2 x BN of the 512 TMEM columns) let the epilogue of one tile overlap
// the MMAs of the next.  Every wait is bounded; a wait that gives up reports
// B200_TIMEOUT through the context's status word and the CTA unwinds (frees TMEM, returns).
//
// The single-thread roles are taken by an elected lane (elect.sync), not by "lane == 0": only then
// does the compiler know that one thread runs the code and keep descriptors and addresses in
// uniform registers.  Measured, 148 CTAs: a tcgen05.mma of 128 x 256 x 16 issued by lane 0 costs
// 142 cycles or more whatever its N, by an elected lane 127 (N = 256), 64 (128), 48 (64).
//
// CG = 2: the CTAs of a pair share one 256 x 256 tile (cta_group::2, issued by the even CTA): each
// loads its own 128 rows of A and half of B's columns, so an SM takes in 32 KB per K step instead
// of 48 (the single-CTA form is bound by that: about 46 B per cycle and SM).
//
// Either operand may be transposed: a K-contiguous operand is loaded as [rows][64 k] boxes
// (K-major descriptor), an M- or N-contiguous one as [64 k][64 rows] boxes (MN-major
// descriptor), so nothing is transposed in memory.  Batches are the third dimension of the maps.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "common.cuh"

namespace cg = cooperative_groups;
using namespace b200;

namespace {

constexpr int BM = 128;
constexpr int BK = 64;          // one 128-byte swizzle row of 16-bit elements
constexpr int kEpilogueWarps = 8;   // two per 32 TMEM lanes, half of the columns each
constexpr int kThreads = 64 + 32 * kEpilogueWarps;
constexpr int kMaxStages = 24;
constexpr int kRowGroup = 8;    // tiles are walked in bands of this many row tiles, so that a wave reuses A and B in L2
constexpr int kStagePitch = 128;                        // bytes of a staged output row; its 16-byte pieces are swizzled by row
constexpr int kStagingBytes = kEpilogueWarps * 32 * kStagePitch;

struct TcArgs {
  void* d;
  const void* bias;
  void* aux;
  int m, n, k;
  int64_t ldd, sd;       // row pitch and batch stride of D and aux
  float alpha, beta;
  int act;
  int ta, tb;
  int tiles_m, tiles_n, batch;
  int stages, stage_bytes;
  int a_rows;            // rows of A in a stage: 128, or all of a smaller m (the MMA reads 128 all the same, but what the
                         // other accumulator rows hold is never stored): a few-row product streams B through a deeper ring
  int bcast_a, bcast_b;  // the operand is the same for every batch
  int split;             // CTAs of a cluster along K (grid.y); 1: persistent CTAs, no cluster
  // WQ: quantised B [n][k] (scales per row and, for int4, offsets)
  const __nv_bfloat16* scale;
  const __nv_bfloat16* offset;
  int scale_ld;          // scales per row: k / 64, or 1
  int scale_vec;         // eight of them may be loaded at once
  int* status;
};

// How B arrives: as 16-bit values by TMA, or quantised, widened into the ring by eight more warps.  The packed weights
// come through a ring of their own (a further warp issues its TMA loads): boxes of 64 bytes of every row, 64-byte swizzle.
// What bounds a step of a 128 x 256 tile is then the widening, about 300 issue slots per scheduler against 508 cycles of MMAs.
// (Packed bytes fetched by the widening threads themselves, each its own row, took 1.05 us a step: 32 lines per load
// instruction, for weights and for scales.)
enum { kWide = 0, kQ4Seq = 1, kQ4Half = 2, kQ8 = 3 };
constexpr int kWidenThreads = 256;
constexpr int kWidenExtra = kWidenThreads + 32;
constexpr int kRawRing = 48 * 1024;
constexpr int kRawBoxBytes = 64;
__host__ __device__ constexpr int RawSlots(int bn) { return kRawRing / (bn * kRawBoxBytes); }

// ---- PTX wrappers --------------------------------------------------------------------
// One lane of the (converged) warp, known as such to the compiler.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// `bar` is a shared::cluster address: with CG = 2 the barrier of the pair's even CTA.
template <int CG>
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  if (CG == 2)
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  if (CG == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
template <int CG>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  if (CG == 2)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on `bar` once the MMAs issued so far have completed; CG = 2: on that barrier in both CTAs of the pair.
template <int CG>
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  if (CG == 2)
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
        "h"(static_cast<uint16_t>(3))
        : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 32 lanes x 32 consecutive columns: thread i of the warp gets lane (base + i), columns c .. c+31
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle.  K-major tile: rows of 128 bytes,
// 8-row groups 1024 bytes apart (SBO), LBO unused.  MN-major tile: boxes of [64 k][64 mn],
// 8-k-row groups 1024 bytes apart (SBO), the next 64 mn (next box) `lbo` bytes on.
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(lbo_bytes >> 4) << 16;
  d |= static_cast<uint64_t>(sbo_bytes >> 4) << 32;
  d |= 1ull << 46;   // descriptor version for this architecture
  d |= 2ull << 61;   // 128-byte swizzle
  return d;
}

// Instruction descriptor for kind::f16: f32 accumulate, A/B format (0 f16, 1 bf16),
// major-ness (0 K-major, 1 MN-major), N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t make_idesc(int ab_format, int a_mn_major, int b_mn_major, int n, int m) {
  return (1u << 4) | (static_cast<uint32_t>(ab_format) << 7) | (static_cast<uint32_t>(ab_format) << 10) |
         (static_cast<uint32_t>(a_mn_major) << 15) | (static_cast<uint32_t>(b_mn_major) << 16) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

template <int BN, int CG>
struct Smem {
  static constexpr int kBCols = BN / CG;             // columns of B in one CTA's shared memory
  static constexpr int kABytes = BM * BK * 2;        // 16 KB
  static constexpr int kBBytes = kBCols * BK * 2;
  static constexpr int kRing = 192 * 1024;           // cut into as many stages as fit (TcArgs::stages)
  static constexpr int kTotal = kRing + kStagingBytes + 1024 /* alignment slack */ + 768 /* barriers */;
  static_assert(kTotal <= 232448, "shared memory of one CTA");
};

template <typename TOut>
struct alignas(16) Vec16 {
  TOut e[16 / sizeof(TOut)];
};

template <typename TOut, int N>
__device__ __forceinline__ void activate(int act, float (&x)[N]) {
  if (sizeof(TOut) == 2) {
    apply_act_16bit<N>(act, x);
  } else if (act != 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = apply_act(act, x[i]);
  }
}

// What is added to alpha * acc for 32 consecutive columns of one row (beta * D and the bias): read before the
// accumulator, so that the two latencies overlap.
template <typename TOut>
__device__ __forceinline__ void addends(const TcArgs& a, const TOut* drow, int col0, float (&x)[32]) {
  const TOut* bias = static_cast<const TOut*>(a.bias);
  constexpr int kVec = 16 / sizeof(TOut);
  const bool full = col0 + 32 <= a.n;
#pragma unroll
  for (int j = 0; j < 32; ++j) x[j] = 0.0f;
  if (a.beta != 0.0f && drow != nullptr) {
    if (full && (reinterpret_cast<uintptr_t>(drow + col0) & 15) == 0) {
#pragma unroll
      for (int j = 0; j < 32; j += kVec) {
        const Vec16<TOut> w = *reinterpret_cast<const Vec16<TOut>*>(drow + col0 + j);
#pragma unroll
        for (int i = 0; i < kVec; ++i) x[j + i] = a.beta * load_as_f32<TOut>(&w.e[i]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < a.n) x[j] = a.beta * load_as_f32<TOut>(drow + col0 + j);
    }
  }
  if (bias != nullptr) {
    if (full && (reinterpret_cast<uintptr_t>(bias + col0) & 15) == 0) {
#pragma unroll
      for (int j = 0; j < 32; j += kVec) {
        const Vec16<TOut> w = *reinterpret_cast<const Vec16<TOut>*>(bias + col0 + j);
#pragma unroll
        for (int i = 0; i < kVec; ++i) x[j + i] += load_as_f32<TOut>(&w.e[i]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < a.n) x[j] += load_as_f32<TOut>(bias + col0 + j);
    }
  }
}

// Where byte b of staged row r lies: 16-byte accesses down a column of rows hit different banks.
__device__ __forceinline__ int staged(int r, int b) { return r * kStagePitch + ((((b >> 4) ^ r) & 7) << 4) + (b & 15); }

// 32 staged rows of kBytes (128 or 64) bytes -> global: 16-byte pieces where rows allow them, else one row per
// instruction in 4-byte words.  A 16-bit row that starts on an odd element is shifted by one (its words then hold the
// upper half of one staged word and the lower half of the next lane's), which leaves single elements at its ends.
template <typename TOut, int kBytes>
__device__ __forceinline__ void store_rows(const uint8_t* st, TOut* out, int64_t ld, int row0, int rows, int col0, int cols, int lane) {
  constexpr int kCols = kBytes / static_cast<int>(sizeof(TOut));
  constexpr int kVec = 16 / static_cast<int>(sizeof(TOut));
  constexpr int kPieces = kBytes / 16, kRowsAtOnce = 32 / kPieces;
  const uintptr_t base = reinterpret_cast<uintptr_t>(out);
  if (cols >= kCols && base % 16 == 0 && ld % kVec == 0) {
#pragma unroll
    for (int i = 0; i < 32 / kRowsAtOnce; ++i) {
      const int r = kRowsAtOnce * i + lane / kPieces, c = lane % kPieces;
      if (r < rows)
        *reinterpret_cast<uint4*>(out + static_cast<int64_t>(row0 + r) * ld + col0 + c * kVec) =
            *reinterpret_cast<const uint4*>(st + staged(r, c * 16));
    }
  } else if (sizeof(TOut) == 2) {
    TOut* o0 = out + static_cast<int64_t>(row0) * ld + col0;
#pragma unroll 8
    for (int r = 0; r < rows; ++r) {
      TOut* o = o0 + static_cast<int64_t>(r) * ld;
      const int odd = static_cast<int>((reinterpret_cast<uintptr_t>(o) >> 1) & 1);
      const uint32_t w = *reinterpret_cast<const uint32_t*>(st + staged(r, (4 * lane) & (kBytes - 1)));
      const uint32_t up = __shfl_down_sync(0xffffffffu, w, 1);
      if (lane < (cols - odd) / 2) *reinterpret_cast<uint32_t*>(o + odd + 2 * lane) = odd ? __byte_perm(w, up, 0x5432) : w;
    }
    if (lane < rows) {
      TOut* o = o0 + static_cast<int64_t>(lane) * ld;
      const int odd = static_cast<int>((reinterpret_cast<uintptr_t>(o) >> 1) & 1);
      if (odd) o[0] = *reinterpret_cast<const TOut*>(st + staged(lane, 0));
      if ((cols - odd) & 1) o[cols - 1] = *reinterpret_cast<const TOut*>(st + staged(lane, 2 * (cols - 1)));
    }
  } else {
#pragma unroll 8
    for (int r = 0; r < rows; ++r)
      if (lane < cols)
        out[static_cast<int64_t>(row0 + r) * ld + col0 + lane] = *reinterpret_cast<const TOut*>(st + staged(r, lane * static_cast<int>(sizeof(TOut))));
  }
}

// The same epilogue for 4 consecutive columns (the split-K reduction, where a warp owns a
// row and its lanes adjacent float4s, so that the reads of the peers' tiles coalesce).
template <typename TOut>
__device__ __forceinline__ void epilogue_quad(const TcArgs& a, const float (&acc)[4], TOut* D, TOut* AUX, int row, int col0) {
  const TOut* bias = static_cast<const TOut*>(a.bias);
  const int64_t o = static_cast<int64_t>(row) * a.ldd + col0;
  float x[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    x[j] = a.alpha * acc[j];
    if (col0 + j < a.n) {
      if (a.beta != 0.0f) x[j] += a.beta * load_as_f32<TOut>(D + o + j);
      if (bias != nullptr) x[j] += load_as_f32<TOut>(bias + col0 + j);
    }
  }
  float y[4] = {x[0], x[1], x[2], x[3]};
  activate<TOut>(a.act, y);
  constexpr size_t kBytes = 4 * sizeof(TOut);
  const bool vec = col0 + 4 <= a.n && (a.ldd % 4 == 0) && (reinterpret_cast<uintptr_t>(D) % kBytes == 0) &&
                   (AUX == nullptr || reinterpret_cast<uintptr_t>(AUX) % kBytes == 0);
  if (vec) {
    struct alignas(kBytes) Pack { TOut e[4]; };
    Pack pd, pa;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      pa.e[j] = store_from_f32<TOut>(x[j]);
      pd.e[j] = store_from_f32<TOut>(y[j]);
    }
    if (AUX != nullptr) *reinterpret_cast<Pack*>(AUX + o) = pa;
    *reinterpret_cast<Pack*>(D + o) = pd;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (col0 + j < a.n) {
        if (AUX != nullptr) AUX[o + j] = store_from_f32<TOut>(x[j]);
        D[o + j] = store_from_f32<TOut>(y[j]);
      }
    }
  }
}

// One arrival on barrier `bar` of CTA `rank`, without ordering this thread's global stores before it (a release
// at cluster scope would wait for them): tcgen05.wait::ld and the tcgen05 fence order what matters here.
__device__ __forceinline__ void mbar_arrive_relaxed(uint64_t* bar, uint32_t rank) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [ra];\n\t}" ::"r"(smem_u32(bar)),
      "r"(rank)
      : "memory");
}

// ---- widening of quantised weights: w = q * s (+ b) rounded once to bf16
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// Nibbles r and r + 4 of v as 128 + q, then q * s + b: q * s is exact, so the fused form rounds once.
__device__ __forceinline__ uint32_t widen_pair(uint32_t v, int r, uint32_t s2, uint32_t b2) {
  const uint32_t m = and_or(v >> (4 * r), 0x000f000fu, 0x43004300u);
  uint32_t q, w;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(q) : "r"(m), "r"(0x43004300u));
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(w) : "r"(q), "r"(s2), "r"(b2));
  return w;
}
// Four int8 as two words of bf16.
__device__ __forceinline__ uint2 widen_bytes(uint32_t v, float s) {
  const uint32_t u = v ^ 0x80808080u;   // q + 128; as the low bits of 2^23 + (q + 128)
  float f[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = (__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7650 + i)) - 8388736.0f) * s;
  return make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
}

struct TileAt {
  int b, tm, tn;
};
__device__ __forceinline__ TileAt tile_at(const TcArgs& a, int tile) {
  const int per = a.tiles_m * a.tiles_n;
  TileAt t;
  t.b = tile / per;
  const int r = tile - t.b * per;
  const int band = r / (kRowGroup * a.tiles_n), in = r - band * kRowGroup * a.tiles_n;
  const int rows = min(kRowGroup, a.tiles_m - band * kRowGroup);
  t.tm = band * kRowGroup + in % rows;
  t.tn = in / rows;
  return t;
}
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(p)), "r"(rank));
  return ra;
}

template <int BN, int CG, typename TOut, int WQ>
__global__ void __launch_bounds__(kThreads + (WQ ? kWidenExtra : 0), 1)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcArgs a,
                   const uint32_t idesc) {
  using S = Smem<BN, CG>;
  const int stages = a.stages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* staging = smem + S::kRing;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + kStagingBytes);
  uint64_t* empty = full + kMaxStages;
  uint64_t* tfull = empty + kMaxStages;
  uint64_t* tempty = tfull + 2;
  uint64_t* raw_full = tempty + 2;
  constexpr int kRawSlots = WQ ? RawSlots(BN) : 1;
  uint64_t* raw_empty = raw_full + kRawSlots;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(raw_empty + kRawSlots);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int num_tiles = a.tiles_m * a.tiles_n * a.batch;
  const int k_iters = (a.k + BK - 1) / BK;
  const int rank = CG == 2 ? static_cast<int>(blockIdx.x & 1) : 0;   // CTA of the pair
  const int tile0 = static_cast<int>(blockIdx.x) / CG, tile_step = static_cast<int>(gridDim.x) / CG;
  const bool solo = CG == 2 || a.split == 1;
  // With K split across a cluster, grid.x is the tile count (one tile per CTA) and CTA
  // blockIdx.y accumulates k steps [ki_begin, ki_end) of it.
  const int ki_begin = solo ? 0 : static_cast<int>(blockIdx.y) * k_iters / a.split;
  const int ki_end = solo ? k_iters : (static_cast<int>(blockIdx.y) + 1) * k_iters / a.split;
  constexpr int kPartLd = BN + 4;          // row pitch (floats) of the partial tile in shared memory
  constexpr uint32_t kTmemCols = 2 * BN;   // two accumulators; a power of two >= 32

  if (tid == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], WQ ? 1 + kWidenThreads / 32 : 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < kRawSlots; ++i) {
      mbar_init(&raw_full[i], 1);
      mbar_init(&raw_empty[i], kWidenThreads / 32);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], CG * kEpilogueWarps);
    }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc<CG>(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cg::this_cluster().sync();   // the pair's barriers exist before anyone arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();               // A, B (and D under beta) may come from the previous kernel
  pdl_launch_dependents();

  if (warp == 0) {
    // ---------------- TMA producer (one lane)
    if (elect_one()) {
      const uint32_t a_bytes = static_cast<uint32_t>(a.a_rows) * BK * 2;
      int s = 0;
      uint32_t parity = 1;   // the first lap waits for nothing
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
        const TileAt t = tile_at(a, tile);
        const int row0 = (t.tm * CG + rank) * BM, col0 = t.tn * BN + rank * S::kBCols;
        const int ba = a.bcast_a ? 0 : t.b, bb = a.bcast_b ? 0 : t.b;
        for (int ki = ki_begin; ki < ki_end; ++ki) {
          if (!mbar_wait_bounded(&empty[s], parity)) {
            report_timeout(a.status, 300 + s);
            ok = false;
            break;
          }
          const uint32_t As = smem_u32(smem + s * a.stage_bytes), Bs = As + a_bytes;
          const uint32_t bar = CG == 2 ? cluster_addr(&full[s], 0) : smem_u32(&full[s]);
          if (rank == 0) mbar_expect_tx(&full[s], WQ ? a_bytes : CG * a.stage_bytes);
          if (!a.ta) {
            tma_load_3d<CG>(As, &tmA, ki * BK, row0, ba, bar);                   // [128 m][64 k]
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)                                      // [64 k][64 m] boxes
              tma_load_3d<CG>(As + j * 8192, &tmA, row0 + j * 64, ki * BK, ba, bar);
          }
          if (WQ) {
            // (B: the widening warps)
          } else if (a.tb) {
            tma_load_3d<CG>(Bs, &tmB, ki * BK, col0, bb, bar);                   // [n][64 k]
          } else {
#pragma unroll
            for (int j = 0; j < S::kBCols / 64; ++j)                               // [64 k][64 n] boxes
              tma_load_3d<CG>(Bs + j * 8192, &tmB, col0 + j * 64, ki * BK, bb, bar);
          }
          if (++s == stages) s = 0, parity ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (one lane; of a pair, the even CTA's)
    if (rank == 0 && elect_one()) {
      int s = 0, tcount = 0;
      uint32_t parity = 0;
      bool ok = true;
      const uint64_t desc_a0 = a.ta ? make_desc(smem_u32(smem), 8192, 1024) : make_desc(smem_u32(smem), 16, 1024);
      const uint32_t b0 = smem_u32(smem) + static_cast<uint32_t>(a.a_rows) * BK * 2;
      const uint64_t desc_b0 = a.tb ? make_desc(b0, 16, 1024) : make_desc(b0, 8192, 1024);
      const uint64_t step_a = a.ta ? 2048 >> 4 : 32 >> 4, step_b = a.tb ? 32 >> 4 : 2048 >> 4;   // 16 k further
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step, ++tcount) {
        const int acc = tcount & 1;
        if (!mbar_wait_bounded(&tempty[acc], ((tcount >> 1) & 1) ^ 1)) {
          report_timeout(a.status, 310 + acc);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int ki = ki_begin; ki < ki_end; ++ki) {
          if (!mbar_wait_bounded(&full[s], parity)) {
            report_timeout(a.status, 320 + s);
            ok = false;
            break;
          }
          tc_fence_after();
          uint64_t da = desc_a0 + static_cast<uint64_t>(s * (a.stage_bytes >> 4));
          uint64_t db = desc_b0 + static_cast<uint64_t>(s * (a.stage_bytes >> 4));
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            umma_f16<CG>(tmem_d, da, db, idesc, (ki > ki_begin || kk > 0) ? 1u : 0u);
            da += step_a;
            db += step_b;
          }
          umma_commit<CG>(&empty[s]);     // the slot is free once these MMAs have read it
          if (++s == stages) s = 0, parity ^= 1;
        }
        if (ok) umma_commit<CG>(&tfull[acc]);
      }
    }
    __syncwarp();
  } else if (WQ && warp == 2 + kEpilogueWarps + kWidenThreads / 32) {
    // ---------------- packed weights (one lane): a box holds kSteps 64-deep steps of every row of the tile
    constexpr int kSteps = WQ == kQ8 ? 1 : 2;
    if (elect_one()) {
      int slot = 0;
      uint32_t parity = 1;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
        const int col0 = tile_at(a, tile).tn * BN;
        for (int ki = ki_begin; ki < ki_end; ki += kSteps) {
          if (!mbar_wait_bounded(&raw_empty[slot], parity)) {
            report_timeout(a.status, 350 + slot);
            ok = false;
            break;
          }
          mbar_expect_tx(&raw_full[slot], BN * kRawBoxBytes);
          tma_load_2d(smem_u32(smem + stages * a.stage_bytes + slot * BN * kRawBoxBytes), &tmB, ki * (kRawBoxBytes / kSteps), col0,
                      smem_u32(&raw_full[slot]));
          if (++slot == kRawSlots) slot = 0, parity ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (WQ && warp >= 2 + kEpilogueWarps) {
    // ---------------- widening warps: a thread owns its part of one row of every 64-deep step (one group of the weights)
    constexpr int kSteps = WQ == kQ8 ? 1 : 2;
    constexpr int kPerRow = kWidenThreads / BN;                                // threads of a row
    constexpr int kBytes = kRawBoxBytes / kSteps / kPerRow;                    // packed bytes of a thread and step
    constexpr int kPieces = kBytes / 16 > 0 ? kBytes / 16 : 1;
    const int wt = tid - kThreads, row = wt / kPerRow, part = wt % kPerRow;
    const uint8_t* raw = smem + stages * a.stage_bytes + row * kRawBoxBytes;
    int s = 0, slot = 0;
    uint32_t parity = 1, raw_parity = 0;
    bool ok = true;
    for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
      const int64_t n = min(tile_at(a, tile).tn * BN + row, a.n - 1);
      const uint16_t* sp = reinterpret_cast<const uint16_t*>(a.scale) + n * a.scale_ld;
      const uint16_t* bp = reinterpret_cast<const uint16_t*>(a.offset) + n * a.scale_ld;
      const bool one_scale = a.scale_ld == 1;
      // scales (and offsets) of eight steps at a time, one such block ahead
      uint4 s8 = make_uint4(0, 0, 0, 0), b8 = s8, s_next = s8, b_next = s8;
      auto load8 = [&](int kb) {
        if (!a.scale_vec) return;
        s_next = __ldg(reinterpret_cast<const uint4*>(sp + kb));
        if (WQ != kQ8) b_next = __ldg(reinterpret_cast<const uint4*>(bp + kb));
      };
      const uint32_t only = one_scale ? __ldg(sp) : 0u;
      load8(ki_begin & ~7);
      for (int kb = ki_begin & ~7; kb < ki_end && ok; kb += 8) {
        s8 = s_next, b8 = b_next;
        if (kb + 8 < ki_end) load8(kb + 8);
        const uint32_t sw[4] = {s8.x, s8.y, s8.z, s8.w}, bw[4] = {b8.x, b8.y, b8.z, b8.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int ki = kb + i;
          if (ki < ki_begin) continue;
          if (ki >= ki_end || !ok) break;
          uint32_t s2, b2;   // the scale and the offset, twice
          if (a.scale_vec) {
            s2 = __byte_perm(sw[i / 2], 0, (i & 1) ? 0x3232 : 0x1010);
            b2 = __byte_perm(bw[i / 2], 0, (i & 1) ? 0x3232 : 0x1010);
          } else {
            s2 = (one_scale ? only : __ldg(sp + ki)) * 0x10001u;
            b2 = WQ == kQ8 ? 0u : __ldg(bp + ki) * 0x10001u;
          }
          const int in_box = kSteps == 2 ? (ki - ki_begin) & 1 : 0;
          if (in_box == 0 && !mbar_wait_bounded(&raw_full[slot], raw_parity)) {
            report_timeout(a.status, 360 + slot);
            ok = false;
            break;
          }
          uint4 v[kPieces];
#pragma unroll
          for (int j = 0; j < kPieces; ++j)
            v[j] = *reinterpret_cast<const uint4*>(raw + slot * BN * kRawBoxBytes + (((in_box * (4 / kSteps) + part * kPieces + j) ^ ((row >> 1) & 3)) << 4));
          if (!mbar_wait_bounded(&empty[s], parity)) {
            report_timeout(a.status, 340 + s);
            ok = false;
            break;
          }
          uint8_t* dst = smem + s * a.stage_bytes + a.a_rows * (BK * 2) + row * 128;
          auto put = [&](int c, const uint4& w) { *reinterpret_cast<uint4*>(dst + ((c ^ (row & 7)) << 4)) = w; };   // chunk c: inputs 8 c ..
          if (WQ == kQ4Seq) {
#pragma unroll
            for (int j = 0; j < kPieces; ++j) {
              const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const uint32_t p0 = widen_pair(w[e], 0, s2, b2), p1 = widen_pair(w[e], 1, s2, b2);
                const uint32_t p2 = widen_pair(w[e], 2, s2, b2), p3 = widen_pair(w[e], 3, s2, b2);
                put(part * (kBytes / 4) + 4 * j + e, make_uint4(__byte_perm(p0, p1, 0x5410), __byte_perm(p2, p3, 0x5410),
                                                               __byte_perm(p0, p1, 0x7632), __byte_perm(p2, p3, 0x7632)));
              }
            }
          } else if (WQ == kQ4Half) {
#pragma unroll
            for (int j = 0; j < kPieces; ++j) {
              // a byte of the group holds inputs i and i + 32
              const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
              for (int e = 0; e < 4; e += 2) {
                uint32_t lo[4], hi[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const uint32_t p0 = widen_pair(w[e + h], 0, s2, b2), p1 = widen_pair(w[e + h], 1, s2, b2);
                  const uint32_t p2 = widen_pair(w[e + h], 2, s2, b2), p3 = widen_pair(w[e + h], 3, s2, b2);
                  lo[2 * h] = __byte_perm(p0, p2, 0x5410), lo[2 * h + 1] = __byte_perm(p0, p2, 0x7632);
                  hi[2 * h] = __byte_perm(p1, p3, 0x5410), hi[2 * h + 1] = __byte_perm(p1, p3, 0x7632);
                }
                const int c = (part * kBytes + 16 * j + 4 * e) / 8;
                put(c, make_uint4(lo[0], lo[1], lo[2], lo[3]));
                put(c + 4, make_uint4(hi[0], hi[1], hi[2], hi[3]));
              }
            }
          } else if (WQ == kQ8) {
            const float sf = bf16_lo(s2);
#pragma unroll
            for (int j = 0; j < kPieces; ++j) {
              const uint2 w0 = widen_bytes(v[j].x, sf), w1 = widen_bytes(v[j].y, sf), w2 = widen_bytes(v[j].z, sf), w3 = widen_bytes(v[j].w, sf);
              put(part * (kBytes / 8) + 2 * j, make_uint4(w0.x, w0.y, w1.x, w1.y));
              put(part * (kBytes / 8) + 2 * j + 1, make_uint4(w2.x, w2.y, w3.x, w3.y));
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads through the async proxy
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[s]);
          if (++s == stages) s = 0, parity ^= 1;
          if (in_box == kSteps - 1 || ki + 1 == ki_end) {
            if (lane == 0) mbar_arrive(&raw_empty[slot]);
            if (++slot == kRawSlots) slot = 0, raw_parity ^= 1;
          }
        }
      }
    }
  } else {
    // ---------------- epilogue warps: TMEM lanes 32 q .. 32 q + 31, columns c_lo .. c_lo + BN / 2 - 1
    const int q = warp & 3;
    const int c_lo = ((warp - 2) >> 2) * (BN / 2);
    uint8_t* st = staging + (warp - 2) * 32 * kStagePitch;
    constexpr int kCols = 128 / static_cast<int>(sizeof(TOut));   // columns gathered per store pass
    constexpr int kPass = kCols < BN / 2 ? kCols : BN / 2;
    constexpr int kVec = 16 / static_cast<int>(sizeof(TOut));
    auto accumulator_free = [&](int acc) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_relaxed(&tempty[acc], 0);
        else mbar_arrive(&tempty[acc]);
      }
    };
    int tcount = 0;
    for (int tile = tile0; tile < num_tiles; tile += tile_step, ++tcount) {
      const TileAt t = tile_at(a, tile);
      const int acc = tcount & 1;
      if (!mbar_wait_bounded(&tfull[acc], (tcount >> 1) & 1)) {
        report_timeout(a.status, 330 + acc);
        break;
      }
      tc_fence_after();
      bool drained = false;
      const uint32_t tmem_row = tmem_base + (static_cast<uint32_t>(32 * q) << 16) + static_cast<uint32_t>(acc * BN);
      if (!solo) {
        // this CTA's K slice only: park the f32 partial in the (now idle) ring
#pragma unroll 1
        for (int c0 = c_lo; c0 < c_lo + BN / 2; c0 += 32) {
          uint32_t v[32];
          tmem_ld_32x32(tmem_row + static_cast<uint32_t>(c0), v);
          float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(smem) + (32 * q + lane) * kPartLd + c0);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            dst[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]),
                                 __uint_as_float(v[4 * j + 3]));
        }
      } else {
        const int row0 = (t.tm * CG + rank) * BM + 32 * q, rows = min(32, a.m - row0);
        TOut* D = static_cast<TOut*>(a.d) + t.b * a.sd;
        TOut* AUX = a.aux != nullptr ? static_cast<TOut*>(a.aux) + t.b * a.sd : nullptr;
        const TOut* drow = lane < rows ? D + static_cast<int64_t>(row0 + lane) * a.ldd : nullptr;
        if (rows > 0) {
#pragma unroll 1
          for (int c0 = c_lo; c0 < c_lo + BN / 2 && t.tn * BN + c0 < a.n; c0 += kPass) {
            const int col0 = t.tn * BN + c0;
#pragma unroll 1
            for (int pass = AUX != nullptr ? 0 : 1; pass < 2; ++pass) {   // 0: the pre-activation to aux, 1: D
#pragma unroll
              for (int h = 0; h < kPass; h += 32) {
                uint32_t v[32];
                float x[32];
                addends<TOut>(a, drow, col0 + h, x);
                tmem_ld_32x32(tmem_row + static_cast<uint32_t>(c0 + h), v);
#pragma unroll
                for (int j = 0; j < 32; ++j) x[j] = fmaf(a.alpha, __uint_as_float(v[j]), x[j]);
                if (pass == 1) activate<TOut>(a.act, x);
#pragma unroll
                for (int j = 0; j < 32; j += kVec) {
                  Vec16<TOut> w;
#pragma unroll
                  for (int i = 0; i < kVec; ++i) w.e[i] = store_from_f32<TOut>(x[j + i]);
                  *reinterpret_cast<Vec16<TOut>*>(st + staged(lane, (h + j) * static_cast<int>(sizeof(TOut)))) = w;
                }
              }
              __syncwarp();
              if (pass == 1 && (c0 + kPass >= c_lo + BN / 2 || col0 + kPass >= a.n)) {   // the last read of this accumulator
                accumulator_free(acc);
                drained = true;
              }
              store_rows<TOut, kPass * static_cast<int>(sizeof(TOut))>(st, pass == 0 ? AUX : D, a.ldd, row0, rows, col0, min(kPass, a.n - col0), lane);
              __syncwarp();
            }
          }
        }
      }
      if (!drained) accumulator_free(acc);
    }
  }
  if (CG == 2) {
    cg::this_cluster().sync();   // the pair's barriers and tensor memory are in use until both are done
  } else if (a.split > 1) {
    // K split: every CTA of the cluster finishes its share of the rows of the
    // tile from all the partial tiles, read through distributed shared memory.
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (warp >= 2 && warp < 2 + kEpilogueWarps) {
      const TileAt t = tile_at(a, blockIdx.x);
      TOut* D = static_cast<TOut*>(a.d) + t.b * a.sd;
      TOut* AUX = a.aux != nullptr ? static_cast<TOut*>(a.aux) + t.b * a.sd : nullptr;
      const int tile_rows = min(BM, a.m - t.tm * BM), rows_per_rank = (tile_rows + a.split - 1) / a.split;
      const float* part = reinterpret_cast<const float*>(smem);
      // a warp per row, lanes on adjacent float4s: 512-byte runs of every peer's tile
      for (int rr = warp - 2; rr < rows_per_rank; rr += kEpilogueWarps) {
        const int r = static_cast<int>(blockIdx.y) * rows_per_rank + rr;
        const int row = t.tm * BM + r;
        if (r >= tile_rows) break;
#pragma unroll
        for (int u = 0; u < BN / 128 + (BN < 128 ? 1 : 0); ++u) {
          const int c = u * 128 + 4 * lane;
          if (c >= BN || t.tn * BN + c >= a.n) continue;
          float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          float4 v[8];
#pragma unroll
          for (int peer = 0; peer < 8; ++peer)   // all the remote loads in flight together
            v[peer] = peer < a.split
                          ? *reinterpret_cast<const float4*>(cluster.map_shared_rank(part, peer) + r * kPartLd + c)
                          : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
          for (int peer = 0; peer < 8; ++peer) {
            sum[0] += v[peer].x;
            sum[1] += v[peer].y;
            sum[2] += v[peer].z;
            sum[3] += v[peer].w;
          }
          epilogue_quad<TOut>(a, sum, D, AUX, row, t.tn * BN + c);
        }
      }
    }
    cluster.sync();   // peers may still be reading this CTA's partial tile
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<CG>(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up through the runtime so that the
// library links nothing but the CUDA runtime.
EncodeTiledFn Encoder() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// A 3-D map over `batch` row-major matrices: `inner` contiguous elements per row, `outer`
// rows `ld` elements apart; boxes of box_inner x box_outer x 1, 128-byte swizzle.
bool MakeMap(CUtensorMap* map, int dtype, const void* base, int64_t inner, int64_t outer, int64_t ld, int64_t batch,
             int64_t batch_stride, int box_inner, int box_outer) {
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer), static_cast<cuuint64_t>(batch)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * 2, static_cast<cuuint64_t>(batch > 1 ? batch_stride : ld * outer) * 2};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(box_inner), static_cast<cuuint32_t>(box_outer), 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = Encoder()(map, dtype == B200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                               3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace
namespace b200 {
// A 2-D map over `rows` rows of bytes; boxes of box_bytes (128 or 64: the span of their swizzle) x box_rows.
bool EncodeByteRows(CUtensorMap* map, const void* base, int64_t row_bytes, int64_t rows, int box_bytes, int box_rows) {
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_bytes), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  return Encoder() != nullptr &&
         Encoder()(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace b200
namespace {

template <int BN, int CG, typename TOut, int WQ>
cudaError_t LaunchTc(const CUtensorMap& ma, const CUtensorMap& mb, const TcArgs& a, uint32_t idesc, int grid,
                     cudaStream_t stream) {
  static_assert(BM * (BN / CG + 4) * 4 <= Smem<BN, CG>::kRing, "partial tile must fit the ring");
  auto kernel = gemm_tc_kernel<BN, CG, TOut, WQ>;
  static std::atomic<uint64_t> ready{0};   // per device: the shared-memory limit is raised
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((ready.load(std::memory_order_relaxed) >> (dev & 63) & 1) == 0) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<BN, CG>::kTotal);
    if (e != cudaSuccess) return e;
    ready.fetch_or(1ull << (dev & 63));
  }
  LaunchCfg lc;
  lc.grid = dim3(CG * grid, a.split, 1);
  lc.block = dim3(kThreads + (WQ ? kWidenExtra : 0));
  lc.smem = Smem<BN, CG>::kTotal;
  lc.stream = stream;
  lc.pdl = true;
  lc.cluster_x = CG;
  lc.cluster_y = a.split;
  return Launch(lc, kernel, ma, mb, a, idesc);
}

// How many clusters of `split` CTAs of this kernel the device holds at once (a GPC takes
// only whole clusters, so this can be well below SMs / split).  Cached per shape of launch.
template <int BN, int CG, typename TOut, int WQ>
int ResidentClusters(int split) {
  static std::mutex mu;
  static int cached[9] = {0};
  std::lock_guard<std::mutex> lock(mu);
  if (cached[split] == 0) {
    auto kernel = gemm_tc_kernel<BN, CG, TOut, WQ>;
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<BN, CG>::kTotal) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(16 * CG, split, 1);
      cfg.blockDim = dim3(kThreads + (WQ ? kWidenExtra : 0));
      cfg.dynamicSmemBytes = Smem<BN, CG>::kTotal;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = CG;
      attr.val.clusterDim.y = split;
      attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) n = 0;
      (void)cudaGetLastError();
    }
    cached[split] = n > 0 ? n : -1;
  }
  return cached[split] > 0 ? cached[split] : 0;
}

template <int BN, int CG, int WQ = kWide>
int ResidentClustersFor(int out_dtype, int split) {
  if (out_dtype == B200_F32) return ResidentClusters<BN, CG, float, WQ>(split);
  if (out_dtype == B200_BF16 || WQ != kWide) return ResidentClusters<BN, CG, __nv_bfloat16, WQ>(split);
  return ResidentClusters<BN, CG, __half, kWide>(split);
}

template <int BN, int CG, int WQ = kWide>
cudaError_t LaunchFor(int out_dtype, const CUtensorMap& ma, const CUtensorMap& mb, const TcArgs& a, uint32_t idesc, int grid,
                      cudaStream_t stream) {
  if (out_dtype == B200_F32) return LaunchTc<BN, CG, float, WQ>(ma, mb, a, idesc, grid, stream);
  if (out_dtype == B200_BF16 || WQ != kWide) return LaunchTc<BN, CG, __nv_bfloat16, WQ>(ma, mb, a, idesc, grid, stream);
  return LaunchTc<BN, CG, __half, kWide>(ma, mb, a, idesc, grid, stream);
}

struct TilePlan {
  int bn = 256, group = 1, split = 1;   // columns of a tile, CTAs of a tile, CTAs along K
  double us = 1e30;
};

// The quantised product: tiles of 128 x 256 or 128 x 128 and the split of K by the same kind of cost model as PlanDense.
constexpr double kWidenStep256 = 0.40, kWidenStep128 = 0.25;   // per 64-deep step of a tile, relative to the epilogues'
template <int WQ>
TilePlan PlanQuantised(const b200_context* ctx, int64_t m, int64_t n, int64_t k, int out_dtype) {
  const int64_t k_iters = k / BK;
  TilePlan p;
  for (int cand : {256, 128}) {
    const double t_iter = cand == 256 ? kWidenStep256 : kWidenStep128, epi = cand == 256 ? 4.0 : 2.3;
    const int64_t tiles = CeilDiv(m, BM) * CeilDiv(n, cand);
    const double whole = static_cast<double>(CeilDiv(tiles, ctx->sm_count)) * std::max(k_iters * t_iter, epi) + epi;
    if (whole < p.us) p.us = whole, p.bn = cand, p.split = 1;
    for (int sp = 2; sp <= 8 && cand == 128; sp *= 2) {
      if (tiles * sp > ctx->sm_count || k_iters / sp < 4) break;
      if (tiles > ResidentClustersFor<128, 1, WQ>(out_dtype, sp)) continue;
      const double cost = static_cast<double>(CeilDiv(k_iters, sp)) * t_iter + 1.5 + epi;
      if (cost < p.us) p.us = cost, p.bn = cand, p.split = sp;
    }
  }
  return p;
}

template <int WQ>
b200_status RunQuantised(b200_context* ctx, cudaStream_t stream, const CUtensorMap& ma, const b200_qmm_params* p, TcArgs a, int out_dtype) {
  const TilePlan plan = PlanQuantised<WQ>(ctx, a.m, a.n, a.k, out_dtype);
  const int bn = plan.bn, split = plan.split;
  a.split = split;
  a.tiles_n = static_cast<int>(CeilDiv(a.n, bn));
  a.stage_bytes = (a.a_rows + bn) * BK * 2;
  a.stages = std::min(kMaxStages, (192 * 1024 - kRawRing) / a.stage_bytes);
  CUtensorMap mb;
  if (!EncodeByteRows(&mb, p->q, p->K * p->bits / 8, p->N, kRawBoxBytes, bn))
    return Stick(ctx, Fail(B200_INTERNAL, "b200_qmm: cuTensorMapEncodeTiled refused the weights"));
  const int64_t tiles = static_cast<int64_t>(a.tiles_m) * a.tiles_n;
  const uint32_t idesc = make_idesc(1, 0, 0, bn, BM);
  const int grid = split > 1 ? static_cast<int>(tiles) : static_cast<int>(std::min<int64_t>(tiles, ctx->sm_count));
  const cudaError_t e = bn == 256 ? LaunchFor<256, 1, WQ>(out_dtype, ma, mb, a, idesc, grid, stream)
                                  : LaunchFor<128, 1, WQ>(out_dtype, ma, mb, a, idesc, grid, stream);
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_qmm (tcgen05) launch: %s", cudaGetErrorString(e)));
  return EndLaunch(ctx, "b200_qmm (tcgen05)");
}

int ARows(int64_t m, int ta) { return ta ? BM : static_cast<int>(std::min<int64_t>(BM, CeilDiv(m, 8) * 8)); }

// Tile shape and K split by a small cost model (microseconds); tiles run in waves over
// the SMs (256 x 256 tiles over pairs of SMs).  When the tiles leave SMs idle, a cluster of
// 2/4/8 CTAs splits one tile's K loop (a serial chain on one SM otherwise) and adds the partial
// tiles through distributed shared memory, for a fixed cost of the cluster barriers and the extra pass.
// straddle: rows of D whose 16-byte pieces are not aligned.
TilePlan PlanDense(const b200_context* ctx, int64_t m, int64_t n, int64_t k, int64_t batch, int ta, int out_dtype, bool straddle) {
  const int64_t k_iters = CeilDiv(k, BK);
  const int a_rows = ARows(m, ta);
  // A k step moves a_rows x 64 of A and bn x 64 of B into an SM at about 0.1 MB/us; the MMAs of a 256-wide
  // tile take 0.27 us.  epi: one tile's epilogue and stores, overlapped with the next tile's loop (measured with K = 64,
  // 8192 x 8192: 43 / 65 / 74 us for the three shapes, about the write limit of HBM; rows whose 128-byte pieces straddle
  // lines take twice as long).
  auto waves_cost = [&](int64_t tiles, int64_t slots, double t_iter, double epi) {
    return static_cast<double>(CeilDiv(tiles, slots)) * std::max(k_iters * t_iter, epi) + epi;
  };
  TilePlan p;
  {
    const int pairs = ResidentClustersFor<256, 2>(out_dtype, 1);
    const int64_t tiles = CeilDiv(m, 2 * BM) * CeilDiv(n, 256) * batch;
    if (pairs > 0 && m > BM) p.us = waves_cost(tiles, pairs, 0.39, straddle ? 6.6 : 3.0), p.group = 2;
  }
  for (int cand : {128, 64}) {
    // 64 columns are 128-byte pieces of B's rows, which stream at about 0.8 of the rate of 256-byte ones
    const double t_iter = (a_rows + cand) * (BK * 2) * (cand == 64 ? 1.25e-5 : 1e-5), epi = cand == 128 ? (straddle ? 4.5 : 2.3) : (straddle ? 3.4 : 1.3);
    const int64_t tiles = CeilDiv(m, BM) * CeilDiv(n, cand) * batch;
    const double whole = waves_cost(tiles, ctx->sm_count, t_iter, epi);
    if (whole < p.us) p.us = whole, p.bn = cand, p.group = 1, p.split = 1;
    for (int sp = 2; sp <= 8; sp *= 2) {
      if (tiles * sp > ctx->sm_count || k_iters / sp < 4) break;
      const int resident = cand == 128 ? ResidentClustersFor<128, 1>(out_dtype, sp) : ResidentClustersFor<64, 1>(out_dtype, sp);
      if (tiles > resident) continue;   // a second wave of clusters would double the time
      const double cost = static_cast<double>(CeilDiv(k_iters, sp)) * t_iter + 1.5 + epi;
      if (cost < p.us) p.us = cost, p.bn = cand, p.group = 1, p.split = sp;
    }
  }
  return p;
}

}  // namespace

namespace b200 {

bool TmaReadable(const b200_operand& x, int64_t batch) {
  // 16-byte aligned bases, row pitches and batch strides that are multiples of 16 bytes
  if (!Aligned(x.ptr, 16) || x.ld % 8 != 0) return false;
  return batch == 1 || x.batch_stride == 0 || (x.batch_stride % 8 == 0 && x.ld > 0 && x.batch_stride % x.ld == 0);
}

bool Tcgen05Supports(const b200_gemm_params* p, const b200_epilogue* epi) {
  (void)epi;
  if (p->a.dtype != B200_BF16 && p->a.dtype != B200_F16) return false;
  if (p->b.dtype != p->a.dtype) return false;
  if (p->k < 1) return false;
  if (Encoder() == nullptr) return false;
  if (!TmaReadable(p->a, p->batch) || !TmaReadable(p->b, p->batch)) return false;
  if (p->m > (1 << 30) || p->n > (1 << 30) || p->k > (1 << 30)) return false;
  return CeilDiv(p->m, BM) * CeilDiv(p->n, 64) * p->batch <= INT32_MAX;
}

b200_status RunTcgen05(b200_context* ctx, cudaStream_t stream, const b200_gemm_params* p, const b200_epilogue* epi) {
  const int ta = p->a.transpose, tb = p->b.transpose;
  const int64_t m = p->m, n = p->n, k = p->k, batch = p->batch;
  const int a_rows = ARows(m, ta);
  const bool straddle = (p->c.ld * DtypeSize(p->c.dtype)) % 16 != 0 || !Aligned(p->c.ptr, 16);
  const TilePlan plan = PlanDense(ctx, m, n, k, batch, ta, p->c.dtype, straddle);
  const int bn = plan.bn, group = plan.group, split = plan.split;
  TcArgs a;
  a.a_rows = a_rows;
  a.stage_bytes = (a_rows + bn / group) * BK * 2;
  a.stages = std::min(kMaxStages, 192 * 1024 / a.stage_bytes);
  a.bcast_a = batch > 1 && p->a.batch_stride == 0;
  a.bcast_b = batch > 1 && p->b.batch_stride == 0;
  const int64_t ba = a.bcast_a ? 1 : batch, bb = a.bcast_b ? 1 : batch;
  CUtensorMap ma, mb;
  bool ok;
  if (!ta) ok = MakeMap(&ma, p->a.dtype, p->a.ptr, k, m, p->a.ld, ba, p->a.batch_stride, BK, a.a_rows);           // A [m][k]
  else ok = MakeMap(&ma, p->a.dtype, p->a.ptr, m, k, p->a.ld, ba, p->a.batch_stride, 64, BK);                     // A stored [k][m]
  if (tb) ok = ok && MakeMap(&mb, p->b.dtype, p->b.ptr, k, n, p->b.ld, bb, p->b.batch_stride, BK, bn / group);     // B stored [n][k]
  else ok = ok && MakeMap(&mb, p->b.dtype, p->b.ptr, n, k, p->b.ld, bb, p->b.batch_stride, 64, BK);               // B [k][n]
  if (!ok) return Stick(ctx, Fail(B200_INTERNAL, "b200_gemm: cuTensorMapEncodeTiled refused the operand layout"));
  a.d = p->c.ptr;
  a.bias = epi->bias;
  a.aux = epi->aux;
  a.m = static_cast<int>(m);
  a.n = static_cast<int>(n);
  a.k = static_cast<int>(k);
  a.ldd = p->c.ld;
  a.sd = batch > 1 ? p->c.batch_stride : 0;
  a.alpha = static_cast<float>(p->alpha);
  a.beta = static_cast<float>(p->beta);
  a.act = epi->act;
  a.ta = ta;
  a.tb = tb;
  a.tiles_m = static_cast<int>(CeilDiv(m, BM * group));
  a.tiles_n = static_cast<int>(CeilDiv(n, bn));
  a.batch = static_cast<int>(batch);
  a.split = split;
  a.status = ctx->dev_status;
  const int64_t tiles = static_cast<int64_t>(a.tiles_m) * a.tiles_n * batch;
  const uint32_t idesc = make_idesc(p->a.dtype == B200_BF16 ? 1 : 0, ta ? 1 : 0, tb ? 0 : 1, bn, BM * group);
  const int out = p->c.dtype;
  cudaError_t e;
  if (group == 2) {
    const int grid = static_cast<int>(std::min<int64_t>(tiles, ResidentClustersFor<256, 2>(out, 1)));
    e = LaunchFor<256, 2>(out, ma, mb, a, idesc, grid, stream);
  } else {
    const int grid = split > 1 ? static_cast<int>(tiles) : static_cast<int>(std::min<int64_t>(tiles, ctx->sm_count));
    if (bn == 128) e = LaunchFor<128, 1>(out, ma, mb, a, idesc, grid, stream);
    else e = LaunchFor<64, 1>(out, ma, mb, a, idesc, grid, stream);
  }
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_gemm (tcgen05) launch: %s", cudaGetErrorString(e)));
  return EndLaunch(ctx, "b200_gemm (tcgen05)");
}

// out = x . dequant(W)^T (+ out, under beta = 1) for quantised weights, widened inside the GEMM: the 16-bit weights
// never exist in memory.  The parameters have passed b200_qmm_validate; false: x does not meet TMA's alignment.
bool QuantisedGemmSupports(const b200_qmm_params* p) {
  const int64_t ldx = p->ldx ? p->ldx : p->K;
  return p->bits != 16 && Encoder() != nullptr && Aligned(p->x, 16) && ldx % 8 == 0 && CeilDiv(p->M, BM) * CeilDiv(p->N, 128) <= INT32_MAX;
}

// Whether dequantising panels of `panel` weight rows and multiplying by those is the faster form: both times estimated (microseconds, cold caches),
// fitted to 144 products of each format, 64 to 8192 rows, at nine shapes between 1024 x 1024 and 24576 x 4096; the estimates are within 7 %
// of what was measured on average, and the form they choose within 0.5 % of the better one (16 % at most).  Dequantising costs per weight, sequential int4 at
// memory speed, the others by a general kernel; the direct form widens the weights again for every 128 rows of x.  Measured, direct / panels (us):
// int4 256 x 4096 -> 4096 31 / 33, 320 rows 41 / 35; 512 x 4096 -> 24576 158 / 167, 640 rows 202 / 169; 256 x 12288 -> 4096 67 / 76, 320 rows
// 108 / 88; int8 per channel 1536 x 4096 -> 4096 118 / 117, 2048 x 4096 -> 24576 652 / 637, 4096 rows 1252 / 955; split-half int4 4096 x 4096 -> 24576 1123 / 1114.
bool PanelsAreFaster(const b200_context* ctx, const b200_qmm_params* p, int64_t panel) {
  const int out = p->epilogue == B200_QMM_OUT_F32_RAW ? B200_F32 : B200_BF16;
  const bool seq = p->bits == 4 && p->nibble_order == 0;
  const TilePlan d = p->bits == 8 ? PlanQuantised<kQ8>(ctx, p->M, p->N, p->K, out)
                                  : (seq ? PlanQuantised<kQ4Seq>(ctx, p->M, p->N, p->K, out) : PlanQuantised<kQ4Half>(ctx, p->M, p->N, p->K, out));
  const int64_t waves = d.split > 1 ? 1 : CeilDiv(CeilDiv(p->M, BM) * CeilDiv(p->N, d.bn), ctx->sm_count);
  const double step = d.bn == 256 ? 0.78 : 0.50, epi = d.bn == 256 ? 4.0 : 2.3;
  const double direct = waves * std::max(CeilDiv(p->K / BK, d.split) * step, 2.0) + epi + 8.0 + (d.split > 1 ? 4.5 : 0.0);
  double gemm = 0.0;
  for (int64_t r = 0; r < p->N; r += panel) gemm += PlanDense(ctx, p->M, std::min(panel, p->N - r), p->K, 1, 0, out, false).us;
  const double weights = static_cast<double>(p->N) * p->K * 1e-6 * (seq ? 0.52 : (p->bits == 4 ? 5.67 : 3.82));
  const double panels = 0.82 * gemm + weights + 12.5 * CeilDiv(p->N, panel);
  return panels < direct;
}

b200_status RunQuantisedGemm(b200_context* ctx, cudaStream_t stream, const b200_qmm_params* p) {
  b200_status s = BeginLaunch(ctx);
  if (s != B200_OK) return s;
  TcArgs a = {};
  const bool f32_out = p->epilogue == B200_QMM_OUT_F32_RAW;
  a.a_rows = static_cast<int>(std::min<int64_t>(BM, CeilDiv(p->M, 8) * 8));
  CUtensorMap ma;
  const int64_t ldx = p->ldx ? p->ldx : p->K;
  if (!MakeMap(&ma, B200_BF16, p->x, p->K, p->M, ldx, 1, 0, BK, a.a_rows))
    return Stick(ctx, Fail(B200_INTERNAL, "b200_qmm: cuTensorMapEncodeTiled refused x"));
  a.d = p->out;
  a.m = static_cast<int>(p->M);
  a.n = static_cast<int>(p->N);
  a.k = static_cast<int>(p->K);
  a.ldd = p->ldo ? p->ldo : p->N;
  a.alpha = 1.0f;
  a.beta = p->epilogue == B200_QMM_ADD_RESIDUAL ? 1.0f : 0.0f;
  a.tb = 1;
  a.tiles_m = static_cast<int>(CeilDiv(p->M, BM));
  a.batch = 1;
  a.scale = static_cast<const __nv_bfloat16*>(p->scale);
  a.offset = static_cast<const __nv_bfloat16*>(p->bias);
  a.scale_ld = static_cast<int>(p->K / p->group);
  a.scale_vec = a.scale_ld % 8 == 0 && Aligned(p->scale, 16) && (p->bits != 4 || Aligned(p->bias, 16));
  a.status = ctx->dev_status;
  const int out = f32_out ? B200_F32 : B200_BF16;
  if (p->bits == 8) return RunQuantised<kQ8>(ctx, stream, ma, p, a, out);
  return p->nibble_order == 0 ? RunQuantised<kQ4Seq>(ctx, stream, ma, p, a, out) : RunQuantised<kQ4Half>(ctx, stream, ma, p, a, out);
}

}  // namespace b200
