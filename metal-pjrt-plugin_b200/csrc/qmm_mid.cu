// Weight-only quantised matmul for 9 to 32 rows of x (batched decoding):
//   out[M, N] = x[M, K] . dequant(W)[N, K]^T, the arithmetic of qmm.cu (f32 sums per group of 64, scale and offset in f32).
//
// What bounds it: issue slots.  Reading the weights once takes 9 us for 24576 x 4096 int4 (HBM); widening, MMAs and scaling
// are about 290 instructions per warp for 32 rows x 64 inputs at 32 rows of x, 14 us if no slot is lost.
//   * A CTA owns a slice of K, whose x it stages once.  From then on its warps are on their own: a warp takes tiles of 32
//     weight rows of that slice, fetches them itself (boxes of 32 rows x 128 bytes, TMA with 128-byte swizzle, into a ring of
//     its own) and keeps the tile's sums in registers, so no barrier is met and no partial tile changes hands.  (Eight warps
//     that shared a 64-row tile along K lost half of the time to the barriers of each tile and to too few warps.)
//   * 32 rows per warp, because a fragment of x read for 16 rows only costs shared memory 1.5 times what HBM takes.
//   * K slices add up in a scratch buffer [slice][N][rows]; a second small kernel sums them in order and stores.
// Measured, 32 rows, before and after: int8 per channel 12288 -> 4096 70 -> 29 us; int4 4096 -> 24576 94 -> 55 us.
#include <cuda.h>

#include <algorithm>

#include "qmm_frag.cuh"
#include "qmm_mid.cuh"

using namespace b200;
using namespace b200::qfrag;

namespace b200 {
// gemm_tcgen05.cu: a 2-D map over `rows` rows of bytes, boxes of box_bytes x box_rows, swizzled over box_bytes
bool EncodeByteRows(CUtensorMap* map, const void* base, int64_t row_bytes, int64_t rows, int box_bytes, int box_rows);
}  // namespace b200

namespace {

constexpr int kMaxWarps = 16;
constexpr int kRows = 32;                   // weight rows of a warp's tile
constexpr int kMaxStages = 8;
constexpr int kBoxBytes = kRows * 128;
constexpr int kStaticSmem = 2048;           // the barriers

struct MidArgs {
  const __nv_bfloat16* scale;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* x;
  const __nv_bfloat16* residual;
  void* out;
  float* scratch;     // [slices][N][8 MB], or null: one slice
  int M, N, K;
  int ldx, ldo;
  int tiles;
  int groups;         // of a slice (the last may hold fewer); slices lie along grid.y
  int stages;
  int scale_ld;
  int x_vec, scale_vec;
  int prologue, epilogue;
  int slices;
  int weights_settled;   // see b200::QmmCaller
  int* status;
};

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&lo)[8], const uint32_t (&hi)[8], int i, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(lo[2 * i]), "r"(hi[2 * i]), "r"(lo[2 * i + 1]), "r"(hi[2 * i + 1]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void tma_rows(void* dst, const CUtensorMap* map, int byte, int row, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(byte), "r"(row), "r"(smem_u32(bar))
      : "memory");
}

// One output element from its sum over K.
__device__ __forceinline__ void store_output(const MidArgs& a, bool per_channel, float v, int m, int n) {
  if (per_channel) v *= ldg_bf16(a.scale + n);
  const size_t o = static_cast<size_t>(m) * a.ldo + n;
  if (a.epilogue == B200_QMM_OUT_F32_RAW) static_cast<float*>(a.out)[o] = v;
  else if (a.epilogue == B200_QMM_OUT_F32) static_cast<float*>(a.out)[o] = bf16_round(v);
  else if (a.epilogue == B200_QMM_ADD_RESIDUAL)
    static_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16_rn(__bfloat162float(a.residual[o]) + bf16_round(v));
  else static_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16_rn(v);
}

// FMT: storage format; MB: batch blocks of 8; GROUPED: a scale (and offset) per 64 inputs, else one per row at the end.
template <int FMT, int MB, bool GROUPED>
__global__ void __launch_bounds__(kMaxWarps * 32, 1) qmm_mid_kernel(const __grid_constant__ CUtensorMap map, const MidArgs a) {
  using F = Fmt<FMT>;
  constexpr int MP = 8 * MB;
  constexpr int kPerBox = 128 / F::kGroupBytes;   // groups of a row in a box
  extern __shared__ uint8_t smem_raw[];
  uint8_t* rings = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t bars[kMaxWarps][kMaxStages];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int threads = static_cast<int>(blockDim.x), warps = threads / 32;
  const int g = lane >> 2, t = lane & 3;
  uint8_t* ring = rings + warp * a.stages * kBoxBytes;
  uint4* xs = reinterpret_cast<uint4*>(rings + warps * a.stages * kBoxBytes);     // [groups][2][MP][4], in register order
  float* xsum = reinterpret_cast<float*>(xs + a.groups * 2 * MP * 4);             // [groups][MP]
  uint32_t* so = reinterpret_cast<uint32_t*>(xsum + a.groups * MP) + warp * a.groups * kRows;   // [groups][kRows] (scale, offset)
  const int g_begin = static_cast<int>(blockIdx.y) * a.groups;
  const int groups = min(a.groups, a.K / kGroupK - g_begin);
  const int boxes = (groups + kPerBox - 1) / kPerBox;
  const int tile0 = static_cast<int>(blockIdx.x) * warps + warp, tile_step = static_cast<int>(gridDim.x) * warps;

  if (lane == 0) {
    for (int s = 0; s < a.stages; ++s) mbar_init(&bars[warp][s], 1);
    mbar_fence_init();
  }
  __syncwarp();
  // The warp's boxes of all its tiles as one sequence; fetches run a whole ring ahead.  Weights that no earlier kernel can
  // still be storing are requested before the wait below.
  if (!a.weights_settled) pdl_wait();
  int f_tile = tile0, f_box = 0, f_slot = 0;
  auto fetch = [&]() {
    if (f_tile >= a.tiles) return;
    if (lane == 0) {
      mbar_expect_tx(&bars[warp][f_slot], kBoxBytes);
      tma_rows(ring + f_slot * kBoxBytes, &map, g_begin * F::kGroupBytes + f_box * 128, f_tile * kRows, &bars[warp][f_slot]);
    }
    if (++f_box == boxes) f_box = 0, f_tile += tile_step;
    if (++f_slot == a.stages) f_slot = 0;
  };
  for (int i = 0; i < a.stages; ++i) fetch();
  // Scales and offsets of the warp's tile: lane r takes row r.
  const bool vec = a.scale_vec && groups % 4 == 0;
  auto scales = [&](int tile) {
    if (!GROUPED || tile >= a.tiles) return;
    const size_t o = static_cast<size_t>(min(tile * kRows + lane, a.N - 1)) * a.scale_ld + g_begin;
    if (vec) {
#pragma unroll 4
      for (int c = 0; c < groups; c += 4) {
        const uint2 sv = __ldg(reinterpret_cast<const uint2*>(a.scale + o + c));
        const uint2 bv = F::kBits == 4 ? __ldg(reinterpret_cast<const uint2*>(a.bias + o + c)) : make_uint2(0, 0);
        so[c * kRows + lane] = __byte_perm(sv.x, bv.x, 0x5410);
        so[(c + 1) * kRows + lane] = __byte_perm(sv.x, bv.x, 0x7632);
        so[(c + 2) * kRows + lane] = __byte_perm(sv.y, bv.y, 0x5410);
        so[(c + 3) * kRows + lane] = __byte_perm(sv.y, bv.y, 0x7632);
      }
    } else {
      for (int c = 0; c < groups; ++c)
        so[c * kRows + lane] = __ldg(reinterpret_cast<const uint16_t*>(a.scale) + o + c) |
                               (F::kBits == 4 ? static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(a.bias) + o + c)) << 16 : 0u);
    }
  };
  scales(tile0);
  pdl_launch_dependents();
  pdl_wait();   // x (and the residual) come from the previous kernel

  // ---- x of the slice in register order: unit (m, group, t) = 16 inputs = two runs of 8 (or one of 16); rows M .. MP - 1 zero
  {
    constexpr bool kOneRun = FMT == kInt4Seq || FMT == kInt8;
    auto load_run = [&](const __nv_bfloat16* p) {
      if (a.x_vec) return __ldg(reinterpret_cast<const uint4*>(p));
      const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
      return make_uint4(__ldg(h) | (static_cast<uint32_t>(__ldg(h + 1)) << 16), __ldg(h + 2) | (static_cast<uint32_t>(__ldg(h + 3)) << 16),
                        __ldg(h + 4) | (static_cast<uint32_t>(__ldg(h + 5)) << 16), __ldg(h + 6) | (static_cast<uint32_t>(__ldg(h + 7)) << 16));
    };
    auto unpack = [&](const uint4& raw, float* dst) {
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        dst[2 * j] = bf16_lo(w[j]);
        dst[2 * j + 1] = bf16_hi(w[j]);
      }
    };
    const bool silu = a.prologue == B200_QMM_PRO_SILU_MUL;   // x is [M, 2K]: gate, then up
    const int units = groups * MP * 4;   // a multiple of the warp size
    constexpr int U = 4;                 // units whose loads are in flight together: their latency is what this part costs
    for (int u0 = tid; u0 < units; u0 += U * threads) {
      uint4 raw[U][2], up[U][2];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int u = u0 + i * threads;
        const int ut = u & 3, um = (u >> 2) % MP, ug = (u >> 2) / MP;
        raw[i][0] = raw[i][1] = up[i][0] = up[i][1] = make_uint4(0, 0, 0, 0);
        if (u < units && um < a.M) {
          const __nv_bfloat16* xr = a.x + static_cast<size_t>(um) * a.ldx + (g_begin + ug) * kGroupK;
          const int run0 = kOneRun ? 16 * ut : 8 * ut, run1 = kOneRun ? 16 * ut + 8 : 32 + 8 * ut;
          raw[i][0] = load_run(xr + run0);
          raw[i][1] = load_run(xr + run1);
          if (silu) {
            up[i][0] = load_run(xr + a.K + run0);
            up[i][1] = load_run(xr + a.K + run1);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int u = u0 + i * threads;
        if (u >= units) break;
        const int ut = u & 3, um = (u >> 2) % MP, ug = (u >> 2) / MP;
        float e[16], sum = 0.0f;
        unpack(raw[i][0], e);
        unpack(raw[i][1], e + 8);
        if (silu) {
          float w[16];
          unpack(up[i][0], w);
          unpack(up[i][1], w + 8);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float sig = bf16_round(__fdividef(1.0f, 1.0f + __expf(-e[j])));   // (as in qmm.cu)
            e[j] = bf16_round(bf16_round(e[j] * sig) * w[j]);
          }
        }
        uint32_t regs[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int k0 = kmap<FMT>(0, r, 0), k1 = kmap<FMT>(0, r, 1);
          const int l0 = kOneRun ? k0 : (k0 & 7) + 8 * (k0 >> 5), l1 = kOneRun ? k1 : (k1 & 7) + 8 * (k1 >> 5);
          regs[r] = pack_bf16(e[l0], e[l1]);
          sum += e[l0] + e[l1];
        }
        xs[((ug * 2 + 0) * MP + um) * 4 + ut] = make_uint4(regs[0], regs[1], regs[2], regs[3]);
        xs[((ug * 2 + 1) * MP + um) * 4 + ut] = make_uint4(regs[4], regs[5], regs[6], regs[7]);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (ut == 0) xsum[ug * MP + um] = sum;
      }
    }
  }
  __syncthreads();   // the last one: from here on the warps are independent

  // this lane's piece of group gb of a box row (swizzled by the row, which is g modulo 8)
  const uint8_t* lane_base = ring + g * 128;
  auto piece = [&](int gb) { return ((gb * F::kGroupBytes) | (t * (F::kBits == 4 ? 8 : 16))) ^ (g << 4); };

  int s = 0;
  uint32_t parity = 0;
  int flying = 0;   // a bounded wait gave up: the boxes that are still to land
  for (int tile = tile0; tile < a.tiles && flying == 0; tile += tile_step) {
    const int n0 = tile * kRows;
    float acc[2][MB][4];
#pragma unroll
    for (int rt = 0; rt < 2; ++rt)
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[rt][mb][i] = 0.0f;
    for (int bx = 0; bx < boxes; ++bx) {
      if (!mbar_wait_bounded(&bars[warp][s], parity)) {
        report_timeout(a.status, 200 + s);
        flying = min(a.stages, boxes - bx + boxes * ((a.tiles - 1 - tile) / tile_step));   // (fetches run a whole ring ahead)
        break;
      }
#pragma unroll
      for (int gb = 0; gb < kPerBox; ++gb) {
        const int gl = bx * kPerBox + gb;
        if (gl < groups) {
          uint32_t w[4][8];   // rows g, g + 8, g + 16, g + 24
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint8_t* p = lane_base + s * kBoxBytes + q * 8 * 128;
            if (F::kBits == 4) {
              const uint2 v = *reinterpret_cast<const uint2*>(p + piece(gb));
              widen<FMT>(make_uint4(v.x, v.y, 0, 0), make_uint4(0, 0, 0, 0), w[q]);
            } else {
              const uint4 v = *reinterpret_cast<const uint4*>(p + piece(gb));
              widen<FMT>(v, F::kBits == 16 ? *reinterpret_cast<const uint4*>(p + (piece(gb) ^ 64)) : v, w[q]);
            }
          }
          float2 sq[4];
          if (GROUPED) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t v = so[gl * kRows + g + 8 * q];
              // int4 registers hold 128 + q: the 128 is folded into the offset
              sq[q] = make_float2(bf16_lo(v), F::kBits == 4 ? fmaf(-128.0f, bf16_lo(v), bf16_hi(v)) : 0.0f);
            }
          }
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) {
            const uint4 v0 = xs[((gl * 2 + 0) * MP + mb * 8 + g) * 4 + t], v1 = xs[((gl * 2 + 1) * MP + mb * 8 + g) * 4 + t];
            const uint32_t xf[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
            if (GROUPED) {
              float d[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
              for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int rt = 0; rt < 2; ++rt) mma(d[rt], w[2 * rt], w[2 * rt + 1], i, xf[2 * i], xf[2 * i + 1]);
              const float2 xq = F::kBits == 4 ? *reinterpret_cast<const float2*>(&xsum[gl * MP + mb * 8 + 2 * t]) : make_float2(0.0f, 0.0f);
#pragma unroll
              for (int rt = 0; rt < 2; ++rt) {
                const float2 p0 = sq[2 * rt], p1 = sq[2 * rt + 1];
                if (F::kBits == 4) {
                  acc[rt][mb][0] = fmaf(p0.x, d[rt][0], fmaf(p0.y, xq.x, acc[rt][mb][0]));
                  acc[rt][mb][1] = fmaf(p0.x, d[rt][1], fmaf(p0.y, xq.y, acc[rt][mb][1]));
                  acc[rt][mb][2] = fmaf(p1.x, d[rt][2], fmaf(p1.y, xq.x, acc[rt][mb][2]));
                  acc[rt][mb][3] = fmaf(p1.x, d[rt][3], fmaf(p1.y, xq.y, acc[rt][mb][3]));
                } else {
                  acc[rt][mb][0] = fmaf(p0.x, d[rt][0], acc[rt][mb][0]);
                  acc[rt][mb][1] = fmaf(p0.x, d[rt][1], acc[rt][mb][1]);
                  acc[rt][mb][2] = fmaf(p1.x, d[rt][2], acc[rt][mb][2]);
                  acc[rt][mb][3] = fmaf(p1.x, d[rt][3], acc[rt][mb][3]);
                }
              }
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int rt = 0; rt < 2; ++rt) mma(acc[rt][mb], w[2 * rt], w[2 * rt + 1], i, xf[2 * i], xf[2 * i + 1]);
            }
          }
        }
      }
      __syncwarp();   // every lane has read the box: its slot is fetched into again
      fetch();
      if (++s == a.stages) s = 0, parity ^= 1;
    }
    if (flying > 0) break;
#pragma unroll
    for (int rt = 0; rt < 2; ++rt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = n0 + rt * 16 + h * 8 + g;
        if (n >= a.N) continue;
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) {
          const int m = mb * 8 + 2 * t;
          const float v0 = acc[rt][mb][2 * h], v1 = acc[rt][mb][2 * h + 1];
          if (a.scratch != nullptr) {
            *reinterpret_cast<float2*>(a.scratch + (static_cast<size_t>(blockIdx.y) * a.N + n) * MP + m) = make_float2(v0, v1);
          } else {
            if (m < a.M) store_output(a, !GROUPED && F::kBits != 16, v0, m, n);
            if (m + 1 < a.M) store_output(a, !GROUPED && F::kBits != 16, v1, m + 1, n);
          }
        }
      }
    if (GROUPED) {
      __syncwarp();
      scales(tile + tile_step);
      __syncwarp();
    }
  }
  // No box may land in this CTA's shared memory once it is gone (one more wait that runs out ends this).
  for (; flying > 0; --flying) {
    if (!mbar_wait_bounded(&bars[warp][s], parity)) break;
    if (++s == a.stages) s = 0, parity ^= 1;
  }
}

// The slices' sums in order, and the epilogue: 32 weight rows per CTA, turned in shared memory so that rows of x are
// written along n.
template <int MP>
__global__ void __launch_bounds__(256) qmm_mid_sum_kernel(const MidArgs a, const int per_channel) {
  __shared__ float tile[32][MP + 1];
  pdl_wait();
  pdl_launch_dependents();
  const int n0 = blockIdx.x * 32;
  for (int i = threadIdx.x; i < 32 * (MP / 4); i += 256) {
    const int r = i / (MP / 4), c = i % (MP / 4) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (n0 + r < a.N) {
      const float* p = a.scratch + static_cast<size_t>(n0 + r) * MP + c;
      const size_t slice = static_cast<size_t>(a.N) * MP;
#pragma unroll 8
      for (int sl = 0; sl < a.slices; ++sl) {
        const float4 q = *reinterpret_cast<const float4*>(p + sl * slice);
        v.x += q.x, v.y += q.y, v.z += q.z, v.w += q.w;
      }
    }
    tile[r][c] = v.x, tile[r][c + 1] = v.y, tile[r][c + 2] = v.z, tile[r][c + 3] = v.w;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * a.M; i += 256) {
    const int r = i % 32, m = i / 32;
    if (n0 + r < a.N) store_output(a, per_channel != 0, tile[r][m], m, n0 + r);
  }
}

struct MidPlan {
  int groups = 0, slices = 0, grid_x = 0, warps = 0, stages = 0;
  size_t smem = 0;
};

// The slices of K and the warps of a CTA (16, or fewer where that spreads a small matrix over more SMs): a slice's x and
// the scales stay in shared memory beside two boxes or more per warp, and the time of the warp with the most tiles is what
// counts.  The microseconds are measured: a group of a tile costs a latency, or its share of the SM's issue slots.
bool MakeMidPlan(int bits, bool grouped, int mb, int64_t N, int64_t K, int sm_count, int max_smem, MidPlan* out) {
  const int total = static_cast<int>(K / kGroupK), tiles = static_cast<int>(CeilDiv(N, kRows)), mp = 8 * mb;
  const int per_box = 128 * 8 / (kGroupK * bits);
  double best = 1e30;
  for (int warps = kMaxWarps; warps >= 4; warps /= 2) {
    const double per_group = std::max({0.2 + 0.05 * mb, 0.014 * mb * warps, 0.0027 * bits * warps});
    int last = 0;
    for (int want = 1; want <= total && want <= sm_count; ++want) {
      const int groups = static_cast<int>(CeilDiv(CeilDiv(total, want), per_box)) * per_box;
      if (groups == last) continue;
      last = groups;
      const int slices = static_cast<int>(CeilDiv(total, groups));
      const size_t fixed = 1024 + static_cast<size_t>(groups) * (mp * 132 + (grouped ? warps * kRows * 4 : 0));
      if (static_cast<size_t>(groups) * mp * 128 > 96 * 1024 || fixed + static_cast<size_t>(2 * warps) * kBoxBytes > static_cast<size_t>(max_smem)) continue;
      const int grid_x = static_cast<int>(std::min<int64_t>(CeilDiv(tiles, warps), std::max(1, sm_count / slices)));
      const double cost = static_cast<double>(CeilDiv(tiles, grid_x * warps)) * (groups * per_group + 1.0) + 0.16 * mb * groups / warps +
                          (slices > 1 ? 2.5 + static_cast<double>(slices) * N * mp * 8 / 5e6 : 0.0);
      if (cost < best) {
        best = cost;
        out->groups = groups;
        out->slices = slices;
        out->grid_x = grid_x;
        out->warps = warps;
        const int units = static_cast<int>(CeilDiv(std::min(groups, total), per_box) * CeilDiv(tiles, grid_x * warps));
        out->stages = std::min({kMaxStages, static_cast<int>((max_smem - fixed) / (static_cast<size_t>(warps) * kBoxBytes)), std::max(units, 2)});
        out->smem = fixed + static_cast<size_t>(out->stages) * warps * kBoxBytes;
      }
    }
  }
  return best < 1e30;
}

size_t PlanScratch(const MidPlan& pl, int mb, int64_t N) { return pl.slices > 1 ? static_cast<size_t>(pl.slices) * N * mb * 8 : 0; }

template <int FMT, int MB, bool GROUPED>
cudaError_t LaunchMid(const MidPlan& pl, const CUtensorMap& map, const MidArgs& a, int max_smem, cudaStream_t stream) {
  auto kernel = qmm_mid_kernel<FMT, MB, GROUPED>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  if (e != cudaSuccess) return e;
  LaunchCfg lc;
  lc.grid = dim3(pl.grid_x, pl.slices);
  lc.block = dim3(pl.warps * 32);
  lc.smem = pl.smem;
  lc.stream = stream;
  lc.pdl = true;
  e = Launch(lc, kernel, map, a);
  if (e != cudaSuccess || a.scratch == nullptr) return e;
  lc.grid = dim3(static_cast<unsigned>(CeilDiv(a.N, 32)));
  lc.block = dim3(256);
  lc.smem = 0;
  return Launch(lc, qmm_mid_sum_kernel<8 * MB>, a, static_cast<int>(!GROUPED && Fmt<FMT>::kBits != 16));
}

template <int FMT, bool GROUPED>
cudaError_t LaunchBatch(int mb, const MidPlan& pl, const CUtensorMap& map, const MidArgs& a, int max_smem, cudaStream_t stream) {
  if (mb == 2) return LaunchMid<FMT, 2, GROUPED>(pl, map, a, max_smem, stream);
  return LaunchMid<FMT, 4, GROUPED>(pl, map, a, max_smem, stream);
}

}  // namespace

namespace b200 {

b200_status QmmMidPlan(const b200_qmm_params* p, int sm_count, int max_smem, int* rows, int* slices, int* mb) {
  MidPlan pl;
  *mb = p->M <= 16 ? 2 : 4;
  if (!MakeMidPlan(p->bits, p->bits == 4 || (p->bits == 8 && p->group == 64), *mb, p->N, p->K, sm_count, max_smem - kStaticSmem, &pl))
    return Fail(B200_UNIMPLEMENTED, "b200_qmm: M=%lld K=%lld does not fit shared memory", static_cast<long long>(p->M), static_cast<long long>(p->K));
  *rows = kRows;
  *slices = pl.slices;
  return B200_OK;
}

size_t QmmMidScratchFloats(const b200_context* ctx, int bits, int group, int64_t M, int64_t N, int64_t K) {
  const int mb = M <= 16 ? 2 : 4;
  MidPlan pl;
  if (!MakeMidPlan(bits, bits == 4 || (bits == 8 && group == 64), mb, N, K, ctx->sm_count, ctx->max_smem_optin - kStaticSmem, &pl)) return 0;
  return PlanScratch(pl, mb, N);
}

b200_status QmmMidRun(b200_context* ctx, cudaStream_t stream, const b200_qmm_params* p, const QmmCaller& caller) {
  const int mb = p->M <= 16 ? 2 : 4;
  const bool grouped = p->bits == 4 || (p->bits == 8 && p->group == 64);
  const int max_smem = ctx->max_smem_optin - kStaticSmem;
  MidPlan pl;
  if (!MakeMidPlan(p->bits, grouped, mb, p->N, p->K, ctx->sm_count, max_smem, &pl))
    return Fail(B200_UNIMPLEMENTED, "b200_qmm: M=%lld K=%lld does not fit shared memory", static_cast<long long>(p->M), static_cast<long long>(p->K));
  CUtensorMap map;
  if (!EncodeByteRows(&map, p->q, p->K * p->bits / 8, p->N, 128, kRows))
    return Stick(ctx, Fail(B200_INTERNAL, "b200_qmm: cuTensorMapEncodeTiled refused the weights"));
  MidArgs a = {};
  a.scale = static_cast<const __nv_bfloat16*>(p->scale);
  a.bias = static_cast<const __nv_bfloat16*>(p->bias);
  a.x = static_cast<const __nv_bfloat16*>(p->x);
  a.residual = static_cast<const __nv_bfloat16*>(p->residual);
  a.out = p->out;
  a.M = static_cast<int>(p->M);
  a.N = static_cast<int>(p->N);
  a.K = static_cast<int>(p->K);
  a.ldx = static_cast<int>(p->ldx ? p->ldx : (p->prologue == B200_QMM_PRO_SILU_MUL ? 2 * p->K : p->K));
  a.ldo = static_cast<int>(p->ldo ? p->ldo : p->N);
  a.tiles = static_cast<int>(CeilDiv(p->N, kRows));
  a.groups = pl.groups;
  a.stages = pl.stages;
  a.slices = pl.slices;
  a.scale_ld = p->bits == 16 ? 0 : static_cast<int>(p->K / p->group);
  a.x_vec = Aligned(p->x, 16) && a.ldx % 8 == 0;
  a.scale_vec = grouped && a.scale_ld % 4 == 0 && pl.groups % 4 == 0 && Aligned(p->scale, 8) && (p->bits != 4 || Aligned(p->bias, 8));   // 8-byte loads
  a.prologue = p->prologue;
  a.epilogue = p->epilogue;
  a.weights_settled = caller.weights_settled;
  a.status = ctx->dev_status;
  void* scratch = nullptr;   // to be given back
  if (pl.slices > 1) {
    const size_t floats = PlanScratch(pl, mb, p->N);
    if (caller.scratch != nullptr) {
      if (floats > caller.scratch_floats) return Fail(B200_RESOURCE_EXHAUSTED, "b200_qmm: %zu floats of scratch, %zu needed", caller.scratch_floats, floats);
      a.scratch = caller.scratch;
    } else {
      // stream-ordered memory of the context's pool (an allocation node under capture)
      const cudaError_t e = cudaMallocFromPoolAsync(&scratch, floats * sizeof(float), ctx->pool, stream);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return Fail(B200_RESOURCE_EXHAUSTED, "b200_qmm: scratch for the slices of K: %s", cudaGetErrorString(e));
      }
      a.scratch = static_cast<float*>(scratch);
    }
  }
  cudaError_t e;
  if (p->bits == 4 && p->nibble_order == 0) e = LaunchBatch<kInt4Seq, true>(mb, pl, map, a, max_smem, stream);
  else if (p->bits == 4) e = LaunchBatch<kInt4Half, true>(mb, pl, map, a, max_smem, stream);
  else if (p->bits == 8 && grouped) e = LaunchBatch<kInt8, true>(mb, pl, map, a, max_smem, stream);
  else if (p->bits == 8) e = LaunchBatch<kInt8, false>(mb, pl, map, a, max_smem, stream);
  else e = LaunchBatch<kBf16, false>(mb, pl, map, a, max_smem, stream);
  if (scratch != nullptr) cudaFreeAsync(scratch, stream);
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_qmm launch: %s", cudaGetErrorString(e)));
  return EndLaunch(ctx, "b200_qmm", pl.slices > 1 ? 2 : 1);
}

}  // namespace b200
