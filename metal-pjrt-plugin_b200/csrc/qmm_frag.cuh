// How the quantised-matmul kernels on mma.sync read weights and order the inputs of a group (qmm.cu, qmm_mid.cu).
#pragma once
#include "common.cuh"

namespace b200 {
namespace qfrag {

constexpr int kGroupK = 64;

enum Format { kInt4Seq = 0, kInt4Half = 1, kInt8 = 2, kBf16 = 3 };

template <int FMT>
struct Fmt {
  static constexpr int kBits = FMT == kInt8 ? 8 : (FMT == kBf16 ? 16 : 4);
  static constexpr int kPad = kBits == 4 ? 32 : 64;           // keeps the quad reads conflict-free
  static constexpr int kGroupBytes = kGroupK * kBits / 8;     // 32 / 64 / 128
};

// Which input (0..63) of a group sits in half `h` of A register `r` (0..7) of
// quad thread `t`.  x is staged in shared memory in exactly this order.
template <int FMT>
__device__ __forceinline__ int kmap(int t, int r, int h) {
  if (FMT == kInt4Seq) return 16 * t + 8 * (r >> 2) + (r & 3) + 4 * h;
  if (FMT == kInt4Half) {
    const int rr = r & 3;
    return 8 * t + 4 * (r >> 2) + (rr >> 1) + 2 * h + 32 * (rr & 1);
  }
  if (FMT == kInt8) return 16 * t + 2 * r + h;
  return 32 * (r >> 2) + 8 * t + 2 * (r & 3) + h;  // bf16: two 16-byte pieces per thread
}

__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// v >> log2(2^32 / pow2).  (Written as a multiply-high by a power of two it would run on the FMA
// pipe, but that instruction measures 4-6 issue cycles per warp on this GPU against about one
// for a plain shift.)
__device__ __forceinline__ uint32_t mulhi_shift(uint32_t v, uint32_t pow2) { return v >> (__clz(pow2) + 1); }

// One thread's raw share of a group of one weight row (int4: 8 bytes, int8: 16, bf16: 16 + 16) as 8 bf16x2 registers.
template <int FMT>
__device__ __forceinline__ void widen(const uint4& w0, const uint4& w1, uint32_t (&a)[8]) {
  if (FMT == kInt4Seq || FMT == kInt4Half) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      a[r] = lop3_and_or(r == 0 ? w0.x : mulhi_shift(w0.x, 1u << (32 - 4 * r)), 0x000f000fu, 0x43004300u);  // bf16 (128 + q)
      a[4 + r] = lop3_and_or(r == 0 ? w0.y : mulhi_shift(w0.y, 1u << (32 - 4 * r)), 0x000f000fu, 0x43004300u);
    }
  } else if (FMT == kInt8) {
    const uint32_t words[4] = {w0.x, w0.y, w0.z, w0.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t u = words[j] ^ 0x80808080u;  // q + 128 in every byte
      // 2^23 + (q + 128) as f32, minus (2^23 + 128): q exactly, no int->float unit
      const float f0 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7650)) - 8388736.0f;
      const float f1 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7651)) - 8388736.0f;
      const float f2 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7652)) - 8388736.0f;
      const float f3 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7653)) - 8388736.0f;
      a[2 * j] = pack_bf16(f0, f1);
      a[2 * j + 1] = pack_bf16(f2, f3);
    }
  } else {
    a[0] = w0.x; a[1] = w0.y; a[2] = w0.z; a[3] = w0.w;
    a[4] = w1.x; a[5] = w1.y; a[6] = w1.z; a[7] = w1.w;
  }
}

}  // namespace qfrag
}  // namespace b200
