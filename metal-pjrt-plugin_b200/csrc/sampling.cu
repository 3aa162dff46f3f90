// Next-token sampling on the device (≙ sample, examples/llm/qwen3.py:395-418): greedy,
// temperature, top-k and top-p (nucleus) over the top-k candidates, so that a decode loop
// reads back 4 bytes per sequence instead of a row of 151936 logits.
//
// The reference draws with jax.random.categorical (Gumbel noise from a threefry key), which
// cannot be reproduced bit for bit outside JAX.  Here the caller supplies one uniform number
// u in [0, 1) per row and the draw is the inverse CDF: the first candidate whose cumulative
// probability exceeds u * (total kept probability).  Candidates are ordered as the reference
// orders them: all logits in vocabulary order when neither top-k nor top-p is set
// (categorical over the row), else the top-k values in descending order, ties by lower
// index first (jax.lax.top_k), of which top-p keeps the smallest prefix whose probability
// reaches top_p (always at least one).
//
// Bound by latency: one pass over the logits is 3 us of HBM for 32 rows of 151936, and one CTA per row
// (which re-read its row from L2 six to ten times and met on single histogram counters) took 158 us for that.
// A cluster of CTAs takes a row (many or short rows: one CTA each, see RowPerCta).  Each reads its share once into shared
// memory, where all later passes run; the CTAs exchange maxima, thresholds and candidates by stores into each other's shared memory.
//   top-k   every thread's maximum is one of kT x cluster groups, so the k-th largest maximum is a lower bound
//           of the k-th largest logit, and hardly more than k logits reach it: those are gathered in the first
//           CTA and sorted there.  The bound is found by bisection over the maxima, which every CTA holds.
//           More than kMaxCand candidates (long runs of equal logits) take an exact radix selection instead.
//   all     the row's exponentials are formed in place; 1024 contiguous chunks are summed one thread each, in
//           the order in which the draw then walks the chosen chunk.
// Against one CTA per row: 32 x 151936, top-k 20 + top-p 158 -> 17 us, whole row 67 -> 20; 32 x 32000, whole row 28 -> 10.
#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;
using namespace b200;

namespace {

constexpr int kT = 1024;
constexpr int kMaxTopK = 1024;
constexpr int kMaxCand = 2048;
constexpr int kMaxCluster = 8;

struct SampleArgs {
  const float* logits;
  const float* uniform;
  int32_t* out;
  int V;
  int chunk;               // ceil(V / kT): the contiguous run of logits one thread sums; a CTA's share is kT / cluster of them
  int stash;               // the share fits shared memory
  float inv_temperature;   // 0: greedy
  int top_k;
  float top_p;
};

// What both kernels use.
struct Common {
  unsigned long long cand[kMaxCand];
  float parts[kT];                     // cluster: sums of all chunks; later the cumulative probabilities
  float s_val[kT / 32];
  int s_idx[kT / 32];
  float warp_tot[kT / 32];
  unsigned hist[256];
  unsigned prefix, krem, count, choice;
};
struct Shared : Common {
  unsigned maxima[kMaxCluster * kT];   // keys of all threads' maxima, of all CTAs
  float cta_max[kMaxCluster];
  int cta_arg[kMaxCluster];
  unsigned warp_cnt[2][kT / 32];
};
constexpr size_t kHeader = (sizeof(Shared) + 15) / 16 * 16;

// order-preserving map of f32 onto u32 (larger float, larger key)
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The largest value of a warp's lanes and its lowest index, in every lane.
__device__ __forceinline__ void best_of_warp(float& v, int& i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) {
      v = ov;
      i = oi;
    }
  }
}

// Inclusive scan over the block's kT threads (deterministic: warp scans, then the warp totals).
__device__ __forceinline__ float block_scan(float v, float* warp_tot, float* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float w = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += n;
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  const float before = warp == 0 ? 0.0f : warp_tot[warp - 1];
  if (total != nullptr) *total = warp_tot[kT / 32 - 1];
  __syncthreads();
  return v + before;
}

// The exact top k of a row by one CTA: the k-th largest key by radix selection (four passes of eight bits), then
// every key above it and the lowest indices of its equals, into cand[0 .. k).
__device__ __forceinline__ void select_exact(Common& sh, const float* x, int V, int k) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    sh.prefix = 0;
    sh.krem = static_cast<unsigned>(k);
  }
  unsigned mask = 0;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int i = tid; i < 256; i += kT) sh.hist[i] = 0;
    __syncthreads();
    const unsigned prefix = sh.prefix;
    for (int i = tid; i < V; i += kT) {
      const unsigned key = fkey(x[i]);
      if ((key & mask) == prefix) atomicAdd(&sh.hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid == 0) {
      unsigned need = sh.krem, seen = 0;
      int b = 255;
      for (; b > 0; --b) {
        if (seen + sh.hist[b] >= need) break;
        seen += sh.hist[b];
      }
      sh.krem = need - seen;
      sh.prefix = prefix | (static_cast<unsigned>(b) << shift);
    }
    mask |= 255u << shift;
    __syncthreads();
  }
  const unsigned thr = sh.prefix, k_eq = sh.krem;   // the k-th largest key; how many of its equals belong to the top k
  // ---- collect: every key above thr (any order, sorted below), and of the keys equal to thr the k_eq lowest indices
  if (tid == 0) sh.count = 0;
  
  __syncthreads();
  const int chunk = (V + kT - 1) / kT;
  const int i0 = min(tid * chunk, V), i1 = min(i0 + chunk, V);
  float n_eq = 0.0f;
  for (int i = i0; i < i1; ++i) {
    const unsigned key = fkey(x[i]);
    if (key > thr) {
      const unsigned slot = atomicAdd(&sh.count, 1u);
      sh.cand[slot] = (static_cast<unsigned long long>(key) << 32) | (0xffffffffu - static_cast<unsigned>(i));
    } else if (key == thr) {
      n_eq += 1.0f;
    }
  }
  const float eq_incl = block_scan(n_eq, sh.warp_tot, nullptr);   // counts up to 2^24 are exact in f32
  {
    unsigned rank = static_cast<unsigned>(eq_incl - n_eq);
    const unsigned base = static_cast<unsigned>(k) - k_eq;     // the keys above thr
    for (int i = i0; i < i1 && rank < k_eq; ++i) {
      if (fkey(x[i]) == thr) {
        sh.cand[base + rank] = (static_cast<unsigned long long>(thr) << 32) | (0xffffffffu - static_cast<unsigned>(i));
        ++rank;
      }
    }
  }
  __syncthreads();
}

// (out of line where it is hardly ever needed; inlined, its atomics and loads know their address spaces)
__device__ __noinline__ void select_exact_cold(Common& sh, const float* x, int V, int k) { select_exact(sh, x, V, k); }

// Reads the CTA's share [lo, hi) of the row (into shared memory where it fits) and returns the thread's maximum and
// the first index that has it (0x7fffffff: nothing above -inf).
template <bool STASH>
__device__ __forceinline__ void read_share(const float* x, int lo, int hi, int chunk, float* stash, float& bv, int& bi) {
  constexpr int U = 16;   // loads in flight per thread
  const bool pad = (chunk & 1) == 0;
  int base = lo + static_cast<int>(threadIdx.x);
  for (; base < hi; base += U * kT) {
    float v[U];
#pragma unroll
    for (int j = 0; j < U; ++j) v[j] = base + j * kT < hi ? __ldg(x + base + j * kT) : -INFINITY;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int i = base + j * kT;
      if (v[j] > bv) {
        bv = v[j];
        bi = i;
      }
      if (STASH && i < hi) {
        const int o = i - lo;
        stash[pad ? o + o / chunk : o] = v[j];
      }
    }
  }
}

// The lowest thread of the block for which `hit` holds -> *choice (0xffffffff before).  One atomic per warp: nearly all threads may hit.
__device__ __forceinline__ void first_thread(bool hit, unsigned* choice) {
  const unsigned m = __ballot_sync(0xffffffffu, hit);
  if (m != 0 && (threadIdx.x & 31) == 0) atomicMin(choice, static_cast<unsigned>(threadIdx.x) + __ffs(m) - 1);
}

// Sorts the gathered candidates and draws among the first k: nucleus, then the inverse CDF.  sh.choice is 0xffffffff.
__device__ __forceinline__ void draw_sorted(Common& sh, const SampleArgs& a, const float* x, float gmax, float u, unsigned n_cand, int row) {
  const int tid = threadIdx.x, k = a.top_k;
  // ---- bitonic sort, descending (value, then lower index first)
  unsigned slots = 32;
  while (slots < n_cand) slots <<= 1;
  for (unsigned i = n_cand + tid; i < slots; i += kT) sh.cand[i] = 0ull;
  __syncthreads();
  for (unsigned size = 2; size <= slots; size <<= 1) {
    for (unsigned stride = size >> 1; stride > 0; stride >>= 1) {
      if (static_cast<unsigned>(tid) < slots / 2) {
        const unsigned i = 2 * tid - (tid & (stride - 1)), j = i + stride;
        const unsigned long long p = sh.cand[i], q = sh.cand[j];
        if ((p < q) == ((i & size) == 0)) {
          sh.cand[i] = q;
          sh.cand[j] = p;
        }
      }
      __syncthreads();
    }
  }
  // ---- probabilities of the sorted candidates, nucleus, draw
  float pj = 0.0f;
  int idx = 0;
  if (tid < k) {
    idx = static_cast<int>(0xffffffffu - static_cast<unsigned>(sh.cand[tid] & 0xffffffffull));
    pj = expf((x[idx] - gmax) * a.inv_temperature);
  }
  float total;
  const float cum = block_scan(pj, sh.warp_tot, &total);
  if (tid < kMaxTopK) sh.parts[tid] = cum;
  // kept: before < top_p * total (the first candidate always is)
  const bool kept = tid < k && (tid == 0 || (cum - pj) < a.top_p * total);
  float kcount;
  block_scan(kept ? 1.0f : 0.0f, sh.warp_tot, &kcount);
  const int kk = max(1, static_cast<int>(kcount));
  const float kept_total = sh.parts[kk - 1];
  const float target = u * kept_total;
  // The first candidate whose cumulative probability exceeds the target.  (Not "the one whose interval holds it": intervals formed
  // from the scan overlap, or leave gaps, in their last bit.)
  first_thread(tid < kk && pj > 0.0f && target < cum, &sh.choice);
  __syncthreads();
  const unsigned at = sh.choice == 0xffffffffu ? static_cast<unsigned>(kk - 1) : sh.choice;   // none: u * total rounded up to the total
  if (static_cast<unsigned>(tid) == at) a.out[row] = idx;
}

// The draw inside a chunk [i0, i1) of the row whose exponentials come from `e`: the first one whose cumulative sum exceeds the target, the last
// one that is not zero where rounding leaves none.  (The sum starts below the target also where the scan has it above: an exponential of zero
// is never the first to exceed it.)
template <typename F>
__device__ __forceinline__ int walk_chunk(int i0, int i1, float before, float target, F e) {
  float c = fminf(before, target);
  for (int i = i0; i < i1; ++i) {
    c += e(i);
    if (target < c) return i;
  }
  int last = i1 - 1;
  while (last > i0 && !(e(last) > 0.0f)) --last;
  return last;
}

// grid = (cluster, rows)
__global__ void __launch_bounds__(kT, 1) sample_kernel(const SampleArgs a) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Shared& sh = *reinterpret_cast<Shared*>(smem_raw);
  float* stash = reinterpret_cast<float*>(smem_raw + kHeader);
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int C = static_cast<int>(gridDim.x), rank = static_cast<int>(blockIdx.x);
  const int V = a.V, chunk = a.chunk;
  const int cpc = kT / C;                        // chunks per CTA
  const int lo = min(rank * cpc * chunk, V), hi = min(lo + cpc * chunk, V);
  // An even pitch between the chunks would put the threads that walk them into the same banks.
  const bool pad = (chunk & 1) == 0;
  const int pitch = pad ? chunk + 1 : chunk;
  cl.barrier_arrive();                           // the peers run before anything is stored into their shared memory
  pdl_wait();
  const float* x = a.logits + static_cast<size_t>(blockIdx.y) * V;

  // ---- maximum and argmax (ties: the lowest index, like jnp.argmax)
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  if (a.stash && a.inv_temperature != 0.0f) read_share<true>(x, lo, hi, chunk, stash, bv, bi);
  else read_share<false>(x, lo, hi, chunk, stash, bv, bi);
  const unsigned mykey = lo + tid < hi ? fkey(bv) : 0u;
  best_of_warp(bv, bi);
  if (lane == 0) {
    sh.s_val[warp] = bv;
    sh.s_idx[warp] = bi;
  }
  if (tid == 0) {
    sh.choice = 0xffffffffu;
    sh.count = 0;
  }
  __syncthreads();
  cl.barrier_wait();
  if (warp == 0) {
    float v = sh.s_val[lane];
    int i = sh.s_idx[lane];
    best_of_warp(v, i);
    if (lane < C) {
      Shared* peer = cl.map_shared_rank(&sh, lane);
      peer->cta_max[rank] = v;
      peer->cta_arg[rank] = i;
    }
  }
  if (a.inv_temperature != 0.0f && a.top_k > 0)
    for (int c = 0; c < C; ++c) cl.map_shared_rank(&sh, c)->maxima[rank * kT + tid] = mykey;
  cl.sync();
  float gmax = sh.cta_max[0];
  int garg = sh.cta_arg[0];
  for (int c = 1; c < C; ++c)
    if (sh.cta_max[c] > gmax) {                  // (equal maxima: the lower CTA has the lower index)
      gmax = sh.cta_max[c];
      garg = sh.cta_arg[c];
    }
  if (garg == 0x7fffffff) garg = 0;              // no logit above -inf
  if (a.inv_temperature == 0.0f) {
    if (rank == 0 && tid == 0) a.out[blockIdx.y] = garg;
    return;
  }
  const float u = a.uniform[blockIdx.y];

  if (a.top_k == 0) {
    // ---- categorical over the whole row, vocabulary order: thread t of the row's kT owns a contiguous chunk
    if (a.stash) {
      const int n = pad ? (hi - lo) + (hi - lo) / chunk : hi - lo;   // (the padding words are never read back)
      for (int o = tid; o < n; o += kT) stash[o] = expf((stash[o] - gmax) * a.inv_temperature);
      __syncthreads();
    }
    if (tid < cpc) {
      const int i0 = min(lo + tid * chunk, V), i1 = min(i0 + chunk, V);
      float part = 0.0f;
      if (a.stash) {
        const float* e = stash + tid * pitch;
#pragma unroll 8
        for (int i = 0; i < i1 - i0; ++i) part += e[i];
      } else {
        for (int i = i0; i < i1; ++i) part += expf((x[i] - gmax) * a.inv_temperature);
      }
      for (int c = 0; c < C; ++c) cl.map_shared_rank(&sh, c)->parts[rank * cpc + tid] = part;
    }
    cl.sync();
    const float part = sh.parts[tid];
    float total;
    const float incl = block_scan(part, sh.warp_tot, &total);
    const float target = u * total;
    // the first chunk that reaches beyond the target (the scan's differences overlap, or leave gaps, in their last bit)
    first_thread(part > 0.0f && target < incl, &sh.choice);
    __syncthreads();
    const unsigned owner = sh.choice;
    if (owner == 0xffffffffu) {
      if (rank == 0 && tid == 0) a.out[blockIdx.y] = garg;   // u * total rounded up to the total
    } else if (owner == static_cast<unsigned>(tid) && tid / cpc == rank) {
      const int i0 = min(tid * chunk, V), i1 = min(i0 + chunk, V);
      const float* e = stash + (tid - rank * cpc) * pitch;
      a.out[blockIdx.y] = a.stash ? walk_chunk(i0, i1, incl - part, target, [&](int i) { return e[i - i0]; })
                                  : walk_chunk(i0, i1, incl - part, target, [&](int i) { return expf((x[i] - gmax) * a.inv_temperature); });
    }
    return;
  }

  // ---- a lower bound of the k-th largest key: the k-th largest of the threads' maxima, or a little below it
  const int k = a.top_k;
  unsigned key[kMaxCluster];
  unsigned kmin = 0xffffffffu, kmax = 0u;
#pragma unroll
  for (int c = 0; c < kMaxCluster; ++c) {
    key[c] = c < C ? sh.maxima[c * kT + tid] : 0u;
    if (c < C) kmin = min(kmin, key[c]), kmax = max(kmax, key[c]);
  }
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  if (lane == 0) {
    sh.warp_cnt[0][warp] = kmin;
    sh.warp_cnt[1][warp] = kmax;
  }
  __syncthreads();
  kmin = __reduce_min_sync(0xffffffffu, sh.warp_cnt[0][lane]);
  kmax = __reduce_max_sync(0xffffffffu, sh.warp_cnt[1][lane]);
  __syncthreads();
  // at least k of the C * kT >= k maxima reach `bound`, fewer reach `above`
  unsigned bound = kmin, above = kmax == 0xffffffffu ? kmax : kmax + 1;
  const unsigned enough = static_cast<unsigned>(k + k / 4 + 16);
  for (int it = 0; above - bound > 1; ++it) {
    const unsigned mid = bound + (above - bound) / 2;
    unsigned n = 0;
#pragma unroll
    for (int c = 0; c < kMaxCluster; ++c)
      if (c < C) n += __popc(__ballot_sync(0xffffffffu, key[c] >= mid));
    if (lane == 0) sh.warp_cnt[it & 1][warp] = n;
    __syncthreads();
    n = __reduce_add_sync(0xffffffffu, sh.warp_cnt[it & 1][lane]);
    if (n >= static_cast<unsigned>(k)) {
      bound = mid;
      if (n <= enough) break;
    } else {
      above = mid;
    }
  }
  // ---- every key that reaches the bound, in any order, into the first CTA
  Shared* first = cl.map_shared_rank(&sh, 0);
  {
    const int n = hi - lo;
    for (int b0 = 0; b0 < n; b0 += kT) {
      const int o = b0 + tid;
      unsigned kk = 0;
      if (o < n) kk = fkey(a.stash ? stash[pad ? o + o / chunk : o] : x[lo + o]);
      const bool hit = o < n && kk >= bound;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (m == 0) continue;
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&first->count, static_cast<unsigned>(__popc(m)));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
      if (hit && at < kMaxCand) first->cand[at] = (static_cast<unsigned long long>(kk) << 32) | (0xffffffffu - static_cast<unsigned>(lo + o));
    }
  }
  cl.sync();
  if (rank != 0) return;
  unsigned n_cand = sh.count;
  __syncthreads();
  if (n_cand > kMaxCand || n_cand < static_cast<unsigned>(k)) {   // (fewer: groups of nothing but NaN)
    select_exact_cold(sh, x, V, k);
    n_cand = static_cast<unsigned>(k);
  }
  draw_sorted(sh, a, x, gmax, u, n_cand, blockIdx.y);
}

// One CTA per row: what many rows take, which fill the GPU without clusters.  The row is read from L2 as often as needed.
__global__ void __launch_bounds__(kT, 2) sample_row_kernel(const SampleArgs a) {
  __shared__ Common sh;
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int V = a.V;
  const float* x = a.logits + static_cast<size_t>(blockIdx.x) * V;
  float bv = -INFINITY;
  int bi = 0x7fffffff;
#pragma unroll 4
  for (int i = tid; i < V; i += kT) {
    const float v = __ldg(x + i);
    if (v > bv) {
      bv = v;
      bi = i;
    }
  }
  best_of_warp(bv, bi);
  if (lane == 0) {
    sh.s_val[warp] = bv;
    sh.s_idx[warp] = bi;
  }
  if (tid == 0) sh.choice = 0xffffffffu;
  __syncthreads();
  bv = sh.s_val[lane];
  bi = sh.s_idx[lane];
  best_of_warp(bv, bi);
  const float gmax = bv;
  const int garg = bi == 0x7fffffff ? 0 : bi;   // no logit above -inf
  if (a.inv_temperature == 0.0f) {
    if (tid == 0) a.out[blockIdx.x] = garg;
    return;
  }
  const float u = a.uniform[blockIdx.x];
  if (a.top_k == 0) {
    const int i0 = min(tid * a.chunk, V), i1 = min(i0 + a.chunk, V);
    float part = 0.0f;
    for (int i = i0; i < i1; ++i) part += expf((x[i] - gmax) * a.inv_temperature);
    float total;
    const float incl = block_scan(part, sh.warp_tot, &total);
    const float target = u * total;
    first_thread(part > 0.0f && target < incl, &sh.choice);
    __syncthreads();
    if (sh.choice == 0xffffffffu) {
      if (tid == 0) a.out[blockIdx.x] = garg;   // u * total rounded up to the total
    } else if (sh.choice == static_cast<unsigned>(tid)) {
      a.out[blockIdx.x] = walk_chunk(i0, i1, incl - part, target, [&](int i) { return expf((x[i] - gmax) * a.inv_temperature); });
    }
    return;
  }
  select_exact(sh, x, V, a.top_k);
  draw_sorted(sh, a, x, gmax, u, static_cast<unsigned>(a.top_k), blockIdx.x);
}

// Which kernel: where rows alone fill the GPU, or a row is too short to share, a cluster's exchanges cost more than they save.
// Measured, one CTA per row / a cluster (us): greedy 8 x 4099 6 / 8, 8 x 32000 12 / 8, 96 x 50257 6 / 10, 256 x 151936 31 / 48; whole row 32 x 8192 5 / 7,
// 37 x 16384 9 / 14, 32 x 32000 24 / 10, 96 x 50257 20 / 32, 256 x 65536 82 / 85; top 50 64 x 8192 28 / 30 (top 20: 33 / 28), 96 x 8192 28 / 44, 96 x 16384
// 42 / 47, 64 x 16384 42 / 33, 256 x 32000 108 / 124, 256 x 65536 187 / 135; top 1000 64 x 8192 38 / 51, 37 x 8192 38 / 35, 96 x 50257 67 / 82,
// 128 x 65536 124 / 110.
bool RowPerCta(int64_t batch, int64_t vocab, const SampleArgs& a) {
  if (a.inv_temperature == 0.0f) return vocab <= 16384 || batch >= (vocab <= 65536 ? 96 : 128);
  if (a.top_k == 0) return vocab <= 8192 || (batch >= 37 && vocab <= 16384) || (batch >= 96 && vocab < 65536) || (batch >= 1024 && vocab <= 65536);
  if (a.top_k >= 256)
    return (batch >= (vocab < 2048 ? 112 : 64) && vocab <= 16384) || (batch >= 96 && vocab < 65536) || (batch >= 512 && vocab <= 65536);
  return (batch >= 80 && vocab <= 8192) || (batch >= 96 && vocab <= 16384) || (batch >= 160 && vocab < 65536);
}

}  // namespace

extern "C" {

b200_status b200_sample(b200_context* ctx, b200_stream stream, const float* logits, int64_t batch, int64_t vocab,
                        float temperature, int32_t top_k, float top_p, const float* uniform, int32_t* out) {
  b200_status s = BeginLaunch(ctx);
  if (s != B200_OK) return s;
  if (temperature < 0.0f) return Fail(B200_INVALID_ARGUMENT, "b200_sample: temperature must be >= 0, got %g", temperature);
  if (batch < 0 || vocab < 0) return Fail(B200_INVALID_ARGUMENT, "b200_sample: negative size");
  if (top_k < 0 || top_k > vocab) return Fail(B200_INVALID_ARGUMENT, "b200_sample: top_k must be in [0, %lld], got %d",
                                              static_cast<long long>(vocab), top_k);
  if (batch == 0) return B200_OK;
  if (vocab == 0) return Fail(B200_INVALID_ARGUMENT, "b200_sample: empty vocabulary");
  if (vocab > (1 << 24)) return Fail(B200_UNIMPLEMENTED, "b200_sample: vocabulary above 2^24");
  if (batch > 65535) return Fail(B200_UNIMPLEMENTED, "b200_sample: more than 65535 rows");
  if (logits == nullptr || out == nullptr) return Fail(B200_INVALID_ARGUMENT, "b200_sample: null buffer");
  if (temperature > 0.0f && uniform == nullptr)
    return Fail(B200_INVALID_ARGUMENT, "b200_sample: sampling needs one uniform number per row");
  if (temperature > 0.0f && top_k > kMaxTopK)
    return Fail(B200_UNIMPLEMENTED, "b200_sample: top_k %d (up to %d)", top_k, kMaxTopK);
  if (temperature > 0.0f && top_k == 0 && top_p < 1.0f)
    return Fail(B200_UNIMPLEMENTED, "b200_sample: top_p without top_k sorts the whole vocabulary; set top_k (up to %d)", kMaxTopK);
  SampleArgs a;
  a.logits = logits;
  a.uniform = uniform;
  a.out = out;
  a.V = static_cast<int>(vocab);
  a.inv_temperature = temperature > 0.0f ? 1.0f / temperature : 0.0f;
  a.top_k = temperature > 0.0f ? top_k : 0;
  a.top_p = top_p;
  // One wave of CTAs where that can be (a CTA's share and tables leave room for one per SM), and at least as many per
  // row as it takes for their shares to fit shared memory.
  a.chunk = static_cast<int>(CeilDiv(vocab, kT));
  LaunchCfg lc;
  lc.stream = stream;
  lc.block = dim3(kT);
  lc.pdl = true;
  cudaError_t e;
  if (RowPerCta(batch, vocab, a)) {
    lc.grid = dim3(static_cast<unsigned>(batch));
    e = Launch(lc, sample_row_kernel, a);
    if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_sample launch: %s", cudaGetErrorString(e)));
    return EndLaunch(ctx, "b200_sample");
  }
  const bool fits4 = kHeader + static_cast<size_t>(kT / 4) * (a.chunk + 1) * sizeof(float) <= static_cast<size_t>(ctx->max_smem_optin);
  const int cluster = batch * 8 <= ctx->sm_count || !fits4 ? 8 : 4;
  const size_t share = static_cast<size_t>(kT / cluster) * (a.chunk + 1) * sizeof(float);
  a.stash = a.inv_temperature != 0.0f && kHeader + share <= static_cast<size_t>(ctx->max_smem_optin);
  lc.grid = dim3(cluster, static_cast<unsigned>(batch));
  lc.cluster_x = cluster;
  lc.smem = kHeader + (a.stash ? share : 0);
  e = cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem_optin);
  if (e == cudaSuccess) e = Launch(lc, sample_kernel, a);
  if (e != cudaSuccess) return Stick(ctx, Fail(B200_INTERNAL, "b200_sample launch: %s", cudaGetErrorString(e)));
  return EndLaunch(ctx, "b200_sample");
}

}  // extern "C"
