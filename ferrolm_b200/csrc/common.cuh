// Shared device helpers: order-preserving (distance, id) keys, the warp-owned
// sorted list used for every top-k, and the reference's exact distance chains.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/ferrovec.h"

typedef unsigned long long u64;

namespace fv {

// ---------------------------------------------------------------------------------------------
// host-side error plumbing
void set_error(const std::string& msg);
int fail(int status, const std::string& msg);

inline const char* base_name(const char* path) {  // the file's name without its directories, for error messages
  const char* b = path;
  for (const char* c = path; *c; ++c)
    if (*c == '/') b = c + 1;
  return b;
}

#define FV_CUDA(expr)                                                                          \
  do {                                                                                         \
    cudaError_t _e = (expr);                                                                   \
    if (_e != cudaSuccess)                                                                     \
      return fv::fail(FV_ERR_CUDA, std::string(#expr) + " (" + fv::base_name(__FILE__) + ":" +  \
                                       std::to_string(__LINE__) + "): " + cudaGetErrorString(_e)); \
  } while (0)

#define FV_TRY(expr)            \
  do {                          \
    int _s = (expr);            \
    if (_s != FV_OK) return _s; \
  } while (0)

inline size_t padded(size_t dim) { return (dim + 7) / 8 * 8; }

// ---------------------------------------------------------------------------------------------
// keys.  Neighbours are ordered by f32::total_cmp on the distance, then by id
// (src/vector/mod.rs:60-64).  Mapping the float's bits to an unsigned integer that
// sorts the same way and putting the id below it turns that order into one u64 compare.
#define FV_EMPTY_KEY 0xFFFFFFFFFFFFFFFFull

__host__ __device__ __forceinline__ uint32_t order_bits(float f) {
#ifdef __CUDA_ARCH__
  uint32_t b = __float_as_uint(f);
#else
  uint32_t b;
  memcpy(&b, &f, 4);
#endif
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__host__ __device__ __forceinline__ float order_bits_to_float(uint32_t k) {
  uint32_t b = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}
__host__ __device__ __forceinline__ u64 make_key(float d, uint32_t id) {
  return (u64(order_bits(d)) << 32) | u64(id);
}
__host__ __device__ __forceinline__ float key_distance(u64 k) { return order_bits_to_float(uint32_t(k >> 32)); }
__host__ __device__ __forceinline__ uint32_t key_id(u64 k) { return uint32_t(k & 0xFFFFFFFFull); }

// Debug build (make EXTRA=-DFV_BOUNDS): the indices kernels gather through (probed cells, list offsets, row ids,
// graph links, vector slots, gathered operand rows) are checked against their extents before the access.  A
// violation is recorded in the translation unit's g_bounds words {count, site, index, extent} and the access is
// skipped; at the end of a search the host turns a non-zero count into FV_ERR_OVERFLOW (bounds_report_*).
// FV_BOUNDS_TU(name) goes once into every .cu with checked kernels.
#if defined(FV_BOUNDS) && defined(__CUDACC__)
static __device__ unsigned long long g_bounds[4];
__device__ __forceinline__ bool idx_ok(unsigned long long i, unsigned long long n, int site) {
  if (i < n) return true;
  if (atomicAdd(&g_bounds[0], 1ull) == 0ull) {
    g_bounds[1] = (unsigned long long)site;
    g_bounds[2] = i;
    g_bounds[3] = n;
  }
  return false;
}
#define FV_IDX_OK(i, n, site) fv::idx_ok((unsigned long long)(i), (unsigned long long)(n), site)
#define FV_BOUNDS_TU(name)                                                                                        \
  namespace fv {                                                                                                  \
  int bounds_report_##name() {                                                                                    \
    unsigned long long h[4] = {0, 0, 0, 0};                                                                       \
    if (cudaMemcpyFromSymbol(h, g_bounds, sizeof(h)) != cudaSuccess) return fail(FV_ERR_CUDA, "bounds words");    \
    if (h[0] == 0) return FV_OK;                                                                                  \
    const unsigned long long z[4] = {0, 0, 0, 0};                                                                 \
    cudaMemcpyToSymbol(g_bounds, z, sizeof(z));                                                                   \
    return fail(FV_ERR_OVERFLOW, std::string("bounds check in " #name ": ") + std::to_string(h[0]) +              \
                                     " violation(s); first at site " + std::to_string(h[1]) + ", index " +         \
                                     std::to_string(h[2]) + ", extent " + std::to_string(h[3]));                   \
  }                                                                                                               \
  }
#else
#define FV_IDX_OK(i, n, site) true
#define FV_BOUNDS_TU(name)                          \
  namespace fv {                                    \
  int bounds_report_##name() { return FV_OK; }      \
  }
#endif

#ifdef __CUDACC__
#define FV_FULL 0xFFFFFFFFu

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// the one dynamic shared-memory array of every kernel
__device__ __forceinline__ unsigned char* dyn_smem() {
  extern __shared__ __align__(1024) unsigned char fv_dyn_smem[];
  return fv_dyn_smem;
}

// Sorts the first `n` keys (a power of two) of `buf` (shared memory) ascending: a bitonic network run by the whole
// block, one barrier per stage.  Called by every thread of the block.
__device__ __forceinline__ void block_sort(u64* buf, int n) {
  for (int k = 2; k <= n; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < (n >> 1); t += blockDim.x) {
        const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));  // the lower index of pair t
        const u64 x = buf[i], y = buf[i | j];
        const bool asc = (i & k) == 0;
        if ((x > y) == asc) {
          buf[i] = y;
          buf[i | j] = x;
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------------------------
// A sorted list of L keys (ascending) owned by ONE warp, in shared or global memory.
// All 32 lanes call every function with the same arguments.
__device__ __forceinline__ void warp_list_init(u64* list, int L) {
  for (int e = lane_id(); e < L; e += 32) list[e] = FV_EMPTY_KEY;
  __syncwarp();
}

// Inserts `key` (must be < list[L-1]) and drops the last entry.  Works from the top chunk of
// 32 entries downwards so that every read sees the list as it was before the call.
__device__ __forceinline__ void warp_list_insert(u64* list, int L, u64 key) {
  const int lane = lane_id();
  for (int c = (L - 1) >> 5; c >= 0; --c) {
    const int e = (c << 5) + lane;
    const u64 cur = (e < L) ? list[e] : FV_EMPTY_KEY;
    const u64 prev = (e > 0 && e <= L) ? list[e - 1] : 0ull;
    __syncwarp();
    if (e < L) {
      u64 nv = cur;
      if (!(cur < key)) nv = (e == 0 || prev < key) ? key : prev;
      list[e] = nv;
    }
    const u64 low = __shfl_sync(FV_FULL, cur, 0);
    __syncwarp();
    if (low < key) break;
  }
}

// Offers the candidates held one per lane (key = FV_EMPTY_KEY for "none") to the list, in lane order.
// Returns the list's last key afterwards (the admission bound).
__device__ __forceinline__ u64 warp_list_offer(u64* list, int L, u64 key, u64 bound) {
  unsigned pending = __ballot_sync(FV_FULL, key < bound);
  while (pending) {
    const int src = __ffs(pending) - 1;
    pending &= pending - 1;
    const u64 k = __shfl_sync(FV_FULL, key, src);
    if (k < bound) {
      warp_list_insert(list, L, k);
      bound = list[L - 1];
    }
  }
  return bound;
}

// ---------------------------------------------------------------------------------------------
// The reference's distance arithmetic (src/kernels.rs:192-231): eight lane accumulators, each a
// chain of fused multiply-adds over every eighth element, then the fixed pairwise lane sum.
__device__ __forceinline__ float hsum8(const float* l) {
  return __fadd_rn(__fadd_rn(__fadd_rn(l[0], l[4]), __fadd_rn(l[2], l[6])),
                   __fadd_rn(__fadd_rn(l[1], l[5]), __fadd_rn(l[3], l[7])));
}

template <bool IS_L2>
__device__ __forceinline__ void dist_step8(float* acc, const float4& a0, const float4& a1, const float4& b0,
                                           const float4& b1) {
  if (IS_L2) {
    float d;
    d = __fsub_rn(a0.x, b0.x); acc[0] = __fmaf_rn(d, d, acc[0]);
    d = __fsub_rn(a0.y, b0.y); acc[1] = __fmaf_rn(d, d, acc[1]);
    d = __fsub_rn(a0.z, b0.z); acc[2] = __fmaf_rn(d, d, acc[2]);
    d = __fsub_rn(a0.w, b0.w); acc[3] = __fmaf_rn(d, d, acc[3]);
    d = __fsub_rn(a1.x, b1.x); acc[4] = __fmaf_rn(d, d, acc[4]);
    d = __fsub_rn(a1.y, b1.y); acc[5] = __fmaf_rn(d, d, acc[5]);
    d = __fsub_rn(a1.z, b1.z); acc[6] = __fmaf_rn(d, d, acc[6]);
    d = __fsub_rn(a1.w, b1.w); acc[7] = __fmaf_rn(d, d, acc[7]);
  } else {
    acc[0] = __fmaf_rn(a0.x, b0.x, acc[0]);
    acc[1] = __fmaf_rn(a0.y, b0.y, acc[1]);
    acc[2] = __fmaf_rn(a0.z, b0.z, acc[2]);
    acc[3] = __fmaf_rn(a0.w, b0.w, acc[3]);
    acc[4] = __fmaf_rn(a1.x, b1.x, acc[4]);
    acc[5] = __fmaf_rn(a1.y, b1.y, acc[5]);
    acc[6] = __fmaf_rn(a1.z, b1.z, acc[6]);
    acc[7] = __fmaf_rn(a1.w, b1.w, acc[7]);
  }
}

// Distance between `a` (shared or global, 16-byte aligned, pd floats) and row `b` (global).
template <bool IS_L2>
__device__ __forceinline__ float exact_distance(const float* __restrict__ a, const float* __restrict__ b, int pd) {
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float4* a4 = reinterpret_cast<const float4*>(a);
  const float4* b4 = reinterpret_cast<const float4*>(b);
#pragma unroll 4
  for (int c = 0; c < pd / 8; ++c) {
    const float4 b0 = __ldg(b4 + 2 * c), b1 = __ldg(b4 + 2 * c + 1);
    const float4 a0 = a4[2 * c], a1 = a4[2 * c + 1];
    dist_step8<IS_L2>(acc, a0, a1, b0, b1);
  }
  const float s = hsum8(acc);
  return IS_L2 ? s : -s;
}

// Sorts one key per lane, ascending, and turns a bitonic sequence of 32 * R keys (place 32 r + lane in e[r]) into an
// ascending one: compare-exchange networks over shuffles.
__device__ __forceinline__ u64 cmp_exchange(u64 v, int stride, bool keep_min) {
  const u64 o = __shfl_xor_sync(FV_FULL, v, stride);
  return (v < o) == keep_min ? v : o;
}
__device__ __forceinline__ u64 warp_sort32(u64 v) {
  const int lane = lane_id();
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) v = cmp_exchange(v, stride, ((lane & stride) == 0) == ((lane & size) == 0));
  return v;
}
template <int R>
__device__ __forceinline__ void bitonic_merge(u64* e) {
#pragma unroll
  for (int s = R >> 1; s > 0; s >>= 1)
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!(r & s)) {
        const u64 x = e[r], y = e[r | s];
        e[r] = x < y ? x : y;
        e[r | s] = x < y ? y : x;
      }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1)
#pragma unroll
    for (int r = 0; r < R; ++r) e[r] = cmp_exchange(e[r], stride, (lane_id() & stride) == 0);
}

// The L best keys in a warp's registers (32 * KR places, L <= 32 * KR), ascending; the last of the L entries sits in
// the last place, the places before the first hold 0.  Both ascending lists of N places, one read backwards: the
// smaller of each pair are the N smallest of both, as a bitonic sequence.  So 32 candidates at a time cost a sort and
// a merge whatever their number, and a candidate alone one shuffle per 32 places; the line between the two is where
// they take equally long.
template <int KR>
struct TopList {
  u64 e[KR];
  __device__ __forceinline__ void init(int L) {
#pragma unroll
    for (int r = 0; r < KR; ++r) e[r] = r * 32 + lane_id() < 32 * KR - L ? 0ull : FV_EMPTY_KEY;
  }
  __device__ __forceinline__ u64 last() const { return __shfl_sync(FV_FULL, e[KR - 1], 31); }
  __device__ __forceinline__ void offer(u64 key, u64& bound) {  // a key per lane, FV_EMPTY_KEY for none
    unsigned pending = __ballot_sync(FV_FULL, key < bound);
    if (__popc(pending) > 6) {
      const u64 c = warp_sort32(key < bound ? key : FV_EMPTY_KEY);
      const u64 back = __shfl_sync(FV_FULL, c, 31 - lane_id());
      e[KR - 1] = min(e[KR - 1], back);
      bitonic_merge<KR>(e);
      bound = last();
      return;
    }
    while (pending) {
      const int src = __ffs(pending) - 1;
      const u64 k = __shfl_sync(FV_FULL, key, src);
#pragma unroll
      for (int r = KR - 1; r >= 0; --r) {
        u64 prev = __shfl_up_sync(FV_FULL, e[r], 1);
        const u64 carry = r > 0 ? __shfl_sync(FV_FULL, e[r > 0 ? r - 1 : 0], 31) : 0ull;
        if (lane_id() == 0) prev = carry;
        if (!(e[r] < k)) e[r] = prev < k ? k : prev;
      }
      bound = last();
      pending = __ballot_sync(FV_FULL, lane_id() > src && key < bound);
    }
  }
  // takes in another list's entries: ascending from place 0 on, FV_EMPTY_KEY behind them
  __device__ __forceinline__ void merge(const u64* c) {
    u64 back[KR];
#pragma unroll
    for (int r = 0; r < KR; ++r) back[r] = __shfl_sync(FV_FULL, c[KR - 1 - r], 31 - lane_id());
#pragma unroll
    for (int r = 0; r < KR; ++r) e[r] = min(e[r], back[r]);
    bitonic_merge<KR>(e);
  }
  // writes the L entries to dst[0 ..]
  __device__ __forceinline__ void store(u64* dst, int L) const {
#pragma unroll
    for (int r = 0; r < KR; ++r) {
      const int i = r * 32 + lane_id() - (32 * KR - L);
      if (i >= 0) dst[i] = e[r];
    }
  }
  // a list of L entries in memory, as merge takes it
  __device__ __forceinline__ static void load(u64* c, const u64* src, int L) {
#pragma unroll
    for (int r = 0; r < KR; ++r) {
      const int i = r * 32 + lane_id();
      c[r] = i < L ? src[i] : FV_EMPTY_KEY;
    }
  }
};

// ---- distances of a run of gathered rows, by LPR lanes per row (32 / LPR rows at a time).  A lane owns 8 / LPR of
// the reference's eight chains (src/kernels.rs:200-231) and the lane sums are added in its pairwise order, so the
// bits are exact_distance's.  With one row per lane every load touches as many lines as there are rows, and a short
// run (the ten unvisited links of a graph node) leaves most lanes idle.  What bounds such a run is its trips to memory
// (about 700 cycles each to L2), so a lane requests U = 16 pieces (128 dimensions of its row) before it works on the
// first; what is left of the row goes in halves.
template <bool IS_L2, int LPR, int U>
__device__ __forceinline__ void group_chunk(const float* __restrict__ a, const float* __restrict__ row, int t, float& c0,
                                            float& c1) {
  if (LPR == 8) {
    float b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) b[u] = __ldg(row + t + 8 * u);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (IS_L2) {
        const float d = __fsub_rn(a[t + 8 * u], b[u]);
        c0 = __fmaf_rn(d, d, c0);
      } else {
        c0 = __fmaf_rn(a[t + 8 * u], b[u], c0);
      }
    }
  } else {
    float2 b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) b[u] = __ldg(reinterpret_cast<const float2*>(row + t + 8 * u));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float2 x = *reinterpret_cast<const float2*>(a + t + 8 * u);
      if (IS_L2) {
        const float d0 = __fsub_rn(x.x, b[u].x), d1 = __fsub_rn(x.y, b[u].y);
        c0 = __fmaf_rn(d0, d0, c0);
        c1 = __fmaf_rn(d1, d1, c1);
      } else {
        c0 = __fmaf_rn(x.x, b[u].x, c0);
        c1 = __fmaf_rn(x.y, b[u].y, c1);
      }
    }
  }
}
template <bool IS_L2, int LPR>
__device__ __forceinline__ float group_distance(const float* __restrict__ a, const float* __restrict__ row, int pd) {
  const int j = lane_id() & (LPR - 1);
  a += LPR == 8 ? j : 2 * j;
  row += LPR == 8 ? j : 2 * j;
  float c0 = 0.f, c1 = 0.f;
  int t = 0;
  for (; t + 128 <= pd; t += 128) group_chunk<IS_L2, LPR, 16>(a, row, t, c0, c1);
  if (pd & 64) {
    group_chunk<IS_L2, LPR, 8>(a, row, t, c0, c1);
    t += 64;
  }
  if (pd & 32) {
    group_chunk<IS_L2, LPR, 4>(a, row, t, c0, c1);
    t += 32;
  }
  for (; t < pd; t += 8) group_chunk<IS_L2, LPR, 1>(a, row, t, c0, c1);
  if (LPR == 8) {
    float s = __fadd_rn(c0, __shfl_xor_sync(FV_FULL, c0, 4));
    s = __fadd_rn(s, __shfl_xor_sync(FV_FULL, s, 2));
    s = __fadd_rn(s, __shfl_xor_sync(FV_FULL, s, 1));
    return IS_L2 ? s : -s;
  }
  // lanes hold (l0,l1) (l2,l3) (l4,l5) (l6,l7): ((l0 + l4) + (l2 + l6)) + ((l1 + l5) + (l3 + l7))
  float s0 = __fadd_rn(c0, __shfl_xor_sync(FV_FULL, c0, 2)), s1 = __fadd_rn(c1, __shfl_xor_sync(FV_FULL, c1, 2));
  s0 = __fadd_rn(s0, __shfl_xor_sync(FV_FULL, s0, 1));
  s1 = __fadd_rn(s1, __shfl_xor_sync(FV_FULL, s1, 1));
  const float s = __fadd_rn(s0, s1);
  return IS_L2 ? s : -s;
}

// The same by eight lanes per row with up to 384 dimensions of it requested before the first is worked on, for kernels with
// the registers for that: one trip to memory instead of one per 128 dimensions (and one more for each odd piece).
template <bool IS_L2>
__device__ __forceinline__ float group_distance_ahead(const float* __restrict__ a, const float* __restrict__ row, int pd) {
  const int j = lane_id() & 7;
  a += j;
  row += j;
  float c = 0.f;
  for (int t0 = 0; t0 < pd; t0 += 384) {
    float b[48];
#pragma unroll
    for (int p = 0; p < 3; ++p)
      if (t0 + 128 * p < pd) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int t = t0 + 128 * p + 8 * u;
          b[16 * p + u] = t < pd ? __ldg(row + t) : 0.f;
        }
      }
#pragma unroll
    for (int p = 0; p < 3; ++p)
      if (t0 + 128 * p < pd) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int t = t0 + 128 * p + 8 * u;
          if (t < pd) {
            const float x = a[t], d = IS_L2 ? __fsub_rn(x, b[16 * p + u]) : x;
            c = __fmaf_rn(d, IS_L2 ? d : b[16 * p + u], c);
          }
        }
      }
  }
  float s = __fadd_rn(c, __shfl_xor_sync(FV_FULL, c, 4));
  s = __fadd_rn(s, __shfl_xor_sync(FV_FULL, s, 2));
  s = __fadd_rn(s, __shfl_xor_sync(FV_FULL, s, 1));
  return IS_L2 ? s : -s;
}

__device__ __forceinline__ float exact_distance(int metric, const float* a, const float* b, int pd) {
  return metric == FV_L2 ? exact_distance<true>(a, b, pd) : exact_distance<false>(a, b, pd);
}
#endif  // __CUDACC__

}  // namespace fv
