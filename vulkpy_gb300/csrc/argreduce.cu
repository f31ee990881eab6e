// argmax / argmin over all elements or along one axis (numpy semantics: the
// first index of the extreme value; a NaN counts as the extreme, so the first
// NaN wins; -0.0 and +0.0 compare equal).  The reference lists these as not
// yet implemented (README.md:73, example/02-nn.py:96 falls back to numpy).
//
// Each candidate is one 64-bit key: an order-preserving image of the value in
// the high word and the complement of the index in the low word, so the
// maximum key is the extreme value at the smallest index and every combine is
// a plain integer max -- associative, so any tree order gives the same answer.
//
// A thread does not build a key per element (about ten instructions: with one
// load each that bound rows of 32768 to 2.3 TB/s): it takes the NaN-passing
// maximum of 16 elements (one instruction each), keeps the best group so far
// and looks up the element in that group once at the end.  8192 x 32768: rows
// 469 -> 151 us, whole 276 -> 152 us (7.0 TB/s).
#include <algorithm>

#include "common.cuh"

namespace vkc {
namespace {

template <bool MIN>
__device__ __forceinline__ uint32_t order_word(float v) {
  if (v != v) return 0xFFFFFFFFu;  // NaN beats every number
  const uint32_t b = __float_as_uint(v == 0.0f ? 0.0f : v);
  const uint32_t o = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  return MIN ? ~o : o;  // NaN handled above, so ~o < 0xFFFFFFFF
}

template <bool MIN>
__device__ __forceinline__ uint64_t make_key(float v, uint32_t i) {
  return ((uint64_t)order_word<MIN>(v) << 32) | (uint64_t)(~i);
}

__device__ __forceinline__ uint64_t kmax(uint64_t a, uint64_t b) { return a > b ? a : b; }

__device__ __forceinline__ uint64_t warp_max(uint64_t k) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) k = kmax(k, __shfl_xor_sync(0xFFFFFFFFu, k, o));
  return k;
}

// Block-wide maximum; every thread gets the result.
__device__ __forceinline__ uint64_t block_max(uint64_t k, uint64_t* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  k = warp_max(k);
  if (lane == 0) sh[w] = k;
  __syncthreads();
  k = lane < nw ? sh[lane] : 0;
  k = warp_max(k);
  __syncthreads();
  return k;
}

constexpr int kThreads = 256;

// max / min that returns NaN when an operand is NaN.
template <bool MIN>
__device__ __forceinline__ float extreme(float a, float b) {
  float r;
  if (MIN) asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  else asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Whether a later group's extreme m replaces the best so far: strictly
// better, or the first NaN.
template <bool MIN>
__device__ __forceinline__ bool replaces(float m, float best) {
  return (MIN ? m < best : m > best) || (m != m && best == best);
}

__device__ __forceinline__ bool is_best(float v, float best) { return v == best || (v != v && best != best); }

template <bool MIN>
constexpr float kWorst = MIN ? INFINITY : -INFINITY;

constexpr int kGroup = 4;  // vectors per group

// A thread's best group: element (at + u nt) W + w for u < U, w < W, or with
// W == 0 the element `at` itself.
struct Scan {
  float best;
  size_t at;
  int w;
  bool any;
};

// Elements t, t + nt, ... of a[0..n) (nt threads) for T = float4 (16-byte
// aligned a; n counts whole float4) or float.
template <bool MIN, class T>
__device__ __forceinline__ Scan scan_groups(const float* __restrict__ a, size_t n, size_t t, size_t nt) {
  constexpr int W = sizeof(T) / 4, U = W == 4 ? kGroup : 4 * kGroup;
  const T* av = reinterpret_cast<const T*>(a);
  Scan s{kWorst<MIN>, t, W, t < n};  // a group of nothing but kWorst is the first one's
  const size_t last = (U - 1) * nt;
  for (size_t i = t; i < n; i += U * nt) {
    T v[U];
    if (i + last < n) {
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = __ldcs(av + i + u * nt);
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = i + u * nt < n ? __ldcs(av + i + u * nt) : v[0];
    }
    float m = kWorst<MIN>;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int w = 0; w < W; ++w) m = extreme<MIN>(m, reinterpret_cast<const float*>(&v[u])[w]);
    if (replaces<MIN>(m, s.best)) {
      s.best = m;
      s.at = i;
    }
  }
  return s;
}

// Thread t of nt over a[0..n): whole float4 when a is aligned, the (at most
// 3) elements after them one by one (nt >= 32).
template <bool MIN>
__device__ __forceinline__ Scan scan(const float* __restrict__ a, size_t n, size_t t, size_t nt) {
  if ((((uintptr_t)a) & 15u) != 0) return scan_groups<MIN, float>(a, n, t, nt);
  const size_t n4 = n / 4;
  Scan s = scan_groups<MIN, float4>(a, n4, t, nt);
  const size_t k = 4 * n4 + t;
  if (k < n && (!s.any || replaces<MIN>(a[k], s.best))) s = Scan{a[k], k, 0, true};
  return s;
}

// The index of the first element of the group at `at` with the value best
// (W floats per load): all the group's loads together, since one after the
// other they are a chain of up to 16 waits for the L2 cache (37 x 257 x 129
// whole 4.9 -> 3.8 us, 64 rows of 4099 3.2 -> 2.2, with the block's two steps in
// 32-bit warp reductions instead of 64-bit shuffles).
template <int W>
__device__ __forceinline__ uint32_t group_first(const float* __restrict__ a, size_t end, size_t at, size_t nt,
                                                float best) {
  constexpr int N = 4 * kGroup;
  float v[N];
  bool in[N];
#pragma unroll
  for (int e = 0; e < N; ++e) {
    const size_t k = W * (at + (size_t)(e / W) * nt) + e % W;
    in[e] = k < end;
    v[e] = in[e] ? a[k] : 0.f;
  }
  uint32_t first = 0xFFFFFFFFu;
#pragma unroll
  for (int e = N - 1; e >= 0; --e)
    if (in[e] && is_best(v[e], best)) first = (uint32_t)(W * (at + (size_t)(e / W) * nt) + e % W);
  return first;
}

__device__ __forceinline__ uint32_t scan_first(const Scan& s, const float* __restrict__ a, size_t n, size_t nt) {
  if (s.w == 0) return (uint32_t)s.at;
  return s.w == 4 ? group_first<4>(a, n / 4 * 4, s.at, nt, s.best) : group_first<1>(a, n, s.at, nt, s.best);
}

// Maximum or minimum over the block's warps (sh: one word per warp, free
// again after the block's next barrier).
template <bool MAX>
__device__ __forceinline__ uint32_t block_word(uint32_t v, uint32_t* sh) {
  auto warp = [](uint32_t x) { return MAX ? __reduce_max_sync(0xFFFFFFFFu, x) : __reduce_min_sync(0xFFFFFFFFu, x); };
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp(v);
  if (lane == 0) sh[w] = v;
  __syncthreads();
  return warp(sh[lane < nw ? lane : 0]);
}

// The best key of a[0..n) over the block: the threads agree on the value
// first, and only those that hold it look for their element.
template <bool MIN>
__device__ __forceinline__ uint64_t block_best(const float* __restrict__ a, size_t n, size_t t, size_t nt,
                                               uint32_t (*sh)[32]) {
  const Scan s = scan<MIN>(a, n, t, nt);
  const uint32_t word = s.any ? order_word<MIN>(s.best) : 0u;
  const uint32_t top = block_word<true>(word, sh[0]);
  const uint32_t at = block_word<false>(s.any && word == top ? scan_first(s, a, n, nt) : 0xFFFFFFFFu, sh[1]);
  return top ? (uint64_t)top << 32 | (uint64_t)(~at) : 0;  // 0: no element at all
}

// Pass 1: each block reduces its share of a[0..n) to one key.
template <bool MIN>
__global__ void __launch_bounds__(kThreads) k_arg_partials(const float* __restrict__ a, size_t n,
                                                           uint64_t* __restrict__ part) {
  __shared__ uint32_t sh[2][32];
  const uint64_t best = block_best<MIN>(a, n, (size_t)blockIdx.x * blockDim.x + threadIdx.x,
                                        (size_t)gridDim.x * blockDim.x, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = best;
}

// Pass 2: one block reduces the partial keys and writes the index.
__global__ void __launch_bounds__(1024) k_arg_final(const uint64_t* __restrict__ part, int m,
                                                   uint32_t* __restrict__ out) {
  __shared__ uint64_t sh[32];
  uint64_t best = 0;
  pdl_wait();
  for (int i = threadIdx.x; i < m; i += blockDim.x) best = kmax(best, part[i]);
  best = block_max(best, sh);
  if (threadIdx.x == 0) out[0] = ~(uint32_t)best;
}

// Along a contiguous axis (post == 1) shorter than 2048: one warp per row,
// the index kept beside the best value (a lane has too few elements for
// groups to pay).
template <bool MIN>
__global__ void __launch_bounds__(kThreads) k_arg_rows_warp(const float* __restrict__ a, size_t rows,
                                                            size_t len, uint32_t* __restrict__ out) {
  const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5);
  const int lane = threadIdx.x & 31;
  for (size_t r = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
    const float* row = a + r * len;
    float best = kWorst<MIN>;
    uint32_t at = lane;
#pragma unroll 4
    for (uint32_t k = lane; k < (uint32_t)len; k += 32) {
      const float v = __ldg(row + k);
      if (replaces<MIN>(v, best)) {
        best = v;
        at = k;
      }
    }
    const bool any = lane < len;
    const uint32_t word = any ? order_word<MIN>(best) : 0u;
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, word);
    at = __reduce_min_sync(0xFFFFFFFFu, any && word == top ? at : 0xFFFFFFFFu);
    if (lane == 0) out[r] = at;
  }
}

// Along a long contiguous axis: one block per row.
template <bool MIN>
__global__ void __launch_bounds__(kThreads) k_arg_rows_block(const float* __restrict__ a, size_t rows,
                                                             size_t len, uint32_t* __restrict__ out) {
  __shared__ uint32_t sh[2][32];
  for (size_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const uint64_t best = block_best<MIN>(a + r * len, len, threadIdx.x, kThreads, sh);
    if (threadIdx.x == 0) out[r] = ~(uint32_t)best;
  }
}

// Strided axis (post > 1): a block covers 32 adjacent columns q of one p and
// splits the axis across its 8 warps-rows; the 8 keys per column are merged
// in shared memory.  Loads are 128-byte coalesced along q.
constexpr int kColsX = 32, kColsY = 8;

template <bool MIN>
__global__ void __launch_bounds__(kColsX* kColsY) k_arg_cols(const float* __restrict__ a, size_t prev,
                                                            size_t len, size_t post,
                                                            uint32_t* __restrict__ out) {
  __shared__ uint64_t sh[kColsY][kColsX];
  const size_t qblocks = (post + kColsX - 1) / kColsX;
  for (size_t b = blockIdx.x; b < prev * qblocks; b += gridDim.x) {
    const size_t p = b / qblocks;
    const size_t q = (b % qblocks) * kColsX + threadIdx.x;
    uint64_t best = 0;
    if (q < post) {
      const float* base = a + p * len * post + q;
      for (size_t k = threadIdx.y; k < len; k += kColsY)
        best = kmax(best, make_key<MIN>(__ldg(base + k * post), (uint32_t)k));
    }
    sh[threadIdx.y][threadIdx.x] = best;
    __syncthreads();
    if (threadIdx.y == 0 && q < post) {
#pragma unroll
      for (int y = 1; y < kColsY; ++y) best = kmax(best, sh[y][threadIdx.x]);
      out[p * post + q] = ~(uint32_t)best;
    }
    __syncthreads();
  }
}

template <bool MIN>
int arg_all(vkc_device_t dev, const float* a, size_t n, uint32_t* out) {
  const unsigned g = stream_grid(dev, (n + 15) / 16, kThreads, 8);
  void* part = nullptr;
  int r = scratch_alloc(dev, (size_t)g * sizeof(uint64_t), &part);
  if (r != VKC_OK) return r;
  k_arg_partials<MIN><<<g, kThreads, 0, dev->stream>>>(a, n, static_cast<uint64_t*>(part));
  r = check_launch("argreduce partials");
  if (r == VKC_OK) {
    const cudaError_t e = launch_second(k_arg_final, dim3(1), dim3(1024), dev->stream, n,
                                        static_cast<const uint64_t*>(part), (int)g, out);
    r = e == cudaSuccess ? check_launch("argreduce final")
                         : set_error(VKC_ERR_CUDA, "argreduce final launch: %s", cudaGetErrorString(e));
  }
  scratch_free(dev, part);
  return r;
}

template <bool MIN>
int arg_axis(vkc_device_t dev, const float* a, size_t prev, size_t len, size_t post, uint32_t* out) {
  if (post == 1) {
    if (len >= 2048) {
      const unsigned g = (unsigned)std::min<size_t>(prev, (size_t)dev->sm_count * 16);
      k_arg_rows_block<MIN><<<g, kThreads, 0, dev->stream>>>(a, prev, len, out);
    } else {
      k_arg_rows_warp<MIN><<<stream_grid(dev, prev * 32, kThreads, 8), kThreads, 0, dev->stream>>>(a, prev, len,
                                                                                                    out);
    }
    return check_launch("argreduce rows");
  }
  const size_t blocks = prev * ((post + kColsX - 1) / kColsX);
  const unsigned g = (unsigned)std::min<size_t>(blocks, (size_t)dev->sm_count * 8);
  k_arg_cols<MIN><<<g, dim3(kColsX, kColsY), 0, dev->stream>>>(a, prev, len, post, out);
  return check_launch("argreduce cols");
}

}  // namespace
}  // namespace vkc

VKC_EXPORT int vkc_arg_reduce_all(vkc_device_t dev, int op, const float* a, size_t n, uint32_t* out) {
  VKC_BIND(dev);
  VKC_REQUIRE(op == VKC_ARGMAX || op == VKC_ARGMIN, "unknown arg-reduction %d", op);
  VKC_REQUIRE(n > 0, "arg-reduction of an empty array");
  VKC_REQUIRE(n <= 0xFFFFFFFFull, "arg-reduction indices are uint32: n must be < 2^32");
  VKC_REQUIRE(a && out, "NULL buffer");
  return op == VKC_ARGMAX ? vkc::arg_all<false>(dev, a, n, out) : vkc::arg_all<true>(dev, a, n, out);
}

VKC_EXPORT int vkc_arg_reduce_axis(vkc_device_t dev, int op, const float* a, size_t prev, size_t axis, size_t post,
                                   uint32_t* out) {
  VKC_BIND(dev);
  VKC_REQUIRE(op == VKC_ARGMAX || op == VKC_ARGMIN, "unknown arg-reduction %d", op);
  VKC_REQUIRE(axis > 0, "arg-reduction along an empty axis");
  VKC_REQUIRE(axis <= 0xFFFFFFFFull, "arg-reduction indices are uint32: the axis must be < 2^32");
  if (prev == 0 || post == 0) return VKC_OK;
  VKC_REQUIRE(a && out, "NULL buffer");
  return op == VKC_ARGMAX ? vkc::arg_axis<false>(dev, a, prev, axis, post, out)
                          : vkc::arg_axis<true>(dev, a, prev, axis, post, out);
}
