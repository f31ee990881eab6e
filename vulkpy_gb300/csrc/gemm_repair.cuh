// The three-part split of fp32 operands for tensor-core products, and the
// recomputation, from the fp32 operands, of the results a three-part
// tensor-core product cannot give: those that came out not finite because an
// operand value is inf, NaN or outside the split's range, or because the sum
// overflows.  Ordered fp32 FMAs over k, as the SIMT GEMM.
#pragma once
#include "gemm_simt.cuh"

#include <cuda_bf16.h>

namespace vkc {

// op(A)(m, k) = ta ? a[k*lda + m] : a[m*lda + k]; op(B)(k, n) = tb ? b[n*ldb + k] : b[k*ldb + n]
struct RepairOperands {
  const float* a = nullptr;  // NULL: nothing to repair with (not a three-part product)
  const float* b = nullptr;
  int64_t lda = 0, ldb = 0, k = 0;
  int ta = 0, tb = 0;
};

namespace {

// x = h + m + l exactly (8 significant bits each), or h NaN for a value the
// three parts cannot hold: inf, NaN, |x| >= 2^127 (h could round to inf) and
// 0 < |x| < 2^-110 (l would fall below bf16's smallest subnormal, 2^-133).
__device__ __forceinline__ void split_bf16_3(float x, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  h = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(h);
  m = __float2bfloat16_rn(r);
  l = __float2bfloat16_rn(r - __bfloat162float(m));
  const float a = fabsf(x);
  if (!(a < 0x1p127f) || (a < 0x1p-110f && a != 0.f)) h = __ushort_as_bfloat16(0x7fffu);
}

__device__ __forceinline__ bool all_finite(float a, float b, float c, float d) {
  return (a * 0.f + b * 0.f) + (c * 0.f + d * 0.f) == 0.f;
}

// Whether this warp's 32 x 32 block of accumulators is finite: the lane's
// row counts if row_in, its first `cols` values.  Warp-uniform result.
__device__ __forceinline__ bool block_finite(const uint32_t (&r)[32], bool row_in, int cols) {
  float t = 0.f;
#pragma unroll
  for (int j = 0; j < 32; ++j) t = fmaf(j < cols ? __uint_as_float(r[j]) : 0.f, 0.f, t);
  return !__any_sync(0xffffffffu, row_in && !(t == 0.f));
}

// One result by itself.
__device__ __noinline__ float repair_dot(const RepairOperands& o, int64_t m, int64_t n) {
  const float* a = o.a + (o.ta ? m : m * o.lda);
  const float* b = o.b + (o.tb ? n * o.ldb : n);
  const int64_t sa = o.ta ? o.lda : 1, sb = o.tb ? 1 : o.ldb;
  float acc = 0.f;
  for (int64_t k = 0; k < o.k; ++k) acc = fmaf(a[k * sa], b[k * sb], acc);
  return acc;
}

// The 32 x 32 block at (m0, n0): 256 threads, four rows of one column each;
// K in steps of 32 through shared memory.  acc[i]: row m0 + 4 (tid / 32) + i,
// column n0 + tid % 32.  The caller synchronises before the next block.
struct RepairSmem {
  float a[32][33], b[32][33];  // [k][row], [k][column]
};
__device__ __forceinline__ void repair_block(const RepairOperands& o, int64_t M, int64_t N, int64_t m0, int64_t n0,
                                             RepairSmem& sm, float (&acc)[4]) {
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = 0.f;
  for (int64_t k0 = 0; k0 < o.k; k0 += 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int slow = ty * 4 + i;  // tx runs along the operand's contiguous index
      const int64_t am = m0 + (o.ta ? tx : slow), ak = k0 + (o.ta ? slow : tx);
      const float va = am < M && ak < o.k ? o.a[o.ta ? ak * o.lda + am : am * o.lda + ak] : 0.f;
      if (o.ta) sm.a[slow][tx] = va;
      else sm.a[tx][slow] = va;
      const int64_t bn = n0 + (o.tb ? slow : tx), bk = k0 + (o.tb ? tx : slow);
      const float vb = bn < N && bk < o.k ? o.b[o.tb ? bn * o.ldb + bk : bk * o.ldb + bn] : 0.f;
      if (o.tb) sm.b[tx][slow] = vb;
      else sm.b[slow][tx] = vb;
    }
    __syncthreads();
    const int kk = (int)(o.k - k0 < 32 ? o.k - k0 : 32);
    for (int k = 0; k < kk; ++k) {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = fmaf(sm.a[k][ty * 4 + i], sm.b[k][tx], acc[i]);
    }
    __syncthreads();
  }
}

// C = act(alpha * acc + beta * C + bias) (* act'(dmask)) for repair_block's values.
__device__ __forceinline__ void repair_store(const float (&acc)[4], int64_t M, int64_t N, int64_t m0, int64_t n0,
                                             float alpha, float beta, float* C, int64_t ldc, const float* bias,
                                             int act, const float* dmask, int dact) {
  const int64_t n = n0 + (threadIdx.x & 31);
  if (n >= N) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t m = m0 + (threadIdx.x >> 5) * 4 + i;
    if (m >= M) continue;
    float v = alpha * acc[i];
    if (beta != 0.f) v += beta * C[m * ldc + n];
    if (bias) v += bias[n];
    if (act == VKC_ACT_RELU) v = fmaxf(v, 0.f);
    else if (act == VKC_ACT_SIGMOID) v = 1.0f / (1.0f + expf(0.0f - v));
    if (dmask) v = act_deriv(v, dmask[m * ldc + n], dact);
    C[m * ldc + n] = v;
  }
}

// The blocks that a GEMM launch left (list[0] of them, numbered along rows of
// 32 x 32 blocks).  Usually none: the launch then reads one word and ends.
__global__ void __launch_bounds__(256)
k_gemm_repair(RepairOperands o, int64_t M, int64_t N, float alpha, float beta, float* C, int64_t ldc,
              const float* bias, int act, const float* dmask, int dact, const uint32_t* list) {
  __shared__ RepairSmem sm;
  pdl_wait();
  pdl_trigger();
  const uint32_t count = list[0], per_row = (uint32_t)((N + 31) / 32);
  for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
    const uint32_t blk = list[1 + i];
    const int64_t m0 = (int64_t)(blk / per_row) * 32, n0 = (int64_t)(blk % per_row) * 32;
    float acc[4];
    repair_block(o, M, N, m0, n0, sm, acc);
    repair_store(acc, M, N, m0, n0, alpha, beta, C, ldc, bias, act, dmask, dact);
  }
}

inline int gemm_repair(vkc_device_t dev, const RepairOperands& o, int64_t M, int64_t N, float alpha, float beta,
                       float* C, int64_t ldc, const GemmEpilogue& epi, const uint32_t* list) {
  const cudaError_t e = launch_pdl(k_gemm_repair, dim3((unsigned)dev->sm_count), dim3(256), 0, dev->stream, o, M, N,
                                   alpha, beta, C, ldc, epi.bias, epi.act, epi.dmask, epi.dact, list);
  if (e != cudaSuccess) return set_error(VKC_ERR_CUDA, "gemm repair launch: %s", cudaGetErrorString(e));
  return check_launch("gemm repair");
}

}  // namespace
}  // namespace vkc
