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

// Operands are scaled by 2^24 for the split, so every float32 below 2^103,
// subnormals included, is the exact sum of three bf16 normals (or zeros) of 8
// significant bits each, and products by 2^48, which the epilogue takes back
// (a result of 2^79 or more overflows on the way and is recomputed).
constexpr float kSplitScale = 0x1p24f, kSplitUnscale = 0x1p-48f;

// 2^24 x = h + m + l exactly, or h NaN for a value the three parts cannot
// hold (inf, NaN, |x| >= 2^103).
__device__ __forceinline__ void split_bf16_3(float x, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  const float v = x * kSplitScale;
  h = __float2bfloat16_rn(v);
  const float r = v - __bfloat162float(h);
  m = __float2bfloat16_rn(r);
  l = __float2bfloat16_rn(r - __bfloat162float(m));
  if (!(fabsf(x) < 0x1p103f)) h = __ushort_as_bfloat16(0x7fffu);
}

// Whether the first `cols` of a lane's N accumulators are finite.
template <int N>
__device__ __forceinline__ bool lane_finite(const float (&r)[N], int cols) {
  float t = 0.f;
#pragma unroll
  for (int j = 0; j < N; ++j) t = fmaf(j < cols ? r[j] : 0.f, 0.f, t);
  return t == 0.f;
}

// The tile at (m0, n0) of the partial sums over k in [k0, k1), into out (M x N),
// by the 256 threads of Sync.
//
// The partial sums are the place for it, since the K ranges share the work: a
// thread per result in the reduction was a chain of all of K (256 x 256 with K =
// 16384 of NaN 2150 us, so 155, FMAs alone 119), and a warp of the GEMM's
// epilogue per 32 rows 1210 us.
template <class Sync>
__device__ __forceinline__ void repair_partial(const RepairOperands& o, int64_t M, int64_t N, int64_t m0, int64_t n0,
                                               int64_t k0, int64_t k1, float* out, SimtSmem& sm) {
  const float* a = o.a + (o.ta ? k0 * o.lda : k0);
  const float* b = o.b + (o.tb ? k0 : k0 * o.ldb);
  const GemmEpilogue none{};
  Sync::sync();  // the previous tile's reads of `sm`
  if (!o.ta && !o.tb)
    simt_tile<false, false, Sync>(M, N, k1 - k0, 1.f, a, o.lda, b, o.ldb, 0.f, out, N, none, nullptr, m0, n0, sm);
  else if (!o.tb)
    simt_tile<true, false, Sync>(M, N, k1 - k0, 1.f, a, o.lda, b, o.ldb, 0.f, out, N, none, nullptr, m0, n0, sm);
  else if (!o.ta)
    simt_tile<false, true, Sync>(M, N, k1 - k0, 1.f, a, o.lda, b, o.ldb, 0.f, out, N, none, nullptr, m0, n0, sm);
  else
    simt_tile<true, true, Sync>(M, N, k1 - k0, 1.f, a, o.lda, b, o.ldb, 0.f, out, N, none, nullptr, m0, n0, sm);
}

// The 128 x 128 tiles that a GEMM launch left (list[0] of them, numbered along
// rows of tiles), by the SIMT GEMM's tile code.  Usually none: the launch then
// reads one word and ends.
template <bool TA, bool TB>
__global__ void __launch_bounds__(kGemmThreads, 2)
k_gemm_repair(RepairOperands o, int64_t M, int64_t N, float alpha, float beta, float* C, int64_t ldc,
              GemmEpilogue epi, const uint32_t* list) {
  __shared__ __align__(16) SimtSmem sm;
  pdl_wait();
  pdl_trigger();
  const uint32_t count = list[0], per_row = (uint32_t)((N + kGemmBN - 1) / kGemmBN);
  for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
    const uint32_t t = list[1 + i];
    __syncthreads();  // the previous tile's reads of `sm` are done
    simt_tile<TA, TB>(M, N, o.k, alpha, o.a, o.lda, o.b, o.ldb, beta, C, ldc, epi, epi.dmask,
                      (int64_t)(t / per_row) * kGemmBM, (int64_t)(t % per_row) * kGemmBN, sm, epi.dact);
  }
}

inline int gemm_repair(vkc_device_t dev, const RepairOperands& o, int64_t M, int64_t N, float alpha, float beta,
                       float* C, int64_t ldc, const GemmEpilogue& epi, const uint32_t* list) {
  auto kern = o.ta ? (o.tb ? k_gemm_repair<true, true> : k_gemm_repair<true, false>)
                   : (o.tb ? k_gemm_repair<false, true> : k_gemm_repair<false, false>);
  const cudaError_t e = launch_pdl(kern, dim3((unsigned)(2 * dev->sm_count)), dim3(kGemmThreads), 0, dev->stream, o, M, N,
                                   alpha, beta, C, ldc, epi, list);
  if (e != cudaSuccess) return set_error(VKC_ERR_CUDA, "gemm repair launch: %s", cudaGetErrorString(e));
  return check_launch("gemm repair");
}

}  // namespace
}  // namespace vkc
