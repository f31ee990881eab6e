// Tensor-core (tcgen05) GEMM for bf16 and split-bf16x3 arithmetic.
#pragma once
#include "common.cuh"
#include "gemm_simt.cuh"

#include <cuda_bf16.h>

namespace vkc {

// K-major bf16 rows (pitch ldk elements, a multiple of 64) of a GEMM result,
// hi = bf16(x) and, for the split mode, lo = bf16(x - hi): the form the
// tensor-core GEMM's operand pre-pass writes, so a following GEMM can take
// the result as its op(A) without a pre-pass of its own.
struct SplitOut {
  __nv_bfloat16* hi;
  __nv_bfloat16* lo;  // NULL in bf16 mode
  int64_t ldk;
};

// C = act(alpha * op(A) op(B) + beta * C + bias) with fp32 A, B, C in memory
// and bf16 (or hi/lo split bf16) tensor-core products accumulated in fp32.
int gemm_tc(vkc_device_t dev, int precision, bool ta, bool tb, int64_t M, int64_t N, int64_t K, float alpha,
            const float* A, int64_t lda, const float* B, int64_t ldb, float beta, float* C, int64_t ldc,
            GemmEpilogue epi);

// Whether a plain fp32 product runs as six bf16 tensor-core products (three
// exact parts per operand) instead of fp32 FMAs in `splits` K ranges.
// The FMA GEMM's time is its chain of K steps (0.115 us per step, 2.5 us of
// launch, 3.5 us more for the reduction of several ranges) until the output
// fills the GPU several times over; the tensor path's three launches cost 8 us
// with one K block.  Measured (us, FMA -> tensor, graph replay): 256 x 256 x
// 64 10.9 -> 9.4, 128^3 17.5 -> 10.4, 300^3 (19 ranges of 16) 12.6 -> 11.2,
// 256^3 (16 ranges of 16) 9.3 -> 10.9, 1024 x 1024 x 48 9.2 -> 9.6, 4096 x
// 4096 x 16 30.6 -> 27.9.  Run call by call the third launch costs another 1.5
// us of host time, hence 96 steps rather than 64.  Unsplit products up to K =
// 256 whose small tiles fit the GPU at once go to k_gemm_small all the same
// (128^3 4.0 us).
inline bool fp32_on_tensor_cores(int64_t M, int64_t N, int64_t K, int splits) {
  if (M < 2 || N < 2 || K < 16) return false;                            // vectors are bound by reading the matrix
  if (M > (1 << 22) || N > (1 << 22) || K >= (1ll << 31)) return false;  // 32-bit tile and row coordinates
  const int64_t chain = (K + splits - 1) / splits;
  return chain + (splits > 1 ? 32 : 0) >= 96 || M * N >= (1 << 24);
}

// The same for the products of layers: vkc_gemm, the grouped GEMM and the
// Dense calls, which agree with one another bit for bit where the single call
// does not split K (the grouped GEMM never does).  Run call by call a layer is
// bound by the host up to about 2^30 (256 x 784 -> 1024 -> 1024 -> 10: 176 us a
// step with FMAs, 191 with the tensor path's extra launches; 4096 x 2048 -> 2048
// forward and backward: 2410 us with FMAs, 637 on the tensor cores).  In a
// graph or a grouped launch, where that cost is gone, the tensor path is the
// faster one from less work on (256 x 1024 x 784: 22.8 -> 14.3 us; a grouped
// step of 64 models 2160 -> 974), but there too the line stays here: in a
// network a ReLU passes another rounding on as another sign wherever a value
// is within it of zero, so that below the line trained models would leave the
// values they have with FMAs (gradients of that grouped step by 4.5e-4, though
// nearer to float64: 7e-5 against 2.8e-4).
inline bool layer_fp32_on_tensor_cores(int64_t M, int64_t N, int64_t K, int splits) {
  return fp32_on_tensor_cores(M, N, K, splits) && M * N * K >= (int64_t(1) << 30);
}

// C = act(alpha * op(A) op(B) + beta * C + bias) (* act'(dmask)) in fp32: on
// the tensor cores or with FMAs, by fp32_on_tensor_cores (layer: by
// layer_fp32_on_tensor_cores).
int gemm_fp32(vkc_device_t dev, bool ta, bool tb, int64_t M, int64_t N, int64_t K, float alpha, const float* A,
              int64_t lda, const float* B, int64_t ldb, float beta, float* C, int64_t ldc, GemmEpilogue epi,
              bool layer = true);

// C *= act'(epi.dmask) as a launch of its own, after a GEMM that could not
// apply it (nn.cu).
int act_deriv_after(vkc_device_t dev, const GemmEpilogue& epi, float* C, int64_t M, int64_t N, int64_t ldc);

// gemm_tc on operands already split ([M][Kp] and [N][Kp] K-major bf16, Kp =
// K rounded up to 64, zero past K); `out` (may be NULL) also receives C in
// that form (pitch out->ldk, zero from N on).  M, N, K > 0.
int gemm_tc_presplit(vkc_device_t dev, int precision, int64_t M, int64_t N, int64_t K, float alpha,
                     const __nv_bfloat16* a_hi, const __nv_bfloat16* a_lo, const __nv_bfloat16* b_hi,
                     const __nv_bfloat16* b_lo, float beta, float* C, int64_t ldc, const GemmEpilogue& epi,
                     const SplitOut* out);

// The operand pre-pass alone: op(A) (M x K, K contiguous iff a_kcontig) and
// op(B)^T (N x K) into K-major bf16 hi (and lo) rows of pitch Kp, one launch.
int tc_split_operands(vkc_device_t dev, const float* A, int64_t M, int64_t lda, bool a_kcontig,
                      __nv_bfloat16* a_hi, __nv_bfloat16* a_lo, const float* B, int64_t N, int64_t ldb,
                      bool b_kcontig, __nv_bfloat16* b_hi, __nv_bfloat16* b_lo, int64_t K, int64_t Kp);

}  // namespace vkc
