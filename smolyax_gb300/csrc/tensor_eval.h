// Contraction of 16-bit split operands, shared by gemm_tc.cu (which defines it)
// and tensor_eval.cu.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "smolyax_gb300.h"
#include "tc_util.cuh"

namespace smx {
namespace tc {

// Second word of a tape entry (first: 128 * slot): the entry's factor 2^f (FP32
// bits), the byte offset of its parent on a stack of 128 bytes per depth, and flags.
constexpr int kPop = 1, kPush = 2, kStackMask = 0xf80, kFactorMask = 0x7f800000;
constexpr int kGroup = 64;  // tape entries (panel columns) per group

// Low parts of the pairs (tc_util.cuh): (v - h) 2^kPairShift, or from v 2^kPairShift.
__device__ __forceinline__ __half pair_low(float v, __half h) {
  return __float2half_rn((v - __half2float(h)) * kPairScale);
}
__device__ __forceinline__ __half2 pair_low_scaled(float2 v, __half2 h) {
  return __float22half2_rn(__ffma2_rn(__half22float2(h), make_float2(-kPairScale, -kPairScale), v));
}
__device__ __forceinline__ __half2 pair_low(float2 v, __half2 h) {
  return pair_low_scaled(__fmul2_rn(v, make_float2(kPairScale, kPairScale)), h);
}

// 16 bytes global -> shared, asynchronously (cp.async.wait_all).
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}

// Basis values of all slots, grow[slot][p], and (drow given) their derivatives,
// p < ldp (a multiple of 32; points past P repeat the last one).
void tensor_basis(const smx_tensor& t, const double* x, int64_t P, int64_t ldx, float* grow, float* drow, int64_t ldp,
                  cudaStream_t st);

constexpr int kTf32 = 0, kBf16 = 1, kF16 = 2;

// What far rows are evaluated from (far_points.cuh).
struct FarPoints {
  const float* rows;  // basis values [slot][gstride]; NULL: no such evaluation
  int64_t gstride;
  const int32_t* col_path;  // [K][4]
  const float* B;           // [N][ldk], zero from K to a multiple of 4
  int64_t ldk;
};

// D [M x N] = sum over 64-column groups q of row_scale[q][m] * (A_q B_q^T), times
// col_scale[n], plus bias[n].  A = Ah + Al, B = Bh + Bl, 16-bit, row-major
// K-contiguous; `splits` slices of K leave partial sums in `partial`
// ([splits][M][N]) that are added in order.
struct SplitGemm {
  int bits;  // kBf16 (no scales) or kF16
  const void *Ah, *Al;
  int64_t lda;
  const void *Bh, *Bl;
  int64_t ldb;
  const float* row_scale;
  int64_t ld_scale;
  const float* col_scale;
  int M, N, K;
  float* D;
  int64_t ldd;  // 0: D is [N / 32][M][32], the columns of 32 together
  const float* bias;
  int* err;
  int splits;
  float* partial;
  bool sliced;     // kF16: A is [ceil(K / 64)][M][64], B [ceil(K / 64)][N][64] (lda, ldb unused)
  int accumulate;  // D += instead of D =
  FarPoints far;   // kF16, row-major: rows of D evaluated apart
};
int split_gemm(const SplitGemm& g, cudaStream_t st);

// Tensor map of a K-contiguous operand or panel: rows x cols, pitch ld
// elements, boxes of box_rows x 128 bytes (128-byte swizzle).
int panel_map(CUtensorMap* tm, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows, int bits);

}  // namespace tc
}  // namespace smx
