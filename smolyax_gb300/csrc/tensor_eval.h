// Contraction of 16-bit split operands, shared by gemm_tc.cu (which defines it)
// and tensor_eval.cu.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace smx {
namespace tc {

constexpr int kTf32 = 0, kBf16 = 1, kF16 = 2;

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
};
int split_gemm(const SplitGemm& g, cudaStream_t st);

// Tensor map of a K-contiguous operand or panel: rows x cols, pitch ld
// elements, boxes of box_rows x 128 bytes (128-byte swizzle).
int panel_map(CUtensorMap* tm, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows, int bits);

}  // namespace tc
}  // namespace smx
