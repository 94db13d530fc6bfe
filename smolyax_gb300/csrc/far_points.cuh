// Rows of the scaled FP16 product whose terms exceed the range of the pairs
// (tensor_eval.cu): the drain warps see each row's scale of every 64-column group, and
// a block evaluates the rows that reach kFarScale once more, over its columns of K, in
// FP32 from the coefficients as they are.
#pragma once

#include <stdint.h>

#include "tensor_eval.h"

namespace smx {
namespace tc {

// Scale of a group whose largest product times its factor 2^f, which brings the entry's
// largest coefficient to [2^13, 2^14), reaches 64 (scale: 2^14 below its power of two).
constexpr float kFarScale = 1.f / 256.f;
constexpr int kFarPts = 8, kFarCols = 512;
constexpr int kFarBytes = kFarPts * kFarCols * 4;  // of shared memory

// D[p][o] = bias[o] + sum of A[p][k] B[o][k] over columns [K0, K1) (K0 a multiple of 4)
// for points p[0 .. kFarPts) and outputs [o0, o1), by all threads of a block: the
// products of kFarCols columns in shared memory (each along its column's slots), a thread
// per output, sums of 64 columns in FP32 and those added in FP64, so that a value depends
// on its point alone.
static __device__ __noinline__ void far_batch(const FarPoints& f, const int (&p)[kFarPts], int K0, int K1, int o0,
                                              int o1, const float* __restrict__ bias, float* __restrict__ D,
                                              int64_t ldd, float* a) {
  for (int o = o0 + int(threadIdx.x); o - int(threadIdx.x) < o1; o += blockDim.x) {
    const float4* b = reinterpret_cast<const float4*>(f.B + int64_t(min(o, o1 - 1)) * f.ldk);
    double sum[kFarPts] = {};
    for (int k0 = K0; k0 < K1; k0 += kFarCols) {
      const int nk = min(kFarCols, (K1 - k0 + 3) / 4 * 4);
      __syncthreads();
      for (int k = threadIdx.x; k < nk; k += blockDim.x) {
        float v[kFarPts];
        const bool in = k0 + k < K1;
#pragma unroll
        for (int i = 0; i < kFarPts; ++i) v[i] = in ? 1.f : 0.f;
        const int4 s4 = in ? __ldg(reinterpret_cast<const int4*>(f.col_path) + k0 + k) : make_int4(-1, -1, -1, -1);
        const unsigned s2[4] = {unsigned(s4.x), unsigned(s4.y), unsigned(s4.z), unsigned(s4.w)};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const unsigned s = (s2[q >> 1] >> (16 * (q & 1))) & 0xffffu;
          if (s == 0xffffu) break;
#pragma unroll
          for (int i = 0; i < kFarPts; ++i) v[i] *= __ldg(f.rows + s * f.gstride + p[i]);
        }
#pragma unroll
        for (int i = 0; i < kFarPts; i += 4)
          *reinterpret_cast<float4*>(a + k * kFarPts + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      }
      __syncthreads();
      if (o >= o1) continue;
      for (int k = 0; k < nk; k += 64) {
        float acc[kFarPts] = {};
#pragma unroll 4
        for (int j = k; j < min(nk, k + 64); j += 4) {
          const float4 b4 = __ldg(b + (k0 + j) / 4);
          const float bk[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int i = 0; i < kFarPts; ++i) acc[i] = fmaf(bk[u], a[(j + u) * kFarPts + i], acc[i]);
        }
#pragma unroll
        for (int i = 0; i < kFarPts; ++i) sum[i] += double(acc[i]);
      }
    }
    if (o < o1)
#pragma unroll
      for (int i = 0; i < kFarPts; ++i)
        D[int64_t(p[i]) * ldd + o] = float(sum[i] + (bias ? double(__ldg(bias + o)) : 0.0));
  }
}

}  // namespace tc
}  // namespace smx
