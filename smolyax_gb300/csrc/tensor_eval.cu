// Tensor-core evaluation of the orthogonal form, many outputs: y = A C + c0 with
// A[p][k] = prod_j phi(z_j), the basis products of the entries of Lambda
// (interpolation.py:264-304 re-expressed over the index set).
//
// Operands are split into two 16-bit parts: FP16 with scales (the default), x ~=
// scale (hi + 2^-11 lo), or BF16 (the caller's faster, less precise choice), x ~=
// hi + lo.  FP16 keeps 11 + 11 significant bits, as the TF32 pair of the 3xTF32
// product does, at twice the tensor rate and half the bytes; its narrow exponent
// range is covered by exact powers of two:
//   u_n  per output       max_k |C[k][n]| 2^-u_n in [1, 2)
//   f_k  per entry        max_n |C[k][n]| 2^(-u_n - f_k) in [2^13, 2^14), so that
//                         A[p][k] 2^f_k is the size of the entry's largest term
//                         (factor 0 for an entry without coefficients)
//   s    per point and group of 64 columns: max |A 2^f| / s in [2^14, 2^15)
// B = C 2^(-u - f) and A 2^f / s are split; the contraction multiplies each
// 64-column partial sum by s as it leaves tensor memory (where it was added
// before) and the result by 2^u_n.  With the low parts scaled (tc_util.cuh) an
// element keeps 22 bits down to 2^-29 of the largest of its group and errs by 2^-51 of
// that one below.  A point's group may serve outputs of very different terms (inputs
// far outside the box that some outputs do not use), so where a point has a term of 2^19
// and more, in units of its output's largest coefficient, the contraction evaluates its
// slice of K in FP32 from the coefficients as they are (far_points.cuh).  For the others
// the pairs err by less than 2^-26 of an output's largest coefficient.
//
// Kernels: basis values of all (dimension, degree) slots [slot][point]; the panel
// A in groups of 64 columns; the contraction (gemm_tc.cu).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "tc_util.cuh"
#include "tensor_eval.h"

namespace {

using namespace smx::tc;

constexpr size_t kSmemMax = 227 * 1024;

// x coordinate in FP32, infinities as NaN (the point's value is then NaN).
__device__ __forceinline__ float x32(double v) {
  const float f = static_cast<float>(v);
  return fabsf(f) == __int_as_float(0x7f800000) ? __int_as_float(0x7fc00000) : f;
}

// Basis rows grow[slot][p] (DERIV: and their derivatives in z, drow) of 32 points x
// 32 dimensions per block: x is read by rows (32 neighbouring dimensions of a
// point) and turned in shared memory, then lane = point.  The dimensions' table
// entries are read beside x, not one after the other by the warps that use them.
// x read and rows written are 160 + 100 MB at 1e5 points x 200 dimensions: 72 us (76
// with derivatives; issue slots 79 % busy), 98 us (108) with the table entries read
// where they are used.  One thread per point ran through all dimensions one after
// the other at first: 69 us at 3001 points x 200 dimensions, now 6.8.
template <bool DERIV>
__global__ void __launch_bounds__(256) tensor_basis_kernel(smx_tensor t, const double* __restrict__ x, int64_t P,
                                                           int64_t ldx, float* __restrict__ grow,
                                                           float* __restrict__ drow, int64_t gstride) {
  __shared__ float z[32][33];
  __shared__ int4 of[32];  // largest degree, first slot, first recurrence pair
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t p0 = blockIdx.x * int64_t(32);
  for (int h0 = blockIdx.y * 32; h0 < t.n_dims; h0 += gridDim.y * 32) {
    const int h = h0 + lane;
    if (h < t.n_dims) {
      const int dim = __ldg(t.dims + h);
      double v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = __ldg(x + min(p0 + warp + 8 * i, P - 1) * ldx + dim);
      const float fa = __ldg(t.fam_a + dim), fb = __ldg(t.fam_b + dim);
      if (warp == 0) of[lane] = make_int4(__ldg(t.dmax + h), __ldg(t.dsoff + h), __ldg(t.fam + dim) * t.max_deg, 0);
#pragma unroll
      for (int i = 0; i < 4; ++i) z[lane][warp + 8 * i] = fmaf(fa, x32(v[i]), fb);
    }
    __syncthreads();
    for (int q = warp; q < 32 && h0 + q < t.n_dims; q += 8) {
      const int4 m = of[q];
      const float2* rec = reinterpret_cast<const float2*>(t.rec) + m.z;
      const float zv = z[q][lane];
      float* to = grow + int64_t(m.y) * gstride + p0 + lane;
      float* td = DERIV ? drow + int64_t(m.y) * gstride + p0 + lane : nullptr;
      float pm1 = 0.f, pc = 1.f, dm1 = 0.f, dc = 0.f;
      for (int n = 0; n < m.x; ++n) {
        const float2 ab = __ldg(rec + n);
        const float pn = ab.x * zv * pc - ab.y * pm1;
        if constexpr (DERIV) {
          const float dn = ab.x * (pc + zv * dc) - ab.y * dm1;
          dm1 = dc, dc = dn;
          td[n * gstride] = dc;
        }
        pm1 = pc, pc = pn;
        to[n * gstride] = pc;
      }
    }
    __syncthreads();
  }
}

// One bulk tensor store of a 64-column x 128-row tile.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tm, const void* src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                   reinterpret_cast<uint64_t>(tm)),
               "r"(c0), "r"(c1), "r"(smem_u32(src))
               : "memory");
}

// Panel: a block of W warps holds 32 points (lane = point) and the basis rows of
// all slots in shared memory; each warp walks its own run of groups of the tape
// (entries in DFS pre-order; two words: the row's byte offset, and factor, stack
// offset and flags).
// An entry is its parent's product, held in a register, times its basis value:
// siblings follow each other, so most entries are one multiplication; an entry
// with children stores its product on a stack by depth (kPush), the first entry
// after a finished subtree (and of every group) reads its parent back (kPop).  The tape is padded in front to whole
// groups, group t of the tape being the columns 64 (n_groups - 1 - t) .. + 63 in
// reversed order (descendants, with small coefficients, precede their
// ancestors); any group may start a run, because `path` lists the slots above its
// first entry.  The 64 values of a group stay in registers until their maximum is
// known, are scaled, split and written as the lane's own 128-byte row of two
// swizzled tiles, which leave by TMA while the next group is walked; the warps
// never wait for each other.  Bound: HBM writes, 4 bytes per value.
// Gauss-Hermite d_in = 100, |Lambda| = 20010, 65536 points: 1.15 ms (4.6 TB/s of
// writes); the TF32 panel it replaces wrote twice the bytes in 3.2 ms.  Measured
// on the way: basis rows read from global memory 3.2 ms (latency), every product
// through the stack 1.35 ms, the tape read from global memory 1.3 - 1.8 ms.  The
// rows are copied with cp.async (no registers between loads and stores): Leja d_in
// = 200, |Lambda| = 5000, 1e5 points 524 us, 554 with loads through registers; the
// scaled low parts are 2 % more issue slots (534 us).
template <bool F16, int W, bool SROWS>
__global__ void __launch_bounds__(32 * W, 1)
    tensor_panel_kernel(const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmL, smx_tensor t,
                        int groups_per_block, const float* __restrict__ grow, int64_t gstride, int64_t P,
                        float* __restrict__ S, int64_t lds) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t* tileH = base + warp * 8192;
  uint8_t* tileL = tileH + 4096;
  uint8_t* ring = base + W * 8192 + warp * 1024;                                       // two tape groups
  float* stk = reinterpret_cast<float*>(base + W * 9216) + warp * (9 * 32) + lane;  // stk[32 d]: first d factors
  float* rows = reinterpret_cast<float*>(base + W * (9216 + 9 * 128));
  const int b0 = blockIdx.x * groups_per_block, nb = min(t.n_groups - b0, groups_per_block);
  const int t0 = b0 + nb * warp / W, t1 = b0 + nb * (warp + 1) / W;
  const int64_t n_pb = (P + 31) / 32;
  for (int64_t pb = blockIdx.y; pb < n_pb; pb += gridDim.y) {
    const int64_t p0 = pb * 32;
    const float* row = SROWS ? rows + lane : grow + p0 + lane;
    const int64_t rs = SROWS ? 32 : gstride;
    if constexpr (SROWS) {
      __syncthreads();  // the previous points' walks are done
      for (int i = warp * 4 + (lane >> 3); i < t.n_slots; i += W * 4)
        copy16(rows + i * 32 + (lane & 7) * 4, grow + i * gstride + p0 + (lane & 7) * 4);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
    }
    if (t0 == t1) continue;
    stk[0] = 1.f;
    for (int i = 0; i < 8; ++i) {
      const int s = __ldg(t.path + t0 * 8 + i);
      if (s < 0) break;
      stk[(i + 1) * 32] = stk[i * 32] * row[s * rs];
    }
    // the warp's next tape group is copied while the current one is walked
    const int4* tape = reinterpret_cast<const int4*>(t.tape) + t0 * (kGroup / 2) + lane;
    auto copy_group = [&](int g) {
      if (g < t1)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(ring + (g & 1) * 512 + lane * 16)),
                     "l"(tape + (g - t0) * (kGroup / 2))
                     : "memory");
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    copy_group(t0);
    const char* rowb = reinterpret_cast<const char*>(row);
    char* stkb = reinterpret_cast<char*>(stk);
    for (int g = t0; g < t1; ++g) {
      copy_group(g + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      const int4* words = reinterpret_cast<const int4*>(ring + (g & 1) * 512);
      float v[kGroup];
      float m = 0.f, cur = 1.f;
#pragma unroll
      for (int k = 0; k < kGroup; k += 4) {
        const int4 wa = words[k / 2], wb = words[k / 2 + 1];
        const int wr[4] = {wa.x, wa.z, wb.x, wb.z}, wf[4] = {wa.y, wa.w, wb.y, wb.w};
        float b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          b[u] = SROWS ? *reinterpret_cast<const float*>(rowb + wr[u]) : row[(wr[u] >> 7) * gstride];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (wf[u] & kPop) cur = *reinterpret_cast<const float*>(stkb + (wf[u] & kStackMask));
          float q = cur * b[u];
          if (wf[u] & kPush) {
            cur = q;
            *reinterpret_cast<float*>(stkb + (wf[u] & kStackMask) + 128) = q;
          }
          if constexpr (F16) q *= __int_as_float(wf[u] & kFactorMask);
          v[k + u] = q;
          m = fmaxf(m, fabsf(q));
        }
      }
      const int q = t.n_groups - 1 - g;  // column group
      float inv = 1.f;
      if constexpr (F16) {
        // power of two that brings the maximum to [2^14, 2^15); products below
        // 2^-100 are left unscaled to the end of the range
        const int e = min(max(__float_as_int(m) >> 23, 27), 254);
        inv = __int_as_float((268 - e) << 23);
        S[int64_t(q) * lds + p0 + lane] = __int_as_float((e - 14) << 23);
      }
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the tiles' previous stores
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) {  // columns 8 i .. 8 i + 7 of the row: values 63 - 8 i, ...
        uint32_t h[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 vv = make_float2(v[63 - 8 * i - 2 * k], v[62 - 8 * i - 2 * k]);
          const float2 ab = __fmul2_rn(vv, make_float2(inv, inv));
          if constexpr (F16) {
            const __half2 hh = __float22half2_rn(ab);
            const __half2 ll = pair_low_scaled(__fmul2_rn(vv, make_float2(inv * kPairScale, inv * kPairScale)), hh);
            h[k] = *reinterpret_cast<const uint32_t*>(&hh);
            l[k] = *reinterpret_cast<const uint32_t*>(&ll);
          } else {
            const __nv_bfloat162 hh = __float22bfloat162_rn(ab);
            const __nv_bfloat162 ll =
                __float22bfloat162_rn(__ffma2_rn(__bfloat1622float2(hh), make_float2(-1.f, -1.f), ab));
            h[k] = *reinterpret_cast<const uint32_t*>(&hh);
            l[k] = *reinterpret_cast<const uint32_t*>(&ll);
          }
        }
        const int at = lane * 128 + ((i ^ (lane & 7)) << 4);
        *reinterpret_cast<uint4*>(tileH + at) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(tileL + at) = make_uint4(l[0], l[1], l[2], l[3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmH, tileH, q * kGroup, int(p0));
        tma_store_2d(&tmL, tileL, q * kGroup, int(p0));
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    }
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

size_t panel_smem(int warps, int slots) { return 1024 + size_t(warps) * (9216 + 9 * 128) + size_t(slots) * 128; }

template <bool F16, int W, bool SROWS>
void launch_panel(const CUtensorMap& tmH, const CUtensorMap& tmL, const smx_tensor& t, const float* grow,
                  int64_t gstride, int64_t m, float* S, int sms, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(tensor_panel_kernel<F16, W, SROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(kSmemMax));
    attr = true;
  }
  // runs of groups per block: the split of the tape with the shortest total of
  // rounds on the SMs x (groups of a warp + about 2 groups' time to load the
  // rows and start)
  const int64_t n_pb = (m + 31) / 32;
  int per = t.n_groups;
  int64_t best = -1;
  for (int segs = 1; segs <= 32 && segs * W <= t.n_groups + W - 1; ++segs) {
    const int p = (t.n_groups + segs - 1) / segs;
    const int64_t blocks = n_pb * ((t.n_groups + p - 1) / p);
    const int64_t cost = ((blocks + sms - 1) / sms) * ((p + W - 1) / W + 2);
    if (best < 0 || cost < best) best = cost, per = p;
  }
  const dim3 grid(unsigned((t.n_groups + per - 1) / per), unsigned(std::min<int64_t>(n_pb, 65535)));
  tensor_panel_kernel<F16, W, SROWS><<<grid, 32 * W, panel_smem(W, SROWS ? t.n_slots : 0), st>>>(
      tmH, tmL, t, per, grow, gstride, m, S, gstride);
}

// 16 warps with the basis rows in shared memory up to ~510 slots, 8 warps up to
// ~1160; beyond, the rows are read through L1.
template <bool F16>
void launch_panel(const CUtensorMap& tmH, const CUtensorMap& tmL, const smx_tensor& t, const float* grow,
                  int64_t gstride, int64_t m, float* S, int sms, cudaStream_t st) {
  if (panel_smem(16, t.n_slots) <= kSmemMax)
    launch_panel<F16, 16, true>(tmH, tmL, t, grow, gstride, m, S, sms, st);
  else if (panel_smem(8, t.n_slots) <= kSmemMax)
    launch_panel<F16, 8, true>(tmH, tmL, t, grow, gstride, m, S, sms, st);
  else
    launch_panel<F16, 16, false>(tmH, tmL, t, grow, gstride, m, S, sms, st);
}

// ---- operands -------------------------------------------------------------------------------
// Per output the power of two of its largest finite coefficient.
__global__ void output_scale_kernel(const float* __restrict__ B, int K, int64_t ldb, float* __restrict__ scale) {
  __shared__ float red[256];
  const float* b = B + int64_t(blockIdx.x) * ldb;
  float m = 0.f;
  for (int k = threadIdx.x; k < K; k += 256) {
    const float a = fabsf(b[k]);
    if (a <= 3.0e38f) m = fmaxf(m, a);
  }
  red[threadIdx.x] = m;
  __syncthreads();
  for (int n = 128; n; n >>= 1) {
    if (threadIdx.x < n) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + n]);
    __syncthreads();
  }
  if (threadIdx.x == 0)
    scale[blockIdx.x] = red[0] > 0.f ? __int_as_float(min(max(__float_as_int(red[0]) >> 23, 1), 253) << 23) : 1.f;
}

__device__ __forceinline__ float scaled(float b, float scale) {
  return b * __int_as_float((254 << 23) - __float_as_int(scale));  // b / scale, scale a power of two
}

// The padded tape: per column k (tape entry j = K - 1 - k) the factor 2^f (1 without
// a B) and the stack flags.  An entry whose coefficients are all zero gets the factor
// 0: its product must not set the scale of its point's group.
__global__ void tape_kernel(const float* __restrict__ B, int N, int K, int64_t ldb, const float* __restrict__ scale,
                            const int32_t* __restrict__ tape, int pad, int2* __restrict__ tape_out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  // padding in front: depth 1, factor 0 (its columns are past K)
  if (k < pad) tape_out[k] = make_int2(0, k == 0 ? kPop : 0);
  if (k >= K) return;
  int factor = 127 << 23;
  if (B) {
    float m = 0.f;
    bool any = false;
    for (int n = 0; n < N; ++n) {
      const float b = B[n * ldb + k], a = fabsf(scaled(b, scale[n]));
      any = any || !(b == 0.f);
      if (a <= 3.0e38f) m = fmaxf(m, a);
    }
    const int e = m > 0.f ? (__float_as_int(m) >> 23) - 127 : 13;
    factor = any ? (min(max(e - 13, -100), 100) + 127) << 23 : 0;
  }
  const int j = K - 1 - k;
  const int w = tape[j], d = w >> 16;
  const int before = j ? tape[j - 1] >> 16 : 0, after = j + 1 < K ? tape[j + 1] >> 16 : 0;
  const int flags = ((pad + j) % kGroup == 0 || before > d ? kPop : 0) | (after == d + 1 ? kPush : 0);
  tape_out[pad + j] = make_int2((w & 0xffff) * 128, factor | ((d - 1) * 128) | flags);
}

__global__ void split_f16_kernel(const float* __restrict__ B, int N, int K, int64_t ldb,
                                 const float* __restrict__ scale, const int2* __restrict__ tape_out, int pad,
                                 __half* __restrict__ Bh, __half* __restrict__ Bl, int64_t ldh) {
  const int64_t n_all = int64_t(N) * K;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n_all; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t n = i / K;
    const int k = int(i - n * K);
    const int factor = tape_out[pad + K - 1 - k].y & kFactorMask;  // 2^f
    const float v = scaled(B[n * ldb + k], scale[n]) * __int_as_float((254 << 23) - factor);
    const __half h = __float2half_rn(v);
    Bh[n * ldh + k] = h;
    Bl[n * ldh + k] = pair_low(v, h);
  }
}

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

struct Layout {  // workspace of one chunk of m points
  int64_t gstride;
  size_t panel, scales, rows, partial, total;
};
Layout layout(const smx_tensor* t, int64_t m) {
  Layout L;
  L.gstride = (m + 127) / 128 * 128;
  L.panel = up256(size_t(m) * t->ldb * 2);
  L.scales = up256(size_t(t->n_groups) * L.gstride * 4);
  L.rows = up256(size_t(t->n_slots) * L.gstride * 4);
  L.partial = t->splits > 1 ? up256(size_t(t->splits) * m * t->d_out * 4) : 0;
  L.total = 2 * L.panel + L.scales + L.rows + L.partial;
  return L;
}

}  // namespace

void smx::tc::tensor_basis(const smx_tensor& t, const double* x, int64_t P, int64_t ldx, float* grow, float* drow,
                           int64_t ldp, cudaStream_t st) {
  const dim3 grid(unsigned(ldp / 32), unsigned(std::min((t.n_dims + 31) / 32, 65535)));
  if (drow)
    tensor_basis_kernel<true><<<grid, 256, 0, st>>>(t, x, P, ldx, grow, drow, ldp);
  else
    tensor_basis_kernel<false><<<grid, 256, 0, st>>>(t, x, P, ldx, grow, nullptr, ldp);
}

extern "C" int smx_tensor_operands(const float* B, int N, int K, int64_t ldb, const int32_t* tape, int32_t* tape_out,
                                   uint16_t* Bh, uint16_t* Bl, int64_t ldh, float* out_scale, void* stream) {
  SMX_REQUIRE(N >= 1 && K >= 1 && ldb >= K && ldh >= K && B && tape && tape_out && Bh && Bl && out_scale,
              "smx_tensor_operands: bad arguments");
  cudaStream_t st = smx::as_stream(stream);
  const int pad = (K + kGroup - 1) / kGroup * kGroup - K;
  output_scale_kernel<<<N, 256, 0, st>>>(B, K, ldb, out_scale);
  tape_kernel<<<smx::grid_for(std::max(K, pad), 128), 128, 0, st>>>(B, N, K, ldb, out_scale, tape, pad,
                                                                    reinterpret_cast<int2*>(tape_out));
  split_f16_kernel<<<smx::grid_for(std::min<int64_t>(int64_t(N) * K, 1 << 24), 256), 256, 0, st>>>(
      B, N, K, ldb, out_scale, reinterpret_cast<const int2*>(tape_out), pad, reinterpret_cast<__half*>(Bh), reinterpret_cast<__half*>(Bl), ldh);
  SMX_LAUNCH_CHECK("smx_tensor_operands");
  return SMX_OK;
}

extern "C" int smx_tensor_tape(const int32_t* tape, int K, int32_t* tape_out, void* stream) {
  SMX_REQUIRE(K >= 1 && tape && tape_out, "smx_tensor_tape: bad arguments");
  const int pad = (K + kGroup - 1) / kGroup * kGroup - K;
  tape_kernel<<<smx::grid_for(std::max(K, pad), 128), 128, 0, smx::as_stream(stream)>>>(nullptr, 0, K, 0, nullptr, tape,
                                                                                       pad, reinterpret_cast<int2*>(tape_out));
  SMX_LAUNCH_CHECK("smx_tensor_tape");
  return SMX_OK;
}

// K slices of the contraction: fixed per plan (a point's value does not depend
// on its batch).  Few outputs leave few tiles, so K is cut as long as the slices
// hold 1024 columns and their partial sums (8 bytes per point, slice and output,
// written and read) stay below an eighth of the panel's bytes.
extern "C" int smx_tensor_splits(int d_out, int K) {
  if (d_out < 1 || K < 1) return 1;
  return std::max(1, std::min({8, K / 1024, K / (8 * d_out)}));
}

// Points per pass: the panel within the memory limit, all scratch (basis rows, scales
// and partial sums too) within 9/8 of it, and at most 65535 tiles of 128 rows (the
// contraction's second grid dimension).
namespace {
constexpr int64_t kMaxPass = int64_t(65535) * 128;
}

extern "C" int64_t smx_tensor_chunk(const smx_tensor* t, double memory_limit_gib) {
  if (!t || t->ldb < 1) return 128;
  const double limit = memory_limit_gib * 1073741824.0, panel = 4.0 * double(t->ldb);
  const double all = panel + 4.0 * t->n_groups + 4.0 * t->n_slots + (t->splits > 1 ? 4.0 * t->splits * t->d_out : 0.0);
  const int64_t fit = int64_t(std::min({limit / panel, 1.125 * limit / all, double(kMaxPass)}));
  return std::max<int64_t>(128, fit / 128 * 128);
}

extern "C" size_t smx_tensor_workspace(const smx_tensor* t, int64_t P) {
  if (!t || P <= 0 || t->chunk < 1) return 0;
  return layout(t, std::min(P, t->chunk)).total;
}

extern "C" int smx_tensor_eval(const smx_tensor* t, const double* x, int64_t P, int64_t ldx, float* y, void* ws,
                               size_t ws_bytes, void* stream) {
  SMX_REQUIRE(t != nullptr, "smx_tensor_eval: null plan");
  SMX_REQUIRE(t->d_in >= 1 && t->d_out >= 1 && t->K >= 0 && t->n_groups == (t->K + kGroup - 1) / kGroup &&
                  t->splits >= 1 && t->chunk >= 1 && t->ldb >= t->K && t->ldb % kGroup == 0,
              "smx_tensor_eval: bad plan sizes");
  SMX_REQUIRE(P >= 0 && ldx >= t->d_in, "smx_tensor_eval: bad sizes");
  SMX_REQUIRE(std::min(P, t->chunk) <= kMaxPass, "smx_tensor_eval: more points per pass than smx_tensor_chunk allows");
  if (P == 0) return SMX_OK;
  SMX_REQUIRE(x && y && t->bias && t->err, "smx_tensor_eval: null pointer");
  SMX_REQUIRE(t->K == 0 || (t->dims && t->dmax && t->dsoff && t->fam && t->fam_a && t->fam_b && t->rec && t->tape &&
                            t->path && t->Bh && t->Bl && (t->bf16 || t->out_scale) &&
                            (!t->B || (t->ldk >= t->K && t->ldk % 4 == 0 && t->col_path))),
              "smx_tensor_eval: incomplete plan");
  SMX_REQUIRE(ws && ws_bytes >= smx_tensor_workspace(t, P) && (reinterpret_cast<uintptr_t>(ws) & 15) == 0,
              "smx_tensor_eval: workspace too small or not 16-byte aligned");
  cudaStream_t st = smx::as_stream(stream);
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return smx::set_error(SMX_ERR_CUDA, "smx_tensor_eval: no device");
  for (int64_t p0 = 0; p0 < P; p0 += t->chunk) {
    const int64_t m = std::min(t->chunk, P - p0);
    const Layout L = layout(t, m);
    uint8_t* w = static_cast<uint8_t*>(ws);
    void* Ah = w;
    void* Al = w + L.panel;
    float* S = reinterpret_cast<float*>(w + 2 * L.panel);
    float* grow = reinterpret_cast<float*>(w + 2 * L.panel + L.scales);
    float* part = reinterpret_cast<float*>(w + 2 * L.panel + L.scales + L.rows);
    int rc;
    if (t->K > 0) {
      tensor_basis(*t, x + p0 * ldx, m, ldx, grow, nullptr, L.gstride, st);
      CUtensorMap tmH, tmL;
      const int bits = t->bf16 ? kBf16 : kF16;
      if ((rc = panel_map(&tmH, Ah, m, t->K, t->ldb, 32, bits)) ||
          (rc = panel_map(&tmL, Al, m, t->K, t->ldb, 32, bits)))
        return rc;
      if (t->bf16)
        launch_panel<false>(tmH, tmL, *t, grow, L.gstride, m, nullptr, sms, st);
      else
        launch_panel<true>(tmH, tmL, *t, grow, L.gstride, m, S, sms, st);
      SMX_LAUNCH_CHECK("smx_tensor_eval panel");
    }
    SplitGemm g{};
    g.bits = t->bf16 ? kBf16 : kF16;
    g.Ah = Ah, g.Al = Al, g.lda = t->ldb;
    g.Bh = t->Bh, g.Bl = t->Bl, g.ldb = t->ldb;
    g.row_scale = t->bf16 ? nullptr : S, g.ld_scale = L.gstride;
    g.col_scale = t->bf16 ? nullptr : t->out_scale;
    g.M = int(m), g.N = t->d_out, g.K = t->K;
    g.D = y + p0 * t->d_out, g.ldd = t->d_out;
    g.bias = t->bias, g.err = t->err;
    g.splits = t->splits, g.partial = part;
    if (t->B && !t->bf16) g.far = FarPoints{grow, L.gstride, t->col_path, t->B, t->ldk};
    if ((rc = split_gemm(g, st))) return rc;
  }
  return SMX_OK;
}
