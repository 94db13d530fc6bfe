// Backward of the tensor-core evaluation, with respect to x:
//   G^T[e][p] = sum_o C[e][o] g[p][o]       (tensor cores, scaled FP16 pairs)
//   dL/dx[p][j] = a_j sum_g phi_g'(z_j) bar[slot (j, g)]
// with bar the adjoints of the basis values under L = sum_e G_e prod phi, and
// dL/dC[e][o] = sum_p A[p][e] g[p][o] further down.  The reference has the dense
// Jacobian instead (interpolation.py:306-345).
//
// Range of G's FP16 pairs (tc_util.cuh): one power of two per point for g (in units of
// the outputs' largest coefficients) and one per entry and 64 outputs for C, so that
// G[e][p] has the accuracy of the TF32 pairs while max |C[e]| max |g[p]| is below 2^29
// times the largest of its terms (outputs in disjoint inputs, 2^29 apart in C g).
//
// G is made transposed in blocks of 32 points, [p / 32][entry][32]: a block of 32
// warps (lane = point) streams its adjoints once, in order, through shared
// memory.  Each entry is two terms, row value * G added to a destination row
// (the adjoint of its last slot; the sum over its parent's children), every
// destination owned by one warp (layout.cu build_walk); the products of whole
// paths are formed only for the few nodes with children, at the end.  No
// adjoint is read, updated and written per path factor in global memory, and
// the order of every sum is fixed.  Traffic that has to be: G^T written and read
// once.  Leja d_in = 200, d_out = 64, |Lambda| = 5000, 1e5 points: the walk takes
// 1.13 ms (56 % of its issue slots and 61 % of the shared-memory pipe busy, the
// bound), G^T 0.32 ms, basis and cotangent 0.10 ms; the TF32 product and the walk
// per path factor through global memory took 0.82 + 3.94 ms.  On the way: terms
// read from global memory by each warp 1.68 ms, two stages of 128 entries 1.46 ms,
// four 1.35 ms; three of 256 halve the steps between chunks.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "tc_util.cuh"
#include "tensor_eval.h"
#include "tile_rule.h"

namespace {

using namespace smx::tc;

constexpr int kStages = 3;  // chunks in flight (layout.cu build_walk sizes them)
constexpr int kWarps = 32;  // owners of destination rows (layout.cu build_walk)
constexpr int kThreads = 32 * kWarps;
constexpr size_t kSmemMax = 227 * 1024;

// Cotangent rows as FP16 pairs: warp per point, v = g * out_scale, one power of
// two per point; columns d_out .. ldo are zero.
__global__ void __launch_bounds__(256) cotangent_kernel(const float* __restrict__ g, int64_t ldg, int64_t P, int d_out,
                                                        int64_t ldo, const float* __restrict__ out_scale,
                                                        __half* __restrict__ hi, __half* __restrict__ lo,
                                                        float* __restrict__ scale) {
  const int lane = threadIdx.x & 31;
  const int64_t p = blockIdx.x * int64_t(8) + (threadIdx.x >> 5);
  if (p >= P) return;
  const float* gp = g + p * ldg;
  float m = 0.f;
  for (int o = lane; o < d_out; o += 32) m = fmaxf(m, fabsf(gp[o] * out_scale[o]));
#pragma unroll
  for (int n = 16; n; n >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, n));
  const int e = min(max(__float_as_int(m) >> 23, 27), 254);
  const float inv = __int_as_float((268 - e) << 23);
  for (int o = lane; o < ldo; o += 32) {
    const float v = o < d_out ? gp[o] * out_scale[o] * inv : 0.f;
    const __half h = __float2half_rn(v);
    hi[p * ldo + o] = h;
    lo[p * ldo + o] = pair_low(v, h);
  }
  if (lane == 0) scale[p] = __int_as_float((e - 14) << 23);
}

// Rows of C: per output the power of two of its largest finite coefficient, 0 for an
// output without any (a constant: its cotangent contributes nothing and must not set
// the scale of its point's cotangents) ...
__global__ void col_scale_kernel(const float* __restrict__ C, int64_t n, int d_out, float* __restrict__ scale) {
  __shared__ float red[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int o = blockIdx.x * 32 + lane;
  float m = 0.f;
  if (o < d_out)
    for (int64_t e = warp; e < n; e += 8) {
      const float a = fabsf(C[e * d_out + o]);
      if (a <= 3.0e38f) m = fmaxf(m, a);
    }
  red[warp][lane] = m;
  __syncthreads();
  if (warp == 0 && o < d_out) {
    for (int w = 1; w < 8; ++w) m = fmaxf(m, red[w][lane]);
    scale[o] = m > 0.f ? __int_as_float(min(max(__float_as_int(m) >> 23, 1), 253) << 23) : 0.f;
  }
}

// ... and per entry and group of 64 outputs the power of two of its largest quotient.
__global__ void split_rows_kernel(const float* __restrict__ C, int64_t n, int d_out, int64_t ldo,
                                  const float* __restrict__ scale, __half* __restrict__ hi, __half* __restrict__ lo,
                                  float* __restrict__ row_scale) {
  const int64_t groups = ldo / 64;
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n * groups) return;
  const int64_t e = i % n, q = i / n;
  auto value = [&](int o) {
    return o < d_out ? C[e * d_out + o] * __int_as_float((254 << 23) - __float_as_int(scale[o])) : 0.f;
  };
  float m = 0.f;
  for (int o = int(q) * 64; o < int(q) * 64 + 64; ++o) {
    const float a = fabsf(value(o));
    if (a <= 3.0e38f) m = fmaxf(m, a);
  }
  const int ex = min(max(__float_as_int(m) >> 23, 27), 254);
  const float inv = __int_as_float((268 - ex) << 23);
  row_scale[q * n + e] = __int_as_float((ex - 14) << 23);
  for (int o = int(q) * 64; o < int(q) * 64 + 64; ++o) {
    const float v = value(o) * inv;
    const __half h = __float2half_rn(v);
    hi[e * ldo + o] = h;
    lo[e * ldo + o] = pair_low(v, h);
  }
}

// ---- G^T = C g^T, few outputs -------------------------------------------------------------
// D[p / 32][entry][32] from R (128 entries a tile) and the cotangents (128 points a
// tile), up to 128 outputs: the contraction is one or two slices of 64, so the
// kernel is bound by writing D and runs as a persistent pipeline.  A block takes a
// run of tiles, entries fastest, so that the points' operand stays in shared
// memory; warp 8 streams R (three stages of TMA), one thread of warp 9 issues the
// MMAs into four accumulators of 128 columns, and warps 0 - 7 drain them (row
// scale per slice, column scale), stage 32 x 32 values and write them by TMA.
// 5120 x 1e5 values from 64 outputs: 331 us (6.2 TB/s of writes); the general
// product, a block per tile with nothing to overlap, took 793 us.
// Every wait is bounded: on timeout the block sets an error code, and once all its
// roles have stopped it waits (bounded) for its copies and MMAs and frees tensor memory.
constexpr int kAdjStages = 3, kAdjAcc = 4, kAdjDrain = 8;
constexpr int kAdjThreads = 32 * (kAdjDrain + 2);
constexpr int kAdjTile = 32 * 1024;  // 128 rows x 64 values, high and low part
constexpr int kAdjMaxSlices = 2;
constexpr int kAdjSmem = kAdjStages * kAdjTile + kAdjMaxSlices * kAdjTile + kAdjDrain * 2 * 4096 + 1024 + 256;

struct AdjArgs {
  int MT, slices, M;
  int64_t tiles;  // point tiles x MT
  const float* row_scale;  // [slice][M]
  const float* col_scale;  // by point, readable to whole tiles of 128
  int* err;
};

__global__ void __launch_bounds__(kAdjThreads, 1)
    adjoint_kernel(const __grid_constant__ CUtensorMap tmRh, const __grid_constant__ CUtensorMap tmRl,
                   const __grid_constant__ CUtensorMap tmGh, const __grid_constant__ CUtensorMap tmGl,
                   const __grid_constant__ CUtensorMap tmD, AdjArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* B = base + kAdjStages * kAdjTile;
  uint8_t* out = B + kAdjMaxSlices * kAdjTile;
  uint64_t* a_full = reinterpret_cast<uint64_t*>(out + kAdjDrain * 2 * 4096);
  uint64_t* a_empty = a_full + kAdjStages;
  uint64_t* b_full = a_empty + kAdjStages;  // [kAdjMaxSlices]
  uint64_t* b_empty = b_full + kAdjMaxSlices;
  uint64_t* acc_full = b_empty + kAdjMaxSlices;
  uint64_t* acc_empty = acc_full + kAdjAcc;
  uint64_t* flush = acc_empty + kAdjAcc;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(flush + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* issued = abort_flag + 1;  // slices of R, points' operands
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = a.slices, nb = kAdjMaxSlices / q;  // buffers of the points' operand
  const int64_t t0 = a.tiles * blockIdx.x / gridDim.x, t1 = a.tiles * (blockIdx.x + 1) / gridDim.x;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kAdjStages; ++i) mbar_init(&a_full[i], 1), mbar_init(&a_empty[i], 1);
    for (int i = 0; i < kAdjMaxSlices; ++i) mbar_init(&b_full[i], 1), mbar_init(&b_empty[i], 1);
    for (int i = 0; i < kAdjAcc; ++i) mbar_init(&acc_full[i], 1), mbar_init(&acc_empty[i], kAdjDrain);
    mbar_init(flush, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kAdjAcc * 128));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  if (warp == kAdjDrain) {
    if (lane == 0) {  // ---- copies
      int64_t last = -1;
      int u = 0, n = 0;
      bool ok = true;
      for (int64_t t = t0; t < t1 && ok; ++t) {
        const int64_t pt = t / a.MT;
        const int mt = int(t - pt * a.MT);
        if (pt != last) {
          const int b = n % nb;
          if (n >= nb && !mbar_wait(&b_empty[b], ((n / nb) & 1) ^ 1, abort_flag)) break;
          mbar_expect_tx(&b_full[b], q * kAdjTile);
          for (int s = 0; s < q; ++s) {
            uint8_t* d = B + (b * q + s) * kAdjTile;
            tma_load_2d(d, &tmGh, s * 64, int(pt * 128), &b_full[b]);
            tma_load_2d(d + kAdjTile / 2, &tmGl, s * 64, int(pt * 128), &b_full[b]);
          }
          last = pt, ++n;
        }
        for (int s = 0; s < q; ++s, ++u) {
          const int i = u % kAdjStages;
          if (u >= kAdjStages && !mbar_wait(&a_empty[i], ((u / kAdjStages) & 1) ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&a_full[i], kAdjTile);
          tma_load_2d(base + i * kAdjTile, &tmRh, s * 64, mt * 128, &a_full[i]);
          tma_load_2d(base + i * kAdjTile + kAdjTile / 2, &tmRl, s * 64, mt * 128, &a_full[i]);
        }
      }
      if (u < int((t1 - t0) * q)) {  // gave up
        atomicExch(a.err, 1);
        *abort_flag = 1;
      }
      issued[0] = u, issued[1] = n;
    }
    __syncwarp();
  } else if (warp == kAdjDrain + 1) {
    if (lane == 0) {  // ---- MMAs
      constexpr uint32_t idesc = idesc_fmt(128, 128, 0u);
      int64_t last = -1;
      int u = 0, n = 0;
      bool ok = true;
      for (int64_t t = t0; t < t1 && ok; ++t) {
        const int64_t pt = t / a.MT;
        if (pt != last) {
          if (n > 0) mma_commit(&b_empty[(n - 1) % nb]);
          ok = mbar_wait(&b_full[n % nb], (n / nb) & 1, abort_flag);
          last = pt, ++n;
        }
        for (int s = 0; s < q && ok; ++s, ++u) {
          const int i = u % kAdjStages, c = u % kAdjAcc;
          if ((u >= kAdjAcc && !mbar_wait(&acc_empty[c], ((u / kAdjAcc) & 1) ^ 1, abort_flag)) ||
              !mbar_wait(&a_full[i], (u / kAdjStages) & 1, abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t ah = smem_u32(base + i * kAdjTile), al = ah + kAdjTile / 2;
          const uint32_t bh = smem_u32(B + (((n - 1) % nb) * q + s) * kAdjTile), bl = bh + kAdjTile / 2;
          mma_pair_slice(tmem + c * 128, ah, al, bh, bl, idesc);
          mma_commit(&a_empty[i]);
          mma_commit(&acc_full[c]);
        }
      }
      if (!ok) {
        atomicExch(a.err, 2);
        *abort_flag = 1;
      }
    }
    __syncwarp();
  } else {
    // ---- drain: rows 32 (warp % 4) .. + 31 of a tile, two of its four blocks of 32 points
    const int quad = warp & 3, half = warp >> 2;
    uint8_t* stage = out + warp * 8192;
    int u = 0, n = 0;
    for (int64_t t = t0; t < t1; ++t, u += q) {
      const int64_t pt = t / a.MT;
      const int e0 = int(t - pt * a.MT) * 128 + quad * 32;
      float rs[kAdjMaxSlices];
      bool ok = true;
#pragma unroll
      for (int s = 0; s < kAdjMaxSlices; ++s) {
        rs[s] = s < q ? __ldg(a.row_scale + int64_t(s) * a.M + min(e0 + lane, a.M - 1)) : 0.f;
        if (s < q) ok = ok && mbar_wait(&acc_full[(u + s) % kAdjAcc], ((u + s) / kAdjAcc) & 1, abort_flag);
      }
      if (!__all_sync(0xffffffffu, ok && !*abort_flag)) {
        if (lane == 0) {
          atomicCAS(a.err, 0, 3);
          *abort_flag = 1;
        }
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
      for (int j = 0; j < 2; ++j, ++n) {
        const int cb = 2 * half + j;
        float v[32];
#pragma unroll
        for (int s = 0; s < kAdjMaxSlices; ++s) {
          if (s >= q) break;
          uint32_t r[32];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
              "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
              : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
                "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
                "=r"(r[30]), "=r"(r[31])
              : "r"(tmem + (uint32_t(quad * 32) << 16) + uint32_t(((u + s) % kAdjAcc) * 128 + cb * 32)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 32; ++i)
            v[i] = s ? fmaf(rs[s], __uint_as_float(r[i]), v[i]) : rs[0] * __uint_as_float(r[i]);
        }
        if (j == 1) {  // the accumulators have been read
          asm volatile("tcgen05.fence::before_thread_sync;");
          __syncwarp();
          if (lane == 0)
            for (int s = 0; s < q; ++s) mbar_arrive(&acc_empty[(u + s) % kAdjAcc]);
        }
        const float4* cs = reinterpret_cast<const float4*>(a.col_scale + pt * 128 + cb * 32);
        uint8_t* buf = stage + (n & 1) * 4096;
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 c = __ldg(cs + i);
          *reinterpret_cast<float4*>(buf + lane * 128 + ((i ^ (lane & 7)) << 4)) =
              make_float4(v[4 * i] * c.x, v[4 * i + 1] * c.y, v[4 * i + 2] * c.z, v[4 * i + 3] * c.w);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (e0 < a.M)
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                             reinterpret_cast<uint64_t>(&tmD)),
                         "r"(0), "r"(e0), "r"(int(pt * 4 + cb)), "r"(smem_u32(buf))
                         : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (*abort_flag) {  // all roles have stopped: wait (bounded) for the copies and MMAs issued
    if (warp == kAdjDrain && lane == 0) {
      for_pending_copies(issued[0], kAdjStages, [&](int s, uint32_t ph) { mbar_wait(&a_full[s], ph, nullptr); });
      for_pending_copies(issued[1], nb, [&](int b, uint32_t ph) { mbar_wait(&b_full[b], ph, nullptr); });
    }
    if (warp == kAdjDrain + 1 && lane == 0) {
      mma_commit(flush);
      mbar_wait(flush, 0, nullptr);
    }
    __syncthreads();
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAdjAcc * 128));
}

// Product of up to 8 slots' values.
__device__ __forceinline__ int4 from_lane(const int4& v, int k) {
  return make_int4(__shfl_sync(0xffffffffu, v.x, k), __shfl_sync(0xffffffffu, v.y, k),
                   __shfl_sync(0xffffffffu, v.z, k), __shfl_sync(0xffffffffu, v.w, k));
}

__device__ __forceinline__ float slot_product(const float* phi, const int4& w4) {
  const unsigned w[4] = {unsigned(w4.x), unsigned(w4.y), unsigned(w4.z), unsigned(w4.w)};
  float v = 1.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const unsigned s = (w[k >> 1] >> (16 * (k & 1))) & 0xffffu;
    if (s == 0xffffu) break;
    v *= phi[s * 32];
  }
  return v;
}

__global__ void __launch_bounds__(kThreads, 1)
    vjp_walk_kernel(smx_tensor t, smx_walk w, const float* __restrict__ grow, const float* __restrict__ drow,
                    int64_t gstride, const float* __restrict__ GT, int64_t P, int* __restrict__ err,
                    double* __restrict__ dx, int64_t lddx) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t p0 = blockIdx.x * int64_t(32), p = p0 + lane;
  const int ns = t.n_slots, nn = w.n_nodes, E = w.chunk;
  float* row = reinterpret_cast<float*>(smem) + lane;  // rows of 32 floats: phi, V, bar, S
  const int row_bar = ns + nn, n_rows = 2 * (ns + nn) + 1;
  const uint32_t bytes = uint32_t(E) * 128, stage_bytes = bytes + uint32_t(w.most) * 8;
  uint8_t* stage = smem + size_t(n_rows) * 128;  // chunks of G, each with its terms
  uint64_t* full = reinterpret_cast<uint64_t*>(stage + kStages * stage_bytes);
  uint64_t* empty = full + kStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kStages);
  int issued = 0;  // chunks, by thread 0
  const uint8_t* G = reinterpret_cast<const uint8_t*>(GT) + blockIdx.x * (int64_t(w.n_chunks) * E * 128);
  auto load_chunk = [&](int c) {
    const int s = c % kStages, t0 = __ldg(w.off + c * 33), n = __ldg(w.off + c * 33 + 32) - t0;
    mbar_expect_tx(&full[s], bytes + n * 8);
    bulk_load(stage + s * stage_bytes, G + int64_t(c) * bytes, bytes, &full[s]);
    bulk_load(stage + s * stage_bytes + bytes, w.term + int64_t(t0) * 2, uint32_t(n) * 8, &full[s]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kWarps);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (; issued < min(kStages, w.n_chunks); ++issued) load_chunk(issued);
  }
  for (int s = warp * 4 + (lane >> 3); s < ns; s += kWarps * 4)
    copy16(row - lane + s * 32 + (lane & 7) * 4, grow + s * gstride + p0 + (lane & 7) * 4);
  for (int s = row_bar + warp; s < n_rows; s += kWarps) row[s * 32] = 0.f;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int n0 = warp; n0 < nn; n0 += kWarps * 32) {  // a lane's load for each of 32 nodes
    const int n = (nn - n0 + kWarps - 1) / kWarps, at = n0 + min(lane, n - 1) * kWarps;
    const int4 path = __ldg(reinterpret_cast<const int4*>(w.node_path) + at);
    for (int k = 0; k < min(32, n); ++k) row[(ns + n0 + k * kWarps) * 32] = slot_product(row, from_lane(path, k));
  }
  __syncthreads();
  // terms of this warp, chunk by chunk; a destination row is only ever touched by
  // its warp, so the warps need not keep step beyond the stages
  uint8_t* rb = smem + lane * 4;
  int t0 = __ldg(w.off + warp), t1 = __ldg(w.off + warp + 1), first = __ldg(w.off);
  bool ok = true;
  for (int c = 0; c < w.n_chunks; ++c) {
    const int s = c % kStages;
    const uint32_t parity = (c / kStages) & 1;
    const uint8_t* gs = stage + s * stage_bytes + lane * 4;
    const int4* term = reinterpret_cast<const int4*>(stage + s * stage_bytes + bytes) + ((t0 - first) >> 1);
    const int n = (t1 - t0) >> 1;
    if (c + 1 < w.n_chunks) {
      const int32_t* o = w.off + (c + 1) * 33;
      t0 = __ldg(o + warp), t1 = __ldg(o + warp + 1), first = __ldg(o);
    }
    const bool got = mbar_test(&full[s], parity) || mbar_wait(&full[s], parity, abort_flag);
    if (!__all_sync(0xffffffffu, got)) {  // bounded: a lost copy ends the block
      *abort_flag = 1;
      break;
    }
    if (n > 0) {  // the next pair's sources are read before this pair's sums are written back
      auto at = [&](unsigned r) { return reinterpret_cast<float*>(rb + r * 128); };
      auto g = [&](int o) { return *reinterpret_cast<const float*>(gs + o); };
      int4 a = term[0];
      float sa = *at(a.x & 0xffff), sb = *at(a.z & 0xffff), ga = g(a.y), gb = g(a.w);
#pragma unroll 2
      for (int i = 1; i <= n; ++i) {
        float *da = at(unsigned(a.x) >> 16), *db = at(unsigned(a.z) >> 16);
        const float va = fmaf(sa, ga, *da), vb = fmaf(sb, gb, *db);
        a = term[min(i, n - 1)];
        sa = *at(a.x & 0xffff), sb = *at(a.z & 0xffff), ga = g(a.y), gb = g(a.w);
        *da = va;
        *db = vb;
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (threadIdx.x == 0 && c + kStages < w.n_chunks) {
      if (mbar_wait(&empty[s], parity, abort_flag)) {
        load_chunk(issued++);  // chunk c + kStages
      } else {
        *abort_flag = 1;  // no further chunk comes: every warp's next wait ends
      }
    }
    __syncwarp();
  }
  __syncthreads();
  if (*abort_flag) {  // leave no copy behind: wait (bounded) for what was issued
    if (threadIdx.x == 0) {
      atomicExch(err, 3);
      for_pending_copies(issued, kStages, [&](int s, uint32_t parity) { mbar_wait(&full[s], parity, nullptr); });
    }
    return;
  }
  // path factors; the slot's adjoint times its derivative in its row of bar
  const int i1 = __ldg(w.warp + warp + 1);
  for (int i0 = __ldg(w.warp + warp); i0 < i1; i0 += 32) {  // a lane's load for each of 32 slots
    const int ni = min(32, i1 - i0);
    const int4 of = __ldg(reinterpret_cast<const int4*>(w.slot) + i0 + min(lane, ni - 1));
    float next = __ldg(drow + __shfl_sync(0xffffffffu, of.x, 0) * gstride + p);
    for (int i = 0; i < ni; ++i) {
      const int4 s = from_lane(of, i);
      const float d = next;
      next = __ldg(drow + __shfl_sync(0xffffffffu, of.x, min(i + 1, ni - 1)) * gstride + p);
      float rest = row[(row_bar + s.x) * 32];
      for (int q0 = s.y; q0 < s.z; q0 += 32) {  // ... and for each of 32 factors
        const int n = min(32, s.z - q0), q = q0 + min(lane, n - 1), r = __ldg(w.row + q);
        const int4 other = __ldg(reinterpret_cast<const int4*>(w.other) + q);
        for (int k = 0; k < n; ++k)
          rest = fmaf(row[__shfl_sync(0xffffffffu, r, k) * 32], slot_product(row, from_lane(other, k)), rest);
      }
      row[(row_bar + s.x) * 32] = rest * d;
    }
  }
  __syncthreads();
  // per dimension the sum over its degrees, turned in the place of phi and V
  float* turn = reinterpret_cast<float*>(smem);  // [n_dims][33]: ends before bar (checked on the host)
  for (int h0 = warp; h0 < t.n_dims; h0 += kWarps * 32) {
    const int n = min(32, (t.n_dims - h0 + kWarps - 1) / kWarps), at = h0 + min(lane, n - 1) * kWarps;
    const int so = __ldg(t.dsoff + at), g = __ldg(t.dmax + at);
    for (int k = 0; k < n; ++k) {
      const float* bar = row + (row_bar + __shfl_sync(0xffffffffu, so, k)) * 32;
      const int gk = __shfl_sync(0xffffffffu, g, k);
      float acc = 0.f;
      for (int m = 0; m < gk; ++m) acc += bar[m * 32];
      turn[(h0 + k * kWarps) * 33 + lane] = acc;
    }
  }
  __syncthreads();
  for (int q = warp; q < 32; q += kWarps) {
    if (p0 + q >= P) break;
    double* out = dx + (p0 + q) * lddx;
#pragma unroll 4
    for (int j = lane; j < t.d_in; j += 32) {
      const int h = __ldg(w.dim_index + j);
      out[j] = h < 0 ? 0.0 : double(__ldg(t.fam_a + j)) * double(turn[h * 33 + q]);
    }
  }
}

// ---- dL/dC = A^T g ---------------------------------------------------------------------
// A^T in slices of 64 points, [p / 64][entry][64] as FP16 pairs with one power of
// two per entry and slice.  Each point's products are multiplied by the power of two of
// its largest cotangent (in units of each output's largest), and the cotangents divided
// by it: the pairs' range (2^29 below the slice's largest at full precision, tc_util.cuh)
// then counts the points' terms A g and not A and g by themselves, which may run against
// each other over the points, and points without a cotangent weigh nothing.  An element
// of dL/dC has the accuracy of the TF32 pairs while its own largest term of a slice is
// within 2^29 of its entry's largest over the outputs (in units of their largest g).  A block of
// W warps holds
// the basis rows of 64 points (two per lane) in shared memory; each warp walks its
// run of tape groups as tensor_panel_kernel does (tensor_eval.cu), but an entry's 64
// values are one register pair per lane, so they are scaled and written at once:
// 128 contiguous bytes per entry and part.  Bound: HBM writes, 4 bytes per value.
// Leja d_in = 200, |Lambda| = 5000, 1e5 points: 0.33 ms (6.1 TB/s of writes, issue
// slots 71 % busy) and 0.32 ms for the product with 64 outputs; one thread per point
// writing TF32 pairs through 400 KB strides took 1.34 ms and its product 0.62 ms.
constexpr float kPointScale = 1.f / 16384.f;
template <int W, int MINB>
__global__ void __launch_bounds__(32 * W, MINB)
    coef_panel_kernel(smx_tensor t, int groups_per_block, const float* __restrict__ grow, int64_t gstride,
                      int64_t n_slices, const float2* __restrict__ pscale, uint32_t* __restrict__ AH,
                      uint32_t* __restrict__ AL, float* __restrict__ S) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t* ring = smem + warp * 1024;  // two tape groups
  uint8_t* stk = smem + W * 1024 + warp * (9 * 256) + lane * 8;  // stk[256 d]: first d factors
  uint8_t* rows = smem + W * (1024 + 9 * 256) + lane * 8;
  const int b0 = blockIdx.x * groups_per_block, nb = min(t.n_groups - b0, groups_per_block);
  const int t0 = b0 + nb * warp / W, t1 = b0 + nb * (warp + 1) / W;
  const int64_t E = int64_t(t.n_groups) * kGroup;
  auto f2 = [](uint8_t* q) -> float2& { return *reinterpret_cast<float2*>(q); };
  for (int64_t sl = blockIdx.y; sl < n_slices; sl += gridDim.y) {
    __syncthreads();  // the previous slice's walks are done
    for (int i = warp * 2 + (lane >> 4); i < t.n_slots; i += W * 2)
      copy16(rows - lane * 8 + i * 256 + (lane & 15) * 16, grow + i * gstride + sl * 64 + (lane & 15) * 4);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (t0 == t1) continue;
    f2(stk) = __ldg(pscale + sl * 32 + lane);  // every product starts with its point's scale
    for (int i = 0; i < 8; ++i) {
      const int s = __ldg(t.path + t0 * 8 + i);
      if (s < 0) break;
      f2(stk + (i + 1) * 256) = __fmul2_rn(f2(stk + i * 256), f2(rows + s * 256));
    }
    const int4* tape = reinterpret_cast<const int4*>(t.tape) + t0 * (kGroup / 2) + lane;
    auto copy_group = [&](int g) {
      if (g < t1)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(ring + (g & 1) * 512 + lane * 16)),
                     "l"(tape + (g - t0) * (kGroup / 2))
                     : "memory");
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    copy_group(t0);
    for (int g = t0; g < t1; ++g) {
      copy_group(g + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      const int4* words = reinterpret_cast<const int4*>(ring + (g & 1) * 512);
      const int64_t e0 = sl * E + g * kGroup;
      float2 cur = make_float2(1.f, 1.f);
      float sc = 0.f;
#pragma unroll 2
      for (int k = 0; k < kGroup; k += 4) {
        const int4 wa = words[k / 2], wb = words[k / 2 + 1];
        const int wr[4] = {wa.x, wa.z, wb.x, wb.z}, wf[4] = {wa.y, wa.w, wb.y, wb.w};
        float2 b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = f2(rows + wr[u] * 2);
        unsigned m[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (wf[u] & kPop) cur = f2(stk + (wf[u] & kStackMask) * 2);
          b[u] = __fmul2_rn(cur, b[u]);
          if (wf[u] & kPush) {
            cur = b[u];
            f2(stk + (wf[u] & kStackMask) * 2 + 256) = cur;
          }
          m[u] = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(b[u].x), fabsf(b[u].y))));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          // power of two that brings the maximum to [2^14, 2^15)
          const int e = min(max(int(m[u] >> 23), 27), 254);
          const float inv = __int_as_float((268 - e) << 23);
          if (lane == ((k + u) & 31)) sc = __int_as_float((e - 14) << 23);
          const float2 v = __fmul2_rn(b[u], make_float2(inv, inv));
          const __half2 h = __float22half2_rn(v);
          const __half2 l = pair_low(v, h);
          AH[(e0 + k + u) * 32 + lane] = *reinterpret_cast<const uint32_t*>(&h);
          AL[(e0 + k + u) * 32 + lane] = *reinterpret_cast<const uint32_t*>(&l);
        }
        if ((k & 31) == 28) S[e0 + (k & 32) + lane] = sc * kPointScale;
      }
    }
  }
}

// Per output the largest finite |g| (bits; `most` starts at zero) and the sum of
// each block's kSumRows points in FP64 ...
constexpr int kSumRows = 512;
__global__ void __launch_bounds__(256) output_most_kernel(const float* __restrict__ g, int64_t ldg, int64_t P, int d_out,
                                                          unsigned* __restrict__ most, double* __restrict__ part) {
  __shared__ float red[8][33];
  __shared__ double sum[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o0 = blockIdx.y * 32; o0 < d_out; o0 += gridDim.y * 32) {
    const int o = o0 + lane;
    const int64_t p1 = min(P, (blockIdx.x + 1) * int64_t(kSumRows));
    float m = 0.f;
    double acc = 0.0;
    if (o < d_out) {
#pragma unroll 8
      for (int64_t p = blockIdx.x * int64_t(kSumRows) + warp; p < p1; p += 8) {
        const float v = __ldg(g + p * ldg + o), a = fabsf(v);
        if (a <= 3.0e38f) m = fmaxf(m, a);
        acc += double(v);
      }
    }
    red[warp][lane] = m;
    sum[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && o < d_out) {
      for (int w = 1; w < 8; ++w) m = fmaxf(m, red[w][lane]), acc += sum[w][lane];
      if (m > 0.f) atomicMax(most + o, __float_as_uint(m));
      part[blockIdx.x * int64_t(d_out) + o] = acc;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ float output_scale(unsigned most) {
  return most ? __int_as_float(min(max(int(most >> 23), 1), 253) << 23) : 1.f;
}

// ... and g / scale transposed in slices of 64 points, [p / 64][output][64], as FP16
// pairs, each point's largest brought to [2^14, 2^15); pscale: what that divided by, times
// kPointScale^-1 (0 for points without a cotangent and past P).
__global__ void __launch_bounds__(256) output_slices_kernel(const float* __restrict__ g, int64_t ldg, int64_t P,
                                                            int d_out, const unsigned* __restrict__ most,
                                                            uint32_t* __restrict__ hi, uint32_t* __restrict__ lo,
                                                            float* __restrict__ pscale, float* __restrict__ scale) {
  __shared__ float tile[64][65];
  __shared__ float red[64][2], inv[64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, oc = threadIdx.x & 63, r0 = threadIdx.x >> 6;
  const int64_t p0 = blockIdx.x * int64_t(64);
  auto value = [&](int64_t p, int o) {
    return p < P && o < d_out
               ? __ldg(g + p * ldg + o) * __int_as_float((254 << 23) - __float_as_int(output_scale(__ldg(most + o))))
               : 0.f;
  };
  if (blockIdx.x == 0)
    for (int o = threadIdx.x; o < d_out; o += 256) scale[o] = output_scale(most[o]);
  for (int r = r0; r < 64; r += 4) {  // two warps per point
    float m = 0.f;
    for (int o0 = 0; o0 < d_out; o0 += 64) {
      const float a = fabsf(value(p0 + r, o0 + oc));
      if (a <= 3.0e38f) m = fmaxf(m, a);
    }
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    if (lane == 0) red[r][warp & 1] = m;
  }
  __syncthreads();
  if (threadIdx.x < 64) {
    const float m = fmaxf(red[threadIdx.x][0], red[threadIdx.x][1]);
    const int e = min(max(__float_as_int(m) >> 23, 27), 254);
    inv[threadIdx.x] = __int_as_float((268 - e) << 23);
    pscale[p0 + threadIdx.x] = m > 0.f ? __int_as_float(e << 23) : 0.f;
  }
  __syncthreads();
  for (int o0 = 0; o0 < d_out; o0 += 64) {
    for (int r = r0; r < 64; r += 4) tile[r][oc] = value(p0 + r, o0 + oc) * inv[r];
    __syncthreads();
    for (int o = warp; o < 64 && o0 + o < d_out; o += 8) {
      const float2 v = make_float2(tile[2 * lane][o], tile[2 * lane + 1][o]);
      const __half2 h = __float22half2_rn(v);
      const __half2 l = pair_low(v, h);
      const int64_t at = (blockIdx.x * int64_t(d_out) + o0 + o) * 32 + lane;
      hi[at] = *reinterpret_cast<const uint32_t*>(&h);
      lo[at] = *reinterpret_cast<const uint32_t*>(&l);
    }
    __syncthreads();
  }
}

// ---- the adjoints' way back to coefficients and nodal values ----------------------------
// Column sums in FP64 in a fixed order: blocks of kSumRows rows (a warp reads whole
// lines: 2^to_log columns by 256 >> to_log row lanes), then the blocks' sums.
constexpr int kSumThreads = 256;

__device__ __forceinline__ double sum_lanes(double v, int to_log, double* red) {
  const int t = threadIdx.x;
  red[t] = v;
  __syncthreads();
  for (int n = kSumThreads >> 1; n >= (1 << to_log); n >>= 1) {
    if (t < n) red[t] += red[t + n];
    __syncthreads();
  }
  return red[t];
}

__global__ void __launch_bounds__(kSumThreads) column_partial_kernel(const double* __restrict__ A, int64_t n, int d,
                                                                     int to_log, double* __restrict__ part) {
  __shared__ double red[kSumThreads];
  const int t = threadIdx.x, o = (int(blockIdx.y) << to_log) + (t & ((1 << to_log) - 1));
  const int64_t r0 = blockIdx.x * int64_t(kSumRows), r1 = min(n, r0 + kSumRows);
  double acc = 0.0;
  if (o < d) {
#pragma unroll 8
    for (int64_t r = r0 + (t >> to_log); r < r1; r += kSumThreads >> to_log) acc += __ldg(A + r * d + o);
  }
  acc = sum_lanes(acc, to_log, red);
  if (t < (1 << to_log) && o < d) part[blockIdx.x * int64_t(d) + o] = acc;
}

// out[o] = sum, or (extra given) out[o] + factor * extra[o] - sum.
__global__ void __launch_bounds__(kSumThreads) column_final_kernel(const double* __restrict__ part, int64_t blocks, int d,
                                                                   int to_log, const double* __restrict__ extra,
                                                                   double factor, double* __restrict__ out) {
  __shared__ double red[kSumThreads];
  const int t = threadIdx.x, o = (int(blockIdx.x) << to_log) + (t & ((1 << to_log) - 1));
  double acc = 0.0;
  if (o < d) {
#pragma unroll 8
    for (int64_t b = t >> to_log; b < blocks; b += kSumThreads >> to_log) acc += __ldg(part + b * d + o);
  }
  acc = sum_lanes(acc, to_log, red);
  if (t < (1 << to_log) && o < d) out[o] = extra ? out[o] + factor * extra[o] - acc : acc;
}

int sum_log(int d) {
  int l = 0;
  while (l < 8 && (1 << l) < d) ++l;
  return l;
}

size_t sum_bytes(int64_t n, int d) { return size_t((n + kSumRows - 1) / kSumRows) * d * sizeof(double); }

// Sums of the blocks' column sums.
void column_finish(const double* part, int64_t blocks, int d, const double* extra, double factor, double* out,
                   cudaStream_t st) {
  const int l = sum_log(d);
  column_final_kernel<<<unsigned((d + (1 << l) - 1) >> l), kSumThreads, 0, st>>>(part, blocks, d, l, extra, factor, out);
}

// Rows of dL/dC from the tape's order (pad rows first) to the entries', in FP64.
__global__ void coef_rows_kernel(const float* __restrict__ rows, int64_t pad, int64_t K, int d,
                                 const int64_t* __restrict__ ent, double* __restrict__ dC) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= K * d) return;
  const int64_t j = i / d;
  dC[__ldg(ent + j) * d + (i - j * d)] = double(rows[(pad + j) * d + (i - j * d)]);
}

// Sums of runs [begin[i], begin[i + 1]) of A (rows row[..] of it, each times its
// weight; or A's rows as they are), in order.  dL/d(nodal values) is two of them:
// runs of at most 64 rows, then the runs of each value, because with nested nodes one
// value may stand in half of all rows.  Leja |Lambda| = 5000, 5000 values x 64
// outputs: 25 + 15 us; a thread through all rows of a value 2.4 ms.  The chain rule
// as a dozen tensor operations (multiply, index_add, sums, ...) cost the host more
// than the GPU: a training step of 1e3 points 0.9 ms, 0.68 with these kernels.
template <bool ROWS>
__global__ void run_sum_kernel(const double* __restrict__ A, const double* __restrict__ weight,
                               const int64_t* __restrict__ row, const int64_t* __restrict__ begin, int64_t n, int d,
                               double* __restrict__ out) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n * d) return;
  const int64_t u = i / d, q1 = __ldg(begin + u + 1);
  const int o = int(i - u * d);
  double acc = 0.0;
#pragma unroll 8
  for (int64_t q = __ldg(begin + u); q < q1; ++q) {
    if constexpr (ROWS) {
      const int64_t r = __ldg(row + q);
      acc = fma(__ldg(weight + r), __ldg(A + r * d + o), acc);
    } else {
      acc += __ldg(A + q * d + o);
    }
  }
  out[i] = acc;
}

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

size_t walk_smem(const smx_tensor* t, const smx_walk& w) {
  return (size_t(2) * (t->n_slots + w.n_nodes) + 1 + size_t(kStages) * w.chunk) * 128 + size_t(kStages) * w.most * 8 + 96;
}

struct Layout {
  int64_t gstride;
  size_t rows, gt, half, scale, total;
};
Layout layout(const smx_tensor* t, const smx_tensor_bwd* b, int64_t m) {
  Layout L;
  L.gstride = (m + 127) / 128 * 128;
  L.rows = up256(size_t(t->n_slots) * L.gstride * 4);
  L.gt = up256(size_t(b->n_rows) * L.gstride * 4);
  L.half = up256(size_t(m) * b->ldo * 2);
  L.scale = up256(size_t(L.gstride) * 4);
  L.total = 2 * L.rows + L.gt + 2 * L.half + L.scale;
  return L;
}

// G^T of m points (adjoint_kernel).
int adjoint_gemm(const smx_tensor& t, const smx_tensor_bwd& b, const __half* gh, const __half* gl, const float* gs,
                 float* GT, int64_t m, int64_t gstride, int sms, cudaStream_t st) {
  PFN_cuTensorMapEncodeTiled_v12000 encode;
  CUtensorMap tRh, tRl, tGh, tGl, tD;
  int rc = tensor_map_encoder(&encode);
  if (rc || (rc = panel_map(&tRh, b.Rh, b.n_rows, b.ldo, b.ldo, 128, kF16)) ||
      (rc = panel_map(&tRl, b.Rl, b.n_rows, b.ldo, b.ldo, 128, kF16)) ||
      (rc = panel_map(&tGh, gh, m, b.ldo, b.ldo, 128, kF16)) || (rc = panel_map(&tGl, gl, m, b.ldo, b.ldo, 128, kF16)))
    return rc;
  const cuuint64_t dims[3] = {32, cuuint64_t(b.n_rows), cuuint64_t(gstride / 32)};
  const cuuint64_t strides[2] = {128, cuuint64_t(b.n_rows) * 128};
  const cuuint32_t box[3] = {32, 32, 1}, estr[3] = {1, 1, 1};
  if (encode(&tD, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, GT, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return smx::set_error(SMX_ERR_CUDA, "smx_tensor_vjp_x: cuTensorMapEncodeTiled failed");
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAdjSmem);
    attr = true;
  }
  AdjArgs a{};
  a.MT = int((b.n_rows + 127) / 128), a.slices = int(b.ldo / 64), a.M = int(b.n_rows);
  a.tiles = (m + 127) / 128 * a.MT;
  a.row_scale = b.row_scale, a.col_scale = gs, a.err = t.err;
  adjoint_kernel<<<unsigned(std::min<int64_t>(a.tiles, sms)), kAdjThreads, kAdjSmem, st>>>(tRh, tRl, tGh, tGl, tD, a);
  SMX_LAUNCH_CHECK("smx_tensor_vjp_x adjoints");
  return SMX_OK;
}

size_t coef_smem(int warps, int slots) { return size_t(warps) * (1024 + 9 * 256) + size_t(slots) * 256; }

struct CoefLayout {  // workspace of one chunk of m points
  int64_t gstride, slices, E;
  size_t panel, scales, rows, cot, pscale, out, dC, partial, total;
};
CoefLayout coef_layout(const smx_tensor* t, int64_t m) {
  CoefLayout L;
  L.gstride = (m + 127) / 128 * 128;
  L.slices = (m + 63) / 64;
  L.E = int64_t(t->n_groups) * kGroup;
  L.panel = up256(size_t(L.slices) * L.E * 128);
  L.scales = up256(size_t(L.slices) * L.E * 4);
  L.rows = up256(size_t(t->n_slots) * L.gstride * 4);
  L.cot = up256(size_t(L.slices) * t->d_out * 128);
  L.pscale = up256(size_t(L.slices) * 256);
  L.out = up256(size_t(t->d_out) * 4);
  L.dC = up256(size_t(L.E) * t->d_out * 4);
  L.partial = t->splits > 1 ? up256(size_t(t->splits) * L.E * t->d_out * 4) : 0;
  L.total = 2 * L.panel + L.scales + L.rows + 2 * L.cot + L.pscale + 2 * L.out + L.dC + L.partial;
  return L;
}

// Sums of g by blocks of kSumRows points, in each chunk.
size_t coef_sum_bytes(const smx_tensor* t, int64_t P) {
  const int64_t whole = P / t->chunk;
  return size_t(whole) * sum_bytes(t->chunk, t->d_out) + sum_bytes(P - whole * t->chunk, t->d_out);
}

template <int W, int MINB>
void launch_coef_panel(const smx_tensor& t, const CoefLayout& L, const float* grow, const float* pscale, uint32_t* AH,
                       uint32_t* AL, float* S, int sms, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(coef_panel_kernel<W, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemMax));
    attr = true;
  }
  // the split of the tape with the shortest total of rounds x (groups of a warp +
  // about 2 groups' time to load the rows and start), as in the evaluation
  int per = t.n_groups;
  int64_t best = -1;
  for (int segs = 1; segs <= 32 && segs * W <= t.n_groups + W - 1; ++segs) {
    const int p = (t.n_groups + segs - 1) / segs;
    const int64_t blocks = L.slices * ((t.n_groups + p - 1) / p);
    const int64_t cost = ((blocks + MINB * sms - 1) / (MINB * sms)) * ((p + W - 1) / W + 2);
    if (best < 0 || cost < best) best = cost, per = p;
  }
  const dim3 grid(unsigned((t.n_groups + per - 1) / per), unsigned(std::min<int64_t>(L.slices, 65535)));
  coef_panel_kernel<W, MINB><<<grid, 32 * W, coef_smem(W, t.n_slots), st>>>(t, per, grow, L.gstride, L.slices,
                                                                            reinterpret_cast<const float2*>(pscale), AH, AL, S);
}

}  // namespace

// Slices of the contraction over the points (tile_rule.h).
extern "C" int smx_tensor_coef_splits(int d_out, int K) {
  if (d_out < 1 || K < 1) return 1;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return choose_slices(K, d_out, sms);
}

extern "C" size_t smx_tensor_vjp_coef_workspace(const smx_tensor* t, int64_t P) {
  if (!t || P <= 0 || t->chunk < 1 || t->K < 1 || coef_smem(16, t->n_slots) > kSmemMax) return 0;
  return up256(coef_sum_bytes(t, P)) + coef_layout(t, std::min(P, t->chunk)).total;
}

extern "C" int smx_tensor_vjp_coef(const smx_tensor* t, const double* x, int64_t P, int64_t ldx, const float* g,
                                   int64_t ldg, const int64_t* ent, const float* rows_given, double* dC, void* ws,
                                   size_t ws_bytes, void* stream) {
  SMX_REQUIRE(t != nullptr, "smx_tensor_vjp_coef: null plan");
  SMX_REQUIRE(t->d_in >= 1 && t->d_out >= 1 && t->K >= 1 && t->n_groups == (t->K + kGroup - 1) / kGroup &&
                  t->splits >= 1 && t->chunk >= 64 && t->chunk % 64 == 0 &&
                  (std::min(P, t->chunk) + 63) / 64 * std::max<int64_t>(64 * t->n_groups, t->d_out) < (int64_t(1) << 31),
              "smx_tensor_vjp_coef: bad plan sizes");
  SMX_REQUIRE(P >= 1 && ldx >= t->d_in && ldg >= t->d_out, "smx_tensor_vjp_coef: bad sizes");
  SMX_REQUIRE(x && g && ent && dC && t->err && t->dims && t->dmax && t->dsoff && t->fam && t->fam_a && t->fam_b && t->rec &&
                  t->tape && t->path,
              "smx_tensor_vjp_coef: null pointer");
  SMX_REQUIRE(coef_smem(16, t->n_slots) <= kSmemMax, "smx_tensor_vjp_coef: the basis rows do not fit in shared memory");
  SMX_REQUIRE(ws && ws_bytes >= smx_tensor_vjp_coef_workspace(t, P) && (reinterpret_cast<uintptr_t>(ws) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(rows_given) & 15) == 0,
              "smx_tensor_vjp_coef: workspace too small or not 16-byte aligned");
  cudaStream_t st = smx::as_stream(stream);
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return smx::set_error(SMX_ERR_CUDA, "smx_tensor_vjp_coef: no device");
  double* sums = static_cast<double*>(ws);  // of g, for the constant's row
  int64_t sum_blocks = 0;
  const size_t first = up256(coef_sum_bytes(t, P)), dC_bytes = coef_layout(t, 1).dC;
  float* rows = reinterpret_cast<float*>(static_cast<uint8_t*>(ws) + first);
  for (int64_t p0 = 0; p0 < P; p0 += t->chunk) {
    const int64_t m = std::min(t->chunk, P - p0);
    const CoefLayout L = coef_layout(t, m);
    uint8_t* q = static_cast<uint8_t*>(ws) + first + dC_bytes;
    auto take = [&](size_t bytes) {
      uint8_t* r = q;
      q += bytes;
      return r;
    };
    uint32_t* AH = reinterpret_cast<uint32_t*>(take(L.panel));
    uint32_t* AL = reinterpret_cast<uint32_t*>(take(L.panel));
    float* S = reinterpret_cast<float*>(take(L.scales));
    float* grow = reinterpret_cast<float*>(take(L.rows));
    uint32_t* gh = reinterpret_cast<uint32_t*>(take(L.cot));
    uint32_t* gl = reinterpret_cast<uint32_t*>(take(L.cot));
    float* pscale = reinterpret_cast<float*>(take(L.pscale));
    unsigned* most = reinterpret_cast<unsigned*>(take(L.out));
    float* scale = reinterpret_cast<float*>(take(L.out));
    if (cudaMemsetAsync(most, 0, size_t(t->d_out) * 4, st) != cudaSuccess)
      return smx::set_error(SMX_ERR_CUDA, "smx_tensor_vjp_coef: memset failed");
    const dim3 ogrid(unsigned((m + kSumRows - 1) / kSumRows), unsigned(std::min((t->d_out + 31) / 32, 65535)));
    output_most_kernel<<<ogrid, 256, 0, st>>>(g + p0 * ldg, ldg, m, t->d_out, most, sums + sum_blocks * t->d_out);
    sum_blocks += ogrid.x;
    output_slices_kernel<<<unsigned(L.slices), 256, 0, st>>>(g + p0 * ldg, ldg, m, t->d_out, most, gh, gl, pscale,
                                                             scale);
    if (rows_given && P <= t->chunk)
      grow = const_cast<float*>(rows_given);
    else
      tensor_basis(*t, x + p0 * ldx, m, ldx, grow, nullptr, L.gstride, st);
    // two blocks of 8 warps per SM while their rows fit (up to ~330 slots), else one of 16
    if (coef_smem(8, t->n_slots) <= (kSmemMax - 2048) / 2)
      launch_coef_panel<8, 2>(*t, L, grow, pscale, AH, AL, S, sms, st);
    else
      launch_coef_panel<16, 1>(*t, L, grow, pscale, AH, AL, S, sms, st);
    SMX_LAUNCH_CHECK("smx_tensor_vjp_coef");
    SplitGemm s{};
    s.bits = kF16;
    s.sliced = true;
    s.Ah = AH, s.Al = AL, s.Bh = gh, s.Bl = gl;
    s.row_scale = S, s.ld_scale = L.E;
    s.col_scale = scale;
    s.M = int(L.E), s.N = t->d_out, s.K = int(L.slices * 64);
    s.D = rows, s.ldd = t->d_out;
    s.err = t->err, s.splits = t->splits, s.partial = reinterpret_cast<float*>(q);
    s.accumulate = p0 > 0;
    const int rc = split_gemm(s, st);
    if (rc) return rc;
  }
  column_finish(sums, sum_blocks, t->d_out, nullptr, 0.0, dC, st);
  coef_rows_kernel<<<smx::grid_for(int64_t(t->K) * t->d_out, 256), 256, 0, st>>>(
      rows, int64_t(t->n_groups) * kGroup - t->K, t->K, t->d_out, ent, dC);
  SMX_LAUNCH_CHECK("smx_tensor_vjp_coef");
  return SMX_OK;
}

extern "C" size_t smx_nodal_adjoint_workspace(int64_t n_values, int64_t n_runs, int d_out) {
  return n_values > 0 && n_runs >= 0 && d_out > 0 ? sum_bytes(n_values, d_out) + size_t(n_runs) * d_out * sizeof(double)
                                                  : 0;
}

extern "C" int smx_nodal_adjoint(const double* Fbar, const double* zeta, int64_t n_values, int64_t n_runs, int d_out,
                                 const int64_t* value_run, const int64_t* run_begin, const int64_t* row,
                                 const double* root, double root_factor, int64_t first, double* out, void* ws,
                                 size_t ws_bytes, void* stream) {
  SMX_REQUIRE(n_values >= 1 && n_runs >= 0 && d_out >= 1 && first >= 0 && first < n_values,
              "smx_nodal_adjoint: bad sizes");
  SMX_REQUIRE(Fbar && zeta && value_run && run_begin && row && root && out, "smx_nodal_adjoint: null pointer");
  SMX_REQUIRE(ws && ws_bytes >= smx_nodal_adjoint_workspace(n_values, n_runs, d_out) &&
                  (reinterpret_cast<uintptr_t>(ws) & 7) == 0,
              "smx_nodal_adjoint: workspace too small or not 8-byte aligned");
  cudaStream_t st = smx::as_stream(stream);
  double* runs = static_cast<double*>(ws);
  if (n_runs)
    run_sum_kernel<true><<<smx::grid_for(n_runs * d_out, 256), 256, 0, st>>>(Fbar, zeta, row, run_begin, n_runs, d_out,
                                                                             runs);
  run_sum_kernel<false><<<smx::grid_for(n_values * d_out, 256), 256, 0, st>>>(runs, nullptr, nullptr, value_run,
                                                                              n_values, d_out, out);
  double* part = runs + n_runs * d_out;
  const int l = sum_log(d_out);
  const int64_t blocks = (n_values + kSumRows - 1) / kSumRows;
  column_partial_kernel<<<dim3(unsigned(blocks), unsigned((d_out + (1 << l) - 1) >> l)), kSumThreads, 0, st>>>(
      out, n_values, d_out, l, part);
  column_finish(part, blocks, d_out, root, root_factor, out + first * d_out, st);
  SMX_LAUNCH_CHECK("smx_nodal_adjoint");
  return SMX_OK;
}

extern "C" int smx_tensor_bwd_operands(const float* C, int64_t n_rows, int d_out, int64_t ldo, uint16_t* Rh,
                                       uint16_t* Rl, float* row_scale, float* out_scale, void* stream) {
  SMX_REQUIRE(n_rows >= 1 && d_out >= 1 && ldo >= d_out && ldo % 64 == 0 && C && Rh && Rl && row_scale && out_scale,
              "smx_tensor_bwd_operands: bad arguments");
  cudaStream_t st = smx::as_stream(stream);
  col_scale_kernel<<<(d_out + 31) / 32, 256, 0, st>>>(C, n_rows, d_out, out_scale);
  split_rows_kernel<<<smx::grid_for(n_rows * (ldo / 64), 128), 128, 0, st>>>(
      C, n_rows, d_out, ldo, out_scale, reinterpret_cast<__half*>(Rh), reinterpret_cast<__half*>(Rl), row_scale);
  SMX_LAUNCH_CHECK("smx_tensor_bwd_operands");
  return SMX_OK;
}

extern "C" size_t smx_tensor_vjp_x_workspace(const smx_tensor* t, const smx_tensor_bwd* b, int64_t P) {
  if (!t || !b || P <= 0 || b->chunk < 1) return 0;
  return layout(t, b, std::min(P, b->chunk)).total;
}

extern "C" int smx_tensor_vjp_x(const smx_tensor* t, const smx_tensor_bwd* b, const double* x, int64_t P, int64_t ldx,
                                const float* g, int64_t ldg, double* dx, int64_t lddx, void* ws, size_t ws_bytes,
                                void* stream) {
  SMX_REQUIRE(t && b, "smx_tensor_vjp_x: null plan");
  SMX_REQUIRE(P >= 0 && ldx >= t->d_in && lddx >= t->d_in && ldg >= t->d_out && b->chunk >= 1 &&
                  b->ldo >= t->d_out && b->ldo % 64 == 0 && b->walk.n_nodes >= 1 && b->walk.chunk >= 1 &&
                  b->n_rows == int64_t(b->walk.n_chunks) * b->walk.chunk && b->n_rows >= t->K && b->n_rows < (1 << 30),
              "smx_tensor_vjp_x: bad sizes");
  if (P == 0) return SMX_OK;
  SMX_REQUIRE(x && g && dx && t->err, "smx_tensor_vjp_x: null pointer");
  const smx_walk& w = b->walk;
  SMX_REQUIRE(t->dims && t->dmax && t->dsoff && t->fam && t->fam_a && t->fam_b && t->rec && b->Rh && b->Rl &&
                  b->row_scale && b->out_scale && w.off && w.term && w.node_path && w.slot && w.warp && w.dim_index,
              "smx_tensor_vjp_x: incomplete plan");
  SMX_REQUIRE(walk_smem(t, w) <= kSmemMax && 33 * int64_t(t->n_dims) <= 32 * (int64_t(t->n_slots) + w.n_nodes),
              "smx_tensor_vjp_x: the walk's rows do not fit in shared memory");
  SMX_REQUIRE(ws && ws_bytes >= smx_tensor_vjp_x_workspace(t, b, P) && (reinterpret_cast<uintptr_t>(ws) & 15) == 0,
              "smx_tensor_vjp_x: workspace too small or not 16-byte aligned");
  cudaStream_t st = smx::as_stream(stream);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(vjp_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemMax));
    attr = true;
  }
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return smx::set_error(SMX_ERR_CUDA, "smx_tensor_vjp_x: no device");
  for (int64_t p0 = 0; p0 < P; p0 += b->chunk) {
    const int64_t m = std::min(b->chunk, P - p0);
    const Layout L = layout(t, b, m);
    uint8_t* q = static_cast<uint8_t*>(ws);
    float* grow = reinterpret_cast<float*>(q);
    float* drow = reinterpret_cast<float*>(q + L.rows);
    float* GT = reinterpret_cast<float*>(q + 2 * L.rows);
    __half* gh = reinterpret_cast<__half*>(q + 2 * L.rows + L.gt);
    __half* gl = reinterpret_cast<__half*>(q + 2 * L.rows + L.gt + L.half);
    float* gs = reinterpret_cast<float*>(q + 2 * L.rows + L.gt + 2 * L.half);
    tensor_basis(*t, x + p0 * ldx, m, ldx, grow, drow, L.gstride, st);
    cotangent_kernel<<<smx::grid_for(m, 8), 256, 0, st>>>(g + p0 * ldg, ldg, m, t->d_out, b->ldo, b->out_scale, gh, gl,
                                                          gs);
    int rc;
    if (b->ldo <= 64 * kAdjMaxSlices) {
      if ((rc = adjoint_gemm(*t, *b, gh, gl, gs, GT, m, L.gstride, sms, st))) return rc;
    } else {
      SplitGemm s{};
      s.bits = kF16;
      s.Ah = b->Rh, s.Al = b->Rl, s.lda = b->ldo;
      s.Bh = gh, s.Bl = gl, s.ldb = b->ldo;
      s.row_scale = b->row_scale, s.ld_scale = b->n_rows;
      s.col_scale = gs;
      s.M = int(b->n_rows), s.N = int(m), s.K = t->d_out;
      s.D = GT, s.ldd = 0;
      s.err = t->err, s.splits = 1;
      if ((rc = split_gemm(s, st))) return rc;
    }
    vjp_walk_kernel<<<smx::grid_for(m, 32), kThreads, walk_smem(t, w), st>>>(*t, w, grow, drow, L.gstride, GT, m,
                                                                              t->err, dx + p0 * lddx, lddx);
    SMX_LAUNCH_CHECK("smx_tensor_vjp_x");
  }
  return SMX_OK;
}
