// Backward of the tensor-core evaluation with respect to x:
//   G^T[e][p] = sum_o C[e][o] g[p][o]       (tensor cores, scaled FP16 pairs)
//   dL/dx[p][j] = a_j sum_g phi_g'(z_j) bar[slot (j, g)]
// with bar the adjoints of the basis values under L = sum_e G_e prod phi.  The
// reference has the dense Jacobian instead (interpolation.py:306-345).
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
// 1.35 ms (60 % of its issue slots and 58 % of the shared-memory pipe busy, the
// bound), G^T 0.84 ms, basis and cotangent 0.14 ms; the TF32 product and the walk
// per path factor through global memory took 0.82 + 3.94 ms.  On the way: terms
// read from global memory by each warp 1.68 ms, two stages instead of four 1.46 ms.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "tc_util.cuh"
#include "tensor_eval.h"

namespace {

using namespace smx::tc;

constexpr int kStages = 4;  // chunks in flight (layout.cu build_walk sizes them)
constexpr int kWarps = 32;  // owners of destination rows (layout.cu build_walk)
constexpr int kThreads = 32 * kWarps;
constexpr size_t kSmemMax = 227 * 1024;

__device__ __forceinline__ float x32(double v) {
  const float f = static_cast<float>(v);
  return fabsf(f) == __int_as_float(0x7f800000) ? __int_as_float(0x7fc00000) : f;
}

// Basis values and their derivatives in z, [slot][p] (as tensor_basis_kernel).
__global__ void __launch_bounds__(256) vjp_basis_kernel(smx_tensor t, const double* __restrict__ x, int64_t P,
                                                        int64_t ldx, float* __restrict__ grow,
                                                        float* __restrict__ drow, int64_t gstride) {
  __shared__ float z[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t p0 = blockIdx.x * int64_t(32);
  for (int h0 = blockIdx.y * 32; h0 < t.n_dims; h0 += gridDim.y * 32) {
    const int h = h0 + lane;
    if (h < t.n_dims) {
      const int dim = __ldg(t.dims + h);
      const float fa = __ldg(t.fam_a + dim), fb = __ldg(t.fam_b + dim);
      for (int r = warp; r < 32; r += 8) z[lane][r] = fmaf(fa, x32(__ldg(x + min(p0 + r, P - 1) * ldx + dim)), fb);
    }
    __syncthreads();
    for (int q = warp; q < 32 && h0 + q < t.n_dims; q += 8) {
      const int hq = h0 + q;
      const int g = __ldg(t.dmax + hq), so = __ldg(t.dsoff + hq);
      const float2* rec = reinterpret_cast<const float2*>(t.rec) + __ldg(t.fam + __ldg(t.dims + hq)) * t.max_deg;
      const float zv = z[q][lane];
      float pm1 = 0.f, pc = 1.f, dm1 = 0.f, dc = 0.f;
      for (int n = 0; n < g; ++n) {
        const float2 ab = __ldg(rec + n);
        const float pn = ab.x * zv * pc - ab.y * pm1;
        const float dn = ab.x * (pc + zv * dc) - ab.y * dm1;
        pm1 = pc, pc = pn, dm1 = dc, dc = dn;
        grow[int64_t(so + n) * gstride + p0 + lane] = pc;
        drow[int64_t(so + n) * gstride + p0 + lane] = dc;
      }
    }
    __syncthreads();
  }
}

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
    lo[p * ldo + o] = __float2half_rn(v - __half2float(h));
  }
  if (lane == 0) scale[p] = __int_as_float((e - 14) << 23);
}

// Rows of C: per output the power of two of its largest finite coefficient ...
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
    scale[o] = m > 0.f ? __int_as_float(min(max(__float_as_int(m) >> 23, 1), 253) << 23) : 1.f;
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
    lo[e * ldo + o] = __float2half_rn(v - __half2float(h));
  }
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
    for (int c = 0; c < min(kStages, w.n_chunks); ++c) load_chunk(c);
  }
  for (int s = warp; s < ns; s += kWarps) row[s * 32] = grow[s * gstride + p];
  for (int s = row_bar + warp; s < n_rows; s += kWarps) row[s * 32] = 0.f;
  __syncthreads();
  for (int n0 = warp; n0 < nn; n0 += kWarps * 32) {  // a lane's load for each of 32 nodes
    const int n = (nn - n0 + kWarps - 1) / kWarps, at = n0 + min(lane, n - 1) * kWarps;
    const int4 path = __ldg(reinterpret_cast<const int4*>(w.node_path) + at);
    for (int k = 0; k < min(32, n); ++k) row[(ns + n0 + k * kWarps) * 32] = slot_product(row, from_lane(path, k));
  }
  __syncthreads();
  // terms of this warp, chunk by chunk; a destination row is only ever touched by
  // its warp, so the warps need not keep step beyond the two stages
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
#pragma unroll 1
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
        load_chunk(c + kStages);
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
      for (int s = 0; s < kStages; ++s)
        if (s < w.n_chunks)
          for (uint32_t ph = 0; ph < 2 && !mbar_wait(&full[s], ph, nullptr); ++ph) {
          }
    }
    return;
  }
  // path factors; the slot's adjoint times its derivative in its row of bar
  for (int i = __ldg(w.warp + warp); i < __ldg(w.warp + warp + 1); ++i) {
    const int4 s = __ldg(reinterpret_cast<const int4*>(w.slot) + i);
    float rest = row[(row_bar + s.x) * 32];
    for (int q0 = s.y; q0 < s.z; q0 += 32) {  // a lane's load for each of 32 factors
      const int n = min(32, s.z - q0), q = q0 + min(lane, n - 1), r = __ldg(w.row + q);
      const int4 other = __ldg(reinterpret_cast<const int4*>(w.other) + q);
      for (int k = 0; k < n; ++k)
        rest = fmaf(row[__shfl_sync(0xffffffffu, r, k) * 32], slot_product(row, from_lane(other, k)), rest);
    }
    row[(row_bar + s.x) * 32] = rest * drow[s.x * gstride + p];
  }
  __syncthreads();
  // per dimension the sum over its degrees, turned in the place of phi and V
  float* turn = reinterpret_cast<float*>(smem);  // [n_dims][33]: ends before bar (checked on the host)
  for (int h = warp; h < t.n_dims; h += kWarps) {
    const int so = __ldg(t.dsoff + h), g = __ldg(t.dmax + h);
    float acc = 0.f;
    for (int n = 0; n < g; ++n) acc += row[(row_bar + so + n) * 32];
    turn[h * 33 + lane] = acc;
  }
  __syncthreads();
  for (int q = warp; q < 32; q += kWarps) {
    if (p0 + q >= P) break;
    double* out = dx + (p0 + q) * lddx;
    for (int j = lane; j < t.d_in; j += 32) {
      const int h = __ldg(w.dim_index + j);
      out[j] = h < 0 ? 0.0 : double(__ldg(t.fam_a + j)) * double(turn[h * 33 + q]);
    }
  }
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
  L.scale = up256(size_t(m) * 4);
  L.total = 2 * L.rows + L.gt + 2 * L.half + L.scale;
  return L;
}

}  // namespace

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
    const dim3 bgrid(unsigned(L.gstride / 32), unsigned(std::min((t->n_dims + 31) / 32, 65535)));
    vjp_basis_kernel<<<bgrid, 256, 0, st>>>(*t, x + p0 * ldx, m, ldx, grow, drow, L.gstride);
    cotangent_kernel<<<smx::grid_for(m, 8), 256, 0, st>>>(g + p0 * ldg, ldg, m, t->d_out, b->ldo, b->out_scale, gh, gl,
                                                          gs);
    SplitGemm s{};
    s.bits = kF16;
    s.Ah = b->Rh, s.Al = b->Rl, s.lda = b->ldo;
    s.Bh = gh, s.Bl = gl, s.ldb = b->ldo;
    s.row_scale = b->row_scale, s.ld_scale = b->n_rows;
    s.col_scale = gs;
    s.M = int(b->n_rows), s.N = int(m), s.K = t->d_out;
    s.D = GT, s.ldd = 0;
    s.err = t->err, s.splits = 1;
    int rc = split_gemm(s, st);
    if (rc) return rc;
    vjp_walk_kernel<<<smx::grid_for(m, 32), kThreads, walk_smem(t, w), st>>>(*t, w, grow, drow, L.gstride, GT, m,
                                                                              t->err, dx + p0 * lddx, lddx);
    SMX_LAUNCH_CHECK("smx_tensor_vjp_x");
  }
  return SMX_OK;
}
