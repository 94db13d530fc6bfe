// Dense Jacobian of the orthogonal form in FP64 (interpolation.py:306-345 over
// barycentric.py:126-229, for Leja and Gauss-Hermite rules).
//
//   J[p][o][j] = sum over entries e of Lambda with e_j = g > 0 of
//                a_j phi_g'(z_j) * A[p][e without j] * C[e][o]
//
// "e without j" is again an entry of the downward closed set, so the products
// A are needed for few distinct rows and are shared by all outputs and
// dimensions.  Per point and output that leaves one multiply-add per (entry,
// active dimension) pair -- 1.1e4 at d_in = 200, |Lambda| = 5000 -- which is
// the bound (2 FP64 multiply-adds per SM clock); every load is hidden behind it.
//
// Kernels:
//   jac_basis  phi[slot][p], a_j phi'[slot][p] of every (dimension, degree)
//              slot, and per dimension whether x_j is a node of the rule
//   jac_rows   A[row][p], product of the row's slots
//   jac_units  the terms are sorted by slot (j, g) and cut into units of at
//              most 128: one block per unit and tile of (points, outputs)
//              leaves phi' * sum in part[unit][p][o].  A thread holds one
//              output and 4 points, lanes run along the outputs (along the
//              points for few outputs), so rows of C are read whole and the
//              products of 4 points by two broadcast 16-byte loads.
//   jac_sum    J[p][o][j] = the sum of the units of j in order, through a
//              32 x 32 tile so that both sides are coalesced; NaN where x_j is
//              a node (the barycentric derivative's value there), 0 for
//              dimensions without entries.
//
// Measured at d_in = 200, d_out = 64, |Lambda| = 5000, 500 points: 0.73 ms
// (0.57 ms of multiply-adds at the FP64 rate) against 45.1 ms for the combination sum (jacobian64_kernel in eval64.cu: every
// summand's tensor once per active dimension, read-modify-writes of J 100 KB
// apart); that kernel serves the other rules and plans without coefficients.
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int kThreads = 128;
constexpr int kPB = 4;        // points per thread
constexpr int kUnit = 128;    // terms per unit, at most
constexpr int kMaxGridY = 65535;

__device__ __forceinline__ double finite_or_nan(double v) {
  const long long b = __double_as_longlong(v);
  return (b & 0x7fffffffffffffffll) == 0x7ff0000000000000ll ? __longlong_as_double(0x7ff8000000000000ll) : v;
}

// Thread: one point and one active dimension h = blockIdx.y.
__global__ void __launch_bounds__(kThreads) jac_basis_kernel(smx_jacobian64 a, const double* __restrict__ x, int64_t P,
                                                             int64_t ldx, int64_t ldp, int h0, double* __restrict__ phi,
                                                             double* __restrict__ dphi, uint8_t* __restrict__ hit) {
  const int64_t p = blockIdx.x * int64_t(kThreads) + threadIdx.x;
  if (p >= ldp) return;
  const int h = h0 + blockIdx.y;
  const int dim = a.dim[h], g = a.deg[h], so = a.soff[h];
  const double xv = x[min(p, P - 1) * ldx + dim];
  const double fa = a.fam_a[dim];
  const double z = fma(fa, finite_or_nan(xv), a.fam_b[dim]);
  double pm1 = 0.0, pc = 1.0, dm1 = 0.0, dc = 0.0;
  const double2* rec = reinterpret_cast<const double2*>(a.rec) + a.fam[dim] * a.max_deg;
  for (int n = 0; n < g; ++n) {
    const double al = rec[n].x, be = rec[n].y;
    const double pn = fma(al * z, pc, -be * pm1);
    const double dn = fma(al, fma(z, dc, pc), -be * dm1);
    pm1 = pc, pc = pn, dm1 = dc, dc = dn;
    phi[(so + n) * ldp + p] = pc;
    dphi[(so + n) * ldp + p] = fa * dc;
  }
  uint8_t on = 0;
  for (int q = a.node_off[h]; q < a.node_off[h + 1]; ++q) on |= __dsub_rn(xv, a.node[q]) == 0.0;
  hit[h * ldp + p] = on;
}

// Thread: one point and 8 rows.
constexpr int kRowsPer = 8;
__global__ void __launch_bounds__(kThreads) jac_rows_kernel(smx_jacobian64 a, const double* __restrict__ phi,
                                                            int64_t ldp, int row0, double* __restrict__ A) {
  const int64_t p = blockIdx.x * int64_t(kThreads) + threadIdx.x;
  if (p >= ldp) return;
  const int r0 = row0 + blockIdx.y * kRowsPer, r1 = min(a.n_rows, r0 + kRowsPer);
  for (int r = r0; r < r1; ++r) {
    double v = 1.0;
    for (int q = a.row_off[r]; q < a.row_off[r + 1]; ++q) v *= phi[a.row_slot[q] * ldp + p];
    A[r * ldp + p] = v;
  }
}

// Block: unit blockIdx.x, outputs (tile0 + blockIdx.y) << lo_log .., points of
// group blockIdx.z.  ldp is a multiple of kPB; rows past P are computed on the
// last point's values and not read by jac_sum.
__global__ void __launch_bounds__(kThreads) jac_units_kernel(smx_jacobian64 a, const double* __restrict__ A,
                                                             const double* __restrict__ dphi, int64_t ldp, int lo_log,
                                                             int tile0, double* __restrict__ part) {
  const int t = threadIdx.x;
  const int o = ((tile0 + int(blockIdx.y)) << lo_log) + (t & ((1 << lo_log) - 1));
  const int64_t p = ((int64_t(blockIdx.z) * (kThreads >> lo_log)) + (t >> lo_log)) * kPB;
  if (o >= a.d_out || p >= ldp) return;
  const int4 u = __ldg(reinterpret_cast<const int4*>(a.unit) + blockIdx.x);  // {t0, t1, slot, dim index}
  const int2* term = reinterpret_cast<const int2*>(a.term);
  double s[kPB] = {};
#pragma unroll 4
  for (int q = u.x; q < u.y; ++q) {
    const int2 tm = __ldg(term + q);  // {row of A, entry}
    const double c = __ldg(a.C + int64_t(tm.y) * a.d_out + o);
    const double2* ar = reinterpret_cast<const double2*>(A + tm.x * ldp + p);
    const double2 v01 = ar[0], v23 = ar[1];
    s[0] = fma(c, v01.x, s[0]);
    s[1] = fma(c, v01.y, s[1]);
    s[2] = fma(c, v23.x, s[2]);
    s[3] = fma(c, v23.y, s[3]);
  }
  const double* d = dphi + u.z * ldp + p;
  double* out = part + (int64_t(blockIdx.x) * ldp + p) * a.d_out + o;
#pragma unroll
  for (int i = 0; i < kPB; ++i) out[int64_t(i) * a.d_out] = d[i] * s[i];
}

// 32 (point, output) pairs x 32 dimensions per block.
__global__ void __launch_bounds__(256) jac_sum_kernel(smx_jacobian64 a, const double* __restrict__ part,
                                                      const uint8_t* __restrict__ hit, int64_t P, int64_t ldp, int j0,
                                                      double* __restrict__ J) {
  __shared__ double tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t npo = P * a.d_out;
  const int64_t po0 = blockIdx.x * int64_t(32);
  const int jb = j0 + int(blockIdx.y) * 32;
  const int64_t po = po0 + tx;
  for (int r = ty; r < 32; r += 8) {
    const int j = jb + r;
    double v = 0.0;
    if (po < npo && j < a.d_in) {
      const int h = a.dim_index[j];
      if (h >= 0) {
        for (int u = a.unit_off[h]; u < a.unit_off[h + 1]; ++u) v += part[u * (ldp * a.d_out) + po];
        if (hit[h * ldp + po / a.d_out]) v = __longlong_as_double(0x7ff8000000000000ll);
      }
    }
    tile[r][tx] = v;
  }
  __syncthreads();
  const int j = jb + tx;
  for (int r = ty; r < 32; r += 8)
    if (po0 + r < npo && j < a.d_in) J[(po0 + r) * a.d_in + j] = tile[tx][r];
}

size_t up16(size_t v) { return (v + 15) / 16 * 16; }
int64_t pad_points(int64_t P) { return (P + kPB - 1) / kPB * kPB; }

}  // namespace

extern "C" size_t smx_jacobian64_workspace(const smx_jacobian64* sp, int64_t P) {
  if (!sp || P <= 0) return 0;
  const size_t ldp = size_t(pad_points(P));
  return (2 * size_t(sp->n_slots) + size_t(sp->n_rows) + size_t(sp->n_units) * sp->d_out) * ldp * sizeof(double) +
         up16(size_t(sp->n_dims) * ldp);
}

extern "C" int smx_jacobian64_eval(const smx_jacobian64* sp, const double* x, int64_t P, int64_t ldx, double* J,
                                   void* ws, size_t ws_bytes, void* stream) {
  SMX_REQUIRE(sp != nullptr, "smx_jacobian64_eval: null plan");
  SMX_REQUIRE(sp->d_in >= 1 && sp->d_out >= 1 && sp->n_dims >= 1 && sp->n_slots >= 1 && sp->n_rows >= 1 &&
                  sp->n_units >= 1 && sp->max_deg >= 1,
              "smx_jacobian64_eval: bad plan sizes");
  SMX_REQUIRE(sp->dim && sp->deg && sp->soff && sp->node_off && sp->node && sp->dim_index && sp->unit_off &&
                  sp->row_off && sp->row_slot && sp->unit && sp->term && sp->C && sp->rec && sp->fam && sp->fam_a && sp->fam_b,
              "smx_jacobian64_eval: incomplete plan");
  SMX_REQUIRE(P >= 0 && ldx >= sp->d_in, "smx_jacobian64_eval: bad sizes");
  if (P == 0) return SMX_OK;
  SMX_REQUIRE(x && J, "smx_jacobian64_eval: null pointer");
  SMX_REQUIRE(ws && ws_bytes >= smx_jacobian64_workspace(sp, P) && (reinterpret_cast<uintptr_t>(ws) & 15) == 0,
              "smx_jacobian64_eval: workspace too small or not 16-byte aligned");
  const int64_t ldp = pad_points(P);
  double* phi = static_cast<double*>(ws);
  double* dphi = phi + sp->n_slots * ldp;
  double* A = dphi + sp->n_slots * ldp;
  double* part = A + sp->n_rows * ldp;
  uint8_t* hit = reinterpret_cast<uint8_t*>(part + int64_t(sp->n_units) * ldp * sp->d_out);
  cudaStream_t st = smx::as_stream(stream);
  const unsigned pb = smx::grid_for(ldp, kThreads);
  auto slices = [](int n) { return unsigned(std::min(n, kMaxGridY)); };
  for (int h0 = 0; h0 < sp->n_dims; h0 += kMaxGridY)
    jac_basis_kernel<<<dim3(pb, slices(sp->n_dims - h0)), kThreads, 0, st>>>(*sp, x, P, ldx, ldp, h0, phi, dphi, hit);
  const int row_blocks = (sp->n_rows + kRowsPer - 1) / kRowsPer;
  for (int b0 = 0; b0 < row_blocks; b0 += kMaxGridY)
    jac_rows_kernel<<<dim3(pb, slices(row_blocks - b0)), kThreads, 0, st>>>(*sp, phi, ldp, b0 * kRowsPer, A);
  int lo_log = 0;
  while (lo_log < 5 && (1 << lo_log) < sp->d_out) ++lo_log;
  const int o_tiles = (sp->d_out + (1 << lo_log) - 1) >> lo_log;
  const int64_t per = int64_t(kThreads >> lo_log) * kPB;  // points per block
  const int64_t groups = (ldp + per - 1) / per;
  SMX_REQUIRE(groups <= kMaxGridY, "smx_jacobian64_eval: too many points in one call");
  for (int c0 = 0; c0 < o_tiles; c0 += kMaxGridY)
    jac_units_kernel<<<dim3(unsigned(sp->n_units), slices(o_tiles - c0), unsigned(groups)), kThreads, 0, st>>>(
        *sp, A, dphi, ldp, lo_log, c0, part);
  const int j_tiles = (sp->d_in + 31) / 32;
  for (int c0 = 0; c0 < j_tiles; c0 += kMaxGridY)
    jac_sum_kernel<<<dim3(smx::grid_for(P * sp->d_out, 32), slices(j_tiles - c0)), 256, 0, st>>>(*sp, part, hit, P, ldp,
                                                                                                c0 * 32, J);
  SMX_LAUNCH_CHECK("smx_jacobian64_eval");
  return SMX_OK;
}
