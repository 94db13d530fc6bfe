// FP64 evaluation path: the reference's combination technique, evaluated
// with the barycentric basis (src/smolyax/barycentric.py) over an unpadded,
// ragged summand layout.
//
//   basis   : Lt[v][p]   normalised barycentric basis value of slot v at point p
//   contract: y[p][o]    offset[o] + sum_s sum_mu F_s[mu][o] prod_i Lt[pair_i, mu_i][p]
//   jacobian: J[p][o][j] derivative of the same sum (one factor replaced by dLt)
//   integral: Q[o]       offset[o] + sum_r qw(r) F[r][o]
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace {

constexpr int kMaxN = 4;   // summands with more active dimensions use the generic path
constexpr int kOC = 4;     // outputs accumulated per pass
constexpr int kMaxGridY = 65535;

// --- barycentric weights (barycentric.py:13-31) ---------------------------------------
__global__ void bary_weights_kernel(int n_pairs, const int32_t* __restrict__ deg, const int32_t* __restrict__ voff,
                                    const double* __restrict__ node, double* __restrict__ w) {
  int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= n_pairs) return;
  const int g = deg[u], o = voff[u];
  for (int b = 0; b <= g; ++b) {
    double acc = 1.0;
    for (int a = 0; a <= g; ++a) {
      double df = __dsub_rn(node[o + a], node[o + b]);
      if (df == 0.0) df = 1.0;
      acc = __dmul_rn(acc, __ddiv_rn(1.0, df));
    }
    w[o + b] = acc;
  }
}

// Normalised barycentric basis of one pair of degree G (no node hit): one
// reciprocal per node difference and one per row sum, kept in registers (FP64
// division is the expensive operation of this kernel on the FP64 pipe).
template <int G>
__device__ __forceinline__ void basis_pair(double xv, const double* __restrict__ nd, const double* __restrict__ bw,
                                           double* __restrict__ Lt, double* __restrict__ dLt, int o, int64_t P,
                                           int64_t p) {
  double r[G + 1], b[G + 1];
  double S = 0.0, Sd = 0.0;
#pragma unroll
  for (int j = 0; j <= G; ++j) {
    r[j] = 1.0 / __dsub_rn(xv, nd[j]);
    b[j] = bw[j] * r[j];
    S += b[j];
    Sd -= b[j] * r[j];
  }
  const double iS = 1.0 / S;
#pragma unroll
  for (int j = 0; j <= G; ++j) {
    const double l = b[j] * iS;
    Lt[int64_t(o + j) * P + p] = l;
    if (dLt) dLt[int64_t(o + j) * P + p] = (-b[j] * r[j]) * iS - l * Sd * iS;
  }
}

// --- basis table (barycentric.py:34-66, normalisation :117; derivative :126-155, :213-219)
__global__ void basis64_kernel(int n_pairs, const int32_t* __restrict__ pdim, const int32_t* __restrict__ pdeg,
                               const int32_t* __restrict__ pvoff, const double* __restrict__ node,
                               const double* __restrict__ bw, const double* __restrict__ x, int64_t P, int64_t ldx,
                               double* __restrict__ Lt, double* __restrict__ dLt, int pairs_per_block) {
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p >= P) return;
  const int u0 = blockIdx.y * pairs_per_block;
  const int u1 = min(n_pairs, u0 + pairs_per_block);
  const double* xp = x + p * ldx;
  const double qnan = __longlong_as_double(0x7ff8000000000000LL);
  for (int u = u0; u < u1; ++u) {
    const int g = pdeg[u], o = pvoff[u];
    const double xv = xp[pdim[u]];
    int hits = 0;
    for (int j = 0; j <= g; ++j) hits += (__dsub_rn(xv, node[o + j]) == 0.0);
    if (hits) {
      // one-hot rule: b_j = [x == xi_j], normalised by the number of hits
      for (int j = 0; j <= g; ++j) {
        const double bj = (__dsub_rn(xv, node[o + j]) == 0.0) ? 1.0 : 0.0;
        Lt[int64_t(o + j) * P + p] = bj / double(hits);
        if (dLt) dLt[int64_t(o + j) * P + p] = qnan;
      }
      continue;
    }
    switch (g) {
      case 0: basis_pair<0>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 1: basis_pair<1>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 2: basis_pair<2>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 3: basis_pair<3>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 4: basis_pair<4>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 5: basis_pair<5>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 6: basis_pair<6>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 7: basis_pair<7>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      case 8: basis_pair<8>(xv, node + o, bw + o, Lt, dLt, o, P, p); break;
      default: {
        double S = 0.0, Sd = 0.0;
        for (int j = 0; j <= g; ++j) {
          const double r = 1.0 / __dsub_rn(xv, node[o + j]);
          const double b = bw[o + j] * r;
          S += b;
          Sd -= b * r;
        }
        const double iS = 1.0 / S;
        for (int j = 0; j <= g; ++j) {
          const double r = 1.0 / __dsub_rn(xv, node[o + j]);
          const double b = bw[o + j] * r;
          const double l = b * iS;
          Lt[int64_t(o + j) * P + p] = l;
          if (dLt) dLt[int64_t(o + j) * P + p] = (-b * r) * iS - l * Sd * iS;
        }
      }
    }
  }
}

// --- contraction --------------------------------------------------------------------------
// Outputs of one row of F (0 past nout): 16-byte loads where the row allows.
template <int OC>
__device__ __forceinline__ void load_row(const double* __restrict__ f, int nout, double (&v)[OC]) {
  if constexpr (OC % 2 == 0) {
    if (nout == OC && (reinterpret_cast<uintptr_t>(f) & 15) == 0) {
#pragma unroll
      for (int q = 0; q < OC; q += 2) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(f + q));
        v[q] = t.x, v[q + 1] = t.y;
      }
      return;
    }
  }
#pragma unroll
  for (int q = 0; q < OC; ++q) v[q] = q < nout ? __ldg(f + q) : 0.0;
}

// Level L of a summand with N active pairs: sum over mu_L of l_L[mu_L] * (inner).
// The innermost level reads rows of F.  `dslot` selects a pair whose basis is
// replaced by its derivative table (jacobian); -1 for evaluation.
template <int OC, int L, int N>
__device__ inline void clevel(const double* __restrict__ Lt, const double* __restrict__ dLt, int dslot, int64_t P,
                              int64_t p, const int (&voff)[kMaxN], const int (&deg)[kMaxN],
                              const double* __restrict__ Fs, int dout, int o0, int nout, int64_t row,
                              double (&acc)[OC]) {
  const int g = deg[L];
  const double* lt = (dslot == L ? dLt : Lt) + int64_t(voff[L]) * P + p;
  if constexpr (L == N - 1 && OC == 1) {
    // innermost level of one output: a dot product with the rows of F, as two
    // interleaved chains (even and odd nodes) so that the FP64 FMA latency overlaps
    const double* fr = Fs + row * (g + 1) * dout + o0;
    double a0[OC], a1[OC];
#pragma unroll
    for (int q = 0; q < OC; ++q) a0[q] = a1[q] = 0.0;
    int j = 0;
    for (; j < g; j += 2) {
      const double l0 = lt[int64_t(j) * P], l1 = lt[int64_t(j + 1) * P];
#pragma unroll
      for (int q = 0; q < OC; ++q) {
        if (q < nout) {
          a0[q] = fma(l0, fr[j * dout + q], a0[q]);
          a1[q] = fma(l1, fr[(j + 1) * dout + q], a1[q]);
        }
      }
    }
    if (j == g) {
      const double l0 = lt[int64_t(j) * P];
#pragma unroll
      for (int q = 0; q < OC; ++q)
        if (q < nout) a0[q] = fma(l0, fr[j * dout + q], a0[q]);
    }
#pragma unroll
    for (int q = 0; q < OC; ++q) acc[q] += a0[q] + a1[q];
  } else {
    for (int j = 0; j <= g; ++j) {
      const double l = lt[int64_t(j) * P];
      double sub[OC];
      if constexpr (L == N - 1) {
        load_row<OC>(Fs + (row * (g + 1) + j) * dout + o0, nout, sub);
      } else {
#pragma unroll
        for (int q = 0; q < OC; ++q) sub[q] = 0.0;
        clevel<OC, L + 1, N>(Lt, dLt, dslot, P, p, voff, deg, Fs, dout, o0, nout, row * (g + 1) + j, sub);
      }
#pragma unroll
      for (int q = 0; q < OC; ++q) acc[q] = fma(l, sub[q], acc[q]);
    }
  }
}

// Generic path (any number of pairs): full product per entry.
template <int OC>
__device__ inline void cgeneric(const double* __restrict__ Lt, const double* __restrict__ dLt, int dslot, int64_t P,
                                int64_t p, const int32_t* __restrict__ pairs, int n,
                                const int32_t* __restrict__ pvoff, const int32_t* __restrict__ pdeg,
                                const double* __restrict__ Fs, int64_t K, int dout, int o0, int nout,
                                double (&acc)[OC]) {
  int mu[SMX_MAX_DEPTH];
  for (int i = 0; i < n; ++i) mu[i] = 0;
  for (int64_t r = 0; r < K; ++r) {
    double w = 1.0;
    for (int i = 0; i < n; ++i) {
      const double* t = (i == dslot ? dLt : Lt);
      w *= t[int64_t(pvoff[pairs[i]] + mu[i]) * P + p];
    }
    const double* fr = Fs + r * dout + o0;
#pragma unroll
    for (int q = 0; q < OC; ++q)
      if (q < nout) acc[q] = fma(w, fr[q], acc[q]);
    for (int i = n - 1; i >= 0; --i) {  // row-major increment, last pair fastest
      if (++mu[i] <= pdeg[pairs[i]]) break;
      mu[i] = 0;
    }
  }
}

// Up to kMaxN pairs, nested.
template <int OC>
__device__ __forceinline__ void contract_nest(const double* __restrict__ Lt, const double* __restrict__ dLt, int dslot,
                                              int64_t P, int64_t p, const int (&voff)[kMaxN], const int (&deg)[kMaxN],
                                              int n, const double* __restrict__ Fs, int dout, int o0, int nout,
                                              double (&acc)[OC]) {
  switch (n) {
    case 1: clevel<OC, 0, 1>(Lt, dLt, dslot, P, p, voff, deg, Fs, dout, o0, nout, 0, acc); break;
    case 2: clevel<OC, 0, 2>(Lt, dLt, dslot, P, p, voff, deg, Fs, dout, o0, nout, 0, acc); break;
    case 3: clevel<OC, 0, 3>(Lt, dLt, dslot, P, p, voff, deg, Fs, dout, o0, nout, 0, acc); break;
    default: clevel<OC, 0, 4>(Lt, dLt, dslot, P, p, voff, deg, Fs, dout, o0, nout, 0, acc); break;
  }
}

template <int OC>
__device__ inline void contract_summand(const double* __restrict__ Lt, const double* __restrict__ dLt, int dslot,
                                        int64_t P, int64_t p, const int32_t* __restrict__ pairs, int n,
                                        const int32_t* __restrict__ pvoff, const int32_t* __restrict__ pdeg,
                                        const double* __restrict__ Fs, int64_t K, int dout, int o0, int nout,
                                        double (&acc)[OC]) {
  if (n > kMaxN) {
    cgeneric<OC>(Lt, dLt, dslot, P, p, pairs, n, pvoff, pdeg, Fs, K, dout, o0, nout, acc);
    return;
  }
  int voff[kMaxN], deg[kMaxN];
#pragma unroll
  for (int i = 0; i < kMaxN; ++i) {
    voff[i] = i < n ? pvoff[pairs[i]] : 0;
    deg[i] = i < n ? pdeg[pairs[i]] : 0;
  }
  contract_nest<OC>(Lt, dLt, dslot, P, p, voff, deg, n, Fs, dout, o0, nout, acc);
}

struct PlanArgs {
  int n_sum, dout, d_in, n_values;
  const int32_t* poff;
  const int32_t* pairs;
  const int64_t* eoff;
  const int32_t* pvoff;
  const int32_t* pdeg;
  const int32_t* pdim;
  const double* F;
  const double* offset;
};

// Evaluation: y[p][o] = offset[o] + sum over all rows r of F of (product of the
// row's basis values at p) * F[r][o].  A cluster of `parts` blocks of kWarps warps
// takes 32 points (lane = point) and up to 8 outputs: the rows are cut into parts x
// kWarps runs of whole summands, one per warp, so that a few thousand points
// already fill the GPU and a basis value is read once for all outputs.  The sums of
// a summand stay nested (pair by pair): with one weight per row its terms lose the
// cancellation inside each dimension, 3 to 4 times the error (2.6 ms instead of
// 3.4, not kept).  The basis values of the points sit in shared memory when
// they fit (SROWS).  Sums are added in a fixed order that does not depend on the
// batch.  Bound: the FP64 pipe,
// 2 multiply-adds per SM clock (0.63 T/s).  Gauss-Hermite d_in = 100, |Lambda| =
// 3545 (19993 rows), 8 outputs: 5000 points 3.4 ms, 50 points 0.36 ms; a thread per
// point and four outputs that ran through all summands took 10.7 and 10.4 ms.  Leja
// d_in = 1000 (50610 rows), one output: 10000 points 14.7 -> 3.6 ms, 1e5 points 38.3
// -> 32.9.  The summands' tables are loaded by lanes, 32 at a time (33 ms; 49 with a
// chain of loads per summand), and sums over them are compensated every kRun: the
// same error or less than the two-level sum before (2.2e-13 after 2.3e-13, 7e-15
// after 1.8e-14); compensated for every summand 5.1 ms.
constexpr int kWarps = 16;
constexpr int kRun = 8;  // summands between two compensated additions
constexpr int kSmemMax = 226 * 1024;

// Blocks per cluster, fixed per plan (a point's value does not depend on its
// batch): up to 8, while a warp's run has 64 rows.  8 blocks for a plan of 32 rows
// took 152 us at 3000 points, one 73; for 4282 rows 7.5 ms at 1e5 points and 160 us
// at 1000, 4 blocks 5.5 ms and 107 us.
int contract_parts(int64_t rows) {
  int parts = 1;
  while (parts < 8 && rows >= int64_t(2 * parts) * kWarps * 64) parts *= 2;
  return parts;
}

// The correction of an infinite or undefined sum is left out, so that the sum stays what it is.
__device__ __forceinline__ double finite_or_zero(double e) {
  return (__double2hiint(e) & 0x7ff00000) == 0x7ff00000 ? 0.0 : e;
}

// sum + v exactly as the new sum and an error that is added to `low`.
__device__ __forceinline__ void two_sum(double& sum, double& low, double v) {
  const double t = __dadd_rn(sum, v), z = __dadd_rn(t, -sum);
  const double e = __dadd_rn(__dadd_rn(sum, -__dadd_rn(t, -z)), __dadd_rn(v, -z));
  low += finite_or_zero(e);
  sum = t;
}

// First summand whose rows begin at or after row r, by a warp.
__device__ __forceinline__ int first_summand(const PlanArgs& a, int64_t r, int lane) {
  int lo = 0, n = a.n_sum;  // answer in [lo, lo + n]
  while (n > 0) {
    const int step = (n + 31) / 32, i = lo + min((lane + 1) * step, n) - 1;
    const unsigned before = __ballot_sync(0xffffffffu, a.eoff[i] < r);
    const int k = __popc(before);  // whole steps before the answer
    if (k == 32) return lo + n;
    lo += k * step;
    n = min(step - 1, n - k * step - 1);
    if (n < 0) n = 0;
  }
  return lo;
}

template <int DO, bool SROWS>
__global__ void __launch_bounds__(32 * kWarps, DO == 1 ? 2 : 1)
    contract_kernel(PlanArgs a, const double* __restrict__ Lt, int64_t P, double* __restrict__ y, int o_base,
                    int parts) {
  extern __shared__ __align__(16) double sm64[];
  double* all = sm64;                         // [parts][DO][32][2] at the first block
  double* rows = all + parts * DO * 64;      // [n_values][32]
  double* own = rows;                         // [kWarps][DO][32], when the rows are done with
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned part;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(part));
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");  // all blocks run: their memory may be written
  const int64_t p0 = (blockIdx.x / parts) * int64_t(32), p = min(p0 + lane, P - 1);
  const int o0 = o_base + int(blockIdx.y) * DO, nout = min(DO, a.dout - o0);
  if constexpr (SROWS) {
#pragma unroll 4
    for (int v = warp; v < a.n_values; v += kWarps) rows[v * 32 + lane] = __ldg(Lt + int64_t(v) * P + p);
    __syncthreads();
  }
  double acc[DO], comp[DO];
#pragma unroll
  for (int o = 0; o < DO; ++o) acc[o] = comp[o] = 0.0;
  const int64_t R = a.n_sum > 0 ? a.eoff[a.n_sum] : 0;
  const int seg = int(part) * kWarps + warp;
  const int s1 = first_summand(a, R * (seg + 1) / (parts * kWarps), lane);
  const int s0 = first_summand(a, R * seg / (parts * kWarps), lane);
  double run[DO];  // up to kRun summands
#pragma unroll
  for (int o = 0; o < DO; ++o) run[o] = 0.0;
  int n_of = 0, voff_of[kMaxN], deg_of[kMaxN];
  int64_t e_of = 0;
  for (int s = s0; s < s1; ++s) {
    const int k = (s - s0) & 31;
    if (k == 0) {  // a lane's loads for each of the next 32 summands
      const int mine = min(s + lane, s1 - 1), q0 = __ldg(a.poff + mine);
      n_of = __ldg(a.poff + mine + 1) - q0;
      e_of = __ldg(a.eoff + mine);
#pragma unroll
      for (int i = 0; i < kMaxN; ++i) {
        const int u = i < n_of ? __ldg(a.pairs + q0 + i) : -1;
        voff_of[i] = u >= 0 ? __ldg(a.pvoff + u) : 0;
        deg_of[i] = u >= 0 ? __ldg(a.pdeg + u) : 0;
      }
    }
    const int n = __shfl_sync(0xffffffffu, n_of, k);
    const int64_t e0 = __shfl_sync(0xffffffffu, e_of, k);
    const double* lt = SROWS ? rows : Lt;
    const int64_t stride = SROWS ? 32 : P, at = SROWS ? lane : p;
    if (n <= kMaxN) {
      int voff[kMaxN], deg[kMaxN];
#pragma unroll
      for (int i = 0; i < kMaxN; ++i) {
        voff[i] = __shfl_sync(0xffffffffu, voff_of[i], k);
        deg[i] = __shfl_sync(0xffffffffu, deg_of[i], k);
      }
      contract_nest<DO>(lt, nullptr, -1, stride, at, voff, deg, n, a.F + e0 * a.dout, a.dout, o0, nout, run);
    } else {
      cgeneric<DO>(lt, nullptr, -1, stride, at, a.pairs + __ldg(a.poff + s), n, a.pvoff, a.pdeg, a.F + e0 * a.dout,
                   __ldg(a.eoff + s + 1) - e0, a.dout, o0, nout, run);
    }
    if ((s - s0) % kRun == kRun - 1 || s + 1 == s1) {
#pragma unroll
      for (int o = 0; o < DO; ++o) {  // compensated
        const double v = __dadd_rn(run[o], -comp[o]), t = __dadd_rn(acc[o], v);
        comp[o] = finite_or_zero(__dadd_rn(__dadd_rn(t, -acc[o]), -v));
        acc[o] = t;
        run[o] = 0.0;
      }
    }
  }
  // the block's warps, then the cluster's blocks, in order
  __syncthreads();
#pragma unroll
  for (int o = 0; o < DO; ++o) own[(warp * DO + o) * 32 + lane] = acc[o];
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  for (int i = threadIdx.x; i < DO * 32; i += 32 * kWarps) {
    double sum = own[i], low = 0.0;
#pragma unroll
    for (int w = 1; w < kWarps; ++w) two_sum(sum, low, own[w * DO * 32 + i]);
    uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(all + 2 * (part * DO * 32 + i)));
    asm volatile("mapa.shared::cluster.u32 %0, %0, 0;" : "+r"(to));
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(to), "d"(sum), "d"(low) : "memory");
  }
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
  if (part != 0) return;
  for (int i = threadIdx.x; i < 32 * nout; i += 32 * kWarps) {
    const int q = i / nout, o = i - q * nout;
    if (p0 + q >= P) break;
    double sum = a.offset[o0 + o], low = 0.0;
    for (int b = 0; b < parts; ++b) {
      const double2 v = reinterpret_cast<const double2*>(all)[(b * DO + o) * 32 + q];
      two_sum(sum, low, v.x);
      low += v.y;
    }
    y[(p0 + q) * a.dout + o0 + o] = sum + low;
  }
}

// Jacobian: J[p][o][dim] += derivative contraction of every summand and every
// active slot.  Each thread owns one point, so the read-modify-writes of its
// row of J never race.
template <int OC>
__global__ void jacobian64_kernel(PlanArgs a, const double* __restrict__ Lt, const double* __restrict__ dLt, int64_t P,
                                  double* __restrict__ J, int o_base) {
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int o0 = o_base + int(blockIdx.y) * OC;
  if (p >= P || o0 >= a.dout) return;
  const int nout = min(OC, a.dout - o0);
  double* Jp = J + p * int64_t(a.dout) * a.d_in;
  for (int s = 0; s < a.n_sum; ++s) {
    const int q0 = a.poff[s], n = a.poff[s + 1] - q0;
    const int64_t e0 = a.eoff[s], K = a.eoff[s + 1] - e0;
    for (int i = 0; i < n; ++i) {
      double acc[OC];
#pragma unroll
      for (int q = 0; q < OC; ++q) acc[q] = 0.0;
      contract_summand<OC>(Lt, dLt, i, P, p, a.pairs + q0, n, a.pvoff, a.pdeg, a.F + e0 * a.dout, K, a.dout, o0, nout,
                       acc);
      const int dim = a.pdim[a.pairs[q0 + i]];
#pragma unroll
      for (int q = 0; q < OC; ++q)
        if (q < nout) Jp[int64_t(o0 + q) * a.d_in + dim] += acc[q];
    }
  }
}

// Integral Q[o] = offset[o] + sum_r qw(r) F[r][o], qw(r) the product of the
// quadrature weights of row r's nodes.  F is read once (the bound; ~11 MB at
// 1.8e5 rows x 8 outputs), so the work is spread over rows: a block takes
// kQuadRows rows, computes their weights into shared memory (one row per
// thread and pass: summand by binary search, node indices by mixed-radix
// division) and sums TO = 2^to_log outputs with 256 / TO row lanes, so that a
// warp reads whole lines of F whatever d_out is; then a fixed-order sum over
// the lanes, and a second launch of the same shape over the blocks' partial
// sums.  Measured at 1.8e5 rows x 8 outputs (Gauss-Hermite d_in = 100,
// |Lambda| = 20010): 21 us a call against 412 us with the kernels before (one
// thread per summand, 4096 rows per block with 8 of 128 threads at work).
constexpr int kQuadRows = 512;
constexpr int kQuadThreads = 256;

// Sum of v over the row lanes of output `t & (TO - 1)`, in a fixed order.
__device__ __forceinline__ double quad_lanes(double v, int to_log, double* red) {
  const int t = threadIdx.x;
  red[t] = v;
  __syncthreads();
  for (int n = kQuadThreads >> 1; n >= (1 << to_log); n >>= 1) {
    if (t < n) red[t] += red[t + n];
    __syncthreads();
  }
  return red[t];
}

__global__ void __launch_bounds__(kQuadThreads) quad_partial_kernel(PlanArgs a, const double* __restrict__ qnode,
                                                                    int64_t R, int to_log, int tile0,
                                                                    double* __restrict__ part) {
  __shared__ double qw[kQuadRows], red[kQuadThreads];
  const int t = threadIdx.x;
  const int64_t r0 = int64_t(blockIdx.x) * kQuadRows;
  const int nr = int(min(R - r0, int64_t(kQuadRows)));
  for (int i = t; i < nr; i += kQuadThreads) {
    const int64_t r = r0 + i;
    int lo = 0, hi = a.n_sum - 1;  // summand s with eoff[s] <= r < eoff[s + 1]
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (a.eoff[mid] <= r) lo = mid; else hi = mid - 1;
    }
    unsigned rest = unsigned(r - a.eoff[lo]);
    double w = 1.0;
    for (int q = a.poff[lo + 1] - 1; q >= a.poff[lo]; --q) {  // last pair fastest
      const int u = a.pairs[q];
      const unsigned m = unsigned(a.pdeg[u] + 1), up = rest / m;
      w *= qnode[a.pvoff[u] + int(rest - up * m)];
      rest = up;
    }
    qw[i] = w;
  }
  __syncthreads();
  const int o = ((tile0 + int(blockIdx.y)) << to_log) + (t & ((1 << to_log) - 1));
  const int lanes = kQuadThreads >> to_log;
  double acc = 0.0;
  if (o < a.dout)
    for (int i = t >> to_log; i < nr; i += lanes) acc = fma(qw[i], a.F[(r0 + i) * a.dout + o], acc);
  acc = quad_lanes(acc, to_log, red);
  if (t < (1 << to_log) && o < a.dout) part[int64_t(blockIdx.x) * a.dout + o] = acc;
}

__global__ void __launch_bounds__(kQuadThreads) quad_reduce_kernel(const double* __restrict__ part, int64_t nchunks,
                                                                   int dout, int to_log,
                                                                   const double* __restrict__ offset,
                                                                   double* __restrict__ Q) {
  __shared__ double red[kQuadThreads];
  const int t = threadIdx.x;
  const int o = (int(blockIdx.x) << to_log) + (t & ((1 << to_log) - 1));
  double acc = 0.0;
  if (o < dout)
    for (int64_t c = t >> to_log; c < nchunks; c += kQuadThreads >> to_log) acc += part[c * dout + o];
  acc = quad_lanes(acc, to_log, red);
  if (t < (1 << to_log) && o < dout) Q[o] = offset[o] + acc;
}

// F rows from unique function values, zeta folded in.
__global__ void assemble_kernel(int n_sum, const int64_t* __restrict__ eoff, const int64_t* __restrict__ zeta,
                                const double* __restrict__ fu, const int64_t* __restrict__ umap,
                                const double* __restrict__ center, int dout, int64_t R, double* __restrict__ F64,
                                float* __restrict__ F32) {
  const int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (idx >= R * dout) return;
  const int64_t r = idx / dout;
  const int o = int(idx - r * dout);
  int lo = 0, hi = n_sum - 1;  // summand s with eoff[s] <= r < eoff[s+1]
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (eoff[mid] <= r) lo = mid; else hi = mid - 1;
  }
  const double v = double(zeta[lo]) * (fu[umap[r] * dout + o] - (center ? center[o] : 0.0));
  F64[idx] = v;
  if (F32) F32[idx] = float(v);
}

PlanArgs args_of(const smx_plan* pl, const double* F) {
  PlanArgs a;
  a.n_sum = pl->n_summands;
  a.dout = pl->d_out;
  a.d_in = pl->d_in;
  a.n_values = int(pl->n_values);
  a.poff = pl->sum_poff;
  a.pairs = pl->sum_pairs;
  a.eoff = pl->sum_eoff;
  a.pvoff = pl->pair_voff;
  a.pdeg = pl->pair_deg;
  a.pdim = pl->pair_dim;
  a.F = F;
  a.offset = pl->offset;
  return a;
}

int check_plan(const smx_plan* pl, const char* who) {
  if (!pl) return smx::set_error(SMX_ERR_ARG, std::string(who) + ": null plan");
  if (pl->d_out < 1 || pl->d_in < 1 || pl->n_summands < 0 || pl->n_values < 0 || pl->n_pairs < 0)
    return smx::set_error(SMX_ERR_ARG, std::string(who) + ": bad plan sizes");
  if (pl->n_summands > 0 && (!pl->sum_poff || !pl->sum_pairs || !pl->sum_eoff || !pl->pair_voff || !pl->pair_deg ||
                             !pl->pair_dim || !pl->F64))
    return smx::set_error(SMX_ERR_ARG, std::string(who) + ": null plan array");
  if (!pl->offset) return smx::set_error(SMX_ERR_ARG, std::string(who) + ": null offset");
  return SMX_OK;
}

template <int DO, bool SROWS>
int launch_contract(const PlanArgs& a, const double* Lt, int64_t P, double* y, int o_base, int passes, int parts,
                    size_t smem, cudaStream_t st) {
  // (with every launch: the attribute belongs to the current device, and the call is cheap)
  if (cudaFuncSetAttribute(contract_kernel<DO, SROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) !=
      cudaSuccess) {
    cudaGetLastError();
    return smx::set_error(SMX_ERR_CUDA, "smx_contract_f64: shared memory of a block refused");
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = unsigned(parts);
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(unsigned((P + 31) / 32 * parts), unsigned(passes));
  cfg.blockDim = dim3(32 * kWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, contract_kernel<DO, SROWS>, a, Lt, P, y, o_base, parts);
  SMX_LAUNCH_CHECK("smx_contract_f64");
  return SMX_OK;
}

// Basis values in shared memory while they fit (up to 770 with 8 outputs).
template <int DO>
int launch_contract(const PlanArgs& a, const double* Lt, int64_t P, double* y, int o_base, int passes, int64_t n_rows,
                    cudaStream_t st) {
  const int parts = contract_parts(n_rows);
  const size_t all = size_t(parts) * DO * 512, own = size_t(kWarps) * DO * 256, rows = size_t(a.n_values) * 256;
  const size_t room = DO == 1 ? kSmemMax / 2 : kSmemMax;  // one output: two blocks per SM
  return all + rows <= room
             ? launch_contract<DO, true>(a, Lt, P, y, o_base, passes, parts, all + std::max(own, rows), st)
             : launch_contract<DO, false>(a, Lt, P, y, o_base, passes, parts, all + own, st);
}

constexpr int kPairsPerBlock = 64;

}  // namespace

extern "C" int smx_bary_weights(int n_pairs, const int32_t* pair_deg, const int32_t* pair_voff, const double* node,
                                double* bweight, void* stream) {
  SMX_REQUIRE(n_pairs >= 0, "smx_bary_weights: negative size");
  if (n_pairs == 0) return SMX_OK;
  SMX_REQUIRE(pair_deg && pair_voff && node && bweight, "smx_bary_weights: null pointer");
  bary_weights_kernel<<<smx::grid_for(n_pairs, 128), 128, 0, smx::as_stream(stream)>>>(n_pairs, pair_deg, pair_voff,
                                                                                         node, bweight);
  SMX_LAUNCH_CHECK("smx_bary_weights");
  return SMX_OK;
}

extern "C" int smx_basis_f64(const smx_plan* pl, const double* x, int64_t P, int64_t ldx, double* Lt, double* dLt,
                             void* stream) {
  int rc = check_plan(pl, "smx_basis_f64");
  if (rc) return rc;
  SMX_REQUIRE(P >= 0 && ldx >= pl->d_in, "smx_basis_f64: bad sizes");
  if (P == 0 || pl->n_pairs == 0) return SMX_OK;
  SMX_REQUIRE(x && Lt && pl->node && pl->bweight, "smx_basis_f64: null pointer");
  // pairs per block: few enough that a small batch fills the GPU
  const int64_t blocks = (P + 127) / 128;
  const int per = int(std::max<int64_t>(1, std::min<int64_t>(kPairsPerBlock, blocks * pl->n_pairs / 1024)));
  dim3 grid(smx::grid_for(P, 128), (pl->n_pairs + per - 1) / per);
  basis64_kernel<<<grid, 128, 0, smx::as_stream(stream)>>>(pl->n_pairs, pl->pair_dim, pl->pair_deg, pl->pair_voff,
                                                           pl->node, pl->bweight, x, P, ldx, Lt, dLt, per);
  SMX_LAUNCH_CHECK("smx_basis_f64");
  return SMX_OK;
}

extern "C" int smx_contract_f64(const smx_plan* pl, const double* Lt, int64_t P, double* y, void* stream) {
  int rc = check_plan(pl, "smx_contract_f64");
  if (rc) return rc;
  SMX_REQUIRE(P >= 0, "smx_contract_f64: negative P");
  if (P == 0) return SMX_OK;
  SMX_REQUIRE(y && (pl->n_summands == 0 || Lt), "smx_contract_f64: null pointer");
  PlanArgs a = args_of(pl, pl->F64);
  // up to 8 outputs per block, as evenly as they divide
  const int passes = (pl->d_out + 7) / 8, DO = (pl->d_out + passes - 1) / passes;
  for (int c0 = 0; c0 < passes; c0 += kMaxGridY) {
    const int n = std::min(kMaxGridY, passes - c0);
    cudaStream_t st = smx::as_stream(stream);
    switch (DO) {
      case 1: rc = launch_contract<1>(a, Lt, P, y, c0, n, pl->n_entries, st); break;
      case 2: rc = launch_contract<2>(a, Lt, P, y, c0 * 2, n, pl->n_entries, st); break;
      case 3: rc = launch_contract<3>(a, Lt, P, y, c0 * 3, n, pl->n_entries, st); break;
      case 4: rc = launch_contract<4>(a, Lt, P, y, c0 * 4, n, pl->n_entries, st); break;
      case 5: rc = launch_contract<5>(a, Lt, P, y, c0 * 5, n, pl->n_entries, st); break;
      case 6: rc = launch_contract<6>(a, Lt, P, y, c0 * 6, n, pl->n_entries, st); break;
      case 7: rc = launch_contract<7>(a, Lt, P, y, c0 * 7, n, pl->n_entries, st); break;
      default: rc = launch_contract<8>(a, Lt, P, y, c0 * 8, n, pl->n_entries, st); break;
    }
    if (rc) return rc;
  }
  return SMX_OK;
}

extern "C" size_t smx_eval_workspace(const smx_plan* pl, int64_t P, int precision) {
  if (!pl || P < 0) return 0;
  if (precision == 32) return pl->fp32 ? smx_fp32_workspace(pl->fp32, P) : 0;
  return size_t(pl->n_values) * size_t(P) * sizeof(double) + 256;
}

extern "C" int smx_eval(const smx_plan* pl, int precision, const double* x, int64_t P, int64_t ldx, void* y, void* ws,
                        size_t ws_bytes, void* stream) {
  int rc = check_plan(pl, "smx_eval");
  if (rc) return rc;
  SMX_REQUIRE(precision == 64 || precision == 32, "smx_eval: precision must be 64 or 32");
  if (precision == 32) {
    if (!pl->fp32)
      return smx::set_error(SMX_ERR_UNSUPPORTED, "smx_eval: precision 32 needs the plan's FP32 form (plan->fp32, "
                                                 "built by smx_fp32_plan_create)");
    return smx_fp32_eval(pl->fp32, x, P, ldx, static_cast<float*>(y), ws, ws_bytes, stream);
  }
  if (pl->fp32 && smx_fp32_plan_has_fp64(pl->fp32))
    return smx_fp32_eval64(pl->fp32, x, P, ldx, static_cast<double*>(y), stream);
  SMX_REQUIRE(ws_bytes >= smx_eval_workspace(pl, P, precision), "smx_eval: workspace too small");
  double* Lt = static_cast<double*>(ws);
  rc = smx_basis_f64(pl, x, P, ldx, Lt, nullptr, stream);
  if (rc) return rc;
  return smx_contract_f64(pl, Lt, P, static_cast<double*>(y), stream);
}

extern "C" size_t smx_jacobian_workspace(const smx_plan* pl, int64_t P) {
  if (!pl || P < 0) return 0;
  return 2 * size_t(pl->n_values) * size_t(P) * sizeof(double) + 256;
}

extern "C" int smx_jacobian(const smx_plan* pl, const double* x, int64_t P, int64_t ldx, double* J, void* ws,
                            size_t ws_bytes, void* stream) {
  int rc = check_plan(pl, "smx_jacobian");
  if (rc) return rc;
  SMX_REQUIRE(P >= 0 && J, "smx_jacobian: bad arguments");
  SMX_REQUIRE(ws_bytes >= smx_jacobian_workspace(pl, P), "smx_jacobian: workspace too small");
  if (P == 0) return SMX_OK;
  cudaStream_t st = smx::as_stream(stream);
  cudaMemsetAsync(J, 0, size_t(P) * pl->d_out * pl->d_in * sizeof(double), st);
  SMX_LAUNCH_CHECK("smx_jacobian memset");
  if (pl->n_summands == 0) return SMX_OK;
  double* Lt = static_cast<double*>(ws);
  double* dLt = Lt + size_t(pl->n_values) * size_t(P);
  rc = smx_basis_f64(pl, x, P, ldx, Lt, dLt, stream);
  if (rc) return rc;
  PlanArgs a = args_of(pl, pl->F64);
  const int oc = pl->d_out == 1 ? 1 : kOC;
  const int chunks = (pl->d_out + oc - 1) / oc;
  for (int c0 = 0; c0 < chunks; c0 += kMaxGridY) {
    const dim3 grid(smx::grid_for(P, 128), unsigned(std::min(kMaxGridY, chunks - c0)));
    if (oc == 1)
      jacobian64_kernel<1><<<grid, 128, 0, st>>>(a, Lt, dLt, P, J, c0);
    else
      jacobian64_kernel<kOC><<<grid, 128, 0, st>>>(a, Lt, dLt, P, J, c0 * kOC);
    SMX_LAUNCH_CHECK("smx_jacobian");
  }
  return SMX_OK;
}

namespace {
int64_t quad_chunks(int64_t R) { return std::max<int64_t>(1, (R + kQuadRows - 1) / kQuadRows); }
}  // namespace

extern "C" size_t smx_integral_workspace(const smx_plan* pl) {
  if (!pl) return 0;
  return size_t(quad_chunks(pl->n_entries)) * pl->d_out * sizeof(double) + 512;
}

extern "C" int smx_integral(const smx_plan* pl, const double* qnode, double* Q, void* ws, size_t ws_bytes,
                            void* stream) {
  int rc = check_plan(pl, "smx_integral");
  if (rc) return rc;
  SMX_REQUIRE(Q && (pl->n_summands == 0 || qnode), "smx_integral: null pointer");
  SMX_REQUIRE(ws_bytes >= smx_integral_workspace(pl), "smx_integral: workspace too small");
  cudaStream_t st = smx::as_stream(stream);
  // outputs per block: the power of two that covers d_out, at most a warp (one
  // 256-byte row segment per warp load)
  int to_log = 0;
  while (to_log < 5 && (1 << to_log) < pl->d_out) ++to_log;
  const unsigned o_tiles = unsigned((pl->d_out + (1 << to_log) - 1) >> to_log);
  double* part = static_cast<double*>(ws);
  int64_t nch = 0;
  if (pl->n_summands > 0 && pl->n_entries > 0) {
    nch = quad_chunks(pl->n_entries);
    PlanArgs a = args_of(pl, pl->F64);
    for (unsigned c0 = 0; c0 < o_tiles; c0 += kMaxGridY)
      quad_partial_kernel<<<dim3(unsigned(nch), std::min<unsigned>(kMaxGridY, o_tiles - c0)), kQuadThreads, 0, st>>>(
          a, qnode, pl->n_entries, to_log, int(c0), part);
  }
  quad_reduce_kernel<<<o_tiles, kQuadThreads, 0, st>>>(part, nch, pl->d_out, to_log, pl->offset, Q);
  SMX_LAUNCH_CHECK("smx_integral");
  return SMX_OK;
}

extern "C" int smx_assemble_F(const smx_plan* pl, const int64_t* sum_zeta, const double* fu, const int64_t* umap,
                              const double* center, double* F64, float* F32, void* stream) {
  SMX_REQUIRE(pl != nullptr, "smx_assemble_F: null plan");
  const int64_t total = pl->n_entries * int64_t(pl->d_out);
  if (total == 0) return SMX_OK;
  SMX_REQUIRE(sum_zeta && fu && umap && F64 && pl->sum_eoff, "smx_assemble_F: null pointer");
  assemble_kernel<<<smx::grid_for(total, 256), 256, 0, smx::as_stream(stream)>>>(
      pl->n_summands, pl->sum_eoff, sum_zeta, fu, umap, center, pl->d_out, pl->n_entries, F64, F32);
  SMX_LAUNCH_CHECK("smx_assemble_F");
  return SMX_OK;
}
