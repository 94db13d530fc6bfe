// Stream evaluator of the orthogonal form: y[p][o] = c0[o] + sum over items of
// v_item(p) * sum over the item's terms of coefficient[o] * row value(p).
//
// One block of 16 warps evaluates a tile of 32 NP points (NP per lane).  The
// tile's rows -- hot basis values, the constant 1, the products of the prefixes
// that cold entries extend -- sit in shared memory as [row][point]; every entry
// of Lambda is one term (row, DO coefficients) of an item, whose factor v is the
// product of at most 8 rows (a hot node) or phi_g(z_j) of a cold dimension.  The
// items are dealt to 16 fixed lists, one per warp, balanced when the tables are
// built; the terms of a list are one contiguous stream of 16-term chunks: 16
// byte offsets of rows (bit 0: last term of its item), then the coefficients.  The warp copies the next chunks into its own ring in
// shared memory (cp.async) while it works on the current one, the next item's
// descriptor and x coordinate are loaded one item ahead, so that no step of
// the sum waits for a global load.  FP32 items are padded to whole groups of 4
// terms, so that the multiply-adds of a group have no branch between them; FP64
// items are not (every term costs).
//
// Why this form.  FP64 (NP = 1): 2 multiply-adds per SM clock are the bound; the
// walk over node, run and term tables it replaces spent half its time on
// chains of dependent loads.  Leja d_in = 1000, |Lambda| = 9999, 20011 points:
// 999 -> 457 us (318 us of multiply-adds, one per entry; the FP64 pipe is 92 %
// busy).  FP32 with 2..15 outputs (NP = 4 with DO = 4, 3 with 8): one row read
// and DO / 4 broadcast coefficient reads feed NP DO multiply-adds per lane, which
// balances the FP32 pipes and the load/store unit.  Gauss-Hermite d_in = 100,
// d_out = 8, |Lambda| = 20010, 50001 points: 6.87 -> 0.61 ms (0.20 ms of
// multiply-adds); 4 points of 8 outputs per lane spilled and took 0.66 ms, 2
// points 0.63 ms.  Each FP32 item's sum is at most 32 terms of plain FP32; items
// are added with compensation.
#pragma once

#include <stdint.h>

#include <type_traits>

#include "common.cuh"

namespace smx {
namespace stream {

constexpr int kLists = 16;  // item lists of a plan, one per warp
constexpr int kThreads = 32 * kLists;
constexpr int kTerms = 16;  // per chunk

// Points per lane: FP64 1; FP32 4, or 3 for 8 outputs (the sums and their
// compensations are 3 registers per point and output: 4 points of 8 outputs
// spill 1.4 loads per term).
template <typename T>
inline __host__ __device__ constexpr int lane_points(int DO) {
  return sizeof(T) == 8 ? 1 : DO == 8 ? 3 : 4;
}
constexpr int kColdItem = 1 << 8, kPlain = 1 << 11;

template <typename T>
constexpr int chunk_bytes(int DO) {
  return 4 * kTerms + kTerms * DO * int(sizeof(T));
}

// Shared memory: rows (at least the reduction's area), then the rings.
template <typename T>
inline __host__ __device__ size_t rows_bytes(int n_rows, int points) {
  const size_t rows = size_t(n_rows) * points * sizeof(T);
  const size_t red = size_t(kLists) * points * 8;
  return ((rows > red ? rows : red) + 15) / 16 * 16;
}

template <typename T>
inline size_t smem_bytes(const smx_stream& s) {
  return rows_bytes<T>(s.n_rows, 32 * lane_points<T>(s.pass)) + size_t(kLists) * 2 * chunk_bytes<T>(s.pass);
}

__device__ __forceinline__ void kahan(float& sum, float& comp, float v) {
  const float y = v - comp;
  const float t = sum + y;
  comp = (t - sum) - y;
  sum = t;
}

__device__ __forceinline__ void copy_chunk(unsigned char* dst, const unsigned char* src, int bytes, int lane) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  for (int i = lane * 16; i < bytes; i += 512)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + i), "l"(src + i) : "memory");
}

// Point of the tile that lane `lane` holds in place i: adjacent points for one
// vector load, or (3 per lane) 32 apart.
template <int NP>
__device__ __forceinline__ int lane_point(int lane, int i) {
  return NP == 3 ? lane + 32 * i : NP * lane + i;
}

// The row values of this lane's points; `at` is the row's address plus the lane's offset.
template <int NP, typename T>
__device__ __forceinline__ void load_row(const unsigned char* at, T (&v)[NP]) {
  if constexpr (NP == 2) {
    const float2 t = *reinterpret_cast<const float2*>(at);
    v[0] = t.x, v[1] = t.y;
  } else if constexpr (NP == 4) {
    const float4 t = *reinterpret_cast<const float4*>(at);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else {
#pragma unroll
    for (int i = 0; i < NP; ++i) v[i] = reinterpret_cast<const T*>(at)[32 * i];
  }
}

// Thread-block clusters: a tile's warp lists may be spread over the blocks of a
// cluster, which add their sums through the first block's shared memory.
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void sync_blocks(int parts) {
  if (parts > 1)
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
  else
    __syncthreads();
}
// Address of the first block's copy of a shared-memory location.
__device__ __forceinline__ uint32_t first_block(const void* p, int parts) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  if (parts > 1) asm volatile("mapa.shared::cluster.u32 %0, %0, 0;" : "+r"(a));
  return a;
}

// Rec: static alpha(family, n), beta(family, n) of the recurrence in T, and
// convert(double): the coordinate in T with infinities as NaN.  The blocks of a
// cluster of `parts` (1, 2, 4 or 8) share the tile: block `part` sums the lists
// part * 16 / parts ..; the value of a point is the same for every split.
template <typename T, int DO, typename Rec>
__device__ __forceinline__ void stream_tile(const smx_stream& a, int d_out, const T* __restrict__ c0,
                                            const double* __restrict__ x, int64_t P, int64_t ldx, T* __restrict__ y,
                                            int pass, int64_t tile, unsigned char* sm, int part = 0, int parts = 1) {
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int NP = lane_points<T>(DO);
  constexpr int kPts = 32 * NP;
  constexpr int CB = chunk_bytes<T>(DO);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* R = reinterpret_cast<T*>(sm);
  unsigned char* ring = sm + rows_bytes<T>(a.n_rows, kPts) + warp * (2 * CB);
  const int64_t p0 = tile * kPts;

  // this block's lists; their streams start before the rows are built
  const int n_lists = kLists / parts, list = part * n_lists + warp;
  const bool works = warp < n_lists;
  const int ch0 = works ? __ldg(a.warp + kLists + 1 + list) : 0;
  const int nch = works ? __ldg(a.warp + kLists + 2 + list) - ch0 : 0;
  const unsigned char* src = reinterpret_cast<const unsigned char*>(a.chunk) + (int64_t(pass) * a.n_chunks + ch0) * CB;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (c < nch) copy_chunk(ring + c * CB, src + int64_t(c) * CB, CB, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // basis values of the hot dimensions
  for (int i = threadIdx.x; i < a.n_hot * kPts; i += kThreads) {
    const int h = i / kPts, q = i % kPts;
    const int4 d4 = __ldg(reinterpret_cast<const int4*>(a.hot) + 2 * h);  // dimension, degree, first row, family
    const double2 ab = __ldg(reinterpret_cast<const double2*>(a.hot) + 2 * h + 1);
    const T xv = Rec::convert(__ldg(x + min(p0 + q, P - 1) * ldx + d4.x));
    const T z = fma(T(ab.x), xv, T(ab.y));
    T pm1 = T(0), pc = T(1);
    for (int n = 0; n < d4.y; ++n) {
      const T pn = fma(Rec::alpha(d4.w, n) * z, pc, -Rec::beta(d4.w, n) * pm1);
      pm1 = pc;
      pc = pn;
      R[(d4.z + n) * kPts + q] = pc;
    }
  }
  __syncthreads();
  // the constant 1 and the prefix products
  for (int i = threadIdx.x; i < a.n_vp * kPts; i += kThreads) {
    const int r = i / kPts, q = i % kPts;
    const int4 s4 = __ldg(reinterpret_cast<const int4*>(a.vp) + r);  // 8 uint16 rows, 0xffff past the last
    const unsigned w[4] = {unsigned(s4.x), unsigned(s4.y), unsigned(s4.z), unsigned(s4.w)};
    T v = T(1);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const unsigned s = (w[k >> 1] >> (16 * (k & 1))) & 0xffffu;
      if (s == 0xffffu) break;
      v = k == 0 ? R[s * kPts + q] : v * R[s * kPts + q];
    }
    R[(a.n_hb + r) * kPts + q] = v;
  }
  __syncthreads();

  T ys[NP][DO], yc[F32 ? NP : 1][F32 ? DO : 1], s[NP][DO];
#pragma unroll
  for (int i = 0; i < NP; ++i)
#pragma unroll
    for (int o = 0; o < DO; ++o) {
      ys[i][o] = T(0);
      if constexpr (F32) yc[i][o] = T(0);
    }

  // items of this warp.  FP64: the descriptors of the current and the next item
  // and the current coordinates are loaded ahead into registers.  FP32 has none
  // to spare: the descriptor and the coordinates are read when the item ends,
  // from L1, where the coordinates are prefetched as the item begins.
  const int4* desc = reinterpret_cast<const int4*>(a.desc) + 2 * (works ? __ldg(a.warp + list) : 0);
  int left = works ? __ldg(a.warp + list + 1) - __ldg(a.warp + list) : 0;
  int open = left;  // items not yet finished
  int4 da = make_int4(0, 0, 0, 0), db = da, na = da, nb = da;
  double xn = 0.0;
  const double* xt = x + p0 * ldx;
  const int last = int(min(P - p0, int64_t(kPts))) - 1;
  auto xat = [&](int i, int dim) { return xt + int64_t(min(lane_point<NP>(lane, i), last)) * ldx + dim; };
  auto fetch = [&]() {
    if constexpr (F32) {
      if (left > 0) {
        const int2 d2 = __ldg(reinterpret_cast<const int2*>(desc));
        if (d2.x & kColdItem) {
#pragma unroll
          for (int i = 0; i < NP; ++i) asm volatile("prefetch.global.L1 [%0];" ::"l"(xat(i, d2.y)));
        }
      }
    } else {
      da = na, db = nb;
      if (left > 0) na = __ldg(desc), nb = __ldg(desc + 1), desc += 2, --left;
      if (da.x & kColdItem) xn = __ldg(xat(0, da.y));
    }
  };
  fetch();
  if constexpr (!F32) fetch();

  // factor of points [I0, I0 + N) of the lane, and the item's sums added
  auto add_points = [&](auto first, auto count) {
    constexpr int I0 = decltype(first)::value, N = decltype(count)::value;
    T v[N];
    if (da.x & kColdItem) {
      const int g = da.x >> 16, fm = (da.x >> 9) & 1;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        T z = Rec::convert(F32 ? __ldg(xat(I0 + i, da.y)) : xn);
        v[i] = z;
        if (da.x & kPlain) continue;  // phi_1 = x: Legendre on [-1, 1], degree 1
        z = fma(T(__hiloint2double(db.y, db.x)), z, T(__hiloint2double(db.w, db.z)));
        T pm1 = T(1), pc = fm == 0 ? z : Rec::alpha(fm, 0) * z;
        for (int n = 1; n < g; ++n) {
          const T pn = fma(Rec::alpha(fm, n) * z, pc, -Rec::beta(fm, n) * pm1);
          pm1 = pc;
          pc = pn;
        }
        v[i] = pc;
      }
    } else {
      const int n = da.x & 0xff;
      const unsigned w[4] = {unsigned(db.x), unsigned(db.y), unsigned(db.z), unsigned(db.w)};
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = T(1);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k >= n) break;
        const T* f = R + int((w[k >> 1] >> (16 * (k & 1))) & 0xffffu) * kPts;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const T fv = f[lane_point<NP>(lane, I0 + i)];
          v[i] = k == 0 ? fv : v[i] * fv;
        }
      }
    }
    if constexpr (F32) {  // pairs of outputs; yc holds minus the compensation
      const float2 m1 = make_float2(-1.f, -1.f);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const int i = I0 + j;
        const float2 vv = make_float2(v[j], v[j]);
#pragma unroll
        for (int o = 0; o < DO; o += 2) {
          const float2 sum = make_float2(ys[i][o], ys[i][o + 1]), comp = make_float2(yc[i][o], yc[i][o + 1]);
          const float2 t = __fadd2_rn(__fmul2_rn(vv, make_float2(s[i][o], s[i][o + 1])), comp);
          const float2 n = __fadd2_rn(sum, t);
          const float2 c = __fadd2_rn(t, __ffma2_rn(n, m1, sum));
          ys[i][o] = n.x, ys[i][o + 1] = n.y, yc[i][o] = c.x, yc[i][o + 1] = c.y;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int o = 0; o < DO; ++o) ys[I0 + j][o] = fma(v[j], s[I0 + j][o], ys[I0 + j][o]);
    }
  };
  // the next item's sum starts at 0, or at the node's own coefficient
  auto start = [&]() {
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
      for (int o = 0; o < DO; ++o) s[i][o] = !F32 && DO == 1 ? T(__hiloint2double(da.w, da.z)) : T(0);
  };
  auto finish = [&]() {
    if constexpr (F32) {
      da = __ldg(desc), db = __ldg(desc + 1), desc += 2, --left;
      add_points(std::integral_constant<int, 0>{}, std::integral_constant<int, 2>{});
      if constexpr (NP > 2) add_points(std::integral_constant<int, 2>{}, std::integral_constant<int, NP - 2>{});
    } else {
      add_points(std::integral_constant<int, 0>{}, std::integral_constant<int, 1>{});
    }
    --open;
    fetch();
    start();
  };

  start();
  const unsigned char* rows = sm + lane_point<NP>(lane, 0) * sizeof(T);
  for (int c = 0; c < nch; ++c) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const unsigned char* buf = ring + (c & 1) * CB;
#pragma unroll 1
    for (int g = 0; g < kTerms / 4; ++g) {
      if (!F32 && open == 0) break;  // padding of the list's last chunk
      // byte offsets of the rows, bit 0: last term of its item
      const uint4 sl = *reinterpret_cast<const uint4*>(buf + 16 * g);
      const unsigned slot[4] = {sl.x, sl.y, sl.z, sl.w};
      const T* cf = reinterpret_cast<const T*>(buf + 4 * kTerms) + 4 * g * DO;
      T r[4][NP];
#pragma unroll
      for (int u = 0; u < 4; ++u) load_row<NP>(rows + (F32 && u < 3 ? slot[u] : slot[u] & ~1u), r[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if constexpr (F32) {
#pragma unroll
          for (int o = 0; o < DO; o += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(cf + u * DO + o);
            const float2 k01 = make_float2(k4.x, k4.y), k23 = make_float2(k4.z, k4.w);
#pragma unroll
            for (int i = 0; i < NP; ++i) {
              const float2 rr = make_float2(r[u][i], r[u][i]);
              const float2 t01 = __ffma2_rn(k01, rr, make_float2(s[i][o], s[i][o + 1]));
              const float2 t23 = __ffma2_rn(k23, rr, make_float2(s[i][o + 2], s[i][o + 3]));
              s[i][o] = t01.x, s[i][o + 1] = t01.y, s[i][o + 2] = t23.x, s[i][o + 3] = t23.y;
            }
          }
        } else {
#pragma unroll
          for (int o = 0; o < DO; ++o)
#pragma unroll
            for (int i = 0; i < NP; ++i) s[i][o] = fma(cf[u * DO + o], r[u][i], s[i][o]);
        }
        if constexpr (!F32)
          if (slot[u] & 1u) finish();
      }
      if constexpr (F32)  // items end with a group of 4 terms
        if (slot[3] & 1u) finish();
    }
    __syncwarp();
    if (c + 2 < nch) copy_chunk(ring + (c & 1) * CB, src + int64_t(c + 2) * CB, CB, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // the lists' sums per point, in a fixed order; as many outputs at a time as
  // fit where the rows were
  constexpr size_t kRed = size_t(kLists) * kPts * 8;
  const int at_once = int(min(size_t(DO), rows_bytes<T>(a.n_rows, kPts) / kRed));  // >= 1
  const uint32_t red = first_block(sm, parts);
  sync_blocks(parts);
  int held = 0;
#pragma unroll
  for (int o = 0; o < DO; ++o) {
    if (pass * DO + o < d_out) {  // block-uniform
      if (works) {
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          const uint32_t at = red + uint32_t(held * kRed) + (list * kPts + lane_point<NP>(lane, i)) * 8;
          if constexpr (F32)
            asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(at), "f"(ys[i][o]), "f"(yc[i][o])
                         : "memory");
          else
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(ys[i][o]) : "memory");
        }
      }
      ++held;
      if (held == at_once || o == DO - 1 || pass * DO + o == d_out - 1) {
        sync_blocks(parts);
        for (int t = threadIdx.x; part == 0 && t < held * kPts; t += kThreads) {
          const int h = t / kPts, q = t % kPts;
          if (p0 + q >= P) continue;
          const int col = pass * DO + o + 1 - held + h;
          const unsigned char* v = sm + h * kRed + q * 8;
          const T base = __ldg(c0 + col);
          T out;
          if constexpr (F32) {
            float sum = 0.f, comp = 0.f;
            for (int w = 0; w < kLists; ++w) {
              const float2 f = *reinterpret_cast<const float2*>(v + w * kPts * 8);
              kahan(sum, comp, f.x);
              kahan(sum, comp, f.y);
            }
            out = base + (sum - comp);
          } else {
            out = base;
            for (int w = 0; w < kLists; ++w) out += *reinterpret_cast<const T*>(v + w * kPts * 8);
          }
          y[(p0 + q) * d_out + col] = out;
        }
        sync_blocks(parts);
        held = 0;
      }
    }
  }
}

// Launch shape of `tiles` tiles x `passes`: the tiles that fill every SM equally
// often run one block each; the rest, or a small batch, run as clusters of up
// to 8 blocks a tile while SMs would stay idle otherwise.
// A second launch costs about kLaunchCycles (its own start and latencies), a tile
// about 256 cycles per chunk (measured at both precisions: 163 us for the 1344
// chunks of a FP32 tile, 100 us for the 633 of a FP64 one), so that a tail is
// split off only where that saves more: 20011 points of the d_in = 1000 plan
// 489 -> 470 us; 10000 points of a plan of 71 chunks 62 us either way.
struct Split {
  int64_t whole, rest;
  int parts;
};
constexpr int64_t kLaunchCycles = 30000;
inline Split split_tiles(int64_t tiles, int passes, int n_chunks, int sms) {
  Split s{tiles, 0, 1};
  const int64_t whole = tiles * passes / sms * sms / passes;
  int parts = 1;
  while (parts < 8 && (tiles - whole) * passes * parts * 2 <= sms) parts *= 2;
  if (parts == 1 || tiles == whole) return s;
  if (whole > 0 && int64_t(n_chunks) * 256 * (parts - 1) / parts < kLaunchCycles) return s;
  s.whole = whole, s.rest = tiles - whole, s.parts = parts;
  return s;
}

// Launches kernel(args..., first tile, parts) over all tiles.
template <typename... KA, typename... Args>
inline int launch(void (*kernel)(KA...), int threads, int64_t tiles, int passes, int n_chunks, size_t smem,
                  cudaStream_t st, const char* who,
                  Args... args) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return set_error(SMX_ERR_CUDA, std::string(who) + ": no device");
  const Split s = split_tiles(tiles, passes, n_chunks, sms);
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  if (s.whole > 0) {
    cfg.gridDim = dim3(unsigned(s.whole), unsigned(passes));
    cudaLaunchKernelEx(&cfg, kernel, args..., int64_t(0), 1);
  }
  if (s.rest > 0) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = unsigned(s.parts);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(s.rest * s.parts), unsigned(passes));
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args..., s.whole, s.parts);
  }
  return check_launch(who);
}

// Checks of the tables' sizes; SMX_OK or an error with a message.
template <typename T>
inline int check(const smx_stream& s, int d_out, const char* who) {
  const std::string w(who);
  if (s.pass != 1 && s.pass != 4 && s.pass != 8) return set_error(SMX_ERR_ARG, w + ": bad stream pass");
  if (s.row_bytes != 32 * lane_points<T>(s.pass) * int(sizeof(T)) || s.n_rows < 1 || s.n_rows > 0x7fff || s.n_hb < 0 || s.n_vp < 1 || s.n_hb + s.n_vp != s.n_rows || s.n_hot < 0 ||
      s.n_chunks < 0 || d_out < 1)
    return set_error(SMX_ERR_ARG, w + ": bad stream sizes");
  if (!s.warp || !s.vp || (s.n_hot && !s.hot) || (s.n_chunks && (!s.chunk || !s.desc)))
    return set_error(SMX_ERR_ARG, w + ": incomplete stream tables");
  return SMX_OK;
}

}  // namespace stream
}  // namespace smx
