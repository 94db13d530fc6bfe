// Inline-PTX helpers of the sm_103a tensor-core kernels (gemm_tc.cu,
// blocked_tc.cu): mbarriers with bounded waits, TMA copies, tcgen05 MMA
// descriptors and issue.  Every wait takes a time limit (%globaltimer) and an
// optional abort flag, so that no kernel spins without bound.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <stdint.h>

namespace smx {
namespace tc {

constexpr uint64_t kWaitNs = 2000000000ull;  // default bound on one wait: 2 s

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Non-blocking test of the phase with the given parity.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded parity wait; false on timeout (after `limit_ns`) or when the abort
// flag is raised.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const volatile int* abort_flag,
                                          uint64_t limit_ns = kWaitNs) {
  const uint32_t a = smem_u32(bar);
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0;; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (abort_flag && *abort_flag) return false;
    if ((it & 255) == 255 && global_ns() - t0 > limit_ns) return false;
  }
}

// Copies go round `stages` buffers, copy c into buffer c % stages in the phase of
// parity (c / stages) & 1.  Calls wait(buffer, parity) for every copy that may be in
// flight after `issued` of them: the last into each buffer (a buffer is filled again
// only once its copy has been read).
template <typename Wait>
__host__ __device__ __forceinline__ void for_pending_copies(int issued, int stages, Wait wait) {
  for (int c = issued > stages ? issued - stages : 0; c < issued; ++c) wait(c % stages, (c / stages) & 1);
}

// 2-D tiled TMA load into shared memory, completion counted on `bar`.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* tm, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

// Contiguous bulk copy global -> shared (16-byte aligned addresses, size a
// multiple of 16), completion counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Shared-memory matrix descriptor of a K-major operand with swizzle span
// `row_bytes` (128, 64 or 32 bytes per row of the swizzle atom; the 8-row
// groups are 8 * row_bytes apart).  tcgen05 descriptor: start address >> 4,
// leading byte offset (unused for swizzled K-major), stride byte offset >> 4,
// version 1 (bit 46), layout type in bits 61-63 (2 = 128-byte swizzle,
// 4 = 64-byte, 6 = 32-byte).
__device__ __forceinline__ uint64_t make_desc_sw(uint32_t saddr, int row_bytes) {
  uint64_t d = 0;
  d |= uint64_t((saddr & 0x3FFFF) >> 4);
  d |= uint64_t(1) << 16;
  d |= uint64_t((8 * row_bytes) >> 4) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(row_bytes == 128 ? 2 : row_bytes == 64 ? 4 : 6) << 61;
  return d;
}

// Instruction descriptor: D = F32, A = B = TF32 (kind::tf32, format 2), BF16
// (kind::f16, format 1) or FP16 (kind::f16, format 0), both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_fmt(int M, int N, uint32_t fmt) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}
__host__ __device__ constexpr uint32_t idesc_mma(int M, int N, bool bf16) { return idesc_fmt(M, N, bf16 ? 1u : 2u); }

template <bool BF16>
__device__ __forceinline__ void mma_op(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  if constexpr (BF16) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
  }
}

// Pairs of FP16 values x = hi + 2^-kPairShift lo: the low part is stored scaled up, so
// that it keeps its 11 bits down to hi's smallest normal number.  With the group's
// largest value in [2^14, 2^15) an element has 22 significant bits down to 2^-29 of
// the largest and errs by 2^-51 of it below (16 bits less range without the shift).
// The products of a high and a low part are added first; the first product of high
// parts then scales the accumulator down by 2^-kPairShift (mma_pair_head).
constexpr int kPairShift = 11;
constexpr float kPairScale = float(1 << kPairShift);

// kind::f16 MMA that multiplies the accumulator by 2^-kPairShift before it adds.
__device__ __forceinline__ void mma_pair_head(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.eq.b32 p, 0, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, %4;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "n"(kPairShift));
}

// One 64-column slice of (Ah + Al)(Bh + Bl) into a fresh accumulator, rows of 128 bytes.
__device__ __forceinline__ void mma_pair_slice(uint32_t tmem_d, uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl,
                                               uint32_t idesc) {
#pragma unroll
  for (int k = 0; k < 128; k += 32) {  // 16 values per MMA
    mma_op<true>(tmem_d, make_desc_sw(ah + k, 128), make_desc_sw(bl + k, 128), idesc, k ? 1u : 0u);
    mma_op<true>(tmem_d, make_desc_sw(al + k, 128), make_desc_sw(bh + k, 128), idesc, 1u);
  }
#pragma unroll
  for (int k = 0; k < 128; k += 32) {
    const uint64_t da = make_desc_sw(ah + k, 128), db = make_desc_sw(bh + k, 128);
    if (k == 0)
      mma_pair_head(tmem_d, da, db, idesc);
    else
      mma_op<true>(tmem_d, da, db, idesc, 1u);
  }
}

// Arrives on `bar` once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// Host: the driver's cuTensorMapEncodeTiled, looked up once (gemm_tc.cu);
// returns SMX_OK or an error code with a message.
int tensor_map_encoder(PFN_cuTensorMapEncodeTiled_v12000* fn);

}  // namespace tc
}  // namespace smx
