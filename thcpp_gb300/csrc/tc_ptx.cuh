// Inline PTX shared by the tcgen05 GEMM kernels: mbarriers, TMA loads, UMMA descriptors,
// tcgen05.mma / commit, TMEM loads, and the host's tensor-map encoder.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>

namespace thc {
namespace {

constexpr int TBM = 128;                       // rows of a CTA tile (UMMA M)
constexpr long long kDrainLimit = 1LL << 22;   // teardown waits after an abort

__device__ __forceinline__ uint32_t su32(const void* p)
{
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(su32(b)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(su32(b)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* b)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(su32(b)) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity)
{
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(su32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: false (and *abort set) when the barrier phase does not complete within
// `limit` polls (the context option "spin_limit"; 0 gives up at once).
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort,
                                          long long limit)
{
  for (long long i = 0; i < limit; i++) {
    if (mbar_try(b, parity)) return true;
    if (*abort) return false;
  }
  *abort = 1;
  return false;
}

// Teardown wait after an abort: polls a phase a bounded number of times, whatever *abort.
__device__ __forceinline__ void mbar_drain(uint64_t* b, uint32_t parity)
{
  for (long long i = 0; i < kDrainLimit; i++)
    if (mbar_try(b, parity)) return;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar)
{
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          su32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(su32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            uint64_t* bar)
{
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
          su32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(su32(bar))
      : "memory");
}

// UMMA shared-memory descriptor, K-major with the rows of one tile BK bf16 (2 BK bytes)
// long: BK = 32 uses the 64-byte swizzle (8-row groups 512 B apart), BK = 16 the 32-byte
// swizzle (groups 256 B apart).
template <int BK>
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr)
{
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;                       // leading byte offset (unused when swizzled)
  d |= (uint64_t)((8 * 2 * BK) >> 4) << 32;     // stride byte offset: one 8-row group
  d |= (uint64_t)1 << 46;                       // descriptor version
  d |= (uint64_t)(BK == 32 ? 4 : 6) << 61;      // layout: 64- or 32-byte swizzle
  return d;
}

// kind::f16 instruction descriptor: D f32, A/B bf16, both K-major, M = 128, N = BN.
template <int BN>
__host__ __device__ constexpr uint32_t idesc()
{
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
         ((uint32_t)(TBM >> 4) << 24);
}

template <int BN>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t acc)
{
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc<BN>()), "r"(acc));
}

// The low word of a descriptor (its address and leading byte offset), and an MMA from the low
// words: the high word is a constant of the layout.
__device__ __forceinline__ uint32_t sdesc_lo(uint32_t saddr)
{
  return ((saddr & 0x3FFFF) >> 4) | (1u << 16);
}

template <int BN, int BK>
__device__ __forceinline__ void umma_lo(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t acc)
{
  constexpr uint32_t hi = (uint32_t)((8 * 2 * BK) >> 4) | (1u << 14) |
                          ((uint32_t)(BK == 32 ? 4 : 6) << 29);
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %4, 0;\n"
      " mov.b64 da, {%1, %5};\n mov.b64 db, {%2, %5};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(a), "r"(b), "r"(idesc<BN>()), "r"(acc), "r"(hi));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                   su32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v)
{
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

// Eight columns at each of two addresses, in flight together.
__device__ __forceinline__ void tmem_ld8x2(uint32_t ta, uint32_t tb, float (&a)[8], float (&b)[8])
{
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]),
        "=f"(a[7]), "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]), "=f"(b[4]), "=f"(b[5]),
        "=f"(b[6]), "=f"(b[7])
      : "r"(ta), "r"(tb)
      : "memory");
}

inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    // The entry point with the ABI of CUDA 12.0, which the PFN type above describes.
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}

}  // namespace
}  // namespace thc
