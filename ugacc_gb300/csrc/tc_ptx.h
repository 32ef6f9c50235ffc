// PTX building blocks of the tcgen05 / TMA / mbarrier kernels (sm_103a): shared by the
// tensor-core GEMMs (tc_gemm.cu) and the fused guess-network kernel (mlp.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdint>

namespace ucc {
namespace tc {

constexpr unsigned long long WAIT_NS = 2000000000ull;  // 2 s per bounded wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait; false if the deadline passed or another warp raised the error flag.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, int* err,
                                          unsigned long long limit_ns = WAIT_NS) {
  if (mbar_test(b, parity)) return true;
  const unsigned long long t0 = gtimer();
  for (uint32_t it = 1;; ++it) {
    if (mbar_test(b, parity)) return true;
    if ((it & 255u) == 0) {
      if (*(volatile int*)err) return false;
      if (gtimer() - t0 > limit_ns) {
        atomicExch(err, 1);
        return false;
      }
    }
  }
}
// Bounded wait that ignores the error flag (used to drain in-flight copies).
__device__ __forceinline__ void mbar_wait_deadline(uint64_t* b, uint32_t parity) {
  const unsigned long long t0 = gtimer();
  while (!mbar_test(b, parity))
    if (gtimer() - t0 > WAIT_NS) return;
}
__device__ __forceinline__ void tma_load(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
// the same by a CTA of a pair (cta_group::2): the bytes land in this CTA's shared memory, the
// completion on a barrier of either CTA of the pair (bar: a shared::cluster address, map_rank)
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// shared::cluster address of this shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// every thread of every CTA of the cluster
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared-memory matrix descriptor: K-major, 128B swizzle, 8-row core groups 1024 B apart
__device__ __forceinline__ uint64_t sdesc(const void* p) {
  const uint64_t a = smem_u32(p);
  return ((a & 0x3FFFFull) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
template <int CG = 1>  // CTAs that work on one MMA (cta_group)
__device__ __forceinline__ void mma_i(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if (CG == 1)
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
  else
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
// arrive on the barrier at this offset (in both CTAs of the pair) once this thread's MMAs complete
template <int CG = 1>
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  if (CG == 1)
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
  else
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
}
// all TMEM columns `cols` of this CTA (of both CTAs of a pair), one warp
template <int CG>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  if (CG == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t cols) {
  if (CG == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
  else
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}
// shared-memory stores of ordinary instructions made visible to the tensor core (async proxy)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// FP32 -> FP64 by moving the bit fields (integer pipe, GB300 has few FP64 units)
__device__ __forceinline__ double f32_bits_to_f64(uint32_t fb) {
  const uint32_t e = (fb >> 23) & 0xFFu, m = fb & 0x7FFFFFu, sgn = fb & 0x80000000u;
  uint32_t ex = e + 896u, mt = m;
  if (e - 1u >= 0xFEu) {  // zero, subnormal, infinite, NaN
    if (e) {
      ex = 0x7FFu;
    } else if (m) {
      const int s = __clz(m) - 8;
      ex = 897u - s;
      mt = (m << s) & 0x7FFFFFu;
    } else {
      ex = 0u;
    }
  }
  return __hiloint2double((int)(sgn | (ex << 20) | (mt >> 3)), (int)(mt << 29));
}

// 32 bytes of a lane, a whole sector, in one access (p: a multiple of 32 bytes)
__device__ __forceinline__ void st_global4(double* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}
__device__ __forceinline__ void ld_global4(const double* p, double* v) {
  asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p) : "memory");
}

// FP64 -> FP32 truncated toward zero by moving the bit fields (relative error below 2^-23,
// integer pipe); zeros keep their sign
__device__ __forceinline__ float f64_to_f32_trunc(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const uint32_t sgn = (uint32_t)(b >> 32) & 0x80000000u;
  const int e = (int)((b >> 52) & 0x7FF) - 1023;
  if (e >= -126 && e <= 127) return __uint_as_float(sgn | ((uint32_t)(e + 127) << 23) | (uint32_t)((b >> 29) & 0x7FFFFFu));
  // beyond FP32's normal range as the conversion instruction rounds, without it: a compiler that
  // evaluates both sides of this branch puts one FP64-pipe conversion on every element
  if (e > 127) return __uint_as_float(sgn | (e == 1024 && (b << 12) ? 0x7FFFFFFFu : 0x7F800000u));
  const int sh = -126 - e + 29;  // >= 30; the FP64 subnormals (e = -1023) come out as zero
  if (sh > 54) return __uint_as_float(sgn);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52), half = 1ull << (sh - 1);
  const unsigned long long q = m >> sh, rem = m & (2 * half - 1);
  return __uint_as_float(sgn | (uint32_t)(q + (rem > half || (rem == half && (q & 1)))));
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {  // tmem_wait before use
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}


}  // namespace tc
}  // namespace ucc
