// Tile of an FP64 (DFMA) product, shared by the single-problem GEMM (dgemm.cu) and the
// grouped GEMM of the batched solver (batch.cu).
//
// What bounds it: GB300 issues two FP64 FMAs per SM clock (1.2 TFLOP/s over 152 SMs), so a
// warp's FMA holds its quarter of the SM for 64 clocks while everything else in the loop
// (shared-memory reads, index arithmetic, cp.async) issues in its shadow.  The only thing
// that counts is how many warp FMAs an SM has to issue: multiply-adds spent on padding, and
// SMs left without work.  So a warp FMA covers an 8 x 4 patch of outputs (lane = 4 row +
// column), a tile is a grid of patches dealt round robin to the warps, and a patch that lies
// outside the matrix is skipped by the whole warp: an M x N output costs ceil(M/8) ceil(N/4)
// patches whatever the tile is.  Small tiles cost nothing here (16 x 16 reads 2 bytes of
// operands per clock and SM), so a launch takes the tile that spreads its patches most
// evenly (dgemm_plan).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "core.h"

namespace ucc {

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = valid ? 8 : 0;  // 0: the 8 bytes are filled with zeros, src is not read
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// WM x WN warps, PM x PN patches of 8 x 4 outputs per warp, K in steps of BK through two
// shared-memory stages filled by cp.async
template <int WM_, int WN_, int PM_, int PN_, int BK_>
struct DTile {
  static constexpr int WM = WM_, WN = WN_, PM = PM_, PN = PN_, BK = BK_;
  static constexpr int BM = 8 * WM * PM, BN = 4 * WN * PN, THREADS = 32 * WM * WN;
  // odd row strides: a k-fast operand's column of a stage falls into different banks
  static constexpr int LDA = BM + 1, LDB = BN + 1, STAGE = BK * (LDA + LDB);
  static constexpr int SMEM = 2 * STAGE;  // doubles

  // one stage: A(0..mrem, 0..krem) and B(0..krem, 0..nrem) relative to the given pointers
  static __device__ __forceinline__ void load(double* st, const double* A, int64_t sAm, int64_t sAk, int mrem,
                                              const double* B, int64_t sBk, int64_t sBn, int nrem, int krem,
                                              bool a_kfast, bool b_nfast) {
    double* As = st;
    double* Bs = st + BK * LDA;
#pragma unroll
    for (int e = threadIdx.x; e < BM * BK; e += THREADS) {
      const int mm = a_kfast ? e / BK : e % BM, kk = a_kfast ? e % BK : e / BM;
      const bool ok = mm < mrem && kk < krem;
      cp_async8(As + kk * LDA + mm, ok ? A + mm * sAm + kk * sAk : A, ok);
    }
#pragma unroll
    for (int e = threadIdx.x; e < BN * BK; e += THREADS) {
      const int nn = b_nfast ? e % BN : e / BK, kk = b_nfast ? e / BN : e % BK;
      const bool ok = nn < nrem && kk < krem;
      cp_async8(Bs + kk * LDB + nn, ok ? B + kk * sBk + nn * sBn : B, ok);
    }
    cp_async_commit();
  }

  // acc += the product of one stage's first kn steps; pm, pn: this warp's patch rows and
  // columns inside the matrix
  template <bool FULL>
  static __device__ __forceinline__ void fma_stage(const double* st, int kn, int pm, int pn, double (&acc)[PM][PN]) {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const double* as = st + (warp / WN) * 8 + lane / 4;
    const double* bs = st + BK * LDA + (warp % WN) * 4 + lane % 4;
#pragma unroll 4
    for (int kk = 0; kk < kn; kk++) {
      double a[PM], b[PN];
#pragma unroll
      for (int i = 0; i < PM; i++) a[i] = as[kk * LDA + i * WM * 8];
#pragma unroll
      for (int j = 0; j < PN; j++) b[j] = bs[kk * LDB + j * WN * 4];
#pragma unroll
      for (int i = 0; i < PM; i++)
#pragma unroll
        for (int j = 0; j < PN; j++)
          if (FULL || (i < pm && j < pn)) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
  }

  // acc = A(0..M, 0..K) B(0..K, 0..N) of this tile (M, N: rows and columns left from its
  // corner, A and B the corner's pointers, K steps in ascending order)
  static __device__ __forceinline__ void product(double* smem, const double* A, int64_t sAm, int64_t sAk,
                                                 const double* B, int64_t sBk, int64_t sBn, int64_t M, int64_t N,
                                                 int64_t K, double (&acc)[PM][PN]) {
    const int warp = threadIdx.x / 32;
    const int mrem = (int)(M < BM ? M : BM), nrem = (int)(N < BN ? N : BN);
    const bool a_kfast = sAk == 1 || (sAm != 1 && sAk < sAm), b_nfast = sBn == 1 || (sBk != 1 && sBn < sBk);
    // patch row i of the warp covers rows 8 (warp / WN + WM i) ..: the count inside the matrix
    const int pr = (mrem + 7) / 8 - warp / WN, pc = (nrem + 3) / 4 - warp % WN;
    const int pm = pr > 0 ? (pr + WM - 1) / WM : 0, pn = pc > 0 ? (pc + WN - 1) / WN : 0;
#pragma unroll
    for (int i = 0; i < PM; i++)
#pragma unroll
      for (int j = 0; j < PN; j++) acc[i][j] = 0.0;
    if (K <= 0) return;
    load(smem, A, sAm, sAk, mrem, B, sBk, sBn, nrem, (int)(K < BK ? K : BK), a_kfast, b_nfast);
    int buf = 0;
    for (int64_t k0 = 0; k0 < K; k0 += BK) {
      const int64_t k1 = k0 + BK;
      if (k1 < K) {
        load(smem + (buf ^ 1) * STAGE, A + k1 * sAk, sAm, sAk, mrem, B + k1 * sBk, sBk, sBn, nrem,
             (int)(K - k1 < BK ? K - k1 : BK), a_kfast, b_nfast);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      const int kn = (int)(K - k0 < BK ? K - k0 : BK);
      if (pm == PM && pn == PN)
        fma_stage<true>(smem + buf * STAGE, kn, pm, pn, acc);
      else if (pm > 0 && pn > 0)
        fma_stage<false>(smem + buf * STAGE, kn, pm, pn, acc);
      __syncthreads();
      buf ^= 1;
    }
  }

  // row / column of this thread's accumulator (i, j) inside the tile
  static __device__ __forceinline__ int row(int i) {
    return ((int)(threadIdx.x / 32) / WN + WM * i) * 8 + (int)(threadIdx.x % 32) / 4;
  }
  static __device__ __forceinline__ int col(int j) {
    return ((int)(threadIdx.x / 32) % WN + WN * j) * 4 + (int)(threadIdx.x % 4);
  }
};

// Four warps per tile (eight, or two interleaved sums per output, time the same within 3 %).
// 16 x 16 takes K in steps of 32: the whole K range of a small product in one or two loads;
// 32 x 32 is the faster one for short K and many tiles (a CTA's start and end count).  A
// 64 x 64 tile was never the fastest.  GEMM device time, events included, with the 64 x 64
// kernel of 256 threads and padded tiles that this replaced -> now: 95 x 95 x 95 96 -> 10.5 us,
// 9216 x 96 x 104 211 -> 162 us (floor 153), 96 x 96 x 6144 316 -> 109 us (floor 94),
// 768^3 -> 761 us (floor 753), 102400 x 160 x 16 616 -> 490 us on 32 x 32 (floor 436).
using DTile32 = DTile<2, 2, 2, 4, 16>;
using DTile16 = DTile<2, 2, 1, 2, 32>;

__device__ __forceinline__ uint32_t dgemm_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void dgemm_cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// element of CTA `rank`'s copy of this shared-memory address
__device__ __forceinline__ double ld_cluster(const double* p, uint32_t rank) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(r) : "memory");
  return v;
}

__device__ __forceinline__ int64_t dgemm_c_offset(const GemmEpilogue& ep, int64_t m, int64_t n) {
  return (ep.msplit ? (m / ep.msplit) * ep.s_mhi + (m % ep.msplit) * ep.s_mlo : m * ep.s_mhi) + n * ep.s_n;
}

// One CTA's share of C = alpha A B + beta C: the tile at (m0, n0), K from k0 over at most kchunk
// steps.  CLUSTER: the zc CTAs of a cluster hold the same tile's K shares, and their partial
// tiles are added through distributed shared memory in rank order, so a split costs no second
// launch and no trip through device memory.
template <class T, bool CLUSTER>
__device__ __forceinline__ void dgemm_cta(double* smem, int rank, int zc, int64_t M, int64_t N, int64_t K, int64_t m0,
                                          int64_t n0, int64_t k0, int64_t kchunk, const double* A, int64_t sAm,
                                          int64_t sAk, const double* B, int64_t sBk, int64_t sBn, double alpha,
                                          double beta, double* C, const GemmEpilogue& epi) {
  const int64_t kn = k0 < K ? (K - k0 < kchunk ? K - k0 : kchunk) : 0;
  double acc[T::PM][T::PN], old[T::PM][T::PN];
  if (!CLUSTER && beta != 0.0) {  // the old values travel while the product runs
#pragma unroll
    for (int i = 0; i < T::PM; i++)
#pragma unroll
      for (int j = 0; j < T::PN; j++) {
        const int64_t m = m0 + T::row(i), n = n0 + T::col(j);
        old[i][j] = m < M && n < N ? C[dgemm_c_offset(epi, m, n)] : 0.0;
      }
  }
  T::product(smem, A + m0 * sAm + k0 * sAk, sAm, sAk, B + k0 * sBk + n0 * sBn, sBk, sBn, M - m0, N - n0, kn, acc);
  if (!CLUSTER) {
#pragma unroll
    for (int i = 0; i < T::PM; i++)
#pragma unroll
      for (int j = 0; j < T::PN; j++) {
        const int64_t m = m0 + T::row(i), n = n0 + T::col(j);
        if (m < M && n < N) {
          const double v = alpha * acc[i][j];
          C[dgemm_c_offset(epi, m, n)] = beta == 0.0 ? v : fma(beta, old[i][j], v);
        }
      }
    return;
  }
  // product() ended with a barrier: its stages are free for the partial tile, [m][n] or
  // [n][m] so that consecutive elements are consecutive in C where one of its indices allows
  const bool mfast = epi.s_n != 1 && !epi.msplit && epi.s_mhi == 1;
#pragma unroll
  for (int i = 0; i < T::PM; i++)
#pragma unroll
    for (int j = 0; j < T::PN; j++)
      smem[mfast ? T::col(j) * T::BM + T::row(i) : T::row(i) * T::BN + T::col(j)] = acc[i][j];
  dgemm_cluster_barrier();
  for (int e = rank * T::THREADS + (int)threadIdx.x; e < T::BM * T::BN; e += zc * T::THREADS) {
    const int64_t m = m0 + (mfast ? e % T::BM : e / T::BN), n = n0 + (mfast ? e / T::BM : e % T::BN);
    if (m >= M || n >= N) continue;
    double* cp = C + dgemm_c_offset(epi, m, n);
    const double o = beta != 0.0 ? *cp : 0.0;
    double s = 0.0;
    for (int q = 0; q < zc; q++) s += ld_cluster(smem + e, (uint32_t)q);
    const double v = alpha * s;
    *cp = beta == 0.0 ? v : fma(beta, o, v);
  }
  dgemm_cluster_barrier();  // no CTA leaves while another still reads its partial tile
}

// `count` products of one shape in a launch
struct GemmShape {
  int64_t M, N, K;
  int count;
};
struct DgemmPlan {
  int shape;   // 0: DTile16, 1: DTile32
  int zc, zg;  // K over the zc CTAs of a cluster, times zg partial products in device memory
};
DgemmPlan dgemm_plan(const std::vector<GemmShape>& probs, bool may_split);

}  // namespace ucc
