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

// An index as one strided run or two (MatView); x < 2^31 as far as a split is used
struct DRun {
  int64_t hi, lo;
  uint32_t split;
  __host__ __device__ __forceinline__ int64_t off(int64_t x) const {
    if (!split) return x * hi;
    const uint32_t q = (uint32_t)x / split;
    return (int64_t)q * hi + (int64_t)((uint32_t)x - q * split) * lo;
  }
  __host__ __device__ __forceinline__ int64_t step() const { return split ? lo : hi; }
};
// Operand: rows (m, or n) x K.  The index arithmetic of two runs costs nothing beside the
// FMAs, and reading an operand in place saves the launch that would gather it.
struct DView {
  const double* p;
  DRun r, k;
  bool kfast;  // neighbouring threads load neighbouring k
};

// WM x WN warps, PM x PN patches of 8 x 4 outputs per warp, K in steps of BK through two
// shared-memory stages filled by cp.async
template <int WM_, int WN_, int PM_, int PN_, int BK_>
struct DTile {
  static constexpr int WM = WM_, WN = WN_, PM = PM_, PN = PN_, BK = BK_;
  static constexpr int BM = 8 * WM * PM, BN = 4 * WN * PN, THREADS = 32 * WM * WN;
  // odd row strides: a k-fast operand's column of a stage falls into different banks
  static constexpr int LDA = BM + 1, LDB = BN + 1, STAGE = BK * (LDA + LDB);
  static constexpr int SMEM = 2 * STAGE;  // doubles

  // one stage: A rows m0.. (mrem of them), B rows n0.. (nrem), K from k0 (krem steps)
  static __device__ __forceinline__ void load(double* st, const DView& A, int64_t m0, int mrem, const DView& B,
                                              int64_t n0, int nrem, int64_t k0, int krem) {
    double* As = st;
    double* Bs = st + BK * LDA;
#pragma unroll
    for (int e = threadIdx.x; e < BM * BK; e += THREADS) {
      const int mm = A.kfast ? e / BK : e % BM, kk = A.kfast ? e % BK : e / BM;
      const bool ok = mm < mrem && kk < krem;
      cp_async8(As + kk * LDA + mm, ok ? A.p + A.r.off(m0 + mm) + A.k.off(k0 + kk) : A.p, ok);
    }
#pragma unroll
    for (int e = threadIdx.x; e < BN * BK; e += THREADS) {
      const int nn = B.kfast ? e / BK : e % BN, kk = B.kfast ? e % BK : e / BN;
      const bool ok = nn < nrem && kk < krem;
      cp_async8(Bs + kk * LDB + nn, ok ? B.p + B.r.off(n0 + nn) + B.k.off(k0 + kk) : B.p, ok);
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

  // acc = the tile at (m0, n0) of an M x N product, K from k0 over kn steps in ascending order
  static __device__ __forceinline__ void product(double* smem, const DView& A, const DView& B, int64_t M, int64_t N,
                                                 int64_t m0, int64_t n0, int64_t k0, int64_t K,
                                                 double (&acc)[PM][PN]) {
    const int warp = threadIdx.x / 32;
    const int mrem = (int)(M - m0 < BM ? M - m0 : BM), nrem = (int)(N - n0 < BN ? N - n0 : BN);
    // patch row i of the warp covers rows 8 (warp / WN + WM i) ..: the count inside the matrix
    const int pr = (mrem + 7) / 8 - warp / WN, pc = (nrem + 3) / 4 - warp % WN;
    const int pm = pr > 0 ? (pr + WM - 1) / WM : 0, pn = pc > 0 ? (pc + WN - 1) / WN : 0;
#pragma unroll
    for (int i = 0; i < PM; i++)
#pragma unroll
      for (int j = 0; j < PN; j++) acc[i][j] = 0.0;
    if (K <= 0) return;
    load(smem, A, m0, mrem, B, n0, nrem, k0, (int)(K < BK ? K : BK));
    int buf = 0;
    for (int64_t kd = 0; kd < K; kd += BK) {
      const int64_t kx = kd + BK;
      if (kx < K) {
        load(smem + (buf ^ 1) * STAGE, A, m0, mrem, B, n0, nrem, k0 + kx, (int)(K - kx < BK ? K - kx : BK));
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      const int kn = (int)(K - kd < BK ? K - kd : BK);
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
  const int64_t mo = ep.msplit ? (m / ep.msplit) * ep.s_mhi + (m % ep.msplit) * ep.s_mlo : m * ep.s_mhi;
  return mo + (ep.nsplit ? (n / ep.nsplit) * ep.s_n + (n % ep.nsplit) * ep.s_nlo : n * ep.s_n);
}

__device__ __forceinline__ unsigned long long dgemm_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Device time of a short GEMM, measured by its own CTAs: the first one to start sets `start`,
// the last one to end adds the difference to `total` and clears the others.  A pair of CUDA
// events costs the stream 4.5 us, more than the median FP64 GEMM of a small solve takes.
__device__ __forceinline__ void dgemm_clock_start(Ctx::DeviceWords* w) {
  if (w && threadIdx.x == 0) atomicCAS(&w->start, 0ull, dgemm_ns());
}
__device__ __forceinline__ void dgemm_clock_stop(Ctx::DeviceWords* w, unsigned int ctas) {
  if (w && threadIdx.x == 0 && atomicAdd(&w->done, 1u) == ctas - 1) {
    const unsigned long long t0 = *(volatile unsigned long long*)&w->start, t1 = dgemm_ns();
    w->total += t1 > t0 ? t1 - t0 : 0ull;
    w->start = 0ull;
    w->done = 0u;
  }
}

// K over zc CTAs of a cluster times zg clusters; the clusters' partial tiles go to part
// [zg][BM * BN] and ticket[rank] counts those that have arrived
struct DSplit {
  int zc, zg, rank, zi;
  int64_t kchunk;
  double* part;
  unsigned int* ticket;
};

// One CTA's share of C = alpha A B + beta C, the tile at (m0, n0).  CLUSTER: the zc CTAs of a
// cluster hold shares of the same tile's K, and their partial tiles are added through
// distributed shared memory in rank order; with zg > 1 the last cluster to finish adds the
// clusters' sums in their order.  So a split needs no second launch.
template <class T, bool CLUSTER>
__device__ __forceinline__ void dgemm_cta(double* smem, const DSplit& z, const DView& A, const DView& B, int64_t M,
                                          int64_t N, int64_t K, int64_t m0, int64_t n0, double alpha, double beta,
                                          double* C, const GemmEpilogue& epi) {
  const int64_t k0 = ((int64_t)z.zi * z.zc + z.rank) * z.kchunk;
  const int64_t kn = k0 < K ? (K - k0 < z.kchunk ? K - k0 : z.kchunk) : 0;
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
  T::product(smem, A, B, M, N, m0, n0, k0, kn, acc);
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
  const bool mfast = epi.s_n != 1 && !epi.msplit && !epi.nsplit && epi.s_mhi == 1;
#pragma unroll
  for (int i = 0; i < T::PM; i++)
#pragma unroll
    for (int j = 0; j < T::PN; j++)
      smem[mfast ? T::col(j) * T::BM + T::row(i) : T::row(i) * T::BN + T::col(j)] = acc[i][j];
  dgemm_cluster_barrier();
  constexpr int kTile = T::BM * T::BN;
  const int e0 = z.rank * T::THREADS + (int)threadIdx.x, step = z.zc * T::THREADS;  // this CTA's elements
  auto store = [&](int e, double s) {
    const int64_t m = m0 + (mfast ? e % T::BM : e / T::BN), n = n0 + (mfast ? e / T::BM : e % T::BN);
    if (m >= M || n >= N) return;
    double* cp = C + dgemm_c_offset(epi, m, n);
    const double v = alpha * s;
    *cp = beta == 0.0 ? v : fma(beta, *cp, v);
  };
  for (int e = e0; e < kTile; e += step) {
    double s = 0.0;
    for (int q = 0; q < z.zc; q++) s += ld_cluster(smem + e, (uint32_t)q);
    if (z.zg > 1)
      z.part[(int64_t)z.zi * kTile + e] = s;
    else
      store(e, s);
  }
  dgemm_cluster_barrier();  // no CTA leaves while another still reads its partial tile
  if (z.zg > 1) {
    __shared__ unsigned int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&z.ticket[z.rank], 1u) == (unsigned)z.zg - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int e = e0; e < kTile; e += step) {
      double s = 0.0;
#pragma unroll 8
      for (int q = 0; q < z.zg; q++) s += __ldcg(z.part + (int64_t)q * kTile + e);
      store(e, s);
    }
    if (threadIdx.x == 0) z.ticket[z.rank] = 0u;
  }
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
DView dgemm_operand(const MatView& v);

}  // namespace ucc
