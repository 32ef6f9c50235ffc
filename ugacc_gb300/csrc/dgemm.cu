// FP64 (DFMA) GEMM over arbitrarily strided operands with a permuting epilogue, so that a
// contraction result lands directly in its tensor layout (no separate transpose pass).
#include <algorithm>
#include <atomic>
#include <memory>

#include "core.h"
#include "dgemm_tile.h"

namespace ucc {

void count_kernel_launch();  // kernels_fp64.cu
void splitk_reduce(Ctx& c, int64_t M, int64_t N, int nsplit, const double* P, double alpha, double beta, double* C,
                   const GemmEpilogue& epi);

namespace {

struct GemmArgs {
  int64_t M, N, K;
  int64_t kchunk;  // K range of one CTA
  int ntn, tiles;  // N tiles, output tiles
  int zc, zg;      // K chunks per tile: zc CTAs of one cluster, zg clusters
  double alpha, beta;
  const double* A;
  int64_t sAm, sAk, bA;
  const double* B;
  int64_t sBk, sBn, bB;
  double* C;  // zg > 1: the partial products [zg][M][N]
  int64_t bC;
  GemmEpilogue epi;
  const GemmPtrs* ptrs;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
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

__device__ __forceinline__ int64_t c_offset(const GemmEpilogue& ep, int64_t m, int64_t n) {
  return (ep.msplit ? (m / ep.msplit) * ep.s_mhi + (m % ep.msplit) * ep.s_mlo : m * ep.s_mhi) + n * ep.s_n;
}

// One output tile per CTA (zc == 1) or per cluster of zc CTAs, each with its share of K: the
// partial tiles are added across the cluster through distributed shared memory in rank
// order, so a split costs no second launch and no trip through device memory.
template <class T, bool CLUSTER>
__global__ void __launch_bounds__(T::THREADS) dgemm_kernel(GemmArgs g) {
  __shared__ double smem[T::SMEM];
  const int rank = CLUSTER ? (int)cluster_rank() : 0;
  const int t = CLUSTER ? (int)blockIdx.x / g.zc : (int)blockIdx.x;
  const int zi = t / g.tiles, tile = t - zi * g.tiles;
  const int64_t m0 = (int64_t)(tile / g.ntn) * T::BM, n0 = (int64_t)(tile % g.ntn) * T::BN;
  const double* A = g.A;
  const double* B = g.B;
  double* C = g.C;
  if (g.ptrs) {
    A = g.ptrs[blockIdx.y].A;
    B = g.ptrs[blockIdx.y].B;
    C = g.ptrs[blockIdx.y].C;
  } else {
    A += (int64_t)blockIdx.y * g.bA;
    B += (int64_t)blockIdx.y * g.bB;
    C += (int64_t)blockIdx.y * g.bC + (int64_t)zi * (g.zg > 1 ? g.M * g.N : 0);
  }
  const int64_t k0 = ((int64_t)zi * g.zc + rank) * g.kchunk;
  const int64_t kn = k0 < g.K ? (g.K - k0 < g.kchunk ? g.K - k0 : g.kchunk) : 0;
  double acc[T::PM][T::PN], old[T::PM][T::PN];
  if (!CLUSTER && g.beta != 0.0) {  // the old values travel while the product runs
#pragma unroll
    for (int i = 0; i < T::PM; i++)
#pragma unroll
      for (int j = 0; j < T::PN; j++) {
        const int64_t m = m0 + T::row(i), n = n0 + T::col(j);
        old[i][j] = m < g.M && n < g.N ? C[c_offset(g.epi, m, n)] : 0.0;
      }
  }
  T::product(smem, A + m0 * g.sAm + k0 * g.sAk, g.sAm, g.sAk, B + k0 * g.sBk + n0 * g.sBn, g.sBk, g.sBn, g.M - m0,
             g.N - n0, kn, acc);
  if (!CLUSTER) {
#pragma unroll
    for (int i = 0; i < T::PM; i++)
#pragma unroll
      for (int j = 0; j < T::PN; j++) {
        const int64_t m = m0 + T::row(i), n = n0 + T::col(j);
        if (m < g.M && n < g.N) {
          const double v = g.alpha * acc[i][j];
          C[c_offset(g.epi, m, n)] = g.beta == 0.0 ? v : fma(g.beta, old[i][j], v);
        }
      }
    return;
  }
  // product() ended with a barrier: its stages are free for the partial tile, [m][n] or
  // [n][m] so that consecutive elements are consecutive in C where one of its indices allows
  const bool mfast = g.epi.s_n != 1 && !g.epi.msplit && g.epi.s_mhi == 1;
#pragma unroll
  for (int i = 0; i < T::PM; i++)
#pragma unroll
    for (int j = 0; j < T::PN; j++)
      smem[mfast ? T::col(j) * T::BM + T::row(i) : T::row(i) * T::BN + T::col(j)] = acc[i][j];
  cluster_barrier();
  for (int e = rank * T::THREADS + (int)threadIdx.x; e < T::BM * T::BN; e += g.zc * T::THREADS) {
    const int64_t m = m0 + (mfast ? e % T::BM : e / T::BN), n = n0 + (mfast ? e / T::BM : e % T::BN);
    if (m >= g.M || n >= g.N) continue;
    double* cp = C + c_offset(g.epi, m, n);
    const double o = g.beta != 0.0 ? *cp : 0.0;
    double s = 0.0;
    for (int q = 0; q < g.zc; q++) s += ld_cluster(smem + e, (uint32_t)q);
    const double v = g.alpha * s;
    *cp = g.beta == 0.0 ? v : fma(g.beta, o, v);
  }
  cluster_barrier();  // no CTA leaves while another still reads its partial tile
}

struct Plan {
  int shape, zc, zg;
};

// The tile and the K split that a launch of `batch` M x N x K products takes: the fewest
// clocks of the busiest SM in the model below (patches x K x 16 clocks of its FP64 pipe), with
// what a split costs: a cluster's two barriers and remote reads, or the partial products in
// device memory and a second launch.  Fitted to a sweep of every (tile, zc, zg) over 20
// shapes from 475 x 19 x 5 to 160 x 160 x 40960; its choice was the fastest or within 5 % of
// it on 18 of them, 9 % on the others.
Plan dgemm_plan(int64_t M, int64_t N, int64_t K, int batch, bool may_split) {
  struct Shape {
    int bm, bn, per;  // tile, FP64 FMAs of one K step in SM clocks
  };
  static const Shape shapes[] = {{DTile16::BM, DTile16::BN, 16 * 8}, {DTile32::BM, DTile32::BN, 16 * 32}};
  constexpr double kSms = 152.0;
  Plan best{1, 1, 1};
  double best_t = 1e300;
  for (int s = 0; s < 2; s++) {
    const double tm = (double)((M + shapes[s].bm - 1) / shapes[s].bm), tn = (double)((N + shapes[s].bn - 1) / shapes[s].bn);
    const double tiles = tm * tn * batch;
    // share of a tile's patches that lie inside the matrix, averaged over the tiles
    const double fill = (double)((M + 7) / 8) * (double)((N + 3) / 4) / (tm * tn * (shapes[s].bm / 8) * (shapes[s].bn / 4));
    for (int zg = 1; zg <= 64; zg *= 2)
      for (int zc = 1; zc <= 8; zc *= 2) {
        const int64_t z = (int64_t)zc * zg;
        if (z > 1 && (!may_split || K < 4 * z)) continue;
        if (zg > 1 && (zc < 8 || 8.0 * M * N * zg > 2e9)) continue;
        const double kc = (double)((K + z - 1) / z);
        const double ctas = tiles * z, full = kc * shapes[s].per;
        // few CTAs per SM: the busiest SM's count of whole tiles, a lone CTA a quarter above the
        // pipe's rate; many: the average plus half a CTA; 700 clocks of each CTA are not covered
        const double waves = ctas / kSms;
        const double load = waves > 4.0   ? (waves + 0.5) * (full * fill + 700.0)
                            : waves > 1.0 ? std::ceil(waves) * (full * 0.5 * (1.0 + fill) + 700.0)
                                          : 1.25 * full + 700.0;
        double t = load + 1500.0 + (zc > 1 ? 1200.0 + 100.0 * zc : 0.0);
        if (zg > 1) t += 7000.0 + 60.0 * zg + (double)M * N * zg * 8.0 / 2000.0;
        if (t < best_t) {
          best_t = t;
          best = Plan{s, zc, zg};
        }
      }
  }
  return best;
}

template <class T>
void launch(Ctx& c, const GemmArgs& g, int batch) {
  const dim3 grid((unsigned)((int64_t)g.tiles * g.zc * g.zg), (unsigned)batch);
  if (g.zc == 1) {
    dgemm_kernel<T, false><<<grid, T::THREADS, 0, c.stream>>>(g);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(T::THREADS);
  cfg.stream = c.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)g.zc;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  UCC_CUDA(cudaLaunchKernelEx(&cfg, dgemm_kernel<T, true>, g));
}

}  // namespace

void dgemm_strided(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm, int64_t sAk,
                   const double* B, int64_t sBk, int64_t sBn, double beta, double* C, const GemmEpilogue& epi,
                   int batch, int64_t bA, int64_t bB, int64_t bC, const GemmPtrs* ptrs) {
  if (M <= 0 || N <= 0 || batch <= 0) return;
  if (Recorder* r = recorder()) {
    UCC_REQUIRE(batch == 1 && !ptrs && epi.msplit == 0, UCC_UNSUPPORTED, "dgemm: form not recordable");
    RecordedOp o;
    o.kind = RecordedOp::kGemm;
    o.M = M, o.N = N, o.K = K, o.sAm = sAm, o.sAk = sAk, o.sBk = sBk, o.sBn = sBn, o.sCm = epi.s_mhi, o.sCn = epi.s_n;
    o.A = A, o.B = B, o.C = C, o.alpha = alpha, o.beta = beta;
    r->ops.push_back(o);
    return;
  }
  UCC_REQUIRE(batch <= 65535, UCC_BAD_ARGS, "dgemm: batch too large");
  UCC_REQUIRE((M + 63) / 64 <= 65535, UCC_BAD_ARGS, "dgemm: M too large");
  const Plan p = dgemm_plan(M, N, K, batch, batch == 1 && !ptrs);
  const int bm = p.shape == 0 ? DTile16::BM : DTile32::BM, bn = p.shape == 0 ? DTile16::BN : DTile32::BN;
  const int64_t ntm = (M + bm - 1) / bm, ntn = (N + bn - 1) / bn, z = (int64_t)p.zc * p.zg;
  UCC_REQUIRE(ntm * ntn * z < ((int64_t)1 << 31), UCC_BAD_ARGS, "dgemm: output too large");
  GemmArgs g{M, N, K, (K + z - 1) / z, (int)ntn, (int)(ntm * ntn), p.zc, p.zg, alpha, beta, A, sAm, sAk, bA, B,
             sBk, sBn, bB, C, bC, epi, ptrs};
  std::unique_ptr<Scratch> part;
  if (p.zg > 1) {  // partial products, added in a fixed order by splitk_reduce
    part = std::make_unique<Scratch>(c, sizeof(double) * M * N * p.zg);
    g.C = part->d();
    g.alpha = 1.0;
    g.beta = 0.0;
    g.epi = GemmEpilogue{0, N, 0, 1};
  }
  cudaEvent_t ev0 = c.take_event(), ev1 = c.take_event();
  cudaEventRecord(ev0, c.stream);
  if (p.shape == 0)
    launch<DTile16>(c, g, batch);
  else
    launch<DTile32>(c, g, batch);
  count_kernel_launch();
  UCC_CUDA(cudaGetLastError());
  if (part) splitk_reduce(c, M, N, p.zg, part->d(), alpha, beta, C, epi);
  cudaEventRecord(ev1, c.stream);
  c.gemm_timers.push_back({ev0, ev1, 2.0 * (double)M * (double)N * (double)K * (double)batch});
  if (c.gemm_timers.size() >= 4096) c.resolve_timers();
}

}  // namespace ucc
