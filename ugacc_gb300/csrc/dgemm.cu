// FP64 (DFMA) GEMM over arbitrarily strided operands with a permuting epilogue, so that a
// contraction result lands directly in its tensor layout (no separate transpose pass).
#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "chain.h"
#include "core.h"
#include "dgemm_tile.h"

namespace ucc {

void count_kernel_launch();  // kernels_fp64.cu
namespace {

struct GemmArgs {
  int64_t M, N, K;
  int64_t kchunk;  // K range of one CTA
  int ntn, tiles;  // N tiles, output tiles
  int zc, zg;      // K chunks per tile: zc CTAs of one cluster, zg clusters
  double alpha, beta;
  DView A, B;
  int64_t bA, bB;
  double* C;
  int64_t bC;
  GemmEpilogue epi;
  const GemmPtrs* ptrs;
  double* part;  // zg > 1: [tiles][zg][tile]
  Ctx::DeviceWords* words;
  bool timed;  // by the kernel itself
};

// One output tile per CTA (zc == 1) or per cluster of zc CTAs (dgemm_cta)
template <class T, bool CLUSTER>
__global__ void __launch_bounds__(T::THREADS) dgemm_kernel(GemmArgs g) {
  __shared__ double smem[T::SMEM];
  chain_enter();
  if (g.timed) dgemm_clock_start(g.words);
  const int rank = CLUSTER ? (int)dgemm_cluster_rank() : 0;
  const int t = CLUSTER ? (int)blockIdx.x / g.zc : (int)blockIdx.x;
  const int tile = t / g.zg, zi = t - tile * g.zg;
  DView A = g.A, B = g.B;
  double* C = g.C;
  if (g.ptrs) {
    A.p = g.ptrs[blockIdx.y].A;
    B.p = g.ptrs[blockIdx.y].B;
    C = g.ptrs[blockIdx.y].C;
  } else {
    A.p += (int64_t)blockIdx.y * g.bA;
    B.p += (int64_t)blockIdx.y * g.bB;
    C += (int64_t)blockIdx.y * g.bC;
  }
  const DSplit z{g.zc, g.zg, rank, zi, g.kchunk, g.part + (int64_t)tile * g.zg * (T::BM * T::BN),
                 g.words ? g.words->tickets + (int64_t)tile * g.zc : nullptr};
  dgemm_cta<T, CLUSTER>(smem, z, A, B, g.M, g.N, g.K, (int64_t)(tile / g.ntn) * T::BM, (int64_t)(tile % g.ntn) * T::BN,
                        g.alpha, g.beta, C, g.epi);
  if (g.timed) dgemm_clock_stop(g.words, gridDim.x * gridDim.y);
}

}  // namespace

DView dgemm_operand(const MatView& v) {
  UCC_REQUIRE(v.rows < ((int64_t)1 << 32) && v.cols < ((int64_t)1 << 32), UCC_BAD_ARGS, "dgemm: extent too large");
  auto run = [](int64_t hi, int64_t split, int64_t lo) { return DRun{hi, lo, (uint32_t)split}; };
  DView d{v.p, run(v.rs_hi, v.rsplit, v.rs_lo), run(v.ks_hi, v.ksplit, v.ks_lo), false};
  d.kfast = d.k.step() == 1 || (d.r.step() != 1 && d.k.step() < d.r.step());
  return d;
}

// The tile and the K split of a launch: the fewest clocks of the busiest SM in the model below
// (patches x K x 16 clocks of its FP64 pipe), with what a split costs: a cluster's two
// barriers and remote reads, or the partial tiles in device memory and their sum.
// Fitted to a sweep of every (tile, zc, zg) over 20 shapes from 475 x 19 x 5 to
// 160 x 160 x 40960; its choice was the fastest or within 5 % of it on 18 of them, 9 % on the
// others.
DgemmPlan dgemm_plan(const std::vector<GemmShape>& probs, bool may_split) {
  struct Shape {
    int bm, bn, per;  // tile, FP64 FMAs of one K step in SM clocks
  };
  static const Shape shapes[] = {{DTile16::BM, DTile16::BN, 16 * 8}, {DTile32::BM, DTile32::BN, 16 * 32}};
  constexpr double kSms = 152.0;
  DgemmPlan best{1, 1, 1};
  double best_t = 1e300;
  int64_t kmax = 0;
  double outputs = 0.0;
  int64_t tiles[2] = {0, 0};
  for (const GemmShape& g : probs) {
    kmax = std::max(kmax, g.K);
    outputs += (double)g.M * g.N * g.count;
    for (int s = 0; s < 2; s++)
      tiles[s] += (g.M + shapes[s].bm - 1) / shapes[s].bm * ((g.N + shapes[s].bn - 1) / shapes[s].bn) * g.count;
  }
  for (int s = 0; s < 2; s++)
    for (int zg = 1; zg <= 64; zg *= 2)
      for (int zc = 1; zc <= 8; zc *= 2) {
        const int64_t z = (int64_t)zc * zg;
        if (z > 1 && (!may_split || kmax < 4 * z)) continue;
        if (zg > 1 && (zc < 8 || tiles[s] * zc > Ctx::DeviceWords::kTickets)) continue;
        double ctas = 0.0, work = 0.0, longest = 0.0;  // CTAs, clocks of all, of the longest one
        for (const GemmShape& g : probs) {
          const double tm = (double)((g.M + shapes[s].bm - 1) / shapes[s].bm);
          const double tn = (double)((g.N + shapes[s].bn - 1) / shapes[s].bn);
          // share of a tile's patches that lie inside the matrix, averaged over the tiles
          const double fill =
              (double)((g.M + 7) / 8) * (double)((g.N + 3) / 4) / (tm * tn * (shapes[s].bm / 8) * (shapes[s].bn / 4));
          const double full = (double)((g.K + z - 1) / z) * shapes[s].per;
          ctas += tm * tn * z * g.count;
          work += tm * tn * z * g.count * (full * fill + 700.0);  // 700 clocks of a CTA are not covered
          longest = std::max(longest, full);
        }
        // few CTAs per SM: the busiest SM's count of average tiles (at least the longest one, a
        // quarter above the pipe's rate when it is alone); many: the average plus half a tile
        const double waves = ctas / kSms;
        const double load = waves > 4.0 ? work / kSms + 0.5 * longest
                                        : std::max(std::ceil(waves) * work / ctas, 1.25 * longest + 700.0);
        double t = load + 1500.0 + (zc > 1 ? 1200.0 + 100.0 * zc : 0.0);
        if (zg > 1) t += 3500.0 + 60.0 * zg + outputs * zg * 16.0 / 2000.0;
        if (t < best_t) {
          best_t = t;
          best = DgemmPlan{s, zc, zg};
        }
      }
  return best;
}

namespace {
template <class T>
void launch(Ctx& c, const GemmArgs& g, int batch) {
  const dim3 grid((unsigned)((int64_t)g.tiles * g.zc * g.zg), (unsigned)batch);
  if (g.zc == 1)
    launch_chained(dgemm_kernel<T, false>, grid, dim3(T::THREADS), c.stream, 1, g);
  else
    launch_chained(dgemm_kernel<T, true>, grid, dim3(T::THREADS), c.stream, (unsigned)g.zc, g);
}

}  // namespace

// GEMMs of at least this many multiply-adds (0.1 ms or more) are timed by a pair of events,
// the others by their own CTAs (dgemm_clock_start)
constexpr double kEventWork = 6e7;

static void dgemm_run(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const DView& A, const DView& B,
                      double beta, double* C, const GemmEpilogue& epi, int batch, int64_t bA, int64_t bB, int64_t bC,
                      const GemmPtrs* ptrs) {
  if (M <= 0 || N <= 0 || batch <= 0) return;
  UCC_REQUIRE(batch <= 65535, UCC_BAD_ARGS, "dgemm: batch too large");
  UCC_REQUIRE((M + 63) / 64 <= 65535, UCC_BAD_ARGS, "dgemm: M too large");
  const DgemmPlan p = dgemm_plan({{M, N, K, batch}}, batch == 1 && !ptrs);
  const int bm = p.shape == 0 ? DTile16::BM : DTile32::BM, bn = p.shape == 0 ? DTile16::BN : DTile32::BN;
  const int64_t ntm = (M + bm - 1) / bm, ntn = (N + bn - 1) / bn, z = (int64_t)p.zc * p.zg;
  UCC_REQUIRE(ntm * ntn * z < ((int64_t)1 << 31), UCC_BAD_ARGS, "dgemm: output too large");
  const double work = (double)M * (double)N * (double)K * (double)batch;
  GemmArgs g{M, N, K, (K + z - 1) / z, (int)ntn, (int)(ntm * ntn), p.zc, p.zg, alpha, beta, A, B,
             bA, bB, C, bC, epi, ptrs, nullptr, c.words(), work < kEventWork};
  std::unique_ptr<Scratch> part;
  if (p.zg > 1) {
    part = std::make_unique<Scratch>(c, sizeof(double) * g.tiles * p.zg * bm * bn);
    g.part = part->d();
  }
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  if (!g.timed) {
    ev0 = c.take_event(), ev1 = c.take_event();
    cudaEventRecord(ev0, c.stream);
  }
  if (p.shape == 0)
    launch<DTile16>(c, g, batch);
  else
    launch<DTile32>(c, g, batch);
  count_kernel_launch();
  UCC_CUDA(cudaGetLastError());
  if (g.timed) {
    c.short_gemm_flops += 2.0 * work;
    c.short_gemm_launches++;
    return;
  }
  cudaEventRecord(ev1, c.stream);
  c.gemm_timers.push_back({ev0, ev1, 2.0 * work});
  if (c.gemm_timers.size() >= 4096) c.resolve_timers();
}

void dgemm_view(Ctx& c, double alpha, const MatView& A, const MatView& B, double beta, double* C,
                const GemmEpilogue& epi) {
  if (Recorder* r = recorder()) {  // an empty product too: all members record the same operations
    RecordedOp o;
    o.kind = RecordedOp::kGemm;
    o.A = A, o.B = B, o.C = C, o.epi = epi, o.alpha = alpha, o.beta = beta;
    r->ops.push_back(o);
    return;
  }
  dgemm_run(c, A.rows, B.rows, A.cols, alpha, dgemm_operand(A), dgemm_operand(B), beta, C, epi, 1, 0, 0, 0, nullptr);
}

void dgemm_strided(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm, int64_t sAk,
                   const double* B, int64_t sBk, int64_t sBn, double beta, double* C, const GemmEpilogue& epi,
                   int batch, int64_t bA, int64_t bB, int64_t bC, const GemmPtrs* ptrs) {
  const MatView a = MatView::strided(A, M, K, sAm, sAk), b = MatView::strided(B, N, K, sBn, sBk);
  if (batch == 1 && !ptrs) return dgemm_view(c, alpha, a, b, beta, C, epi);
  UCC_REQUIRE(!recorder(), UCC_UNSUPPORTED, "dgemm: form not recordable");
  dgemm_run(c, M, N, K, alpha, dgemm_operand(a), dgemm_operand(b), beta, C, epi, batch, bA, bB, bC, ptrs);
}

}  // namespace ucc
