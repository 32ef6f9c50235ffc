// Mixed-precision tensor-core GEMM for sm_103a (tcgen05 + TMEM + TMA).
//
// C[m][n] (FP64, strided, alpha/beta, permuting epilogue) =
//     sum_k  Ahi[m][k] Bhi[n][k] + Ahi[m][k] Blo[n][k] + Alo[m][k] Bhi[n][k]
// where x = hi + lo with hi = bf16(x), lo = bf16(x - hi): the two-term split product of
// FP64 operands, accumulated in FP32 in tensor memory (gemm_kernel); and FP64-accurate
// products of exact bf16 digits (sliced_gemm_kernel, sliced_short_kernel below).
//
// gemm_kernel (one CTA per SM, persistent over 128 x bn output tiles, bn up to 256; with two M
// tiles or more the CTAs work in pairs, cta_group::2, on 256 rows):
//   warp 0      TMA producer (one thread): K blocks of 64 of A (128 rows) and B (bn rows, a pair's
//               CTA half of them), 128B swizzle; a two-part stage holds hi and lo of both
//   warp 1      MMA issuer (one thread, rank 0 of a pair): kind::f16, M = 128 or 256, K = 16
//   warps 2-5   epilogue: tcgen05.ld 32x32b.x32 -> FP64 alpha/beta -> global
//   smem ring of up to 4 stages (full/empty mbarriers), two TMEM accumulators (2 x 256 columns) so
//   the epilogue of one tile, or of one pass over K, overlaps the MMAs of the next.
// Every mbarrier wait is bounded (globaltimer deadline); on expiry the kernel raises a
// device error flag, the other warps see it and leave their loops, loads and MMAs in flight are
// awaited, TMEM is released and the host reports UCC_DEVICE_TIMEOUT.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <cstring>
#include <map>
#include <tuple>

#include "cc.h"
#include "chain.h"
#include "core.h"
#include "tc_ptx.h"

namespace ucc {

void count_kernel_launch();  // kernels_fp64.cu
// C(epi) = alpha * sum_z P[z] + beta * C(epi) (kernels_fp64.cu)
void splitk_reduce(Ctx& c, int64_t M, int64_t N, int nsplit, const double* P, double alpha, double beta, double* C,
                   const GemmEpilogue& epi);

namespace tc {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4, THREADS = 192;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
constexpr uint32_t TMEM_COLS = 2 * BN;
constexpr size_t SMEM_BYTES = 1024 + (size_t)STAGES * (A_BYTES + B_BYTES) + 256;
// N tile for N output columns: the fewest tiles of at most 256 columns, each a multiple of
// 32 (N = 320 takes two tiles of 160 rather than 256 + 64)
inline int pick_bn(int64_t N) {
  const int64_t nt = (N + 255) / 256;
  return (int)(((N + nt - 1) / nt + 31) / 32 * 32);
}
// CTAs per cluster for a launch with mtiles M tiles: pairs that work on one N tile whenever
// there are two M tiles to pair (the B maps then have boxes of bn / 2 rows)
inline int cluster_m(int mtiles) { return mtiles >= 2 ? 2 : 1; }

// gemm_kernel: an operand ring of 216 KB (four 48 KB stages, or fused stages of
// A_hi | A_lo | B_hi | B_lo), then the barriers
constexpr size_t GEMM_RING = 216 * 1024;
constexpr size_t GEMM_SMEM_BYTES = 1024 + GEMM_RING + 256;
// instruction descriptor, kind::f16: D f32 (bit 4), A bf16 (bits 7-9 = 1), B bf16
// (bits 10-12 = 1), both K-major, N>>3 at bits 17-22, M>>4 at bits 24-28; the CTAs of a pair
// work on M = 256 rows together
__device__ __forceinline__ uint32_t idesc_of(int cm, int bn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(cm * BM >> 4) << 24);
}

struct Params {
  int M, N, kblocks, mtiles, ntiles;
  int bn;  // N tile: the MMA's N and the B box rows (a multiple of 32 up to 256)
  double alpha, beta;
  double* C;
  GemmEpilogue epi;
  int* err;
  // batched problems of one shape (0 = a single problem): problem p reads A rows from
  // a_row0[p] and B rows from b_row0[p] of the tensor maps and writes C + c_off[p]
  int nprob;
  const int* a_row0;
  const int* b_row0;
  const int64_t* c_off;
  // split-K (single problem only): chunk z covers K blocks [z*kchunk, (z+1)*kchunk) of each
  // of the three split products and writes a plain [M][N] FP64 partial at C + z*M*N
  int ksplit, kchunk;
  // nterms = 2 (batched problems only): a second product accumulated into the same tile,
  // A from the second pair of tensor maps at rows a_row1[p], B at rows b_row1[p], for the
  // problems p < npair
  int nterms, npair;
  const int* a_row1;
  const int* b_row1;
  // C32 != null: FP32 output C32[off] = alpha * acc (+ C32[off] when beta != 0), no FP64
  // work in the epilogue (GB300 issues ~4 FP64 operations per clock per SM)
  float* C32;
  // nparts = 3: operands split hi + mid + lo (third maps), six products hi.hi, hi.mid,
  // mid.hi, hi.lo, mid.mid, lo.hi (representation error ~2^-25 instead of ~2^-17)
  int nparts;
  // kc > 0: the K range of every tile runs in chunks of kc K blocks, each chunk's FP32
  // accumulator added into the FP64 output by the epilogue (the first with beta, the
  // rest with 1), which bounds the FP32 accumulation chain; FP64 output only
  int kc;
  // fused (two parts): one ring stage holds A_hi, A_lo, B_hi and B_lo of a K block
  // and the three products are issued from it (a third less operand traffic than one
  // stage per product); nst stages of stage_bytes each
  int fused, nst, stage_bytes;
  // tblk > 0 (FP32 output of the (T) tuple GEMMs, alpha 1, beta 0): W3 in the blocked
  // layout of w3_block_offset with tblk blocks per index; the strides s_mhi, s_mlo, s_n
  // (nv^2, nv or 1, msplit = nv) say which of a, b, c each index is
  int tblk = 0;
};

// v[p] <- v[p ^ k] for 0 <= k < 8: three conditional swaps (selects, no indexed registers)
__device__ __forceinline__ void xor_swap8(float (&v)[8], int k) {
#pragma unroll
  for (int bit = 1; bit < 8; bit <<= 1) {
    const bool s = (k & bit) != 0;
#pragma unroll
    for (int e = 0; e < 8; e++)
      if ((e & bit) == 0) {
        const float lo = v[e], hi = v[e | bit];
        v[e] = s ? hi : lo;
        v[e | bit] = s ? lo : hi;
      }
  }
}

// the split products of one K block: (A part, B part), part 0 = hi, 1 = lo (2 parts) or
// 0 = hi, 1 = mid, 2 = lo (3 parts)
__device__ __forceinline__ void seg_parts(int nparts, int seg, int& pa, int& pb) {
  if (nparts == 3) {  // A parts 0,0,1,0,1,2 and B parts 0,1,0,2,1,0, two bits per segment
    pa = (2320 >> (2 * seg)) & 3;
    pb = (388 >> (2 * seg)) & 3;
  } else {
    pa = seg == 2 ? 1 : 0;
    pb = seg == 1 ? 1 : 0;
  }
}

// N tiles per raster band: the tiles of one problem run band by band, and inside a band M
// group by M group with the band's N tiles fastest, so that the ~150 tiles in flight at a
// time cover about a dozen M groups x RASTER_N N tiles: each A tile is then read by
// RASTER_N concurrent tiles and each B tile by a dozen, mostly from L2 (walking M fastest
// over a whole column of tiles shared B only and re-read every A tile from DRAM once per N
// tile).
constexpr int RASTER_N = 8;
__device__ __forceinline__ void raster(int mgroups, int ntiles, int tl, int& mg, int& nt) {
  const int band = tl / (mgroups * RASTER_N);
  const int w = min(RASTER_N, ntiles - band * RASTER_N);  // N tiles in this band
  const int r = tl - band * mgroups * RASTER_N;
  mg = r / w;
  nt = band * RASTER_N + (r - mg * w);
}

// Work item -> (problem or K chunk pb, M tile group mg, N tile nt).  Batched problems run
// M-group-major: all problems and N tiles of one M group before the next, so that the
// problems of a launch that share an A operand (the (T) tuples of one occupied index) read
// each A tile from L2 instead of DRAM.  One problem (or its split-K chunks) runs
// chunk-major, each chunk in raster bands.
__device__ __forceinline__ void tile_coords(const Params& p, int mgroups, int tile, int& pb, int& mg, int& nt) {
  if (p.nprob) {
    const int per_m = p.nprob * p.ntiles;
    mg = tile / per_m;
    const int r = tile - mg * per_m;
    pb = r / p.ntiles;
    nt = r - pb * p.ntiles;
  } else {
    const int tiles_per = mgroups * p.ntiles;
    pb = tile / tiles_per;
    raster(mgroups, p.ntiles, tile - pb * tiles_per, mg, nt);
  }
}

// The loads of a pair's ring complete on rank 0's barriers, and rank 0 waits for those of the stages
// that it issued itself.  After a wait that ran out its peer can be up to a ring ahead, with loads in
// flight into its own shared memory that nobody waits for.  So both producers leave their count of
// issued stages with both CTAs (issued[rank], before the cluster's last barrier), and when the
// counts differ rank 0 expects and awaits the peer's surplus, `bytes` a stage, before either leaves.
// Without an error the counts are equal and nothing more is done.
__device__ __forceinline__ void pair_tell(int64_t* issued, int rank, int64_t n) {
  issued[rank] = n;
  asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(map_rank(issued + rank, (uint32_t)(rank ^ 1))), "l"(n)
               : "memory");
}
__device__ __forceinline__ void pair_drain(uint64_t* full, int nst, const int64_t* issued, int rank, uint32_t bytes) {
  const int64_t n0 = issued[0], n1 = issued[1];
  if (n0 == n1) return;
  if (rank == 0 && threadIdx.x == 0)
    for (int64_t n = n0; n < n1; n++) {
      mbar_expect_tx(&full[n % nst], bytes);
      mbar_wait_deadline(&full[n % nst], (uint32_t)((n / nst) & 1));
    }
  cluster_sync();
}

// CM CTAs per cluster along M (1 or 2).  With CM = 2 the two CTAs of a cluster work as a pair
// (cta_group::2) on M tiles 2j and 2j+1 of one N tile: each CTA's ring holds its own 128 rows
// of A and half of the B tile's rows (the B tensor maps have boxes of bn / 2 rows), rank 0
// issues MMAs of 256 rows that read both rings, and each CTA's tensor memory gets its own
// 128 rows of the result.  Rank 0's full barriers count the bytes of both CTAs' loads, its
// MMA commits arrive on the empty and accumulator barriers of both, and both epilogues
// release an accumulator on rank 0's barrier.
//
// What bounds it is the shared-memory port (128 bytes per SM clock), which TMA writes and
// operand reads share: a 128 x 256 x 16 MMA (128 clocks) reads 12 KB, and filling the ring
// with a whole B tile per CTA adds 96 KB per three products of a K block (1536 clocks), 160
// bytes per clock together; as a pair it is 8 KB and 64 KB, 106 bytes.
template <int CM>
__global__ void __launch_bounds__(THREADS, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap mAhi, const __grid_constant__ CUtensorMap mAlo,
                const __grid_constant__ CUtensorMap mBhi, const __grid_constant__ CUtensorMap mBlo,
                const __grid_constant__ CUtensorMap mA2hi, const __grid_constant__ CUtensorMap mA2lo,
                const __grid_constant__ CUtensorMap mAmid, const __grid_constant__ CUtensorMap mBmid, Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_BYTES;
  uint64_t* full = (uint64_t*)(smem + GEMM_RING);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* mdone = tempty + 2;  // every MMA of this CTA has completed (before TMEM is released)
  int64_t* issued_of = (int64_t*)(mdone + 1);  // stages issued by the CTAs of a pair
  uint32_t* tslot = (uint32_t*)(issued_of + 2);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int nst = p.fused ? p.nst : STAGES;  // ring stages (at most STAGES)
  const int rank = CM > 1 ? (int)cluster_rank() : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 128 * CM);  // the epilogues of both CTAs, on rank 0's barrier
    }
    mbar_init(mdone, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc<CM>(tslot, TMEM_COLS);
  fence_before();
  __syncthreads();
  fence_after();
  if (CM > 1) cluster_sync();  // the peer's barriers exist before loads, commits or arrivals reach them
  const uint32_t tmem = *tslot;
  // M tiles in groups of CM (one per CTA of the cluster); the clusters walk the groups
  const int mgroups = (p.mtiles + CM - 1) / CM;
  const int tiles_per = mgroups * p.ntiles;
  const int ntile = tiles_per * (p.nprob ? p.nprob : (p.ksplit > 1 ? p.ksplit : 1));
  const int cid = blockIdx.x / CM, ncl = gridDim.x / CM;
  const int bh = p.bn / CM;  // B rows this CTA loads
  // ring items per K block and term: one fused stage, or one stage per split product
  const int nseg = p.fused ? 1 : (p.nparts == 3 ? 6 : 3);
  const uint32_t b_tile = (uint32_t)(bh * BK * 2);
  // K chunks of one tile (in-kernel chunking) and the K blocks of chunk ch
  const int nch = p.kc > 0 ? (p.kblocks + p.kc - 1) / p.kc : 1;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int64_t issued = 0;
      bool ok = true;
      for (int tile = cid; tile < ntile && ok; tile += ncl) {
        int pb, mg, nt;
        tile_coords(p, mgroups, tile, pb, mg, nt);
        const int mt = mg * CM + rank;
        const int ar0 = (p.nprob ? p.a_row0[pb] : 0) + mt * BM;
        const int br0 = (p.nprob ? p.b_row0[pb] : 0) + nt * p.bn + rank * bh;
        const int terms = p.nterms > 1 && pb < p.npair ? 2 : 1;
        const int ar1 = terms > 1 ? p.a_row1[pb] + mt * BM : 0;
        const int br1 = terms > 1 ? p.b_row1[pb] + nt * p.bn + rank * bh : 0;
        for (int ch = 0; ch < nch && ok; ch++) {
          int k0 = 0, kn = p.kblocks;
          if (p.ksplit > 1) {
            k0 = pb * p.kchunk;
            kn = min(p.kblocks - k0, p.kchunk);
          } else if (p.kc > 0) {
            k0 = ch * p.kc;
            kn = min(p.kblocks - k0, p.kc);
          }
          for (int kb = 0; kb < terms * nseg * kn; kb++) {
            if (!mbar_wait(&empty[stage], phase ^ 1u, p.err)) {
              ok = false;
              break;
            }
            const int term = kb / (nseg * kn), w = kb - term * nseg * kn;
            const int seg = w / kn, kk = (k0 + w - seg * kn) * BK;
            // rank 0 counts the bytes of the pair's loads
            const uint32_t fbar = CM > 1 ? map_rank(&full[stage], 0) : 0u;
            auto load = [&](uint8_t* dst, const CUtensorMap* map, int row) {
              if (CM == 1)
                tma_load(dst, map, &full[stage], kk, row);
              else
                tma_load_pair(dst, map, fbar, kk, row);
            };
            if (p.fused) {  // A_hi | A_lo | B_hi | B_lo of K block kk
              uint8_t* st = smem + (size_t)stage * p.stage_bytes;
              if (rank == 0) mbar_expect_tx(&full[stage], CM * ((uint32_t)(2 * A_BYTES) + 2 * b_tile));
              load(st, term == 0 ? &mAhi : &mA2hi, term == 0 ? ar0 : ar1);
              load(st + A_BYTES, term == 0 ? &mAlo : &mA2lo, term == 0 ? ar0 : ar1);
              load(st + 2 * A_BYTES, &mBhi, term == 0 ? br0 : br1);
              load(st + 2 * A_BYTES + b_tile, &mBlo, term == 0 ? br0 : br1);
            } else {
              int pa, pbp;
              seg_parts(p.nparts, seg, pa, pbp);
              const CUtensorMap* ma = term == 0 ? (pa == 0 ? &mAhi : (pa == 1 && p.nparts == 3) ? &mAmid : &mAlo)
                                                : (pa == 0 ? &mA2hi : &mA2lo);
              const CUtensorMap* mb = pbp == 0 ? &mBhi : (pbp == 1 && p.nparts == 3) ? &mBmid : &mBlo;
              if (rank == 0) mbar_expect_tx(&full[stage], CM * ((uint32_t)A_BYTES + b_tile));
              load(sA + stage * A_BYTES, ma, term == 0 ? ar0 : ar1);
              load(sB + stage * B_BYTES, mb, term == 0 ? br0 : br1);
            }
            ++issued;
            if (++stage == nst) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      // the last ring loads must have landed before the CTA may exit (matters only on an
      // error path; normally the epilogue's final wait already implies it); rank 0's barriers
      // see the loads of both (pair_drain)
      if (rank == 0)
        for (int64_t n = issued > nst ? issued - nst : 0; n < issued; n++)
          mbar_wait_deadline(&full[n % nst], (uint32_t)((n / nst) & 1));
      if (CM > 1) pair_tell(issued_of, rank, issued);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank != 0) {
      mbar_wait_deadline(mdone, 0);  // rank 0 issues the pair's MMAs
    } else if (lane == 0) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      const uint32_t idesc = idesc_of(CM, p.bn);
      for (int tile = cid; tile < ntile && ok; tile += ncl) {
        int terms = 1;
        if (p.nterms > 1) {
          int pb, mg, nt;
          tile_coords(p, mgroups, tile, pb, mg, nt);
          terms = pb < p.npair ? 2 : 1;
        }
        for (int ch = 0; ch < nch && ok; ch++) {
          int kn = p.kblocks;
          if (p.ksplit > 1)
            kn = min(p.kblocks - (tile / tiles_per) * p.kchunk, p.kchunk);
          else if (p.kc > 0)
            kn = min(p.kblocks - ch * p.kc, p.kc);
          if (!mbar_wait(&tempty[acc], aphase ^ 1u, p.err)) {
            ok = false;
            break;
          }
          fence_after();
          const uint32_t d = tmem + (uint32_t)(acc * BN);
          for (int kb = 0; kb < terms * nseg * kn; kb++) {
            if (!mbar_wait(&full[stage], phase, p.err)) {
              ok = false;
              break;
            }
            fence_after();
            if (p.fused) {  // hi.hi, hi.lo, lo.hi from one stage
              uint8_t* st = smem + (size_t)stage * p.stage_bytes;
              const uint64_t ahi = sdesc(st), alo = sdesc(st + A_BYTES);
              const uint64_t bhi = sdesc(st + 2 * A_BYTES), blo = sdesc(st + 2 * A_BYTES + b_tile);
#pragma unroll
              for (int pr = 0; pr < 3; pr++) {
                const uint64_t ad = pr == 2 ? alo : ahi, bd = pr == 1 ? blo : bhi;
#pragma unroll
                for (int k = 0; k < BK / 16; k++)
                  mma_i<CM>(d, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (kb | pr | k) != 0);
              }
            } else {
              const uint64_t ad = sdesc(sA + stage * A_BYTES), bd = sdesc(sB + stage * B_BYTES);
#pragma unroll
              for (int k = 0; k < BK / 16; k++)  // +32 bytes along K per 16-element step
                mma_i<CM>(d, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (kb | k) != 0);
            }
            mma_commit<CM>(&empty[stage]);
            if (++stage == nst) {
              stage = 0;
              phase ^= 1u;
            }
          }
          mma_commit<CM>(&tfull[acc]);
          if (++acc == 2) {
            acc = 0;
            aphase ^= 1u;
          }
        }
      }
      // on an error path the loop may end with MMAs still running: wait for all of them
      // before the CTA releases tensor memory
      mma_commit<CM>(mdone);
      mbar_wait_deadline(mdone, 0);
    }
  } else {
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    int acc = 0;
    uint32_t aphase = 0;
    const GemmEpilogue ep = p.epi;
    bool ok = true;
    for (int tile = cid; tile < ntile && ok; tile += ncl)
    for (int kch = 0; kch < nch; kch++) {
      int pb, mg, nt;
      tile_coords(p, mgroups, tile, pb, mg, nt);
      const int mt = mg * CM + rank;
      const int64_t coff = p.nprob ? p.c_off[pb] : (p.ksplit > 1 ? (int64_t)pb * p.M * p.N : 0);
      if (!mbar_wait(&tfull[acc], aphase, p.err)) {
        ok = false;
        break;
      }
      fence_after();
      const int64_t m = (int64_t)mt * BM + q * 32 + lane;
      const int64_t mo = ep.msplit ? (m / ep.msplit) * ep.s_mhi + (m % ep.msplit) * ep.s_mlo : m * ep.s_mhi;
      // later K chunks of a tile add onto the earlier ones
      const double alpha = p.alpha, beta = kch == 0 ? p.beta : 1.0;
      // columns contiguous and every row on a 32-byte boundary (the same for all lanes)
      const bool sectors = ep.s_n == 1 && ((reinterpret_cast<uintptr_t>(p.C + coff) & 31u) == 0) &&
                           ep.s_mhi % 4 == 0 && (!ep.msplit || ep.s_mlo % 4 == 0);
      for (int ch = 0; ch < p.bn / 32; ch++) {
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN + ch * 32), r);
        if (m < p.M) {
          const int64_t n0 = (int64_t)nt * p.bn + ch * 32;
          // with beta != 0 all 32 old values are loaded before the first store, so the
          // loads are in flight together instead of each waiting behind a store that
          // might alias it
          if (p.C32 && p.tblk) {
            // blocked W3: each index placed by its linear stride (nv^2 a, nv b, 1 c)
            const int64_t nvv = ep.msplit, hi = m / nvv, lo = m % nvv, T = p.tblk;
            const int rn = ep.s_n == 1 ? 2 : (ep.s_n == nvv ? 1 : 0);
            const int rh = ep.s_mhi == 1 ? 2 : (ep.s_mhi == nvv ? 1 : 0);
            float* Cw = p.C32 + coff;
            if (rn == 2 && n0 + 32 <= p.N) {
              // the 32 columns are c: four 8-wide c blocks, each a contiguous 32 bytes
              // holding element z at z ^ k, stored as two float4 after the same swap
              const int64_t a = rh == 0 ? hi : lo, b = rh == 0 ? lo : hi;
              const int x = (int)(a & 7), y = (int)(b & 7), k = (5 * y) & 7;
              float* base = Cw + (((a >> 3) * T + (b >> 3)) * T) * 512 + 64 * x + 8 * (y ^ x);
#pragma unroll
              for (int g = 0; g < 4; g++) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = __uint_as_float(r[8 * g + e]);
                xor_swap8(v, k);
                float4* dst = reinterpret_cast<float4*>(base + ((n0 >> 3) + g) * 512);
                dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                dst[1] = make_float4(v[4], v[5], v[6], v[7]);
              }
            } else {
              // the 32 columns are four 8-wide blocks of one index (n0 % 32 == 0): the
              // offset is a block part, linear in the block, plus one of eight in-block
              // offsets fixed by the row (32-bit: a tuple's blocks hold < 2^31 floats)
              const int rl = 3 - rn - rh;
              const int fa = (int)(rh == 0 ? hi : (rl == 0 ? lo : 0)), fb = (int)(rh == 1 ? hi : (rl == 1 ? lo : 0));
              const int fc = (int)(rh == 2 ? hi : (rl == 2 ? lo : 0)), nb0 = (int)(n0 >> 3), Ti = (int)T;
              const int bA = rn == 0 ? nb0 : fa >> 3, bB = rn == 1 ? nb0 : fb >> 3, bC = rn == 2 ? nb0 : fc >> 3;
              const int blk0 = ((bA * Ti + bB) * Ti + bC) * 512;
              const int gstride = (rn == 0 ? Ti * Ti : (rn == 1 ? Ti : 1)) * 512;
              int loc[8];
#pragma unroll
              for (int e = 0; e < 8; e++) {
                const int x = rn == 0 ? e : (fa & 7), y = rn == 1 ? e : (fb & 7), z = rn == 2 ? e : (fc & 7);
                loc[e] = 64 * x + 8 * (y ^ x) + (z ^ ((5 * y) & 7));
              }
#pragma unroll
              for (int j = 0; j < 32; j++)
                if (n0 + j < p.N) Cw[blk0 + (j >> 3) * gstride + loc[j & 7]] = __uint_as_float(r[j]);
            }
          } else if (p.C32) {
            float* Cf = p.C32 + coff + mo;
            const float af = (float)alpha;
            if (ep.s_n == 1 && beta == 0.0 && af == 1.0f && n0 + 32 <= p.N &&
                ((reinterpret_cast<uintptr_t>(Cf + n0) & 15u) == 0)) {
              // a lane's 32 columns are contiguous: 16-byte stores, 8 per lane instead of 32
              float4* dst = reinterpret_cast<float4*>(Cf + n0);
#pragma unroll
              for (int j = 0; j < 8; j++)
                dst[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                     __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
            } else {
              float old[32];
#pragma unroll
              for (int j = 0; j < 32; j++) old[j] = (beta != 0.0 && n0 + j < p.N) ? Cf[(n0 + j) * ep.s_n] : 0.f;
#pragma unroll
              for (int j = 0; j < 32; j++)
                if (n0 + j < p.N) Cf[(n0 + j) * ep.s_n] = fmaf(af, __uint_as_float(r[j]), old[j]);
            }
          } else if (alpha == 1.0 && (beta == 0.0 || beta == 1.0)) {
            double* Cb = p.C + coff + mo;
            double old[32];
            if (sectors && n0 + 32 <= p.N) {
              // a lane's 32 columns are eight whole sectors.  Written element by element, in
              // quarters of 32 lanes' sectors, the epilogue bounded products with a short K:
              // 25600 x 2560 x 200 took 537 us and takes 293, 4864 x 6144 x 2048 281 and 203
              if (beta != 0.0) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) ld_global4(Cb + n0 + j, old + j);
#pragma unroll
                for (int j = 0; j < 32; j++) old[j] += f32_bits_to_f64(r[j]);
              } else {
#pragma unroll
                for (int j = 0; j < 32; j++) old[j] = f32_bits_to_f64(r[j]);
              }
#pragma unroll
              for (int j = 0; j < 32; j += 4) st_global4(Cb + n0 + j, old[j], old[j + 1], old[j + 2], old[j + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; j++) old[j] = (beta != 0.0 && n0 + j < p.N) ? Cb[(n0 + j) * ep.s_n] : 0.0;
#pragma unroll
              for (int j = 0; j < 32; j++)
                if (n0 + j < p.N) {
                  const double v = f32_bits_to_f64(r[j]);
                  Cb[(n0 + j) * ep.s_n] = beta != 0.0 ? old[j] + v : v;
                }
            }
          } else {
            double* Cb = p.C + coff + mo;
#pragma unroll
            for (int j = 0; j < 32; j++) {
              const int64_t n = n0 + j;
              if (n < p.N) {
                double* cp = Cb + n * ep.s_n;
                const double v = alpha * (double)__uint_as_float(r[j]);
                *cp = (beta == 0.0) ? v : fma(beta, *cp, v);
              }
            }
          }
        }
      }
      fence_before();
      if (CM == 1)
        mbar_arrive(&tempty[acc]);
      else
        mbar_arrive_cluster(map_rank(&tempty[acc], 0));
      if (++acc == 2) {
        acc = 0;
        aphase ^= 1u;
      }
    }
  }
  fence_before();
  __syncthreads();
  // no CTA leaves while MMAs may still read its ring, its peer arrive on its barriers or loads be in flight
  if (CM > 1) {
    cluster_sync();
    pair_drain(full, nst, issued_of, rank, p.fused ? (uint32_t)(2 * A_BYTES) + 2 * b_tile : (uint32_t)A_BYTES + b_tile);
  }
  if (warp == 1) {
    fence_after();
    tmem_dealloc<CM>(tmem, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------
// FP64 GEMM from exact BF16 slices (the error-free splitting of Ozaki, Ogita, Oishi and
// Rump, Numer. Algorithms 59 (2012) 95-118, with base-2^SB digits, SB = 6).
//
// Every operand row r is scaled by 2^-e_r (e_r = ilogb(max_k |x_rk|) + 2, so the scaled
// row lies in (-1/2, 1/2)) and written as S balanced base-2^SB digits,
//   x_rk = 2^e_r sum_{s<S} d_s(r,k) 2^-SB(s+1),  |d_s| <= 2^(SB-1) = 32,
// stored pre-scaled as bf16 slices d_s 2^-SB(s+1) (exact: small integers times a power of
// two).  A product of an A slice s and a B slice t is an integer times 2^-SB(s+t+2), at most
// 2^10 in magnitude, so any sum of up to 2^14 such products with the same s+t is exact in
// the FP32 tensor-memory accumulator.  The kernel therefore accumulates, per output tile,
// "units": for each order g = s+t < gex, every pair (s, g-s) over a K range of at most
// 2^14 / (g+1) elements (exact), and one tail unit with all pairs of order gex..S-1 over the
// whole K range (FP32, its terms are ~2^-SB gex smaller than the leading ones).  The
// epilogue adds each unit into the FP64 output as
//   C[m][n] += alpha 2^(e_m + e_n) acc,
// the first unit of a tile applying beta.  Pairs with s+t >= S are dropped (truncation
// ~2^-SB S relative to max|A_m.| max|B_.n|).  Fewer, wider digits (SB = 7) would need 20 %
// fewer products but 4x more units, and the global read-modify-write of every unit's
// epilogue is what limits this kernel.
// ------------------------------------------------------------------------------------
struct SParams {
  int M, N, kblocks, mtiles, ntiles;
  int bn;              // N tile (a multiple of 32 up to 256): the MMA's N and the B box rows
  int S, gex;          // slices per operand; orders below gex are accumulated exactly
  int a_rows, b_rows;  // rows per slice in the slice arrays (slice s of row r at s * rows + r)
  double alpha, beta;
  double* C;
  GemmEpilogue epi;
  const int* ea;  // row exponents of A and B
  const int* eb;
  int* err;
  int ksplit, kchunk;  // split-K into FP64 partials at C + z*M*N (alpha 1, beta 0)
  int klast;           // sliced_short_kernel: 16-element K steps of the last K block that hold data
};

struct SUnit {
  int g0, g1, kb0, kb1;  // orders [g0, g1], K blocks [kb0, kb1)
};

constexpr int SB = 6;                                           // bits per digit
constexpr int kSlices = 9;  // digits per operand of the full-precision product (9 x 6 = 54 bits)
constexpr int SEXACT_KB = (1 << (24 - 2 * (SB - 1))) / BK;     // K blocks of one pair per exact unit

// K blocks per exact unit of order g: (g+1) pairs x kc blocks x 64 <= 2^(24 - 2(SB-1)) products
__device__ __forceinline__ int sunit_kc(int g) { return max(1, SEXACT_KB / (g + 1)); }

__device__ __forceinline__ int sunit_count(int S, int gex, int kn) {
  int u = gex < S ? 1 : 0;
  for (int g = 0; g < gex; g++) {
    const int kc = sunit_kc(g);
    u += (kn + kc - 1) / kc;
  }
  return u;
}

__device__ __forceinline__ SUnit sunit_at(int S, int gex, int k0, int kn, int u) {
  for (int g = 0; g < gex; g++) {
    const int kc = sunit_kc(g), nu = (kn + kc - 1) / kc;
    if (u < nu) return SUnit{g, g, k0 + u * kc, k0 + min((u + 1) * kc, kn)};
    u -= nu;
  }
  return SUnit{gex, S - 1, k0, k0 + kn};
}

__device__ __forceinline__ int sunit_items(const SUnit& U) {
  int pairs = 0;
  for (int g = U.g0; g <= U.g1; g++) pairs += g + 1;
  return pairs * (U.kb1 - U.kb0);
}

__device__ __forceinline__ double pow2i(int e) {  // 2^e for -1022 <= e <= 1023
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// ring stages of the sliced kernel, of A_BYTES + B_BYTES / cm each
constexpr int sliced_stages(int cm) { return cm == 2 ? 6 : STAGES; }
static_assert(6 * (A_BYTES + B_BYTES / 2) <= STAGES * (A_BYTES + B_BYTES), "the pair's ring fits the same space");
// shared memory of the sliced kernel: the operand ring, barriers, and a 32 x 33 FP32
// transpose buffer per epilogue warp
constexpr size_t SLICED_SMEM_BYTES = SMEM_BYTES + 4 * 32 * 33 * sizeof(float);

// CM = 2: as gemm_kernel<2>, the two CTAs of a cluster work as a pair on neighbouring M tiles,
// each with its own A rows and half of every B slice tile in its ring.  Every slice product of
// a K block is its own ring item, so the shared-memory port sees 96 bytes of fill and 96 of
// operand reads per clock without the pair (two thirds of the MMA rate at best) and 64 and 64
// as a pair; half tiles of B also leave room for six stages instead of four.
template <int CM>
__global__ void __launch_bounds__(THREADS, 1)
    sliced_gemm_kernel(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, SParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * (A_BYTES + B_BYTES));
  uint64_t* empty = full + sliced_stages(2);
  uint64_t* tfull = empty + sliced_stages(2);
  uint64_t* tempty = tfull + 2;
  uint64_t* mdone = tempty + 2;  // every MMA of this CTA has completed (before TMEM is released)
  int64_t* issued_of = (int64_t*)(mdone + 1);  // stages issued by the CTAs of a pair
  uint32_t* tslot = (uint32_t*)(issued_of + 2);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int rank = CM > 1 ? (int)cluster_rank() : 0;
  constexpr int NST = sliced_stages(CM), STAGE = A_BYTES + B_BYTES / CM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 128 * CM);
    }
    mbar_init(mdone, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc<CM>(tslot, TMEM_COLS);
  fence_before();
  __syncthreads();
  fence_after();
  if (CM > 1) cluster_sync();
  const uint32_t tmem = *tslot;
  const int mgroups = (p.mtiles + CM - 1) / CM;
  const int tiles_per = mgroups * p.ntiles;
  const int ntile = tiles_per * (p.ksplit > 1 ? p.ksplit : 1);
  const int cid = blockIdx.x / CM, ncl = gridDim.x / CM;
  const int bh = p.bn / CM;
  // K range of a tile: the whole K, or chunk z of a split-K launch
  auto krange = [&](int tile, int& k0, int& kn) {
    k0 = 0;
    kn = p.kblocks;
    if (p.ksplit > 1) {
      k0 = (tile / tiles_per) * p.kchunk;
      kn = min(p.kblocks - k0, p.kchunk);
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int64_t issued = 0;
      bool ok = true;
      for (int tile = cid; tile < ntile && ok; tile += ncl) {
        int mg, ntl;
        raster(mgroups, p.ntiles, tile % tiles_per, mg, ntl);
        const int m0 = (mg * CM + rank) * BM, n0 = ntl * p.bn + rank * bh;
        int k0, kn;
        krange(tile, k0, kn);
        const int nu = sunit_count(p.S, p.gex, kn);
        for (int u = 0; u < nu && ok; u++) {
          const SUnit U = sunit_at(p.S, p.gex, k0, kn, u);
          for (int g = U.g0; g <= U.g1 && ok; g++)
            for (int s = 0; s <= g && ok; s++)
              for (int kb = U.kb0; kb < U.kb1; kb++) {
                if (!mbar_wait(&empty[stage], phase ^ 1u, p.err)) {
                  ok = false;
                  break;
                }
                uint8_t* st = smem + (size_t)stage * STAGE;
                const int arow = s * p.a_rows + m0, brow = (g - s) * p.b_rows + n0;
                if (rank == 0) mbar_expect_tx(&full[stage], (uint32_t)(CM * A_BYTES + p.bn * BK * 2));
                if (CM == 1) {
                  tma_load(st, &mA, &full[stage], kb * BK, arow);
                  tma_load(st + A_BYTES, &mB, &full[stage], kb * BK, brow);
                } else {
                  const uint32_t fbar = map_rank(&full[stage], 0);
                  tma_load_pair(st, &mA, fbar, kb * BK, arow);
                  tma_load_pair(st + A_BYTES, &mB, fbar, kb * BK, brow);
                }
                ++issued;
                if (++stage == NST) {
                  stage = 0;
                  phase ^= 1u;
                }
              }
        }
      }
      if (rank == 0)
        for (int64_t n = issued > NST ? issued - NST : 0; n < issued; n++)
          mbar_wait_deadline(&full[n % NST], (uint32_t)((n / NST) & 1));
      if (CM > 1) pair_tell(issued_of, rank, issued);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank != 0) {
      mbar_wait_deadline(mdone, 0);
    } else if (lane == 0) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      const uint32_t idesc = idesc_of(CM, p.bn);
      for (int tile = cid; tile < ntile && ok; tile += ncl) {
        int k0, kn;
        krange(tile, k0, kn);
        const int nu = sunit_count(p.S, p.gex, kn);
        for (int u = 0; u < nu && ok; u++) {
          const int items = sunit_items(sunit_at(p.S, p.gex, k0, kn, u));
          if (!mbar_wait(&tempty[acc], aphase ^ 1u, p.err)) {
            ok = false;
            break;
          }
          fence_after();
          const uint32_t d = tmem + (uint32_t)(acc * BN);
          for (int kb = 0; kb < items; kb++) {
            if (!mbar_wait(&full[stage], phase, p.err)) {
              ok = false;
              break;
            }
            fence_after();
            const uint8_t* st = smem + (size_t)stage * STAGE;
            const uint64_t ad = sdesc(st), bd = sdesc(st + A_BYTES);
#pragma unroll
            for (int k = 0; k < BK / 16; k++)
              mma_i<CM>(d, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (kb | k) != 0);
            mma_commit<CM>(&empty[stage]);
            if (++stage == NST) {
              stage = 0;
              phase ^= 1u;
            }
          }
          mma_commit<CM>(&tfull[acc]);
          if (++acc == 2) {
            acc = 0;
            aphase ^= 1u;
          }
        }
      }
      mma_commit<CM>(mdone);  // as in gemm_kernel: no MMA in flight when TMEM is released
      mbar_wait_deadline(mdone, 0);
    }
  } else {
    const int q = warp & 3;
    int acc = 0;
    uint32_t aphase = 0;
    const GemmEpilogue ep = p.epi;
    bool ok = true;
    const int nch = p.bn / 32;
    for (int tile = cid; tile < ntile && ok; tile += ncl) {
      int mg, nt;
      raster(mgroups, p.ntiles, tile % tiles_per, mg, nt);
      const int mt = mg * CM + rank;
      const int64_t coff = p.ksplit > 1 ? (int64_t)(tile / tiles_per) * p.M * p.N : 0;
      int k0, kn;
      krange(tile, k0, kn);
      const int nu = sunit_count(p.S, p.gex, kn);
      const int64_t mw = (int64_t)mt * BM + q * 32;  // first row of this warp
      const int64_t m = mw + lane;
      auto moff = [&](int64_t mm) {
        return ep.msplit ? (mm / ep.msplit) * ep.s_mhi + (mm % ep.msplit) * ep.s_mlo : mm * ep.s_mhi;
      };
      const int64_t mo = moff(m);
      // alpha 2^e_m; the column factor 2^e_n is added to its exponent field (|e| <= 500 and
      // 2^-20 <= |alpha| <= 2^20 keep the result normal)
      const long long sa = m < p.M ? __double_as_longlong(p.alpha * pow2i(p.ea[m])) : 0;
      // lanes run along the rows when those are contiguous in C; otherwise the 32 x 32 block
      // is transposed through shared memory so that lanes run along the columns
      const bool rows_contiguous = ep.msplit == 0 && ep.s_mhi == 1;
      float* tsm = reinterpret_cast<float*>(smem + STAGES * (A_BYTES + B_BYTES) + 256) + (warp - 2) * 32 * 33;
      for (int u = 0; u < nu; u++) {
        if (!mbar_wait(&tfull[acc], aphase, p.err)) {
          ok = false;
          break;
        }
        fence_after();
        const bool first = u == 0;
        const bool load_old = !(first && p.beta == 0.0);
        for (int ch = 0; ch < nch; ch++) {
          uint32_t r[32];
          tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN + ch * 32), r);
          const int64_t n0 = (int64_t)nt * p.bn + ch * 32;
          if (rows_contiguous) {
            if (m < p.M) {
              double* Cb = p.C + coff + mo;
#pragma unroll
              for (int h = 0; h < 32; h += 16) {  // 16 columns at a time: loads in flight together
                double old[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                  old[j] = 0.0;
                  if (n0 + h + j < p.N && load_old) {
                    old[j] = Cb[(n0 + h + j) * ep.s_n];
                    if (first) old[j] *= p.beta;
                  }
                }
#pragma unroll
                for (int j = 0; j < 16; j++)
                  if (n0 + h + j < p.N) {
                    const double f = __longlong_as_double(sa + ((long long)p.eb[n0 + h + j] << 52));
                    Cb[(n0 + h + j) * ep.s_n] = fma(f32_bits_to_f64(r[h + j]), f, old[j]);
                  }
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; j++) tsm[lane * 33 + j] = __uint_as_float(r[j]);
            __syncwarp();
            const int64_t n = n0 + lane;  // this lane's column
            const bool nok = n < p.N;
            const long long ebs = nok ? (long long)p.eb[n] << 52 : 0;
            double* Cn = p.C + coff + n * ep.s_n;
#pragma unroll
            for (int h = 0; h < 32; h += 16) {
              double old[16];
#pragma unroll
              for (int i = 0; i < 16; i++) {
                old[i] = 0.0;
                if (nok && mw + h + i < p.M && load_old) {
                  old[i] = Cn[moff(mw + h + i)];
                  if (first) old[i] *= p.beta;
                }
              }
#pragma unroll
              for (int i = 0; i < 16; i++) {
                const long long sai = __shfl_sync(0xffffffffu, sa, h + i);
                if (nok && mw + h + i < p.M)
                  Cn[moff(mw + h + i)] = fma(f32_bits_to_f64(__float_as_uint(tsm[(h + i) * 33 + lane])),
                                             __longlong_as_double(sai + ebs), old[i]);
              }
            }
            __syncwarp();
          }
        }
        fence_before();
        if (CM == 1)
          mbar_arrive(&tempty[acc]);
        else
          mbar_arrive_cluster(map_rank(&tempty[acc], 0));
        if (++acc == 2) {
          acc = 0;
          aphase ^= 1u;
        }
      }
    }
  }
  fence_before();
  __syncthreads();
  if (CM > 1) {  // as in gemm_kernel
    cluster_sync();
    pair_drain(full, NST, issued_of, rank, (uint32_t)(A_BYTES + bh * BK * 2));
  }
  if (warp == 1) {
    fence_after();
    tmem_dealloc<CM>(tmem, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------
// The same product for a short K (at most kShortK elements): the accumulators of all S orders of
// a 128 x SN tile stay in tensor memory (at most nine of SN columns), so a K block's slices of
// both operands are loaded once for all its S (S + 1) / 2 products, and the output is written
// once, not once per order.  The ring kernel above reads an A and a B tile from L2 for each
// product and passes over C eight times; at K = 256 the passes (FP64 multiply-adds on a pipe of
// two per clock, a trip to memory each) took ten times the products' time.
//
// An MMA of 128 rows takes 130 to 150 clocks however few columns it has (measured with SN = 32
// and 64), so one MMA does several slices of B: they lie one after the other in shared memory,
// 128 SN bytes each, and A slice s times slices t0 .. t1 of B as one operand of (t1 - t0 + 1) SN
// rows lands in the columns of orders s + t0 .. s + t1, which are neighbours too.  SN = 48 (two
// groups of 4 and 5 slices, 14 MMAs for 45 products), 32 (8 and 1) or 16 (all nine at once).
//
// The epilogue needs no FP64 operation but the add onto an old value: the accumulators are
// integers below 2^22 in units of 2^-SB(g+2) (K (g+1) 2^10).  A 64-bit integer sum of them, in
// quarters of the last order but one's unit (2^-56 of the row and column maxima's product at
// nine digits; below 448 2^54 of those), is turned into a double by its bit fields.  All
// accumulators of a tile are read and released before C is touched, so the writes overlap the
// next tile's products.
//
// Every slice has its own slot and barriers.  A K block's products run by rows, A slice s with B
// slices 0 .. S-1-s, from s = S-1 down: A slices free up one by one and are loaded again under
// the rest.  All B slices are in use until row 0 ends, so the ones that the next K block begins
// with (all of them where they fit, the first four at SN = 48) have two slots.
//
// Measured (kernel alone, nine digits): 8192 x 8192 x 256 1.56 ms (2.81 with one MMA per
// product), 200000 x 16 x 160 0.14 ms (0.42; 0.56 on the ring kernel); a K block takes 8.7
// thousand clocks where its 56 MMAs need 7.2.
// ------------------------------------------------------------------------------------
constexpr int kShortK = 448, kShortThreads = 64 + 512;
constexpr int short_double(int sn) { return sn == 48 ? 4 : kSlices; }  // B slices with two slots
constexpr int short_group(int sn) { return sn == 48 ? 4 : 256 / sn; }  // B slices of the first MMA of a row
constexpr size_t short_smem(int sn) {
  return 1024 + (size_t)kSlices * A_BYTES + (size_t)(kSlices + short_double(sn)) * sn * BK * 2 + 768;
}
static_assert(short_smem(48) <= 227 * 1024 && short_smem(32) <= 227 * 1024, "nine slices of both operands");
static_assert((kSlices - short_group(48)) * 48 <= 256, "the second group is one MMA");

// V 2^e as a double (round to nearest, ties away), integer operations only while the result
// is a normal number
__device__ __forceinline__ double fixed_to_f64(long long v, int e) {
  if (v == 0) return 0.0;
  const unsigned long long u = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = __clzll((long long)u);
  const unsigned long long m = u << lz, sgn = (unsigned long long)v & 0x8000000000000000ull;
  const unsigned long long mant = (m >> 11) + ((m >> 10) & 1ull);  // 2^52 .. 2^53: adds 1 (or 2) to the exponent
  const int ex = 1022 + 63 - lz + e;
  if (ex > 0 && ex < 2045) return __longlong_as_double((long long)(sgn | (((unsigned long long)ex << 52) + mant)));
  const double d = __longlong_as_double((long long)(sgn | ((1022ull << 52) + mant)));  // times 2^(63 - lz + e)
  const int h = (63 - lz + e) / 2;
  return d * pow2i(h) * pow2i(63 - lz + e - h);
}

template <int SN>
__global__ void __launch_bounds__(kShortThreads, 1)
    sliced_short_kernel(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB, SParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int kB = SN * BK * 2, DB = short_double(SN), G0 = short_group(SN);
  constexpr int NBUF = 2 * kSlices * SN <= 512 ? 2 : 1;  // two sets of accumulators where they fit
  uint8_t* sA = smem;
  uint8_t* sB = smem + kSlices * A_BYTES;
  uint64_t* fullA = (uint64_t*)(sB + (kSlices + DB) * kB);
  uint64_t* fullB = fullA + kSlices;  // by slot: slice t < DB of K block n at t + (n & 1) DB, else DB + t
  uint64_t* emptyA = fullB + 2 * kSlices;
  uint64_t* emptyB = emptyA + kSlices;
  uint64_t* tfull = emptyB + 2 * kSlices;
  uint64_t* tempty = tfull + 2;
  uint64_t* mdone = tempty + 2;
  uint32_t* tslot = (uint32_t*)(mdone + 1);
  // slot of slice t in the CTA's K block n, and the parity of the slot's use there
  auto bslot = [](int t, uint32_t n) { return t < DB ? t + (int)(n & 1u) * DB : DB + t; };
  auto bpar = [](int t, uint32_t n) { return (t < DB ? n >> 1 : n) & 1u; };
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, S = p.S;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSlices; s++) {
      mbar_init(&fullA[s], 1);
      mbar_init(&emptyA[s], 1);
    }
    for (int s = 0; s < kSlices + DB; s++) {
      mbar_init(&fullB[s], 1);
      mbar_init(&emptyB[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 512);
    }
    mbar_init(mdone, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc<1>(tslot, 512);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tslot;
  const int ntile = p.mtiles * p.ntiles;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t n = 0;  // K blocks of this CTA so far, over all its tiles
      bool ok = true;
      int part = 0;    // loads of K block n that were issued (fewer than 2 S only after an error)
      for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
        int mt, nt;
        raster(p.mtiles, p.ntiles, tile, mt, nt);
        for (int kb = 0; kb < p.kblocks && ok; kb++) {
          part = 0;
          for (int i = 0; i < S; i++) {  // A slice S-1-i and B slice i in the order of their first use
            const int s = S - 1 - i, bs = bslot(i, n);
            if (!(ok = mbar_wait(&emptyA[s], (n & 1u) ^ 1u, p.err))) break;
            mbar_expect_tx(&fullA[s], A_BYTES);
            tma_load(sA + s * A_BYTES, &mA, &fullA[s], kb * BK, s * p.a_rows + mt * BM);
            part++;
            if (!(ok = mbar_wait(&emptyB[bs], bpar(i, n) ^ 1u, p.err))) break;
            mbar_expect_tx(&fullB[bs], (uint32_t)kB);
            tma_load(sB + bs * kB, &mB, &fullB[bs], kb * BK, i * p.b_rows + nt * SN);
            part++;
          }
          if (ok) n++;
        }
      }
      if (!ok) {
        // the loads in flight must land before the CTA exits: a slot's last load is that of the
        // broken K block n (the first `part` of its loads), or the one before it in that slot
        for (int i = 0; i < S; i++) {
          const int s = S - 1 - i;
          const bool a = 2 * i < part, b = 2 * i + 1 < part;
          if (a || n >= 1) mbar_wait_deadline(&fullA[s], (a ? n : n - 1) & 1u);
          const uint32_t gap = i < DB ? 2 : 1;  // K blocks between two uses of a B slot
          if (b || n >= gap) mbar_wait_deadline(&fullB[bslot(i, n)], bpar(i, b ? n : n - gap));
          if (i < DB && n >= 1) mbar_wait_deadline(&fullB[bslot(i, n - 1)], bpar(i, n - 1));
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t n = 0, aphase = 0;
      int buf = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < ntile && ok; tile += gridDim.x) {
        if (!mbar_wait(&tempty[buf], aphase ^ 1u, p.err)) break;
        fence_after();
        const uint32_t d0 = tmem + (uint32_t)(buf * kSlices * SN);
        for (int kb = 0; kb < p.kblocks && ok; kb++, n++) {
          const int ksteps = kb == p.kblocks - 1 ? p.klast : BK / 16;
          for (int s = S - 1; s >= 0; s--) {
            const int cnt = S - s;  // B slices of this row; order s + t of the tile in columns (s + t) SN
            if (!(ok = mbar_wait(&fullA[s], n & 1u, p.err) &&
                       mbar_wait(&fullB[bslot(cnt - 1, n)], bpar(cnt - 1, n), p.err)))
              break;
            fence_after();
            const uint64_t ad = sdesc(sA + s * A_BYTES);
            for (int t0 = 0; t0 < cnt; t0 += t0 == 0 ? G0 : kSlices) {
              const int nt = min(cnt - t0, t0 == 0 ? G0 : kSlices);
              const uint64_t bd = sdesc(sB + bslot(t0, n) * kB);
              const uint32_t d = d0 + (uint32_t)((s + t0) * SN);
              for (int k = 0; k < ksteps; k++) {
                if (kb == 0 && k == 0 && t0 == 0) {  // order s begins here, the later ones have begun
                  mma_i(d, ad, bd, idesc_of(1, SN), 0u);
                  if (nt > 1)
                    mma_i(d + (uint32_t)SN, ad, bd + (uint64_t)(kB >> 4), idesc_of(1, (nt - 1) * SN), 1u);
                } else {
                  mma_i(d, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc_of(1, nt * SN), 1u);
                }
              }
              if (s == 0)
                for (int t = t0; t < t0 + nt; t++) mma_commit(&emptyB[bslot(t, n)]);
            }
            mma_commit(&emptyA[s]);
          }
        }
        if (!ok) break;
        mma_commit(&tfull[buf]);
        if (++buf == NBUF) {
          buf = 0;
          aphase ^= 1u;
        }
      }
      mma_commit(mdone);  // no MMA in flight when TMEM is released
      mbar_wait_deadline(mdone, 0);
    }
  } else {
    // warps 2 .. 17: the tile's rows of lane quarter q, SN / 4 columns each
    const int q = warp & 3, part = (warp - 2) / 4, lsb = -SB * S - 2;
    constexpr int NC = SN / 4;
    uint32_t aphase = 0;
    int buf = 0;
    const GemmEpilogue ep = p.epi;
    // a power-of-two alpha goes into the exponent
    const long long ab = __double_as_longlong(p.alpha);
    const bool apow2 = (ab & 0xFFFFFFFFFFFFFll) == 0;
    const int aexp = apow2 ? (int)((ab >> 52) & 0x7FF) - 1023 : 0;
    const bool rows_contiguous = ep.msplit == 0 && ep.s_mhi == 1;
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
      int mt, nt;
      raster(p.mtiles, p.ntiles, tile, mt, nt);
      if (!__all_sync(0xffffffffu, mbar_wait(&tfull[buf], aphase, p.err))) break;
      fence_after();
      long long v[NC];
      // n = acc 2^(SB (g + 2)), exact, by adding 1.5 2^23
      auto whole = [&](uint32_t x, int g) {
        const float sc = __int_as_float((127 + SB * (g + 2)) << 23);
        return __float_as_int(fmaf(__uint_as_float(x), sc, 12582912.f)) - 0x4B400000;
      };
#pragma unroll
      for (int c0 = 0; c0 < NC; c0 += 4) {
        const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * kSlices * SN + part * NC + c0);
        uint32_t r[kSlices][4];  // by order from the last one, r[0]; orders that fewer digits lack stay unread
#pragma unroll
        for (int u = 0; u < kSlices; u++)
          if (u < S) tmem_ld4(base + (uint32_t)((S - 1 - u) * SN), r[u]);
        tmem_wait();
        // orders in pairs from the most significant: w = 2^SB n_hi + n_lo in 32 bits, then 64-bit
        // sums; the pairs end at the last order but one, then the last in quarters of its unit
#pragma unroll
        for (int j = 0; j < 4; j++) {
          long long x = 0;
#pragma unroll
          for (int u = 8; u >= 2; u -= 2) {
            int w = 0;
            if (u < S) w = whole(r[u][j], S - 1 - u) * (1 << SB);
            if (u - 1 < S) w += whole(r[u - 1][j], S - u);
            x = u == 8 ? (long long)w : x * (1ll << (2 * SB)) + w;
          }
          v[c0 + j] = x * 4 + ((whole(r[0][j], S - 1) + 8) >> 4);
        }
      }
      fence_before();
      mbar_arrive(&tempty[buf]);
      if (++buf == NBUF) {
        buf = 0;
        aphase ^= 1u;
      }
      const int64_t m = (int64_t)mt * BM + q * 32 + lane, n0 = (int64_t)nt * SN + part * NC;
      if (m < p.M && n0 < p.N) {
        const int em = p.ea[m] + lsb + aexp;
        const int ncol = (int)(p.N - n0 < NC ? p.N - n0 : NC);
        double* Cm = p.C + (ep.msplit ? (m / ep.msplit) * ep.s_mhi + (m % ep.msplit) * ep.s_mlo : m * ep.s_mhi) +
                     n0 * ep.s_n;
        auto value = [&](int j) {
          const double d = fixed_to_f64(v[j], em + p.eb[n0 + j]);
          return apow2 ? (ab < 0 ? -d : d) : p.alpha * d;
        };
        if (!rows_contiguous && ep.s_n == 1 && ncol == NC && ((uintptr_t)Cm & 15) == 0) {
          double2* C2 = reinterpret_cast<double2*>(Cm);  // a lane's columns are contiguous: 16-byte accesses
          double2 old[NC / 2];
          if (p.beta != 0.0) {
#pragma unroll
            for (int j = 0; j < NC / 2; j++) old[j] = C2[j];
          }
#pragma unroll
          for (int j = 0; j < NC / 2; j++) {
            double2 x = make_double2(value(2 * j), value(2 * j + 1));
            if (p.beta == 1.0) {
              x.x += old[j].x;
              x.y += old[j].y;
            } else if (p.beta != 0.0) {
              x.x = fma(p.beta, old[j].x, x.x);
              x.y = fma(p.beta, old[j].y, x.y);
            }
            C2[j] = x;
          }
        } else {
          double old[NC];
#pragma unroll
          for (int j = 0; j < NC; j++) old[j] = p.beta != 0.0 && j < ncol ? Cm[j * ep.s_n] : 0.0;
#pragma unroll
          for (int j = 0; j < NC; j++)
            if (j < ncol) {
              const double x = value(j);
              Cm[j * ep.s_n] = p.beta == 0.0 ? x : p.beta == 1.0 ? old[j] + x : fma(p.beta, old[j], x);
            }
        }
      }
      __syncwarp();
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    tmem_dealloc<1>(tmem, 512);
  }
}

__device__ __forceinline__ bool mv_kcontig(const MatView& v) { return (v.ksplit ? v.ks_lo : v.ks_hi) == 1; }

// Offsets of 32 rows and 64 columns of an operand: one division per element of the two index
// lists instead of up to two per matrix element, which bounded the passes below.
struct TileOffsets {
  int64_t r[32], k[64];
};
__device__ __forceinline__ int64_t mv_off(int64_t i, int64_t split, int64_t hi, int64_t lo) {
  if (!split) return i * hi;
  const uint32_t s = (uint32_t)min(split, (int64_t)INT32_MAX), q = (uint32_t)i / s;  // extents are below 2^31
  return (int64_t)q * hi + (int64_t)((uint32_t)i - q * s) * lo;
}
__device__ __forceinline__ void row_offsets(const MatView& x, int64_t r0, TileOffsets& o, int tid) {
  if (tid < 32) o.r[tid] = mv_off(r0 + tid, x.rsplit, x.rs_hi, x.rs_lo);
}
__device__ __forceinline__ void col_offsets(const MatView& x, int64_t k0, int64_t* k, int tid) {
  if (tid >= 64 && tid < 128) k[tid - 64] = mv_off(k0 + tid - 64, x.ksplit, x.ks_hi, x.ks_lo);
}

// row maxima |x| of a rows x cols FP64 view as bit patterns (non-negative doubles order
// like their bits, so the maximum is an integer one); block (x, y) covers 32 rows and the
// K range [x kchunk, (x+1) kchunk) (kchunk a multiple of 64), lanes along k (sk == 1) or along
// the rows (transposed views), and merges into amax (zeroed by the caller) with one atomicMax
// per row; a single chunk writes its rows' maxima.  Reading bounds it, with eight loads per
// thread in flight: 6.6e6 elements (rows and columns of two strided runs) take 20 us, and took
// 48 us with divisions for each element and K chunks of 1024.
__global__ void slice_absmax_kernel(MatView x, int64_t kchunk, unsigned long long* amax) {
  chain_enter();
  constexpr int kCols = 512;  // columns of an offset list
  __shared__ unsigned long long t[8][32];
  __shared__ int64_t ro[32], ko[kCols];
  const bool single = gridDim.x == 1, kc = mv_kcontig(x);
  const int64_t r0 = (int64_t)blockIdx.y * 32, k0 = (int64_t)blockIdx.x * kchunk;
  const int64_t k1 = min(x.cols, k0 + kchunk);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
  const int nr = (int)min((int64_t)32, x.rows - r0);
  const unsigned long long absmask = 0x7FFFFFFFFFFFFFFFull;
  if (tid < 32) ro[tid] = mv_off(r0 + tid, x.rsplit, x.rs_hi, x.rs_lo);
  unsigned long long mm[4] = {0, 0, 0, 0};
  for (int64_t kt = k0; kt < k1; kt += kCols) {
    const int nk = (int)min((int64_t)kCols, k1 - kt);
    __syncthreads();
    for (int j = tid; j < nk; j += 256) ko[j] = mv_off(kt + j, x.ksplit, x.ks_hi, x.ks_lo);
    __syncthreads();
#pragma unroll 2
    for (int j0 = 0; j0 < nk; j0 += 64) {
      unsigned long long v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int i = kc ? ty + 8 * (q / 2) : tx, j = j0 + (kc ? tx + 32 * (q % 2) : ty + 8 * q);
        v[q] = i < nr && j < nk ? (unsigned long long)__double_as_longlong(x.p[ro[i] + ko[j]]) & absmask : 0;
      }
#pragma unroll
      for (int q = 0; q < 8; q++) mm[q / 2] = max(mm[q / 2], v[q]);
    }
  }
  if (kc) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = ty + 8 * q;
      for (int o = 16; o > 0; o >>= 1) mm[q] = max(mm[q], __shfl_xor_sync(0xffffffffu, mm[q], o));
      if (tx == 0 && i < nr) {
        if (single)
          amax[r0 + i] = mm[q];
        else if (mm[q])
          atomicMax(amax + r0 + i, mm[q]);
      }
    }
  } else {
    t[ty][tx] = max(max(mm[0], mm[1]), max(mm[2], mm[3]));
    __syncthreads();
    if (ty == 0 && tx < nr) {
      unsigned long long m = t[0][tx];
      for (int i = 1; i < 8; i++) m = max(m, t[i][tx]);
      if (single)
        amax[r0 + tx] = m;
      else if (m)
        atomicMax(amax + r0 + tx, m);
    }
  }
}

// The 32 x 64 tile at (r0, k0) of an operand in pairs of neighbouring columns: v0[q], v1[q] are
// elements (ty + 8 q, 2 tx) and (ty + 8 q, 2 tx + 1), zero outside the matrix.  Rows with unit
// stride are read directly, others along the rows, through shared memory; either way a
// thread's eight loads are in flight together.  The split of 6.6e6 elements into two parts took
// 39 us (2 TB/s) with a division or two per element, one load at a time ahead of its shared
// store, and an FP64-pipe conversion per element; it takes 20 us.  The slicing into nine digits
// took 40 us and takes 34 us (5 TB/s).
struct TileStage {
  TileOffsets off;
  double t[32][65];
};
__device__ __forceinline__ void load_pairs(TileStage& s, const MatView& x, int64_t r0, int64_t k0, double (&v0)[4],
                                           double (&v1)[4]) {
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
  row_offsets(x, r0, s.off, tid);
  col_offsets(x, k0, s.off.k, tid);
  __syncthreads();
  const int nr = (int)min((int64_t)32, x.rows - r0), nk = (int)min((int64_t)64, x.cols - k0);
  if (mv_kcontig(x)) {
    const int64_t c0 = s.off.k[2 * tx], c1 = s.off.k[2 * tx + 1];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = ty + 8 * q;
      v0[q] = i < nr && 2 * tx < nk ? x.p[s.off.r[i] + c0] : 0.0;
      v1[q] = i < nr && 2 * tx + 1 < nk ? x.p[s.off.r[i] + c1] : 0.0;
    }
  } else {
    const double* p = x.p + s.off.r[tx];
    double v[8];  // all eight loads before the first store, which might alias them
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = tx < nr && ty + 8 * q < nk ? p[s.off.k[ty + 8 * q]] : 0.0;
#pragma unroll
    for (int q = 0; q < 8; q++) s.t[tx][ty + 8 * q] = v[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) v0[q] = s.t[ty + 8 * q][2 * tx], v1[q] = s.t[ty + 8 * q][2 * tx + 1];
  }
}

// row exponent from the row maximum: e = ilogb(max) + 2 (max/2^e in [1/4, 1/2)), clamped
// below at -500; a row maximum >= 2^498 sets *range (the caller falls back to FP64)
__device__ __forceinline__ int slice_exponent(unsigned long long bits, int* range) {
  const int be = (int)((bits >> 52) & 0x7FF);
  if (be == 0) return -500;  // zero or subnormal row maximum
  const int e = be - 1023 + 2;
  if (e > 500) {
    atomicExch(range, 1);
    return 500;
  }
  return max(e, -500);
}

// x 2^(bits-e) rounded to an integer (|result| < 2^(bits-1) since |x| < 2^(e-1); bits <= 56),
// from the bit fields of x with integer operations only
__device__ __forceinline__ long long slice_fixed(double x, int e, int bits) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int E = (int)((b >> 52) & 0x7FF);
  const long long mant = (long long)(b & 0xFFFFFFFFFFFFFull) | (E ? (1ll << 52) : 0ll);
  const int shift = max(E, 1) - 1075 + bits - e;  // x = mant 2^(max(E,1) - 1075)
  long long v;
  if (shift >= 0)
    v = mant << shift;
  else if (shift > -63)
    v = (mant + (1ll << (-shift - 1))) >> (-shift);
  else
    v = 0;
  return (b >> 63) ? -v : v;
}

// digits: slices[s][r][k] = bf16(d_s 2^-SB(s+1)) for r < rows_p (zero past rows), k < kp
// (zero past cols), the balanced base-2^SB digits of x 2^(SB S - e) (least significant s = S-1);
// e[r] written by the blocks of the first K tile.  32 x 64 tiles through shared memory:
// reads coalesced along whichever stride is 1; each thread then slices two neighbouring
// elements of a row and stores each digit pair as one bf16x2 (a warp writes 128
// contiguous bytes of a slice plane per store; kp is a multiple of 64).
__global__ void slice_digits_kernel(MatView x, int64_t rows_p, int64_t kp, const unsigned long long* amax, int S,
                                    __nv_bfloat16* slices, int* e_out, int* range) {
  chain_enter();
  __shared__ TileStage st;
  const int64_t rows = x.rows, r0 = (int64_t)blockIdx.y * 32, k0 = (int64_t)blockIdx.x * 64;
  const int tx = threadIdx.x, ty = threadIdx.y;
  double v0[4], v1[4];
  load_pairs(st, x, r0, k0, v0, v1);
  const size_t plane2 = (size_t)rows_p * kp / 2;  // a slice plane in bf16 pairs
  constexpr int H = 1 << (SB - 1);
#pragma unroll
  for (int q4 = 0; q4 < 4; q4++) {
    const int64_t r = r0 + ty + 8 * q4, k = k0 + 2 * tx;
    if (r >= rows_p) continue;
    const int e = r < rows ? slice_exponent(amax[r], range) : 0;
    if (k == 0 && r < rows) e_out[r] = e;
    long long X0 = r < rows ? slice_fixed(v0[q4], e, SB * S) : 0;
    long long X1 = r < rows ? slice_fixed(v1[q4], e, SB * S) : 0;
    __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(slices + (size_t)r * kp + k);
    // digit s (|d| <= 2^(SB-1)): a 32-bit conversion, exact, and exact in bf16 after the
    // power-of-2 scale
    // (the sum 1.5 2^23 + d as bits, scaled and shifted by one exact FMA: an integer conversion
    // runs at a quarter of the rate)
    auto put = [&](int s, int d0, int d1) {
      const float sc = __int_as_float((127 - SB * (s + 1)) << 23), off = -12582912.0f * sc;
      dst[(size_t)s * plane2] = __floats2bfloat162_rn(fmaf(__int_as_float(0x4B400000 + d0), sc, off),
                                                      fmaf(__int_as_float(0x4B400000 + d1), sc, off));
    };
    if (S >= 6) {
      // balanced digits in 32-bit arithmetic: the low 30 bits hold the 5 least significant
      // digits, whose carry out (0 or 1) joins the high part for the other S - 5
      int lo0 = (int)(X0 & 0x3FFFFFFFll), hi0 = (int)(X0 >> 30);
      int lo1 = (int)(X1 & 0x3FFFFFFFll), hi1 = (int)(X1 >> 30);
      int s = S - 1;
      for (int q = 0; q < 5; q++, s--) {
        const int d0 = ((lo0 + H) & (2 * H - 1)) - H, d1 = ((lo1 + H) & (2 * H - 1)) - H;  // in [-H, H)
        lo0 = (lo0 - d0) >> SB;
        lo1 = (lo1 - d1) >> SB;
        put(s, d0, d1);
      }
      hi0 += lo0;
      hi1 += lo1;
      for (; s > 0; s--) {
        const int d0 = ((hi0 + H) & (2 * H - 1)) - H, d1 = ((hi1 + H) & (2 * H - 1)) - H;
        hi0 = (hi0 - d0) >> SB;
        hi1 = (hi1 - d1) >> SB;
        put(s, d0, d1);
      }
      put(0, hi0, hi1);  // what remains: |d| <= H
    } else {
      for (int s = S - 1; s >= 0; s--) {
        long long d0, d1;
        if (s > 0) {
          d0 = ((X0 + H) & (2 * H - 1)) - H;  // balanced digit in [-H, H)
          d1 = ((X1 + H) & (2 * H - 1)) - H;
          X0 = (X0 - d0) >> SB;
          X1 = (X1 - d1) >> SB;
        } else {
          d0 = X0;  // what remains: |d| <= H
          d1 = X1;
        }
        put(s, (int)d0, (int)d1);
      }
    }
  }
}

// FP64 rows x cols view (strides sr, sk) -> bf16 hi/lo [rows][kp], zero padded to kp
// (mid != null: three parts, x = hi + mid + lo, each the bf16 rounding of what remains)
// 32 x 64 tiles through shared memory: reads coalesced along whichever stride is 1 (sk == 1:
// along k, otherwise along the rows); each thread splits two neighbouring elements of a row
// and stores each part as one bf16x2 (128 contiguous bytes per warp store; kp is a
// multiple of 64).  Two parts are formed in FP32 (x truncated to FP32 first, from its bit
// fields: 2^-23, far below the lo part's 2^-17), three parts in FP64.
__global__ void __launch_bounds__(256, 6) split_kernel(MatView x, int64_t kp, __nv_bfloat16* hi, __nv_bfloat16* lo, __nv_bfloat16* mid) {
  chain_enter();
  __shared__ TileStage st;
  const int64_t rows = x.rows, k0 = (int64_t)blockIdx.x * 64;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int64_t r0 = (int64_t)blockIdx.y * 32; r0 < rows; r0 += (int64_t)gridDim.y * 32) {  // row tiles
  __syncthreads();
  double w0[4], w1[4];
  load_pairs(st, x, r0, k0, w0, w1);
#pragma unroll
  for (int q4 = 0; q4 < 4; q4++) {
    const int64_t r = r0 + ty + 8 * q4, k = k0 + 2 * tx;
    if (r >= rows) continue;
    const int64_t o2 = (r * kp + k) / 2;  // bf16 pair index
    const double v0 = w0[q4], v1 = w1[q4];
    if (mid) {
      const __nv_bfloat16 h0 = __double2bfloat16(v0), h1 = __double2bfloat16(v1);
      double r0d = v0 - (double)__bfloat162float(h0), r1d = v1 - (double)__bfloat162float(h1);
      const __nv_bfloat16 m0 = __double2bfloat16(r0d), m1 = __double2bfloat16(r1d);
      r0d -= (double)__bfloat162float(m0);
      r1d -= (double)__bfloat162float(m1);
      reinterpret_cast<__nv_bfloat162*>(hi)[o2] = __halves2bfloat162(h0, h1);
      reinterpret_cast<__nv_bfloat162*>(mid)[o2] = __halves2bfloat162(m0, m1);
      reinterpret_cast<__nv_bfloat162*>(lo)[o2] = __halves2bfloat162(__double2bfloat16(r0d), __double2bfloat16(r1d));
    } else {
      const float f0 = f64_to_f32_trunc(v0), f1 = f64_to_f32_trunc(v1);
      const __nv_bfloat16 h0 = __float2bfloat16_rn(f0), h1 = __float2bfloat16_rn(f1);
      reinterpret_cast<__nv_bfloat162*>(hi)[o2] = __halves2bfloat162(h0, h1);
      reinterpret_cast<__nv_bfloat162*>(lo)[o2] =
          __halves2bfloat162(__float2bfloat16_rn(f0 - __bfloat162float(h0)), __float2bfloat16_rn(f1 - __bfloat162float(h1)));
    }
  }
  }
}

// The bounded-wait path of the pipelines above, exercised on its own: thread 0 waits, with
// the same mbar_wait and the given limit, on a barrier that nothing arrives on, so the wait
// runs out, raises the error flag and the kernel returns; the host then sees the flag
// exactly as after a stalled GEMM pipeline.
__global__ void wait_selftest_kernel(int* err, unsigned long long limit_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait(&bar, 0, err, limit_ns);
}

// ------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------
struct Split {
  __nv_bfloat16* hi = nullptr;
  __nv_bfloat16* lo = nullptr;
  __nv_bfloat16* mid = nullptr;  // three-part splits only
  std::unique_ptr<Scratch> tmp;  // storage of a temporary (non-constant) operand
  int64_t rows = 0, kp = 0;
  CUtensorMap mhi, mlo, mmid;  // tensor maps of the last box_rows asked for (maps_for)
  int map_rows = 0;
  ~Split() {
    if (tmp) return;
    if (hi) cudaFree(hi);
    if (lo) cudaFree(lo);
    if (mid) cudaFree(mid);
  }
};

// an operand as S exact bf16 slices [S][rows_p][kp] with row exponents (sliced FP64 GEMM)
struct Sliced {
  __nv_bfloat16* d = nullptr;
  int* e = nullptr;
  std::unique_ptr<Scratch> tmp;  // storage of a temporary (non-constant) operand
  int64_t rows = 0, rows_p = 0, kp = 0;
  int S = 0;
  CUtensorMap map;  // for boxes of map_rows rows (slice_map)
  int map_rows = 0;
  ~Sliced() {
    if (!tmp) {
      if (d) cudaFree(d);
      if (e) cudaFree(e);
    }
  }
};

// an operand of the caches: the view (pointer, shape, strides), the box rows and the parts
using Key = std::tuple<const double*, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int, int>;
static Key make_key(const MatView& v, int box_rows, int parts) {
  return Key{v.p, v.rows, v.cols, v.rsplit, v.rs_hi, v.rs_lo, v.ksplit, v.ks_hi, v.ks_lo, box_rows, parts};
}
struct Triples;
struct Cache {
  std::map<Key, std::unique_ptr<Split>> ops;
  std::map<Key, std::unique_ptr<Sliced>> sliced;
  int* range = nullptr;    // device flag: a sliced operand row maximum beyond the range (sticky)
  int* pinned = nullptr;   // host copies of err and range (tc_check)
  bool unchecked = false;  // launches since the last check
  bool sattr_set = false;
  int max_pairs_sliced = 0;  // clusters of two sliced_gemm_kernel CTAs resident at once
  std::shared_ptr<Triples> triples;
  int* err = nullptr;
  int sms = 0;
  bool attr_set = false;
  int max_pairs = 0;  // clusters of two gemm_kernel CTAs resident at once
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  ~Cache() {
    if (err) cudaFree(err);  // err and range share one allocation
    if (pinned) cudaFreeHost(pinned);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
  }
};

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* f = nullptr;
    UCC_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q));
    UCC_REQUIRE(q == cudaDriverEntryPointSuccess && f, UCC_CUDA_ERROR, "cuTensorMapEncodeTiled unavailable");
    fn = (PFN_cuTensorMapEncodeTiled_v12000)f;
  }
  return fn;
}

static void make_map(CUtensorMap* m, void* base, int64_t rows, int64_t kp, int box_rows) {
  cuuint64_t dims[2] = {(cuuint64_t)kp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)kp * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  CUresult r = encode_fn()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  UCC_REQUIRE(r == CUDA_SUCCESS, UCC_CUDA_ERROR, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
}

static Cache& cache(Ctx& c) {
  if (!c.tc_cache) {
    auto* k = new Cache;
    c.tc_cache = std::shared_ptr<void>(k, [](void* p) { delete static_cast<Cache*>(p); });
    UCC_CUDA(cudaMalloc(&k->err, 2 * sizeof(int)));
    UCC_CUDA(cudaMemset(k->err, 0, 2 * sizeof(int)));
    k->range = k->err + 1;
    UCC_CUDA(cudaMallocHost(&k->pinned, 2 * sizeof(int)));
    k->pinned[0] = k->pinned[1] = 0;
    UCC_CUDA(cudaDeviceGetAttribute(&k->sms, cudaDevAttrMultiProcessorCount, c.device));
    UCC_CUDA(cudaEventCreate(&k->ev0));
    UCC_CUDA(cudaEventCreate(&k->ev1));
  }
  return *static_cast<Cache*>(c.tc_cache.get());
}

// the operand's tensor maps for boxes of box_rows x 64
static Split* maps_for(Split* s, int box_rows, int parts) {
  if (s->map_rows != box_rows) {
    make_map(&s->mhi, s->hi, s->rows, s->kp, box_rows);
    make_map(&s->mlo, s->lo, s->rows, s->kp, box_rows);
    if (parts == 3) make_map(&s->mmid, s->mid, s->rows, s->kp, box_rows);
    s->map_rows = box_rows;
  }
  return s;
}

// split (and cache when the source is a constant block) a rows x cols FP64 operand
static Split* prepare(Ctx& c, const MatView& x, int box_rows, std::unique_ptr<Split>& temp, int parts = 2) {
  Cache& k = cache(c);
  const bool constant = c.is_constant(x.p);
  const int64_t rows = x.rows, cols = x.cols;
  UCC_REQUIRE(rows < INT32_MAX && cols < INT32_MAX, UCC_BAD_ARGS, "tensor-core GEMM: operand too large");
  // the split data does not depend on the box a launch reads it with (maps_for)
  const Key key = make_key(x, 0, parts);
  if (constant) {
    auto it = k.ops.find(key);
    if (it != k.ops.end()) return maps_for(it->second.get(), box_rows, parts);
  }
  auto s = std::make_unique<Split>();
  s->rows = rows;
  s->kp = (cols + BK - 1) / BK * BK;
  const size_t plane = sizeof(__nv_bfloat16) * rows * s->kp;  // a multiple of 128 bytes
  if (constant) {
    UCC_CUDA(cudaMalloc(&s->hi, plane));
    UCC_CUDA(cudaMalloc(&s->lo, plane));
    if (parts == 3) UCC_CUDA(cudaMalloc(&s->mid, plane));
  } else {  // stream-ordered pool: no device synchronisation per temporary
    s->tmp = std::make_unique<Scratch>(c, plane * (parts == 3 ? 3 : 2));
    s->hi = static_cast<__nv_bfloat16*>(s->tmp->p);
    s->lo = reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(s->tmp->p) + plane);
    if (parts == 3) s->mid = reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(s->tmp->p) + 2 * plane);
  }
  launch_chained(split_kernel, dim3((unsigned)(s->kp / 64), (unsigned)std::min<int64_t>((rows + 31) / 32, 65535)),
                 dim3(32, 8), c.stream, 1, x, s->kp, s->hi, s->lo, s->mid);
  count_kernel_launch();
  UCC_CUDA(cudaGetLastError());
  maps_for(s.get(), box_rows, parts);
  Split* raw = s.get();
  if (constant)
    k.ops[key] = std::move(s);
  else
    temp = std::move(s);
  return raw;
}

// the slices' tensor map for boxes of box_rows x 64
static Sliced* slice_map(Sliced* s, int box_rows) {
  if (s->map_rows != box_rows) {
    make_map(&s->map, s->d, (int64_t)s->S * s->rows_p, s->kp, box_rows);
    s->map_rows = box_rows;
  }
  return s;
}

// slice (and cache when the source is a constant block and memory allows) a rows x cols
// FP64 operand, the slice arrays padded to 32 rows and read with boxes of box_rows rows (the
// last tile's box may reach into the next slice: rows or columns that no output uses).
// A cached operand always holds all kSlices digits: a product with S < kSlices digits reads
// the leading S of them (they differ from x by less than one unit of digit S-1, like an
// S-digit split).  nullptr when the slices do not fit in free memory.
static Sliced* slice_prepare(Ctx& c, const MatView& x, int box_rows, int S, std::unique_ptr<Sliced>& temp,
                             bool allow_cache) {
  Cache& k = cache(c);
  bool constant = allow_cache && c.is_constant(x.p);
  const int64_t rows = x.rows, cols = x.cols;
  UCC_REQUIRE(rows < INT32_MAX && cols < INT32_MAX, UCC_BAD_ARGS, "sliced GEMM: operand too large");
  const Key key = make_key(x, 0, kSlices);
  if (constant) {
    auto it = k.sliced.find(key);
    if (it != k.sliced.end()) return slice_map(it->second.get(), box_rows);
    S = kSlices;
  }
  auto s = std::make_unique<Sliced>();
  s->rows = rows;
  s->rows_p = (rows + 31) / 32 * 32;
  s->kp = (cols + BK - 1) / BK * BK;
  s->S = S;
  const size_t nel = (size_t)S * s->rows_p * s->kp;
  size_t free_b = 0, total_b = 0;
  UCC_CUDA(cudaMemGetInfo(&free_b, &total_b));
  const double need = 2.0 * nel + 4.0 * rows;
  // a cached copy keeps a tenth of the memory free for the solver; a temporary 2 GB
  if (constant && need > (double)free_b - 0.1 * (double)total_b) constant = false;
  if (!constant && need > (double)free_b - 2e9) return nullptr;
  if (constant) {
    UCC_CUDA(cudaMalloc(&s->d, sizeof(__nv_bfloat16) * nel));
    UCC_CUDA(cudaMalloc(&s->e, sizeof(int) * rows));
  } else {
    s->tmp = std::make_unique<Scratch>(c, sizeof(__nv_bfloat16) * nel + sizeof(int) * rows + 16);
    s->d = static_cast<__nv_bfloat16*>(s->tmp->p);
    s->e = reinterpret_cast<int*>(static_cast<char*>(s->tmp->p) + ((sizeof(__nv_bfloat16) * nel + 15) / 16) * 16);
  }
  Scratch amax(c, sizeof(unsigned long long) * rows);
  // K chunks of >= 256 elements, enough blocks to cover the SMs a few times
  const int64_t rblocks = (rows + 31) / 32;
  const int64_t want = std::max<int64_t>(1, (int64_t)k.sms * 8 / rblocks);
  const int64_t kchunk = (std::max<int64_t>(256, (cols + want - 1) / want) + 63) / 64 * 64;
  const dim3 blk(32, 8);
  const unsigned nchunks = (unsigned)((cols + kchunk - 1) / kchunk);
  unsigned long long* am = static_cast<unsigned long long*>(amax.p);
  if (nchunks > 1) UCC_CUDA(cudaMemsetAsync(am, 0, sizeof(unsigned long long) * rows, c.stream));
  launch_chained(slice_absmax_kernel, dim3(nchunks, (unsigned)rblocks), blk, c.stream, 1, x, kchunk, am);
  count_kernel_launch();
  launch_chained(slice_digits_kernel, dim3((unsigned)(s->kp / 64), (unsigned)(s->rows_p / 32)), blk, c.stream, 1, x,
                 s->rows_p, s->kp, am, S, s->d, s->e, k.range);
  count_kernel_launch();
  UCC_CUDA(cudaGetLastError());
  slice_map(s.get(), box_rows);
  Sliced* raw = s.get();
  if (constant)
    k.sliced[key] = std::move(s);
  else
    temp = std::move(s);
  return raw;
}

}  // namespace tc

namespace tc {
static void set_sliced_attrs(Cache& k) {
  if (k.sattr_set) return;
  UCC_CUDA(cudaFuncSetAttribute(sliced_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)SLICED_SMEM_BYTES));
  UCC_CUDA(cudaFuncSetAttribute(sliced_gemm_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)SLICED_SMEM_BYTES));
  UCC_CUDA(cudaFuncSetAttribute(sliced_short_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)short_smem(32)));
  UCC_CUDA(cudaFuncSetAttribute(sliced_short_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)short_smem(16)));
  UCC_CUDA(cudaFuncSetAttribute(sliced_short_kernel<48>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)short_smem(48)));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * k.sms);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SLICED_SMEM_BYTES;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  UCC_CUDA(cudaOccupancyMaxActiveClusters(&n, sliced_gemm_kernel<2>, &cfg));
  k.max_pairs_sliced = std::max(1, n);
  k.sattr_set = true;
}

// The N tile and the K split of a single product: the least of a time model over N tiles of 32 to
// 256 columns and splits z,
//   waves * sum over units of max(items t(bn), e(bn)),  waves = ceil(tiles z / slots),
// with t the time of a ring item (a K block: three products of the split form, one of the
// sliced) measured at 4864 x 6144 x 2048 on full waves, and e that of an epilogue pass: 33 ns a
// column for the split form's one (a 64-bit operation per element on two per clock), 120 ns for
// each of the sliced form's (it reads and writes C again per unit).  z > 1 adds the partial
// products' way through memory at about 4 TB/s.  An MMA's time hardly falls below 128 columns,
// so narrow tiles pay only where they fill a wave.  The rule before (the widest tile that wastes
// no column, the split with the fewest waves) counted neither: 2560^3 ran as z = 3 of
// 256-column tiles, 237 us split and 2154 us sliced at nine digits; in two waves of 192-column
// tiles it is 126 (three passes over K) and 1272, and 160 x 40960 x 2048 at nine digits 2586 -> 1510.
//
// chain: the most K blocks that one accumulation in tensor memory may cover (accumulation_blocks;
// kblocks where it does not matter).  z splits obey it; so do, where C is cheap to pass over
// again (in_place), kc K blocks per pass with the passes added in C in FP64: a pass is added
// behind the next one's products, which a z split's partial products are not (2560^3 in one
// pass, with an accumulation nearly three times too long, took 74 us; 4000^3 220, in two 240 us).
struct TilePlan {
  int bn, z, kc;  // N tile, K split, K blocks per pass (0: one pass)
};
static TilePlan plan_tiles(int64_t M, int64_t N, int kblocks, int cm, int slots, const double (&t)[8], double products,
                           int units, int min_blocks, int chain, bool in_place) {
  // ring items per K block of unit u: order u of the sliced form, the tail the rest
  auto unit_items = [&](int u) { return u + 1 < units ? u + 1.0 : products - 0.5 * u * (u + 1); };
  TilePlan best{256, 1, 0};
  double best_us = 1e300;
  auto take = [&](double us, const TilePlan& p) {
    if (us < best_us) best_us = us, best = p;
  };
  const double groups = cm == 2 ? (double)(((M + BM - 1) / BM + 1) / 2) : (double)((M + BM - 1) / BM);
  const double mb = 8e-6 * (double)M * N;
  std::vector<int> zs = {1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 16, 20, 24, 32, 40, 48, 64, 96, 128, 192, 256};
  const int passes = (kblocks + chain - 1) / chain;
  zs.push_back(passes);
  for (int bn = 256; bn >= 32; bn -= 32) {
    const double nt = (double)((N + bn - 1) / bn);
    if (bn > 32 && N <= bn - 32) continue;  // a whole step of padding
    const double epi = (units > 1 ? 0.12 : 0.033) * bn;
    for (int z : zs) {
      const int kb = (kblocks + z - 1) / z;
      if (kb > chain) continue;
      if (z > 1 && z != passes && (kblocks / z < min_blocks || 8.0 * (double)M * N * z > 2e9)) continue;
      double tile = 0.0;
      for (int u = 0; u < units; u++) tile += std::max(unit_items(u) * kb * t[bn / 32 - 1], epi);
      double us = std::ceil(groups * nt * z / slots) * tile + epi;
      if (units > 1 && mb * z > 100.0) us = std::max(us, mb * z * 2.0 * units / 4.0);
      if (z > 1) us += 5.0 + mb * ((units > 1 ? 2.0 : 1.0) * z + z + 2.0) / 4.0;
      take(us, TilePlan{bn, z, 0});
    }
    if (passes > 1 && in_place) {
      const int kc = (kblocks + passes - 1) / passes;
      const double tile = passes * std::max(products * kc * t[bn / 32 - 1], 2.0 * epi);
      take(std::max(std::ceil(groups * nt / slots) * tile + epi, mb * 2.0 * passes / 4.0), TilePlan{bn, 1, kc});
    }
  }
  return best;
}

// K blocks that one FP32 accumulation of a split product may cover.  The tensor core truncates
// its sums: at operands of one sign an accumulation over K elements loses 4.4e-9 K of the
// result, which passes the 4.6e-6 that two bf16 parts leave near K = 1000.  These are the lengths
// that the mixed form's stated accuracy was measured with: K in the number of parts (of at
// least four blocks) that gives tiles as wide as possible the fewest waves of CTAs, one more part
// only for a 5 % gain.  Lengths from time alone were up to five times as long, and so were the
// errors (relative, normal / uniform operands):
//   2560 x 2560 x 2560     896 elements 5.4e-6 / 3.4e-6,  2560 elements 9.9e-6 / 1.3e-5
//   15440 x 136 x 12880   2624 elements 1.0e-5 / 1.3e-5, 12880 elements 4.5e-5 / 8.7e-5
//   160 x 160 x 40960      576 elements 4.9e-6 / 2.3e-6,  1280 elements 6.3e-6 / 5.6e-6
static int accumulation_blocks(int64_t M, int64_t N, int kblocks, int sms) {
  if (kblocks < 8) return kblocks;
  const int bn = pick_bn(N);
  const int64_t tiles = (M + BM - 1) / BM * ((N + bn - 1) / bn);
  const int zmax =
      (int)std::min<int64_t>(std::min<int64_t>(kblocks / 4, 256), std::max<int64_t>(1, 8LL * sms / tiles));
  int z = 1;
  double best = (double)((tiles + sms - 1) / sms);
  for (int y = 2; y <= zmax && 8.0 * M * N * y <= 2e9; y++) {
    const double waves = (double)((tiles * y + sms - 1) / sms) / y;
    if (waves < 0.95 * best) best = waves, z = y;
  }
  return (kblocks + z - 1) / z;
}
// microseconds of a ring item by columns / 32: a fused K block of the split form, a slice product
constexpr double kSplitItem[8] = {0.56, 0.61, 0.66, 0.79, 0.94, 1.10, 1.28, 1.46};
constexpr double kSliceItem[8] = {0.269, 0.276, 0.290, 0.306, 0.329, 0.364, 0.406, 0.450};
}  // namespace tc

// the smallest GEMM the sliced FP64 GEMM takes
constexpr double kSlicedMinWork = 3e7;

static bool sliced_gemm_part(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const MatView& A,
                             const MatView& B, double beta, double* C, const GemmEpilogue& epi, int S, bool allow_cache,
                             bool& wrote);

// A: M x K, B: N x K (rows = the output's columns)
bool sliced_gemm_run(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const MatView& A, const MatView& B,
                     double beta, double* C, const GemmEpilogue& epi, int S) {
  bool wrote = false;
  const bool ok = sliced_gemm_part(c, M, N, K, alpha, A, B, beta, C, epi, S, true, wrote);
  // a false return lets the caller redo the whole product in FP64, so no chunk may have been
  // written by then
  UCC_REQUIRE(ok || !wrote, UCC_BAD_ARGS, "sliced GEMM: operand outside the sliced range after partial output");
  return ok;
}

bool sliced_gemm_run(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm, int64_t sAk,
                     const double* B, int64_t sBk, int64_t sBn, double beta, double* C, const GemmEpilogue& epi,
                     int S) {
  return sliced_gemm_run(c, M, N, K, alpha, MatView::strided(A, M, K, sAm, sAk), MatView::strided(B, N, K, sBn, sBk),
                         beta, C, epi, S);
}

// one sliced product, or the longer of M and N (else K) in halves when the slices exceed one
// launch's limits or the free memory (chunks are sliced as temporaries; a chunk boundary must
// not split a two-stride run)
static bool sliced_gemm_part(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const MatView& A,
                             const MatView& B, double beta, double* C, const GemmEpilogue& epi, int S, bool allow_cache,
                             bool& wrote) {
  using namespace tc;
  UCC_REQUIRE(S >= 2 && SB * S <= 56, UCC_BAD_ARGS, "sliced GEMM: 2 to 9 slices");
  const double aa = std::fabs(alpha);
  if (!(aa >= 0x1p-20 && aa <= 0x1p20) || M > INT32_MAX || N > INT32_MAX) return false;
  // a short K: the kernel that keeps every order in tensor memory (tiles of 48 columns, 32 or 16 for
  // a thin product); otherwise the ring kernel with the N tile and K split of plan_tiles
  const bool short_k = K <= kShortK;
  Cache& k = cache(c);
  set_sliced_attrs(k);
  // neighbouring M tiles pair up in clusters (boxes of bn / 2 rows of B)
  const int cm = short_k ? 1 : cluster_m((int)((M + BM - 1) / BM));
  TilePlan plan{N > 32 ? 48 : N > 16 ? 32 : 16, 1, 0};
  if (!short_k)
    plan = plan_tiles(M, N, (int)((K + BK - 1) / BK), cm, cm == 2 ? k.max_pairs_sliced : k.sms, kSliceItem,
                      0.5 * S * (S + 1), std::max(1, S - 2) + 1, 8, (int)((K + BK - 1) / BK), false);
  const int bn = plan.bn;
  {
    const int64_t Mp = (M + 31) / 32 * 32, Np = (N + 31) / 32 * 32, kp = (K + BK - 1) / BK * BK;
    auto cached = [&](const MatView& x) { return allow_cache && k.sliced.count(make_key(x, 0, kSlices)) != 0; };
    const double needA = cached(A) ? 0.0 : 2.0 * S * (double)Mp * kp;
    const double needB = cached(B) ? 0.0 : 2.0 * S * (double)Np * kp;
    size_t free_b = 0, total_b = 0;
    UCC_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const bool too_big = (double)S * Mp >= 2e9 || (double)S * Np >= 2e9 || Np / 32 > 65535 || Mp / 32 > 65535 ||
                         needA + needB > (double)free_b - 4e9;
    if (too_big) {
      MatView x1, x2, y1, y2;
      if (needB >= needA && N > bn) {
        const int64_t n1 = ((N + 1) / 2 + bn - 1) / bn * bn;
        if (B.sub_rows(0, n1, x1) && B.sub_rows(n1, N - n1, x2))
          return sliced_gemm_part(c, M, n1, K, alpha, A, x1, beta, C, epi, S, false, wrote) &&
                 sliced_gemm_part(c, M, N - n1, K, alpha, A, x2, beta, C + n1 * epi.s_n, epi, S, false, wrote);
      }
      const int64_t unit = epi.msplit ? (int64_t)BM * epi.msplit : BM;  // row chunks keep the row split whole
      if (M > unit && needA >= needB) {
        const int64_t m1 = ((M + 1) / 2 + unit - 1) / unit * unit;
        if (m1 < M && A.sub_rows(0, m1, x1) && A.sub_rows(m1, M - m1, x2)) {
          const int64_t off = epi.msplit ? (m1 / epi.msplit) * epi.s_mhi : m1 * epi.s_mhi;
          return sliced_gemm_part(c, m1, N, K, alpha, x1, B, beta, C, epi, S, false, wrote) &&
                 sliced_gemm_part(c, M - m1, N, K, alpha, x2, B, beta, C + off, epi, S, false, wrote);
        }
      }
      // both operands short and K long (or little memory left): K in halves, the second
      // accumulating onto the first
      if (K >= 2 * 4096) {
        const int64_t k1 = ((K + 1) / 2 + BK - 1) / BK * BK;
        if (A.sub_cols(0, k1, x1) && A.sub_cols(k1, K - k1, x2) && B.sub_cols(0, k1, y1) &&
            B.sub_cols(k1, K - k1, y2))
          return sliced_gemm_part(c, M, N, k1, alpha, x1, y1, beta, C, epi, S, false, wrote) &&
                 sliced_gemm_part(c, M, N, K - k1, alpha, x2, y2, 1.0, C, epi, S, false, wrote);
      }
      return false;
    }
  }
  cudaEvent_t ev0 = c.take_event(), ev1 = c.take_event();
  UCC_CUDA(cudaEventRecord(ev0, c.stream));  // the time includes the slicing of non-cached operands
  std::unique_ptr<Sliced> ta, tb;
  Sliced* a = slice_prepare(c, A, BM, S, ta, allow_cache);
  const CUtensorMap amap = a ? a->map : CUtensorMap{};  // copied: A and B may be one cached operand
  Sliced* b = a ? slice_prepare(c, B, bn / cm, S, tb, allow_cache) : nullptr;
  if (!a || !b) {
    c.event_pool.push_back(ev0);
    c.event_pool.push_back(ev1);
    return false;
  }
  const CUtensorMap bmap = b->map;
  wrote = true;
  SParams p;
  p.M = (int)M;
  p.N = (int)N;
  p.bn = bn;
  p.kblocks = (int)(a->kp / BK);
  p.mtiles = (int)((M + BM - 1) / BM);
  p.ntiles = (int)((N + bn - 1) / bn);
  p.S = S;
  p.gex = std::max(1, S - 2);
  p.a_rows = (int)a->rows_p;
  p.b_rows = (int)b->rows_p;
  p.alpha = alpha;
  p.beta = beta;
  p.C = C;
  p.epi = epi;
  p.ea = a->e;
  p.eb = b->e;
  p.err = k.err;
  p.ksplit = 1;
  p.kchunk = p.kblocks;
  p.klast = (int)((K - (int64_t)(p.kblocks - 1) * BK + 15) / 16);
  const int tiles = p.mtiles * p.ntiles;
  std::unique_ptr<Scratch> part;
  // FP64 partial products of the K chunks, added in a fixed order
  const int ks = plan.z;
  {
    if (ks > 1) {
      p.kchunk = (p.kblocks + ks - 1) / ks;
      p.ksplit = (p.kblocks + p.kchunk - 1) / p.kchunk;
      part = std::make_unique<Scratch>(c, sizeof(double) * M * N * p.ksplit);
      p.C = part->d();
      p.alpha = 1.0;
      p.beta = 0.0;
      p.epi.msplit = 0;
      p.epi.s_mhi = N;
      p.epi.s_n = 1;
    }
  }
  if (short_k) {
    const int grid = std::min(tiles, k.sms);
    if (bn == 16)
      sliced_short_kernel<16><<<grid, kShortThreads, short_smem(16), c.stream>>>(amap, bmap, p);
    else if (bn == 32)
      sliced_short_kernel<32><<<grid, kShortThreads, short_smem(32), c.stream>>>(amap, bmap, p);
    else
      sliced_short_kernel<48><<<grid, kShortThreads, short_smem(48), c.stream>>>(amap, bmap, p);
  } else if (cm == 1) {
    sliced_gemm_kernel<1><<<std::min(tiles * p.ksplit, k.sms), THREADS, SLICED_SMEM_BYTES, c.stream>>>(amap, bmap,
                                                                                                        p);
  } else {
    const int groups = (p.mtiles + 1) / 2 * p.ntiles * p.ksplit;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * std::min(groups, k.max_pairs_sliced));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SLICED_SMEM_BYTES;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    UCC_CUDA(cudaLaunchKernelEx(&cfg, sliced_gemm_kernel<2>, amap, bmap, p));
  }
  count_kernel_launch();
  c.stats.sliced_gemm_launches++;
  UCC_CUDA(cudaGetLastError());
  if (part) splitk_reduce(c, M, N, p.ksplit, part->d(), alpha, beta, C, epi);
  UCC_CUDA(cudaEventRecord(ev1, c.stream));
  // no synchronisation: temporaries are freed in stream order, the time is resolved with the
  // other GEMM timers and the status flags are read at the next synchronisation (tc_check)
  c.gemm_timers.push_back({ev0, ev1, 2.0 * (double)M * (double)N * (double)K, 2, 0.5 * S * (S + 1)});
  if (c.gemm_timers.size() >= 4096) c.resolve_timers();
  k.unchecked = true;
  return true;
}

namespace tc {
// ring layout of a two-part launch: fused stages (A_hi | A_lo | B_hi | B_lo), as many as fit
static void set_fused(Params& p, bool fused, int cm) {
  p.fused = fused ? 1 : 0;
  p.stage_bytes = 2 * A_BYTES + 2 * p.bn * BK * 2 / cm;
  p.nst = fused ? (int)std::min<size_t>(STAGES, GEMM_RING / (size_t)p.stage_bytes) : STAGES;
}

static void set_gemm_attrs(Cache& k) {
  if (k.attr_set) return;
  UCC_CUDA(cudaFuncSetAttribute(gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_BYTES));
  UCC_CUDA(cudaFuncSetAttribute(gemm_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_BYTES));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * k.sms);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = GEMM_SMEM_BYTES;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  UCC_CUDA(cudaOccupancyMaxActiveClusters(&n, gemm_kernel<2>, &cfg));
  k.max_pairs = std::max(1, n);
  k.attr_set = true;
}

// one persistent launch over `work` tiles (output tiles x problems or K chunks): one CTA
// per SM, or pairs of CTAs in clusters when cm = 2
static void launch_gemm(Ctx& c, Cache& k, int cm, int work, const CUtensorMap& ahi, const CUtensorMap& alo,
                        const CUtensorMap& bhi, const CUtensorMap& blo, const CUtensorMap& a2hi,
                        const CUtensorMap& a2lo, const CUtensorMap& amid, const CUtensorMap& bmid, const Params& p) {
  set_gemm_attrs(k);
  if (cm == 1) {
    gemm_kernel<1><<<std::min(work, k.sms), THREADS, GEMM_SMEM_BYTES, c.stream>>>(ahi, alo, bhi, blo, a2hi, a2lo,
                                                                                  amid, bmid, p);
  } else {
    const int groups = (p.mtiles + 1) / 2 * p.ntiles * (p.nprob ? p.nprob : (p.ksplit > 1 ? p.ksplit : 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * std::min(groups, k.max_pairs));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = GEMM_SMEM_BYTES;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    UCC_CUDA(cudaLaunchKernelEx(&cfg, gemm_kernel<2>, ahi, alo, bhi, blo, a2hi, a2lo, amid, bmid, p));
  }
  count_kernel_launch();
  c.stats.tc_gemm_launches++;
  UCC_CUDA(cudaGetLastError());
}
}  // namespace tc

// A: M x K, B: N x K (rows = the output's columns)
void tc_gemm_run(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const MatView& A, const MatView& B,
                 double beta, double* C, const GemmEpilogue& epi, int parts, int kc) {
  using namespace tc;
  UCC_REQUIRE(parts == 2 || parts == 3, UCC_BAD_ARGS, "tensor-core GEMM: 2 or 3 split parts");
  Cache& k = cache(c);
  set_gemm_attrs(k);
  std::unique_ptr<Split> ta, tb;
  const int cm = cluster_m((int)((M + BM - 1) / BM));
  // K chunks of one tile summed in FP64 (kc) are not split further
  const int kblocks = (int)((K + BK - 1) / BK);
  const bool chunks = kc > 0 && kc < kblocks;
  // rows of C in whole sectors, or lanes along its contiguous rows
  const bool in_place = parts == 2 && ((epi.s_n == 1 && (reinterpret_cast<uintptr_t>(C) & 31u) == 0 && epi.s_mhi % 4 == 0 &&
                                        (!epi.msplit || epi.s_mlo % 4 == 0)) ||
                                       (epi.s_mhi == 1 && !epi.msplit));
  const TilePlan plan = plan_tiles(M, N, kblocks, cm, cm == 2 ? k.max_pairs : k.sms, kSplitItem, parts == 2 ? 1.0 : 2.0,
                                   1, chunks ? kblocks + 1 : 4,
                                   chunks ? kblocks : accumulation_blocks(M, N, kblocks, k.sms), in_place);
  const int bn = plan.bn;
  // the maps are copied at once: A and B may be one cached operand read with two boxes
  Split* a = prepare(c, A, BM, ta, parts);
  const CUtensorMap a_hi = a->mhi, a_lo = a->mlo, a_mid = a->mmid;
  Split* b = prepare(c, B, bn / cm, tb, parts);
  const CUtensorMap b_hi = b->mhi, b_lo = b->mlo, b_mid = b->mmid;
  Params p;
  p.M = (int)M;
  p.N = (int)N;
  p.kblocks = (int)(a->kp / BK);
  p.mtiles = (int)((M + BM - 1) / BM);
  p.bn = bn;
  p.ntiles = (int)((N + bn - 1) / bn);
  p.alpha = alpha;
  p.beta = beta;
  p.C = C;
  p.epi = epi;
  p.err = k.err;
  p.nprob = 0;
  p.a_row0 = p.b_row0 = nullptr;
  p.c_off = nullptr;
  p.ksplit = 1;
  p.kchunk = p.kblocks;
  const int tiles = p.mtiles * p.ntiles;
  std::unique_ptr<Scratch> part;
  p.kc = chunks ? kc : plan.kc;
  {
    // FP64 partial products of the K chunks, added in a fixed order
    const int ks = plan.z;
    if (ks > 1) {
      p.kchunk = (p.kblocks + ks - 1) / ks;
      p.ksplit = (p.kblocks + p.kchunk - 1) / p.kchunk;
      part = std::make_unique<Scratch>(c, sizeof(double) * M * N * p.ksplit);
      p.C = part->d();
      p.alpha = 1.0;
      p.beta = 0.0;
      p.epi.msplit = 0;
      p.epi.s_mhi = N;
      p.epi.s_n = 1;
    }
  }
  cudaEvent_t ev0 = c.take_event(), ev1 = c.take_event();
  UCC_CUDA(cudaEventRecord(ev0, c.stream));
  p.nterms = 1;
  p.npair = 0;
  p.a_row1 = p.b_row1 = nullptr;
  p.C32 = nullptr;
  p.nparts = parts;
  set_fused(p, parts == 2, cm);
  launch_gemm(c, k, cm, tiles * p.ksplit, a_hi, a_lo, b_hi, b_lo, a_hi, a_lo, parts == 3 ? a_mid : a_hi,
              parts == 3 ? b_mid : b_hi, p);
  if (part) splitk_reduce(c, M, N, p.ksplit, part->d(), alpha, beta, C, epi);
  UCC_CUDA(cudaEventRecord(ev1, c.stream));
  // no synchronisation (see sliced_gemm_part)
  c.gemm_timers.push_back({ev0, ev1, 2.0 * (double)M * (double)N * (double)K, 1});
  if (c.gemm_timers.size() >= 4096) c.resolve_timers();
  k.unchecked = true;
}

// the status of the tensor-core launches since the last check, after a synchronisation of
// the stream: a pipeline wait that timed out, or a sliced operand whose row maximum is
// beyond 2^498 (the product of such rows is not formed; FP64 covers them)
void tc_check(Ctx& c) {
  if (!c.tc_cache) return;
  tc::Cache& k = *static_cast<tc::Cache*>(c.tc_cache.get());
  if (!k.unchecked) return;
  // the flags are sticky: one copy per check (a copy behind every launch, with the idle time on
  // both its sides, and plain launches of the split and slicing passes took 3.9 of the 162.7 ms
  // of a mixed CCSD(T) solve at no=16/nv=160)
  UCC_CUDA(cudaMemcpyAsync(k.pinned, k.err, 2 * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  UCC_CUDA(cudaStreamSynchronize(c.stream));
  k.unchecked = false;
  const int herr = k.pinned[0], hrange = k.pinned[1];
  if (!herr && !hrange) return;
  UCC_CUDA(cudaMemsetAsync(k.err, 0, 2 * sizeof(int), c.stream));
  UCC_CUDA(cudaStreamSynchronize(c.stream));
  if (herr) throw Error(UCC_DEVICE_TIMEOUT, "tensor-core GEMM: a pipeline wait timed out");
  throw Error(UCC_BAD_ARGS, "sliced FP64 GEMM: an operand row maximum is beyond 2^498; use PRECISION FP64");
}

// drops the cached operands made from the n doubles at p
void tc_forget(Ctx& c, const double* p, size_t n) {
  if (!c.tc_cache) return;
  tc::Cache& k = *static_cast<tc::Cache*>(c.tc_cache.get());
  auto erase = [&](auto& m) {
    for (auto it = m.begin(); it != m.end();) {
      const double* q = std::get<0>(it->first);
      it = q >= p && q < p + n ? m.erase(it) : std::next(it);
    }
  };
  erase(k.ops);
  erase(k.sliced);
}

// a device-side wait of limit_ns that nothing completes: the kernel returns once it runs
// out and the status check that follows every tensor-core launch reports
// UCC_DEVICE_TIMEOUT; the stream and the context stay usable
void wait_selftest(Ctx& c, unsigned long long limit_ns) {
  tc::Cache& k = tc::cache(c);
  tc::wait_selftest_kernel<<<1, 32, 0, c.stream>>>(k.err, limit_ns);
  count_kernel_launch();
  UCC_CUDA(cudaGetLastError());
  k.unchecked = true;
  tc_check(c);
}

void tc_gemm_run(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm, int64_t sAk,
                 const double* B, int64_t sBk, int64_t sBn, double beta, double* C, const GemmEpilogue& epi, int parts,
                 int kc) {
  tc_gemm_run(c, M, N, K, alpha, MatView::strided(A, M, K, sAm, sAk), MatView::strided(B, N, K, sBn, sBk), beta, C,
              epi, parts, kc);
}

void tc_gemm_run(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm, int64_t sAk,
                 const double* B, int64_t sBk, int64_t sBn, double beta, double* C, const GemmEpilogue& epi) {
  tc_gemm_run(c, M, N, K, alpha, A, sAm, sAk, B, sBk, sBn, beta, C, epi, 2, 0);
}

bool tc_eligible(int64_t M, int64_t N, int64_t K) {
  // small problems stay on the FP64 path; the tensor tile is 128 x 256 x 64.  A small
  // output with a long K (a reduction such as Fmi, 32 x 32 x 3.3e6 at no=32/nv=320:
  // 6.7 GFLOP, ~6 ms on the FP64 pipe) runs split-K over the SMs despite its mostly empty tile
  const bool reduction = K >= 65536 && (double)M * N * K >= 1e9;
  if ((std::max(M, N) < 64 && !reduction) || K < 16 || (double)M * N * K < 1e7) return false;
  return M <= INT32_MAX && N <= INT32_MAX;
}

// C (strides sCm, sCn) = alpha A B + beta C with A: M x K and B: N x K views; a short M becomes
// the narrow N tile of C^T = B^T A^T so that the long side fills the 128-row MMA tile
void tc_gemm_oriented(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const MatView& A, const MatView& B,
                      double beta, double* C, int64_t sCm, int64_t sCn, int parts, int kc) {
  GemmEpilogue epi;
  epi.msplit = 0;
  if (M <= 256 && N > M) {
    epi.s_mhi = sCn;
    epi.s_n = sCm;
    tc_gemm_run(c, N, M, K, alpha, B, A, beta, C, epi, parts, kc);
  } else {
    epi.s_mhi = sCm;
    epi.s_n = sCn;
    tc_gemm_run(c, M, N, K, alpha, A, B, beta, C, epi, parts, kc);
  }
}

void tc_gemm_oriented(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm,
                      int64_t sAk, const double* B, int64_t sBk, int64_t sBn, double beta, double* C, int64_t sCm,
                      int64_t sCn, int parts, int kc) {
  tc_gemm_oriented(c, M, N, K, alpha, MatView::strided(A, M, K, sAm, sAk), MatView::strided(B, N, K, sBn, sBk), beta,
                   C, sCm, sCn, parts, kc);
}

// FP64-accurate GEMM on the tensor cores (sliced operands) for the FP64 work of the MIXED
// form; false when the problem is too small for it or outside its exponent range
bool sliced_gemm(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const MatView& A, const MatView& B,
                 double beta, double* C, int64_t sCm, int64_t sCn) {
  // K < 48 (contractions over the occupied indices of most problems) stays on the FP64 pipe.  The line was
  // drawn when every order's sum took a pass over the output: the K = 16 contractions of no=16/nv=160 made its
  // sweeps slower here (203 -> 220 ms per solve), and so did the K = 32 ones of no=32/nv=320.
  // sliced_short_kernel would be the faster one now (25600 x 2560 x 16: 0.77 ms against 1.92, K = 47 0.79 against
  // 5.16), but nine digits of the row and column maxima leave 5.7e-16 of the result at K = 16 and the
  // FP64 multiply-adds 1.0e-16, so moving these contractions would cost accuracy
  if (K < 48 || (double)M * N * K < kSlicedMinWork || M > INT32_MAX || N > INT32_MAX) return false;
  // the output must fill at least 1/16 of its 128 x (N rounded to 32) tiles
  const int64_t lo = std::min(M, N), hi = std::max(M, N);
  if (16.0 * (double)lo * hi < (double)((hi + 127) / 128 * 128) * (double)((lo + 31) / 32 * 32)) return false;
  GemmEpilogue epi;
  epi.msplit = 0;
  // a record sweep's products carry the digits its anchor needs; everything else all of them
  const int digits = c.anchors.mode == 1 ? std::min(tc::kSlices, std::max(2, c.anchors.digits)) : tc::kSlices;
  if (M <= 256 && N > M) {  // the short side becomes the (narrow) N tile
    epi.s_mhi = sCn;
    epi.s_n = sCm;
    return sliced_gemm_run(c, N, M, K, alpha, B, A, beta, C, epi, digits);
  }
  epi.s_mhi = sCm;
  epi.s_n = sCn;
  return sliced_gemm_run(c, M, N, K, alpha, A, B, beta, C, epi, digits);
}

bool sliced_gemm(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm, int64_t sAk,
                 const double* B, int64_t sBk, int64_t sBn, double beta, double* C, int64_t sCm, int64_t sCn) {
  return sliced_gemm(c, M, N, K, alpha, MatView::strided(A, M, K, sAm, sAk), MatView::strided(B, N, K, sBn, sBk), beta,
                     C, sCm, sCn);
}

bool mixed_gemm(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const MatView& A, const MatView& B, double beta,
                double* C, int64_t sCm, int64_t sCn) {
  if (!tc_eligible(M, N, K)) return false;
  tc_gemm_oriented(c, M, N, K, alpha, A, B, beta, C, sCm, sCn, 2, 0);
  return true;
}

bool mixed_gemm(Ctx& c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t sAm, int64_t sAk,
                const double* B, int64_t sBk, int64_t sBn, double beta, double* C, int64_t sCm, int64_t sCn) {
  return mixed_gemm(c, M, N, K, alpha, MatView::strided(A, M, K, sAm, sAk), MatView::strided(B, N, K, sBn, sBk), beta,
                    C, sCm, sCn);
}

// ------------------------------------------------------------------------------------
// (T) on the tensor cores: A_x^T = [<xe|ab> ; -t2[x][m][a][b]] stacked over x as
// [no*nv^2][K'] and B_yz^T = [t2[y][z][c][e] ; <zy|mc>] stacked over (y,z) as [no^2*nv][K']
// (K' = nv + no padded to 64), split once per (T) call; each of the six terms of a tuple
// batch is one batched launch whose problems are the tuples of the batch.
// ------------------------------------------------------------------------------------
namespace tc {
// dst[(row0 + r) * ld + col0 + k] (hi/lo) = scale * src[(r / rsplit) * sr_hi + (r % rsplit) * sr + k*sk],
// r < rows, k < cols; 32x32 tiles through shared memory so that the destination rows are
// written coalesced
__global__ void split_into_kernel(int64_t rows, int64_t cols, const double* src, int64_t rsplit, int64_t sr_hi,
                                  int64_t sr, int64_t sk, double scale, __nv_bfloat16* hi, __nv_bfloat16* lo,
                                  int64_t ld, int64_t row0, int64_t col0) {
  chain_enter();
  __shared__ double t[32][33];
  const int64_t r0 = (int64_t)blockIdx.y * 32, k0 = (int64_t)blockIdx.x * 32;
  double v[4];  // all loads before the first store, which might alias them
  const int64_t rl = r0 + threadIdx.x;
  const double* p = src + (rl / rsplit) * sr_hi + (rl % rsplit) * sr;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int64_t k = k0 + threadIdx.y + 8 * q;
    v[q] = rl < rows && k < cols ? p[k * sk] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < 4; q++) t[threadIdx.y + 8 * q][threadIdx.x] = scale == 1.0 ? v[q] : scale * v[q];
  __syncthreads();
  for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
    const int64_t r = r0 + yy, k = k0 + threadIdx.x;
    if (r < rows && k < cols) {
      // in FP32 from the truncated value (2^-23, below the lo part's 2^-17): no FP64 pipe work
      const float f = f64_to_f32_trunc(t[threadIdx.x][yy]);
      const __nv_bfloat16 h = __float2bfloat16_rn(f);
      const int64_t o = (row0 + r) * ld + col0 + k;
      hi[o] = h;
      lo[o] = __float2bfloat16_rn(f - __bfloat162float(h));
    }
  }
}

struct Triples {
  Split A, A2, B;  // A2: A with its (a,b) row pairs in (b,a) order
  int bn = BN;     // N tile over the virtual index c (pick_bn)
  int* d_arow = nullptr;
  int* d_brow = nullptr;
  int64_t* d_coff = nullptr;
  ~Triples() {
    if (d_arow) cudaFree(d_arow);
    if (d_brow) cudaFree(d_brow);
    if (d_coff) cudaFree(d_coff);
  }
};

static void split_into(Ctx& c, int64_t rows, int64_t cols, const double* src, int64_t sr, int64_t sk, double scale,
                       Split& dst, int64_t row0, int64_t col0, int64_t rsplit = 0, int64_t sr_hi = 0) {
  dim3 grid((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32));
  UCC_REQUIRE(grid.y <= 65535, UCC_BAD_ARGS, "split_into: too many rows");
  if (rsplit <= 0) rsplit = rows;  // one level: r * sr
  launch_chained(split_into_kernel, grid, dim3(32, 8), c.stream, 1, rows, cols, src, rsplit, sr_hi, sr, sk, scale,
                 dst.hi, dst.lo, dst.kp, row0, col0);
  count_kernel_launch();
  UCC_CUDA(cudaGetLastError());
}

static void alloc_split(Split& s, int64_t rows, int64_t kp, cudaStream_t st) {
  s.rows = rows;
  s.kp = kp;
  UCC_CUDA(cudaMalloc(&s.hi, sizeof(__nv_bfloat16) * rows * kp));
  UCC_CUDA(cudaMalloc(&s.lo, sizeof(__nv_bfloat16) * rows * kp));
  UCC_CUDA(cudaMemsetAsync(s.hi, 0, sizeof(__nv_bfloat16) * rows * kp, st));
  UCC_CUDA(cudaMemsetAsync(s.lo, 0, sizeof(__nv_bfloat16) * rows * kp, st));
}
}  // namespace tc

bool mixed_triples_prepare(Ctx& c, int max_batch) {
  using namespace tc;
  const int64_t no = c.no, nv = c.nv, nv2 = nv * nv, kp = (nv + no + BK - 1) / BK * BK;
  if (nv < 64) return false;  // small virtual spaces stay on the FP64 path
  Cache& k = cache(c);
  k.triples.reset();  // of a call that ran out of memory
  auto T = std::make_shared<Triples>();
  alloc_split(T->A, no * nv2, kp, c.stream);
  alloc_split(T->A2, no * nv2, kp, c.stream);
  alloc_split(T->B, no * no * nv, kp, c.stream);
  const double* t2 = c.get("T").p + no * nv;
  const double* Vovvv = c.get("Vovvv").p;
  const double* Vooov = c.get("Vooov").p;
  for (int64_t x = 0; x < no; x++) {
    split_into(c, nv2, nv, Vovvv + x * nv * nv2, 1, nv2, 1.0, T->A, x * nv2, 0);   // <xe|ab>
    split_into(c, nv2, no, t2 + x * no * nv2, 1, nv2, -1.0, T->A, x * nv2, nv);   // -t2[x][m][a][b]
    // the same rows in (b,a) order: row b*nv + a
    split_into(c, nv2, nv, Vovvv + x * nv * nv2, nv, nv2, 1.0, T->A2, x * nv2, 0, nv, 1);
    split_into(c, nv2, no, t2 + x * no * nv2, nv, nv2, -1.0, T->A2, x * nv2, nv, nv, 1);
  }
  split_into(c, no * no * nv, nv, t2, nv, 1, 1.0, T->B, 0, 0);  // t2[y][z][c][e]
  for (int64_t y = 0; y < no; y++)
    for (int64_t z = 0; z < no; z++)  // <zy|mc>
      split_into(c, nv, no, Vooov + (z * no + y) * no * nv, 1, nv, 1.0, T->B, (y * no + z) * nv, nv);
  make_map(&T->A.mhi, T->A.hi, T->A.rows, kp, BM);
  make_map(&T->A.mlo, T->A.lo, T->A.rows, kp, BM);
  make_map(&T->A2.mhi, T->A2.hi, T->A2.rows, kp, BM);
  make_map(&T->A2.mlo, T->A2.lo, T->A2.rows, kp, BM);
  T->bn = pick_bn(nv);
  // M = nv^2 rows per tuple: always two or more M tiles, so the launches pair CTAs that
  // share the B tile (boxes of bn / 2 rows)
  make_map(&T->B.mhi, T->B.hi, T->B.rows, kp, T->bn / 2);
  make_map(&T->B.mlo, T->B.lo, T->B.rows, kp, T->bn / 2);
  UCC_CUDA(cudaMalloc(&T->d_arow, sizeof(int) * 6 * max_batch));  // 3 term pairs x 2 terms
  UCC_CUDA(cudaMalloc(&T->d_brow, sizeof(int) * 6 * max_batch));
  UCC_CUDA(cudaMalloc(&T->d_coff, sizeof(int64_t) * 3 * max_batch));
  k.triples = T;
  set_gemm_attrs(k);
  return true;
}

void mixed_triples_release(Ctx& c) {
  UCC_CUDA(cudaStreamSynchronize(c.stream));
  tc::cache(c).triples.reset();
}

// W3 of nb tuples as three FP32 partial arrays, one per pair of terms: pair pq writes
// W3 + (pq * nb + b) * S for tuple b with beta 0 (no read-modify-write of W3 in the
// epilogue), S = nv^3 in the plain [a][b][c] layout (tblk = 0) or tblk^3 * 512 in the
// blocked layout of w3_block_offset; triples_energy_f32 adds the three while staging its
// tiles.  The launches go out back to back with their own row tables; the caller
// synchronises.
bool mixed_triples_batch(Ctx& c, int nb, const int* tuples, float* W3, int tblk, bool halves) {
  using namespace tc;
  Cache& k = cache(c);
  Triples& T = *k.triples;
  const int64_t no = c.no, nv = c.nv, nv2 = nv * nv, nv3 = nv2 * nv;
  const int64_t per = tblk ? (int64_t)tblk * tblk * tblk * 512 : nv3;  // floats per tuple and partial
  UCC_REQUIRE(!tblk || (tblk >= (nv + 7) / 8 && per < ((int64_t)1 << 31)), UCC_BAD_ARGS,
              "mixed (T): blocked W3 needs whole 8-wide blocks and < 2^31 floats per tuple");
  TriplesTerm terms[6];
  triples_terms(nv, terms);
  // The six terms in pairs that write the same W3 layout: one term of a pair uses
  // A's natural (a,b) rows, the other the (b,a) copy, so that one tile accumulates both
  // in tensor memory; every pair's fastest-varying output row index has W3 stride 1 or
  // its column index does.
  // halves: with i == j the terms 5, 4, 3 are 0, 1, 2 with a and b exchanged, with j == k the terms
  // 1, 5, 4 are 0, 2, 3 with b and c exchanged.  Such a tuple's arrays then hold S with
  // W3 = S + S(exchanged): term 0 and the second pair (array 2 is not written), or the first
  // pair and term 3 (array 1 is not); the energy kernels add the exchange in registers.  15 % of
  // the products go at no = 16, 12 % at no = 20, 8 % at no = 32 (CCSD(T) no=16/nv=160
  // 148.3 -> 146.6 ms, no=20/nv=200 409.7 -> 402.5 ms).  Half tuples come last in a launch, so a
  // problem's number tells how many terms it has.
  // In the last pair the (b,a) copy comes first: a half tuple takes a pair's first term alone.
  const int pairs[3][2] = {{0, 5}, {1, 2}, {3, 4}};
  std::vector<int> both[3], one[3];  // tuples with both terms of a pair, with the first
  for (int b = 0; b < nb; b++) {
    const int* ijk = tuples + 3 * b;
    const bool ij = halves && ijk[0] == ijk[1], jk = halves && !ij && ijk[1] == ijk[2];
    (ij ? one : both)[0].push_back(b);
    if (!jk) both[1].push_back(b);
    if (!ij) (jk ? one : both)[2].push_back(b);
  }
  std::vector<int> arow, brow;
  std::vector<int64_t> coff;
  for (int pq = 0; pq < 3; pq++) {
    for (const auto* l : {&both[pq], &one[pq]})
      for (int b : *l) coff.push_back(((int64_t)pq * nb + b) * per);
    auto rows = [&](const TriplesTerm& tm, const std::vector<int>& l) {
      for (int b : l) {
        const int* ijk = tuples + 3 * b;
        arow.push_back((int)(ijk[tm.x] * nv2));
        brow.push_back((int)((ijk[tm.y] * no + ijk[tm.z]) * nv));
      }
    };
    rows(terms[pairs[pq][0]], both[pq]);
    rows(terms[pairs[pq][0]], one[pq]);
    rows(terms[pairs[pq][1]], both[pq]);
  }
  UCC_CUDA(cudaMemcpyAsync(T.d_coff, coff.data(), sizeof(int64_t) * coff.size(), cudaMemcpyHostToDevice, c.stream));
  UCC_CUDA(cudaMemcpyAsync(T.d_arow, arow.data(), sizeof(int) * arow.size(), cudaMemcpyHostToDevice, c.stream));
  UCC_CUDA(cudaMemcpyAsync(T.d_brow, brow.data(), sizeof(int) * brow.size(), cudaMemcpyHostToDevice, c.stream));
  cudaEvent_t ev0 = c.take_event(), ev1 = c.take_event();
  UCC_CUDA(cudaEventRecord(ev0, c.stream));
  size_t row = 0, off = 0;
  for (int pq = 0; pq < 3; pq++) {
    const int n2 = (int)both[pq].size(), n = n2 + (int)one[pq].size();
    if (!n) continue;
    const TriplesTerm& t0 = terms[pq == 2 ? 4 : pairs[pq][0]];  // output strides for A's natural rows
    Params p;
    p.M = (int)nv2;
    p.N = (int)nv;
    p.kblocks = (int)(T.A.kp / BK);
    p.mtiles = (int)((nv2 + BM - 1) / BM);
    p.bn = T.bn;
    p.ntiles = (int)((nv + T.bn - 1) / T.bn);
    p.alpha = 1.0;
    p.beta = 0.0;
    p.C = nullptr;
    p.C32 = W3;  // W3 in FP32: its rounding (~6e-8) is far below the split products' (~5e-6)
    p.tblk = tblk;
    p.epi.msplit = nv;
    p.epi.s_mhi = t0.su;
    p.epi.s_mlo = t0.sv;
    p.epi.s_n = t0.sw;
    p.err = k.err;
    p.nprob = n;
    p.ksplit = 1;
    p.kchunk = p.kblocks;
    p.nterms = n2 ? 2 : 1;
    p.npair = n2;
    p.a_row0 = T.d_arow + row;
    p.b_row0 = T.d_brow + row;
    p.a_row1 = T.d_arow + row + n;
    p.b_row1 = T.d_brow + row + n;
    p.c_off = T.d_coff + off;
    row += (size_t)n + n2;
    off += n;
    const int tiles = p.mtiles * p.ntiles * n;
    p.nparts = 2;
    p.kc = 0;
    set_fused(p, true, 2);
    const Split &A0 = pq == 2 ? T.A2 : T.A, &A1 = pq == 2 ? T.A : T.A2;
    launch_gemm(c, k, 2, tiles, A0.mhi, A0.mlo, T.B.mhi, T.B.mlo, A1.mhi, A1.mlo, A0.mhi, T.B.mhi, p);
  }
  UCC_CUDA(cudaEventRecord(ev1, c.stream));
  // timed with the other GEMMs (resolved lazily), `row` products of one term each; the status flags are read
  // at the next check
  c.gemm_timers.push_back({ev0, ev1, 2.0 * (double)row * (double)nv2 * (double)nv * (double)(nv + no), 1});
  if (c.gemm_timers.size() >= 4096) c.resolve_timers();
  k.unchecked = true;
  return true;
}

}  // namespace ucc
