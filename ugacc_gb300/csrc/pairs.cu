// Amplitude passes on tiles and pairs (pairs.h) for one problem: packing of the ladder
// operators and amplitudes, the ring terms' combinations, the doubles residual's assembly.
#include <algorithm>

#include "chain.h"
#include "core.h"
#include "pairs.h"

namespace ucc {

void count_kernel_launch();  // kernels_fp64.cu

namespace {

const dim3 kBlock(32, 8);

int64_t tile_pairs(int nv) {
  const int64_t nt = (nv + 31) / 32;
  return nt * (nt + 1) / 2;
}
dim3 tile_grid(int64_t tiles, int64_t rows) {
  return dim3((unsigned)tiles, (unsigned)std::min<int64_t>(std::max<int64_t>(rows, 1), 65535));
}
void launched(const char* what) {
  count_kernel_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw Error(UCC_CUDA_ERROR, std::string(what) + ": " + cudaGetErrorString(e));
}

// Row pair (x <= y) of an [nv]^4 block H, MODE as in pack_vvvv.  The HBAR forms (modes 1 and 2)
// add the slice (y, x); with an FP64 square root and two divisions per element they took
// 24 ms at nv = 160, a per-element pass over 6.6e8 packed elements.
template <int MODE>
__global__ void pack_vvvv_kernel(int nv, const double* __restrict__ H, double* Vp, double* Vm) {
  __shared__ TileBuf s;
  const int64_t nv2 = (int64_t)nv * nv, np = (nv2 + nv) / 2, nm = (nv2 - nv) / 2;
  for (int64_t R = blockIdx.y; R < np; R += gridDim.y) {
    int x, y;
    pair_of(R, x, y);
    pack_slice_tile(s, nv, 1.0, H + ((int64_t)x * nv + y) * nv2, MODE == 0 ? nullptr : H + ((int64_t)y * nv + x) * nv2,
                    MODE != 1, MODE == 1 && x == y, Vp + R * np,
                    x < y ? Vm + ((int64_t)y * (y - 1) / 2 + x) * nm : nullptr, (int)blockIdx.x);
  }
}

// every (m, a) slice of <ma|ef>
__global__ void pack_rows_kernel(int64_t rows, int nv, const double* __restrict__ H, double* Vp, double* Vm) {
  __shared__ TileBuf s;
  const int64_t nv2 = (int64_t)nv * nv, np = (nv2 + nv) / 2, nm = (nv2 - nv) / 2;
  for (int64_t R = blockIdx.y; R < rows; R += gridDim.y)
    pack_slice_tile(s, nv, 1.0, H + R * nv2, nullptr, true, false, Vp + R * np, Vm + R * nm, (int)blockIdx.x);
}

__global__ void pack_tau_kernel(int no, int nv, const double* tau, double* Tp, double* Tm) {
  chain_enter();
  __shared__ TileBuf s;
  const int64_t op = (int64_t)no * (no + 1) / 2;
  for (int64_t R = blockIdx.y; R < op; R += gridDim.y) pack_tau_tile(s, no, nv, tau, Tp, Tm, (int)blockIdx.x, R);
}

__global__ void ring_kernel(int no, int nv, const double* t1, const double* t2, double* X, double* P, double* S) {
  chain_enter();
  __shared__ TileBuf s;
  const int64_t slices = (int64_t)no * no;
  for (int64_t R = blockIdx.y; R < slices; R += gridDim.y) ring_tile(s, no, nv, t1, t2, X, P, S, (int)blockIdx.x, R);
}

__global__ void assemble_kernel(int no, int nv, const double* V, const double* S, int64_t ldS, const double* A,
                                int64_t ldA, const double* Rh, const double* H, double* R2) {
  chain_enter();
  __shared__ TileBuf s;
  const int64_t op = (int64_t)no * (no + 1) / 2;
  for (int64_t R = blockIdx.y; R < op; R += gridDim.y)
    assemble_tile(s, no, nv, V, S, ldS, A, ldA, Rh, H, R2, (int)blockIdx.x, R);
}

__global__ void unpack_z_kernel(int no, int nv, const double* S, int64_t ldS, const double* A, int64_t ldA, double* Z) {
  chain_enter();
  const int64_t n = (int64_t)no * no * no * nv;
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x)
    Z[x] = z_element(no, nv, S, ldS, A, ldA, x);
}

// R2[ijab] += alpha * unpack_pair
template <class I>
__global__ void unpack_ladder_kernel(int no, int nv, double alpha, const double* S, const double* A, double* R2) {
  chain_enter();
  const I n = (I)no * no * nv * nv;
  for (I x = (I)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (I)gridDim.x * blockDim.x)
    R2[x] = fma(alpha, unpack_pair<I>(no, nv, S, A, x), R2[x]);
}
unsigned grid_for(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 32)); }

}  // namespace

void pack_vvvv(Ctx& c, int nv, int mode, const double* H, double* Vp, double* Vm) {
  UCC_REQUIRE(!recorder(), UCC_UNSUPPORTED, "not recordable");
  const dim3 grid = tile_grid(tile_pairs(nv), (int64_t)nv * (nv + 1) / 2);
  if (mode == 0)
    pack_vvvv_kernel<0><<<grid, kBlock, 0, c.stream>>>(nv, H, Vp, Vm);
  else if (mode == 1)
    pack_vvvv_kernel<1><<<grid, kBlock, 0, c.stream>>>(nv, H, Vp, Vm);
  else
    pack_vvvv_kernel<2><<<grid, kBlock, 0, c.stream>>>(nv, H, Vp, Vm);
  launched("pack_vvvv");
}

void pack_ovvv(Ctx& c, int no, int nv, const double* H, double* Vp, double* Vm) {
  UCC_REQUIRE(!recorder(), UCC_UNSUPPORTED, "not recordable");
  const int64_t rows = (int64_t)no * nv;
  pack_rows_kernel<<<tile_grid(tile_pairs(nv), rows), kBlock, 0, c.stream>>>(rows, nv, H, Vp, Vm);
  launched("pack_ovvv");
}

static void record(RecordedOp::Kind kind, int no, int nv, const std::vector<const double*>& src,
                   const std::vector<double*>& dst, double alpha = 1.0) {
  RecordedOp o;
  o.kind = kind;
  o.d[0] = no, o.d[1] = nv;
  o.alpha = alpha;
  std::copy(src.begin(), src.end(), o.src);
  std::copy(dst.begin(), dst.end(), o.dst);
  recorder()->ops.push_back(o);
}

void pack_tau(Ctx& c, int no, int nv, const double* tau, double* Tp, double* Tm) {
  if (recorder()) return record(RecordedOp::kPackTau, no, nv, {tau}, {Tp, Tm});
  launch_chained(pack_tau_kernel, tile_grid(tile_pairs(nv), (int64_t)no * (no + 1) / 2), kBlock, c.stream, 1, no, nv,
                 tau, Tp, Tm);
  launched("pack_tau");
}

void ring_amplitudes(Ctx& c, int no, int nv, const double* t1, const double* t2, double* X, double* P, double* S) {
  if (recorder()) return record(RecordedOp::kRing, no, nv, {t1, t2}, {X, P, S});
  const int64_t nt = (nv + 31) / 32;
  launch_chained(ring_kernel, tile_grid(nt * nt, (int64_t)no * no), kBlock, c.stream, 1, no, nv, t1, t2, X, P, S);
  launched("ring_amplitudes");
}

void assemble_r2(Ctx& c, int no, int nv, const double* V, const double* S, int64_t ldS, const double* A, int64_t ldA,
                 const double* Rh, const double* H, double* R2) {
  if (recorder()) return record(RecordedOp::kAssemble, no, nv, {V, S, A, Rh, H}, {R2});
  launch_chained(assemble_kernel, tile_grid(tile_pairs(nv), (int64_t)no * (no + 1) / 2), kBlock, c.stream, 1, no, nv, V,
                 S, ldS, A, ldA, Rh, H, R2);
  launched("assemble_r2");
}

void unpack_z(Ctx& c, int no, int nv, const double* S, const double* A, double* Z) {
  if (recorder()) return record(RecordedOp::kUnpackZ, no, nv, {S, A}, {Z});
  const PairLd ld(no, nv);
  launch_chained(unpack_z_kernel, grid_for((int64_t)no * no * no * nv), 256, c.stream, 1, no, nv, S, ld.s, A, ld.a, Z);
  launched("unpack_z");
}

void unpack_ladder(Ctx& c, int no, int nv, double alpha, const double* S, const double* A, double* R2) {
  UCC_REQUIRE(!recorder(), UCC_UNSUPPORTED, "not recordable");
  const int64_t n = (int64_t)no * no * nv * nv;
  if (n + 152 * 32 * 256 < ((int64_t)1 << 31))
    launch_chained(unpack_ladder_kernel<uint32_t>, grid_for(n), 256, c.stream, 1, no, nv, alpha, S, A, R2);
  else
    launch_chained(unpack_ladder_kernel<int64_t>, grid_for(n), 256, c.stream, 1, no, nv, alpha, S, A, R2);
  launched("unpack_ladder");
}

}  // namespace ucc
