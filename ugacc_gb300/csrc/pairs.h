// Device code of the pair-symmetric particle ladder, shared by the single-problem kernels
// (kernels_fp64.cu) and the batched ones (batch.cu).  Pairs p <= q are numbered
// q(q+1)/2 + p, strict pairs p < q are numbered q(q-1)/2 + p.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ucc {

// Packs a source whose (x, y) slice is one contiguous nv x nv block t = src + (x * nx + y) * nv^2
// (tau: x, y = i, j; <ab|ef>: x, y = a, b):
//   P[x<=y][e<=f] = h (t[e][f] + t[f][e]) (e < f), t[e][e] (e == f)
//   M[x<y][e<f]   = h (t[e][f] - t[f][e])
// with h = 1/2 (tau) or 1 (<ab|ef>).  A block of 32 x 8 threads takes tile pair tp and row
// pair R: it stages the 32 x 32 tile (E, F) of t and the transposed tile (F, E) in shared
// memory, both read along rows, and writes the packed elements along e (contiguous in both
// outputs for fixed f); the pair indices come from a per-block decode instead of an FP64
// square root per element (GB300's FP64 pipe made the per-element form run at 0.44-0.77 TB/s).
__device__ __forceinline__ void pack_pairs_tile(int nx, int nv, double h, const double* __restrict__ src, double* P,
                                                double* M, int tp, int64_t R) {
  __shared__ double A[32][33], B[32][33];
  const int64_t vp = (int64_t)nv * (nv + 1) / 2, vm = (int64_t)nv * (nv - 1) / 2;
  // tile pair (E <= F): F (F + 1) / 2 + E
  int F = 0;
  while ((F + 1) * (F + 2) / 2 <= tp) F++;
  const int E = tp - F * (F + 1) / 2;
  // row pair (x <= y): y (y + 1) / 2 + x
  int y = (int)((sqrtf(8.0f * (float)R + 1.0f) - 1.0f) * 0.5f);
  while ((int64_t)(y + 1) * (y + 2) / 2 <= R) y++;
  while ((int64_t)y * (y + 1) / 2 > R) y--;
  const int x = (int)(R - (int64_t)y * (y + 1) / 2);
  const double* t = src + ((int64_t)x * nx + y) * (int64_t)nv * nv;
  const int e0 = E * 32, f0 = F * 32, tx = threadIdx.x, ty = threadIdx.y;
  for (int r = ty; r < 32; r += 8) {
    const int ea = e0 + r, fa = f0 + tx;  // A[r][tx] = t[e0 + r][f0 + tx]
    A[r][tx] = (ea < nv && fa < nv) ? t[(int64_t)ea * nv + fa] : 0.0;
    const int fb = f0 + r, eb = e0 + tx;  // B[tx][r] = t[f0 + r][e0 + tx]: B[e][f] = t[f][e]
    B[tx][r] = (fb < nv && eb < nv) ? t[(int64_t)fb * nv + eb] : 0.0;
  }
  __syncthreads();
  double* Prow = P + R * vp;
  double* Mrow = x < y ? M + ((int64_t)y * (y - 1) / 2 + x) * vm : nullptr;
  for (int c = ty; c < 32; c += 8) {  // f = f0 + c, e = e0 + tx along the lanes
    const int f = f0 + c, e = e0 + tx;
    if (f >= nv || e > f) continue;
    const double a = A[tx][c], b = B[tx][c];
    Prow[(int64_t)f * (f + 1) / 2 + e] = e == f ? a : h * (a + b);
    if (Mrow && e < f) Mrow[(int64_t)f * (f - 1) / 2 + e] = h * (a - b);
  }
}

// Element x of [no][no][nv][nv] from the packed S and A: S[(i,j) sorted][(a,b) sorted] +
// sign * A[...], sign = (-1)^[i>j] (-1)^[a>b], A = 0 on i == j or a == b
template <class I>
__device__ __forceinline__ double unpack_pair(int no, int nv, const double* __restrict__ S,
                                              const double* __restrict__ A, I x) {
  const I v_ = (I)nv, o_ = (I)no, vp = v_ * (v_ + 1) / 2, vm = v_ * (v_ - 1) / 2;
  const I b = x % v_;
  I r = x / v_;
  const I a = r % v_;
  r /= v_;
  const I j = r % o_, i = r / o_;
  const I i0 = i < j ? i : j, j0 = i < j ? j : i, a0 = a < b ? a : b, b0 = a < b ? b : a;
  double v = S[(int64_t)(j0 * (j0 + 1) / 2 + i0) * vp + b0 * (b0 + 1) / 2 + a0];
  if (i != j && a != b) {
    const double am = A[(int64_t)(j0 * (j0 - 1) / 2 + i0) * vm + b0 * (b0 - 1) / 2 + a0];
    v += ((i > j) != (a > b)) ? -am : am;
  }
  return v;
}

}  // namespace ucc
