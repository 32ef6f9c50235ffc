// Device code of the amplitude passes that work on 32 x 32 tiles of a (x, y) slice of a
// [n][n][nv][nv] array and on its transposed tile: packing to pairs, the ring terms' amplitude
// combinations and the assembly of the doubles residual.  Shared by the single-problem kernels
// (pairs.cu) and the batched ones (batch.cu); a block has 32 x 8 threads.
//
// Pairs p <= q are numbered q(q+1)/2 + p, strict pairs p < q are numbered q(q-1)/2 + p.
// The passes are HBM-bound; the pair numbers of a tile and a slice come from one decode per
// block, since an FP64 square root per element would keep GB300's FP64 pipe (two operations
// per SM clock) busier than the memory.  The functions are inlined into kernels whose first
// statement waits for the kernel before (chain.h), so no pointer is __restrict__; each loads what a
// thread needs of a tile before its first store, which might alias it.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ucc {

// p <= q of pair number R (q + 1 < 2^15 or so: float is close enough for the search)
__device__ __forceinline__ void pair_of(int64_t R, int& p, int& q) {
  int j = (int)((sqrtf(8.0f * (float)R + 1.0f) - 1.0f) * 0.5f);
  while ((int64_t)(j + 1) * (j + 2) / 2 <= R) j++;
  while ((int64_t)j * (j + 1) / 2 > R) j--;
  q = j;
  p = (int)(R - (int64_t)j * (j + 1) / 2);
}

struct TileBuf {
  double a[32][33], b[32][33];
};

// Packs one slice over its tile pair tp = (E <= F), W[e][f] = t[e][f] (+ u[f][e] with u):
//   P[e<=f] = h (W[e][f] + W[f][e]), W[e][e] where e == f (keep_diag) or 2h W[e][e] (not);
//             W[e][f] itself with `plain`
//   M[e<f]  = h (W[e][f] - W[f][e])   (M may be null)
// written along e, which is contiguous in both for a fixed f.
__device__ __forceinline__ void pack_slice_tile(TileBuf& s, int nv, double h, const double* t,
                                                const double* u, bool keep_diag, bool plain, double* P,
                                                double* M, int tp) {
  int E, F;
  pair_of(tp, E, F);
  const int e0 = E * 32, f0 = F * 32, tx = threadIdx.x, ty = threadIdx.y;
  double va[4], vb[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int ea = e0 + ty + 8 * q, fa = f0 + tx, fb = f0 + ty + 8 * q, eb = e0 + tx;
    va[q] = ea < nv && fa < nv ? t[(int64_t)ea * nv + fa] : 0.0;
    vb[q] = fb < nv && eb < nv ? t[(int64_t)fb * nv + eb] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    s.a[ty + 8 * q][tx] = va[q];  // a[e][f] = t[e][f]
    s.b[tx][ty + 8 * q] = vb[q];  // b[e][f] = t[f][e]
  }
  if (u) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int ea = e0 + ty + 8 * q, fa = f0 + tx, fb = f0 + ty + 8 * q, eb = e0 + tx;
      va[q] = ea < nv && fa < nv ? u[(int64_t)ea * nv + fa] : 0.0;
      vb[q] = fb < nv && eb < nv ? u[(int64_t)fb * nv + eb] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) s.b[ty + 8 * q][tx] += va[q];  // W[f][e] has u[e][f]
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) s.a[tx][ty + 8 * q] += vb[q];  // W[e][f] has u[f][e]
  }
  __syncthreads();
  for (int c = ty; c < 32; c += 8) {  // f = f0 + c, e = e0 + tx along the lanes
    const int f = f0 + c, e = e0 + tx;
    if (f >= nv || e > f) continue;
    const double a = s.a[tx][c], b = s.b[tx][c];
    P[(int64_t)f * (f + 1) / 2 + e] = plain || (keep_diag && e == f) ? a : h * (a + b);
    if (M && e < f) M[(int64_t)f * (f - 1) / 2 + e] = h * (a - b);
  }
  __syncthreads();  // the buffers are free for the next slice
}

// tau[i<=j] -> Tp, Tm (h = 1/2) over row pair R and tile pair tp
__device__ __forceinline__ void pack_tau_tile(TileBuf& s, int no, int nv, const double* tau, double* Tp, double* Tm,
                                              int tp, int64_t R) {
  int x, y;
  pair_of(R, x, y);
  const int64_t nv2 = (int64_t)nv * nv, vp = (nv2 + nv) / 2, vm = (nv2 - nv) / 2;
  pack_slice_tile(s, nv, 0.5, tau + ((int64_t)x * no + y) * nv2, nullptr, true, false, Tp + R * vp,
                  x < y ? Tm + ((int64_t)y * (y - 1) / 2 + x) * vm : nullptr, tp);
}

// The ring terms' combinations of one slice (i, j), tile (E, F) of all nt^2 tiles:
//   X[ijef] = t2/2 + t1[ie] t1[jf];  P[ijef] = t2[ijfe] - X[ijef];  S[ijef] = t2 - t2[ijfe]/2
__device__ __forceinline__ void ring_tile(TileBuf& s, int no, int nv, const double* t1,
                                          const double* t2, double* X, double* P, double* S, int tile,
                                          int64_t slice) {
  const int nt = (nv + 31) / 32, e0 = tile / nt * 32, f0 = tile % nt * 32, tx = threadIdx.x, ty = threadIdx.y;
  const int64_t base = slice * (int64_t)nv * nv;
  const double* t = t2 + base;
  const double* ti = t1 + slice / no * nv;
  const double* tj = t1 + slice % no * nv;
  const int f = f0 + tx;
  const double tjf = f < nv ? tj[f] : 0.0;
  double vb[4], v[4], ti4[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int fb = f0 + ty + 8 * q, eb = e0 + tx, e = e0 + ty + 8 * q;
    vb[q] = fb < nv && eb < nv ? t[(int64_t)fb * nv + eb] : 0.0;
    v[q] = e < nv && f < nv ? t[(int64_t)e * nv + f] : 0.0;
    ti4[q] = e < nv ? ti[e] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < 4; q++) s.b[tx][ty + 8 * q] = vb[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int r = ty + 8 * q, e = e0 + r;
    if (e >= nv || f >= nv) continue;
    const int64_t o = (int64_t)e * nv + f;
    const double w = s.b[r][tx], x = fma(0.5, v[q], ti4[q] * tjf);
    X[base + o] = x;
    P[base + o] = w - x;
    S[base + o] = fma(-0.5, w, v[q]);
  }
  __syncthreads();
}

// The doubles residual of the slices (i <= j) and (j, i), tile pair (A <= B):
//   R2[ijab] = V[ijab] + (S + sign A)[ij][ab] + Q[ijab] + Q[jiba],  Q = Rh + H/2 + H(ijba)
// with S [pairs i<=j][ldS] and A [pairs i<j][ldA] on the pairs a<=b and a<b (sign = -1 when
// exactly one of i > j, a > b holds; A = 0 on i == j or a == b; S null: no such term).  One value goes to ijab and
// jiba and one to ijba and jiab, so R2 is exactly symmetric whatever the rounding of Rh and H:
// in the antisymmetric sector the Jacobi step of the solver does not damp.
__device__ __forceinline__ void assemble_tile(TileBuf& s, int no, int nv, const double* V,
                                              const double* S, int64_t ldS, const double* A,
                                              int64_t ldA, const double* Rh, const double* H,
                                              double* R2, int tp, int64_t R) {
  int ta, tb, i, j;
  pair_of(tp, ta, tb);
  pair_of(R, i, j);
  const int a0 = ta * 32, b0 = tb * 32, tx = threadIdx.x, ty = threadIdx.y;
  const int64_t nv2 = (int64_t)nv * nv, ij = ((int64_t)i * no + j) * nv2, ji = ((int64_t)j * no + i) * nv2;
  const double* Srow = S + R * ldS;
  const double* Arow = A + ((int64_t)j * (j - 1) / 2 + i) * ldA;  // read for i < j only
  double u1[4], u2[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {  // along a: the transposed elements and the packed ones
    const int b = b0 + ty + 8 * q, a = a0 + tx;
    u1[q] = u2[q] = 0.0;
    if (b < nv && a <= b) {
      const int64_t o = (int64_t)b * nv + a;
      const double h3 = H[ij + o], h2 = H[ji + o];
      const double sp = S ? Srow[(int64_t)b * (b + 1) / 2 + a] : 0.0;
      const double am = S && i < j && a < b ? Arow[(int64_t)b * (b - 1) / 2 + a] : 0.0;
      u1[q] = (fma(0.5, h2, Rh[ji + o]) + h3) + (sp + am);
      u2[q] = (fma(0.5, h3, Rh[ij + o]) + h2) + (sp - am);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    s.a[tx][ty + 8 * q] = u1[q];
    s.b[tx][ty + 8 * q] = u2[q];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int r = ty + 8 * q, a = a0 + r, b = b0 + tx;
    if (b < nv && a <= b) {
      const int64_t o = (int64_t)a * nv + b;
      const double h1 = H[ij + o], h4 = H[ji + o];
      u1[q] = ((fma(0.5, h1, Rh[ij + o]) + h4) + s.a[r][tx]) + V[ij + o];
      u2[q] = ((fma(0.5, h4, Rh[ji + o]) + h1) + s.b[r][tx]) + V[ji + o];
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int r = ty + 8 * q, a = a0 + r, b = b0 + tx;
    if (b < nv && a <= b) {
      const int64_t o = (int64_t)a * nv + b;
      R2[ij + o] = u1[q];
      if (i < j) R2[ji + o] = u2[q];
      s.a[r][tx] = u1[q];
      s.b[r][tx] = u2[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = ty; r < 32; r += 8) {
    const int b = b0 + r, a = a0 + tx;
    if (b < nv && a < b) {
      const int64_t o = (int64_t)b * nv + a;
      R2[ji + o] = s.a[tx][r];
      if (i < j) R2[ij + o] = s.b[tx][r];
    }
  }
  __syncthreads();
}

// Element x of Z[m][b][i][j] = (S + sign A)[(i,j) sorted][off + mb], off the number of packed
// ladder columns before the (m,b) ones
__device__ __forceinline__ double z_element(int no, int nv, const double* S, int64_t ldS,
                                            const double* A, int64_t ldA, int64_t x) {
  const int64_t oo = (int64_t)no * no, mb = x / oo;
  const int y = (int)(x - mb * oo), i = y / no, j = y - i * no;
  const int p = i < j ? i : j, q = i < j ? j : i;
  const int64_t nv2 = (int64_t)nv * nv;
  double v = S[((int64_t)q * (q + 1) / 2 + p) * ldS + (nv2 + nv) / 2 + mb];
  if (i != j) {
    const double am = A[((int64_t)q * (q - 1) / 2 + p) * ldA + (nv2 - nv) / 2 + mb];
    v += i > j ? -am : am;
  }
  return v;
}

// Element x of [no][no][nv][nv] from the packed S and A (see assemble_tile)
template <class I>
__device__ __forceinline__ double unpack_pair(int no, int nv, const double* S,
                                              const double* A, I x) {
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
