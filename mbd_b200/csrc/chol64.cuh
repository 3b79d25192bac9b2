// Cholesky factor and inverse of one 64 x 64 block in shared memory by a CTA
// of 128 or 256 threads, and the FP64 tensor-core product they are built on
// (k_cholflow.cu, k_cg.cu).
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"

namespace mbd {
namespace {

constexpr int NB = kCholNB;      // 64
constexpr int FS = NB + 4;       // row stride of 64-wide shared blocks: a half-warp's 8 x 4 fragment loads hit 16 bank pairs

// D = A B + D with A 8x4 (row), B 4x8 (col), D 8x8 in FP64:
// a = A[lane/4][lane%4], b = B[lane%4][lane/4], d = D[lane/4][2*(lane%4) + {0,1}].
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// ---- the 64 x 64 diagonal block -------------------------------------------
// S (row stride FS) holds the updated block's lower triangle, overwritten
// with L; X receives L^-1 (zeros above the diagonal).  Eight 8-column panels:
// warp 0 factors a panel (two rows per lane, the pivot row's entries by
// shuffles), all warps then update the next panel's columns, and while warp 0
// factors on, the other seven update the rest and build the inverse behind
// it.  Bound by the chain of 64 pivots (reciprocal square root, product,
// shuffle).  The code is kept small on purpose: straight-line 32-column
// panels ran at the instruction fetch's pace (58 000 cycles a block; 29 000 now, 2 300 a panel).

// The shift stays apart from the diagonal (whose updates then round at the
// source matrix's size, not at the shift's) and is added to form the pivot;
// the logarithm of (x + shift) / (c2 + shift) is log1p((x - c2) * ref).
struct DiagShift {
  double shift, c2, ref;
};

__device__ __forceinline__ void panel8(double* S, int s, int lane, double shift, int col0, int n, int* bad,
                                       double* dinv, double* diagx) {
  const int r0 = 8 * s + lane, r1 = r0 + 32;
  double a0[8], a1[8];
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    double2 v = make_double2(0.0, 0.0), w = v;
    if (r0 < NB) v = *reinterpret_cast<const double2*>(S + r0 * FS + 8 * s + j);
    if (r1 < NB) w = *reinterpret_cast<const double2*>(S + r1 * FS + 8 * s + j);
    a0[j] = v.x;
    a0[j + 1] = v.y;
    a1[j] = w.x;
    a1[j + 1] = w.y;
  }
  // the chain pivot -> rsqrt -> entry below it -> next pivot: a lane forms its
  // own next pivot (its diagonal entry before the shift is kept for the
  // logarithm), the sign test is on the pivot's high word
  double x = a0[0];
  double piv = x + shift;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    if (lane == c) diagx[8 * s + c] = x;
    piv = __shfl_sync(0xffffffffu, piv, c);
    if ((unsigned)(__double2hiint(piv) - 0x00100000) >= 0x7fe00000u) {
      // not SPD (or NaN): the first failing column; factor on with a unit pivot
      if (*bad == 0 && col0 + 8 * s + c < n) *bad = col0 + 8 * s + c + 1;
      piv = 1.0;
    }
    const double inv = rsqrt(piv);
    const double u = a0[c] * inv;
    if (c < 7) {
      x = fma(-u, u, a0[c + 1]);
      piv = fma(-u, u, a0[c + 1] + shift);
    }
    const double l0 = lane > c ? u : 0.0;   // L's own diagonal is not needed, only its reciprocal
    const double l1 = a1[c] * inv;
    if (lane == c) dinv[8 * s + c] = inv;
#pragma unroll
    for (int j = c + 1; j < 8; ++j) {
      const double lj = __shfl_sync(0xffffffffu, l0, j);
      a0[j] = fma(-l0, lj, a0[j]);
      a1[j] = fma(-l1, lj, a1[j]);
    }
    a0[c] = l0;
    a1[c] = l1;
  }
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    if (r0 < NB) *reinterpret_cast<double2*>(S + r0 * FS + 8 * s + j) = make_double2(a0[j], a0[j + 1]);
    if (r1 < NB) *reinterpret_cast<double2*>(S + r1 * FS + 8 * s + j) = make_double2(a1[j], a1[j + 1]);
  }
}

// C(i, j) -= L(i, s) L(j, s)^T, 8 x 8 blocks; one warp.
__device__ __forceinline__ void update8(double* S, int i, int j, int s, int g, int q) {
  double2* c = reinterpret_cast<double2*>(S + (8 * i + g) * FS + 8 * j + 2 * q);
  double2 v = *c;
#pragma unroll
  for (int kk = 0; kk < 8; kk += 4)
    dmma(v.x, v.y, -S[(8 * i + g) * FS + 8 * s + kk + q], S[(8 * j + g) * FS + 8 * s + kk + q]);
  *c = v;
}

// The same for two block rows at once.
__device__ __forceinline__ void update8x2(double* S, int i0, int i1, int j, int s, int g, int q) {
  double2* c0 = reinterpret_cast<double2*>(S + (8 * i0 + g) * FS + 8 * j + 2 * q);
  double2* c1 = reinterpret_cast<double2*>(S + (8 * i1 + g) * FS + 8 * j + 2 * q);
  const double *a0 = S + (8 * i0 + g) * FS + 8 * s + q, *a1 = S + (8 * i1 + g) * FS + 8 * s + q;
  const double* b = S + (8 * j + g) * FS + 8 * s + q;
  double2 v0 = *c0, v1 = *c1;
  const double b0 = b[0], b1 = b[4], x0 = a0[0], y0 = a0[4], x1 = a1[0], y1 = a1[4];
  dmma(v0.x, v0.y, -x0, b0);
  dmma(v1.x, v1.y, -x1, b0);
  dmma(v0.x, v0.y, -y0, b1);
  dmma(v1.x, v1.y, -y1, b1);
  *c0 = v0;
  *c1 = v1;
}

// X(s, s) = L(s, s)^-1, a column per lane; one warp.
__device__ __forceinline__ void inverse8(const double* S, const double* dinv, double* X, int s, int lane) {
  double x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    x[i] *= dinv[8 * s + i];
#pragma unroll
    for (int k = i + 1; k < 8; ++k) x[k] = fma(-S[(8 * s + k) * FS + 8 * s + i], x[i], x[k]);
  }
  if (lane < 8)
#pragma unroll
    for (int i = 0; i < 8; ++i) X[(8 * s + i) * FS + 8 * s + lane] = x[i];
}

// X(s, j) = -X(s, s) sum_{k=j}^{s-1} L(s, k) X(k, j); one warp.
__device__ __forceinline__ void inverse_row8(const double* S, double* X, int s, int j, int g, int q) {
  double2 w = make_double2(0.0, 0.0);
  for (int kk = 8 * j; kk < 8 * s; kk += 4) dmma(w.x, w.y, S[(8 * s + g) * FS + kk + q], X[(kk + q) * FS + 8 * j + g]);
  double2* out = reinterpret_cast<double2*>(X + (8 * s + g) * FS + 8 * j + 2 * q);
  *out = w;
  __syncwarp();
  double2 v = make_double2(0.0, 0.0);
#pragma unroll
  for (int kk = 0; kk < 8; kk += 4)
    dmma(v.x, v.y, -X[(8 * s + g) * FS + 8 * s + kk + q], X[(8 * s + kk + q) * FS + 8 * j + g]);
  __syncwarp();
  *out = v;
}

// Factors S and inverts the factor into X; dinv, diagx: 64 doubles each.
// All THREADS threads of the CTA.
template <int THREADS>
__device__ __forceinline__ void diag_factor(double* S, double* X, double* dinv, double* diagx, int tid, int col0,
                                            int n, int* bad, double shift) {
  constexpr int W = THREADS / 32;
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  for (int e = tid; e < NB * FS / 2; e += THREADS) reinterpret_cast<double2*>(X)[e] = make_double2(0.0, 0.0);
  __syncthreads();
#pragma unroll 1
  for (int s = 0; s < 10; ++s) {
    // warp 0: panel s, while there is one.  The others: what panel s - 1 does to
    // the columns past s, the inverse of diagonal block s - 1, row s - 2 of the inverse
    const int h = s < 8 ? warp - 1 : warp, nh = s < 8 ? W - 1 : W;
    if (h < 0) {
      panel8(S, s, lane, shift, col0, n, bad, dinv, diagx);
    } else {
      if (h == 0 && s >= 1 && s <= 8) inverse8(S, dinv, X, s - 1, lane);
      for (int j = nh - 1 - h; j < s - 2; j += nh) inverse_row8(S, X, s - 2, j, g, q);
      if (s >= 1 && s < 8) {
        int t = nh - 1 - h;   // tiles (i, j), s < j <= i < 8, dealt from the last warp down
        for (int j = s + 1; j < 8; ++j)
          for (int i = j; i < 8; ++i)
            if (--t < 0) {
              update8(S, i, j, s - 1, g, q);
              t = nh - 1;
            }
      }
    }
    __syncthreads();
    if (s < 7) {   // panel s on the columns of panel s + 1
      const int i = s + 1 + warp;
      if (W < 7 && i + W < 8) {
        update8x2(S, i, i + W, s + 1, s, g, q);
      } else if (i < 8) {
        update8(S, i, s + 1, s, g, q);
      }
      __syncthreads();
    }
  }
}

}  // namespace
}  // namespace mbd
