// Block conjugate gradients for the relay system of every frequency at once:
// A(iw_f) X_f = B with B = [I3; ...; I3] (3N x 3), A lower-stored FP64 --
// the solve of get_screened_alpha (UTILS.f90:469-473) by iteration instead of
// PDPOTRF/PDPOTRS, for the MIXED_LEARNED mode.
//
// Preconditioner M^-1: the exact inverses of the 64 x 64 diagonal tiles of A
// (block Jacobi over tiles; the atoms are in spatial order, so a tile holds
// about 21 neighbouring atoms and their strongest couplings).  Iteration (O'Leary's block CG, 3 right-hand sides, one
// recurrence per frequency):
//   Q = A P;  alpha = (P^T Q)^-1 (Z^T R);  X += P alpha;  R -= Q alpha
//   Z = M^-1 R;  beta = (Z_old^T R_old)^-1 (Z^T R);  P = Z + P beta
// Four launches per iteration, all frequencies at once (grid.y = f):
//   strip      partials of A P (k_strip.cu; the lower half serves both triangles)
//   cg_rows    Q = sum of the partials of each 64-row block; partials of P^T Q
//   cg_update  alpha; X, R, Z = M^-1 R of one 64-row tile per CTA; partials
//              of Z^T R, R^T R
//   cg_dir     beta; P; convergence test ||R||_F^2 <= tol2, after which every
//              later launch returns at once for that frequency
// The 3x3 sums are added in one fixed order by every CTA, so all CTAs of a
// launch take the same decisions.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "chol64.cuh"
#include "kernels.h"
#include "strip.cuh"

namespace mbd {
namespace {

constexpr int CT = kStripRows;   // tile edge (rows)
constexpr int AT = 64;       // atoms per CTA in the per-atom kernels
constexpr int kRed = 10;     // per-CTA partial sums: a 3x3 matrix and one scalar
// state[f][kCgState]: [0] stop (0 run, 1 converged, 2 breakdown, 3 negative
// curvature), [1] iterations, [2..10] Z^T R (even iterations), [11..19] Z^T R
// (odd), [20] R^T R, [kCgIndefinite] 1 when the relay matrix is shown not to
// be positive definite
constexpr int kZR0 = 2, kRR = 20;

// out = m^-1 (3x3, row-major) by cofactors; false when singular or not finite.
__device__ __forceinline__ bool inv3(const double* m, double* out) {
  const double c00 = m[4] * m[8] - m[5] * m[7];
  const double c01 = m[5] * m[6] - m[3] * m[8];
  const double c02 = m[3] * m[7] - m[4] * m[6];
  const double det = m[0] * c00 + m[1] * c01 + m[2] * c02;
  if (!(fabs(det) > 0.0) || !isfinite(det)) return false;
  const double id = 1.0 / det;
  out[0] = c00 * id;
  out[1] = (m[2] * m[7] - m[1] * m[8]) * id;
  out[2] = (m[1] * m[5] - m[2] * m[4]) * id;
  out[3] = c01 * id;
  out[4] = (m[0] * m[8] - m[2] * m[6]) * id;
  out[5] = (m[2] * m[3] - m[0] * m[5]) * id;
  out[6] = c02 * id;
  out[7] = (m[1] * m[6] - m[0] * m[7]) * id;
  out[8] = (m[0] * m[4] - m[1] * m[3]) * id;
  return true;
}

// True when the symmetric part of m (3x3, row-major) has a clearly negative
// pivot in its LDL^T factorisation: some combination p of the search
// directions has p^T A p < 0, which no positive definite A allows.  Pivots
// within 1e-10 of the trace count as a (rank) breakdown, not as a proof.
__device__ __forceinline__ bool negative_curvature(const double* m) {
  const double a = m[0], b = 0.5 * (m[1] + m[3]), c = 0.5 * (m[2] + m[6]);
  const double d = m[4], e = 0.5 * (m[5] + m[7]), f = m[8];
  const double tol = 1e-10 * (fabs(a) + fabs(d) + fabs(f));
  if (a < -tol) return true;
  if (!(a > tol)) return false;
  const double d2 = d - b * b / a;
  if (d2 < -tol) return true;
  if (!(d2 > tol)) return false;
  const double e2 = e - b * c / a;
  const double d3 = f - c * c / a - e2 * e2 / d2;
  return d3 < -tol;
}

__device__ __forceinline__ void mul3(const double* a, const double* b, double* c) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) c[3 * i + j] = a[3 * i] * b[j] + a[3 * i + 1] * b[3 + j] + a[3 * i + 2] * b[6 + j];
}

// Sum of `cnt` partial records (kRed doubles each) in a fixed order by warp 0;
// the totals land in out[0..kRed) (shared memory) for the whole CTA.
__device__ void sum_records(const double* rec, int cnt, double* out) {
  if (threadIdx.x < 32) {
    double acc[kRed];
#pragma unroll
    for (int q = 0; q < kRed; ++q) acc[q] = 0.0;
    for (int k = threadIdx.x; k < cnt; k += 32)
#pragma unroll
      for (int q = 0; q < kRed; ++q) acc[q] += rec[(size_t)k * kRed + q];
#pragma unroll
    for (int q = 0; q < kRed; ++q) {
      double v = acc[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (threadIdx.x == 0) out[q] = v;
    }
  }
  __syncthreads();
}

// CTA-wide sums of vals[0..kRed) into dst (global), fixed order.
__device__ void cta_record(const double* vals, double* sm /* [kRed][32] */, double* dst) {
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int nw = (blockDim.x + 31) / 32;
#pragma unroll
  for (int q = 0; q < kRed; ++q) {
    double v = vals[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sm[q * 32 + warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < kRed) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += sm[threadIdx.x * 32 + w];
    dst[threadIdx.x] = s;
  }
}

__device__ __forceinline__ bool stopped(const CgArgs& a, int f) { return a.state[f * kCgState] != 0.0; }

// Minv[f][I] = inverse of the diagonal tile A_II (rows beyond n: the
// identity) = W^T W with W = L^-1 of its Cholesky factor (chol64.cuh), the
// product on the FP64 tensor cores.  A tile that is not positive definite
// gets the identity (the iteration then cannot converge and the residual gate
// sends the geometry to the direct solve).  Bound by the factor's chain of 64
// pivots; a column-at-a-time factor with dot products by single threads took
// 153 us a launch (300-atom clusters) against 28.
constexpr int kTileInvThreads = 256;
constexpr size_t kTileInvSmem = sizeof(double) * 2 * NB * FS;
__global__ void __launch_bounds__(kTileInvThreads) cg_tile_inv_kernel(CgArgs a) {
  extern __shared__ __align__(16) double dsm[];
  __shared__ double s_dinv[NB], s_diagx[NB];
  __shared__ int s_bad;
  double* S = dsm;
  double* X = dsm + NB * FS;
  const int I = blockIdx.x, f = blockIdx.y, tid = threadIdx.x;
  const double* A = a.A + (size_t)f * a.a_stride;
  for (int e = tid; e < NB * NB; e += kTileInvThreads) {
    const int r = e / NB, c = e % NB, gr = I * NB + r, gc = I * NB + c;
    S[r * FS + c] = (c <= r && gr < a.n) ? A[(size_t)gr * a.ld + gc] : (r == c ? 1.0 : 0.0);
  }
  if (tid == 0) s_bad = 0;
  __syncthreads();
  diag_factor<kTileInvThreads>(S, X, s_dinv, s_diagx, tid, 0, NB, &s_bad, 0.0);
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  double o[8][2];
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j][0] = o[j][1] = 0.0;
  for (int kk = 8 * warp; kk < NB; kk += 4) {   // W is lower triangular: k >= max(row, column)
    const double af = X[(kk + q) * FS + 8 * warp + g];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (8 * j <= kk + 3) dmma(o[j][0], o[j][1], af, X[(kk + q) * FS + 8 * j + g]);
  }
  double* M = a.Minv + ((size_t)f * a.nt + I) * NB * NB;
  const int row = 8 * warp + g;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 8 * j + 2 * q;
    if (s_bad) {
      o[j][0] = row == c ? 1.0 : 0.0;
      o[j][1] = row == c + 1 ? 1.0 : 0.0;
    }
    *reinterpret_cast<double2*>(M + row * NB + c) = make_double2(o[j][0], o[j][1]);
  }
}

// Row sums y = (A v) of 64-row block I from the partials that strip_kernel<T>
// left on `ctas` CTAs.  init: R = B - y.  Otherwise Q = y and the block's
// partial of P^T Q goes to red[f][I].
template <typename T>
__global__ void __launch_bounds__(192) cg_rows_kernel(CgArgs a, int init, int ctas) {
  const int I = blockIdx.x, f = blockIdx.y;
  if (stopped(a, f)) return;
  __shared__ double sm[kRed * 32];
  const int tid = threadIdx.x;
  const int r = tid / 3, q = tid % 3;
  const int gr = I * CT + r;
  const double y = strip_row_sum<T>(a.partial, a.state, a.batch, a.nt, f, I, ctas, r, q);
  const bool live = gr < a.n;
  const size_t o = (size_t)f * a.ystride + (size_t)gr * 3;
  if (init) {
    if (live) a.R[o + q] = ((gr % 3) == q ? 1.0 : 0.0) - y;
    return;
  }
  if (live) a.Q[o + q] = y;
  double vals[kRed];
#pragma unroll
  for (int k = 0; k < kRed; ++k) vals[k] = 0.0;
  if (live) {
    // thread (row, q) adds P[row][c] Q[row][q] to entry (c, q)
#pragma unroll
    for (int c = 0; c < 3; ++c) vals[3 * c + q] = a.P[o + c] * y;
  }
  cta_record(vals, sm, a.red + ((size_t)f * a.nt + I) * kRed);
}

// One thread per (atom, rhs column): loads the atom's 3x3 block of v.
__device__ __forceinline__ void load_block(const double* v, size_t base, int i, double* out) {
#pragma unroll
  for (int k = 0; k < 9; ++k) out[k] = v[base + (size_t)9 * i + k];
}

// Shared memory of the per-tile preconditioner step.
struct TileSmem {
  double Ms[CT][CT + 1];   // M^-1 of the tile
  double Rs[CT][3], Zs[CT][3];
  double red[kRed * 32];
};

// Thread (r, q) of a 192-thread CTA on 64-row tile I of frequency f holds
// R(64 I + r, q) in rv (0 beyond n): Z = M^-1 R on the tile (written to a.Z,
// and to a.P when also_p), then the CTA's partials of Z^T R and R^T R.
__device__ void tile_precondition(const CgArgs& a, int f, int I, double rv, bool also_p, TileSmem& S) {
  const int tid = threadIdx.x, r = tid / 3, q = tid % 3;
  const double* Mg = a.Minv + ((size_t)f * a.nt + I) * CT * CT;
  for (int e = tid; e < CT * CT / 2; e += blockDim.x) {
    const double2 v = reinterpret_cast<const double2*>(Mg)[e];
    const int rr = (2 * e) / CT, cc = (2 * e) % CT;
    S.Ms[rr][cc] = v.x;
    S.Ms[rr][cc + 1] = v.y;
  }
  S.Rs[r][q] = rv;
  __syncthreads();
  double z0 = 0.0, z1 = 0.0;   // two accumulation chains
#pragma unroll 8
  for (int k = 0; k < CT; k += 2) {
    z0 += S.Ms[r][k] * S.Rs[k][q];
    z1 += S.Ms[r][k + 1] * S.Rs[k + 1][q];
  }
  const double z = z0 + z1;
  S.Zs[r][q] = z;
  const int gr = I * CT + r;
  if (gr < a.n) {
    const size_t o = (size_t)f * a.ystride + (size_t)gr * 3 + q;
    a.Z[o] = z;
    if (also_p) a.P[o] = z;
  }
  __syncthreads();
  double vals[kRed];
#pragma unroll
  for (int k = 0; k < kRed; ++k) vals[k] = 0.0;
  // (Z^T R)(c, q) = sum_rows Z[row][c] R[row][q]
#pragma unroll
  for (int c = 0; c < 3; ++c) vals[3 * c + q] = S.Zs[r][c] * rv;
  vals[9] = rv * rv;
  cta_record(vals, S.red, a.red2 + ((size_t)f * a.nt + I) * kRed);
}

// init: Z = M^-1 R, P = Z on one 64-row tile; partials of Z^T R and R^T R.
__global__ void __launch_bounds__(192) cg_init_tiles_kernel(CgArgs a) {
  const int I = blockIdx.x, f = blockIdx.y;
  if (stopped(a, f)) return;
  __shared__ TileSmem S;
  const int r = threadIdx.x / 3, q = threadIdx.x % 3, gr = I * CT + r;
  const double rv = gr < a.n ? a.R[(size_t)f * a.ystride + (size_t)gr * 3 + q] : 0.0;
  tile_precondition(a, f, I, rv, true, S);
}

// Between the phases: frequencies stopped as converged (1) or broken down
// (2) run again, negative curvature (3) stays; the first phase's iteration
// count is kept in kCgPhase1Iters.  Must run before any kernel that tests
// the stop flag in the restart.
__global__ void cg_reopen_kernel(CgArgs a) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= a.batch) return;
  double* st = a.state + f * kCgState;
  st[kCgPhase1Iters] = st[1];
  if (st[0] == 1.0 || st[0] == 2.0) st[0] = 0.0;
}

// init: Z^T R and R^T R into the state; stop when already converged.
__global__ void cg_init_final_kernel(CgArgs a, int nb) {
  const int f = blockIdx.x;
  __shared__ double tot[kRed];
  if (stopped(a, f)) return;
  sum_records(a.red2 + (size_t)f * nb * kRed, nb, tot);
  if (threadIdx.x == 0) {
    double* st = a.state + f * kCgState;
    for (int k = 0; k < 9; ++k) st[kZR0 + k] = tot[k];
    st[kRR] = tot[9];
    st[1] = 0.0;
    if (tot[9] <= a.tol2) st[0] = 1.0;
  }
}

// alpha = (P^T Q)^-1 (Z^T R); X += P alpha; R -= Q alpha on one 64-row
// tile; Z = M^-1 R; partials of Z^T R (new) and R^T R into red2.
__global__ void __launch_bounds__(192) cg_update_kernel(CgArgs a, int it) {
  const int I = blockIdx.x, f = blockIdx.y;
  if (stopped(a, f)) return;
  __shared__ double tot[kRed];
  __shared__ double s_alpha[9];
  __shared__ int s_indef;
  __shared__ TileSmem S;
  sum_records(a.red + (size_t)f * a.nt * kRed, a.nt, tot);
  if (threadIdx.x == 0) {
    const double* zr = a.state + f * kCgState + kZR0 + 9 * (it & 1);
    double pq[9], ipq[9], al[9];
    for (int k = 0; k < 9; ++k) pq[k] = tot[k];
    // P^T A P with a negative direction: A is not positive definite (the
    // reference's unchecked PDPOTRF info, UTILS.f90:469).  Every CTA sees the
    // same sums and stops; CTA 0 records it and ends this frequency's solve.
    s_indef = negative_curvature(pq) ? 1 : 0;
    if (s_indef && I == 0) {
      double* st = a.state + f * kCgState;
      st[kCgIndefinite] = 1.0;
      st[0] = 3.0;
    }
    if (inv3(pq, ipq)) {
      mul3(ipq, zr, al);
    } else {
      for (int k = 0; k < 9; ++k) al[k] = 0.0;
    }
    for (int k = 0; k < 9; ++k) s_alpha[k] = al[k];
  }
  __syncthreads();
  if (s_indef) return;
  const int r = threadIdx.x / 3, q = threadIdx.x % 3, gr = I * CT + r;
  double rv = 0.0;
  if (gr < a.n) {
    const size_t o = (size_t)f * a.ystride + (size_t)gr * 3;
    double x = a.X[o + q], rr = a.R[o + q];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      x += a.P[o + c] * s_alpha[3 * c + q];
      rr -= a.Q[o + c] * s_alpha[3 * c + q];
    }
    a.X[o + q] = x;
    a.R[o + q] = rr;
    rv = rr;
  }
  tile_precondition(a, f, I, rv, false, S);
}

// beta = (Z^T R)_old^-1 (Z^T R)_new; P = Z + P beta; convergence test.
__global__ void __launch_bounds__(AT) cg_dir_kernel(CgArgs a, int it) {
  const int f = blockIdx.y;
  if (stopped(a, f)) return;
  __shared__ double tot[kRed];
  __shared__ double s_beta[9];
  __shared__ int s_done;
  sum_records(a.red2 + (size_t)f * a.nt * kRed, a.nt, tot);   // one record per 64-row tile
  double* st = a.state + f * kCgState;
  if (threadIdx.x == 0) {
    const double* zr_old = st + kZR0 + 9 * (it & 1);
    double zo[9], izo[9], zn[9], be[9];
    for (int k = 0; k < 9; ++k) {
      zo[k] = zr_old[k];
      zn[k] = tot[k];
    }
    int done = 0;
    if (tot[9] <= a.tol2) {
      done = 1;
    } else if (!inv3(zo, izo)) {
      done = 2;
    } else {
      mul3(izo, zn, be);
      for (int k = 0; k < 9; ++k) s_beta[k] = be[k];
    }
    s_done = done;
    if (blockIdx.x == 0) {
      double* zr_new = st + kZR0 + 9 * ((it + 1) & 1);
      for (int k = 0; k < 9; ++k) zr_new[k] = zn[k];
      st[kRR] = tot[9];
      st[1] = (double)(it + 1);
    }
  }
  __syncthreads();
  if (s_done) {
    // every CTA reads the old flag at entry; CTA 0 raises it after its own
    // update, so no CTA of this launch sees it change
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) st[0] = (double)s_done;
    return;
  }
  const int i = blockIdx.x * AT + threadIdx.x;
  if (i < a.N) {
    const size_t base = (size_t)f * a.ystride;
    double Z[9], P[9], t[9];
    load_block(a.Z, base, i, Z);
    load_block(a.P, base, i, P);
    mul3(P, s_beta, t);
#pragma unroll
    for (int k = 0; k < 9; ++k) a.P[base + 9 * (size_t)i + k] = Z[k] + t[k];
  }
}

// ---- all iterations of a phase in one launch -------------------------------
// One thread-block cluster per frequency runs the FP32-pass iterations of
// launch_cg_iteration to the end, with a cluster barrier where that has a
// launch boundary: a converged frequency leaves at once, and a geometry costs
// the host one launch a phase instead of four an iteration (a batch of 256
// clusters issued 91 000 launches, 430 ms of host time).  Every CTA takes the
// 3 x 3 decisions from the same records in the same order, so the cluster
// stays uniform.
//
// Matrix pass: a CTA owns 64-row blocks in pairs from both ends (equal work)
// and forms their products whole -- its rows up to the diagonal, then the
// columns below it, 16 rows or columns to a warp -- so no partial sums leave
// the CTA and nothing is reduced across lanes until a warp has swept its row.
// An entry off the diagonal blocks is read twice (by its row's and its
// column's owner): matrices of this size stay in L2, and the symmetric sweep
// tried first spent more on the exchange than on the products.  Sums as in
// strip_kernel<float>: four products in FP32, everything beyond in FP64.
// P is kept in shared memory of every CTA in FP32, written by its owners
// through the cluster.
constexpr int CLT = 256;

// A warp's matrix chunks (32 lanes x 4 loads of 16 bytes) on their way, each
// lane's own: a sweep is bound by the bytes it has in flight.
constexpr int kRing = 4;

// P in shared memory: per row (x, y, z, 0), and the three columns apart.
struct PShared {
  float4* row;     // [nt * 64 + 32]
  float* col[3];   // [nt * 64 + 32] each
};
__host__ __device__ constexpr size_t p_shared_rows(int nt) { return (size_t)nt * CT + 32; }
size_t p_shared_bytes(int nt) {
  return p_shared_rows(nt) * (sizeof(float4) + 3 * sizeof(float)) + sizeof(float4) * kRing * 4 * CLT;
}

// d[4][3] over lanes that differ in the bits OFF, OFF/2, OFF/4: afterwards
// out holds the sums of element ((lane / (OFF/2)) & 3).
template <int OFF>
__device__ __forceinline__ void scatter4(double (&d)[4][3], int lane, double (&out)[3]) {
  const bool u1 = lane & OFF, u2 = lane & (OFF / 2);
  double e[2][3];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double send = u1 ? d[t][q] : d[t + 2][q], keep = u1 ? d[t + 2][q] : d[t][q];
      e[t][q] = keep + __shfl_xor_sync(0xffffffffu, send, OFF);
    }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double send = u2 ? e[0][q] : e[1][q], keep = u2 ? e[1][q] : e[0][q];
    const double v = keep + __shfl_xor_sync(0xffffffffu, send, OFF / 2);
    out[q] = v + __shfl_xor_sync(0xffffffffu, v, OFF / 4);
  }
}

// out[16][3] = A[r0 .. r0 + 16)[0 .. diagonal] P, the diagonal included.
// Lane: four columns of 32 (cg) and four rows (rg).  Rows past n repeat row
// n - 1; their sums are not used.
__device__ __forceinline__ void rows_task(const float* A, int ld, int n, const PShared& ps, int r0, int lane,
                                          float4* ring, double* out) {
  const int cg = lane & 7, rg = lane >> 3;
  const float* Ar[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) Ar[t] = A + (size_t)min(r0 + 4 * rg + t, n - 1) * ld + 4 * cg;
  double rs[4][3];
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int q = 0; q < 3; ++q) rs[t][q] = 0.0;
  const int chunks = r0 / 32 + 1;              // the last holds the diagonal
  auto issue = [&](int c) {
    if (c < chunks)
#pragma unroll
      for (int t = 0; t < 4; ++t) ring_copy(ring + ((c & (kRing - 1)) * 4 + t) * 32 + lane, Ar[t] + 32 * c);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < kRing - 1; ++c) issue(c);
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
    float4 v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = ring[((c & (kRing - 1)) * 4 + t) * 32 + lane];
    issue(c + kRing - 1);
    const int gc = 32 * c + 4 * cg;
    if (c + 1 == chunks) {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int r = r0 + 4 * rg + t;
        if (gc > r) v[t].x = 0.f;
        if (gc + 1 > r) v[t].y = 0.f;
        if (gc + 2 > r) v[t].z = 0.f;
        if (gc + 3 > r) v[t].w = 0.f;
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const float4 x = *reinterpret_cast<const float4*>(ps.col[q] + gc);
      const unsigned long long x01 = pack2(x.x, x.y), x23 = pack2(x.z, x.w);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float lo, hi;
        unpack2(fma2(pack2(v[t].z, v[t].w), x23, mul2(pack2(v[t].x, v[t].y), x01)), lo, hi);
        rs[t][q] += widen(lo + hi);
      }
    }
  }
  double y[3];
  scatter4<4>(rs, lane, y);
  if ((lane & 1) == 0) {
    double* o = out + (4 * rg + ((lane >> 1) & 3)) * 3;
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = y[q];
  }
}

// out[16][3] = (A[below the diagonal .. n)[c0 .. c0 + 16))^T P.  Lane: four
// columns (cg) and every eighth row.  P is zero past n.
__device__ __forceinline__ void cols_task(const float* A, int ld, int n, const PShared& ps, int c0, int lane,
                                          float4* ring, double* out) {
  const int cg = lane & 3, rp = lane >> 2;
  const float* Ac = A + c0 + 4 * cg;
  double cs[4][3];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int q = 0; q < 3; ++q) cs[k][q] = 0.0;
  const int chunks = (n - c0 + 31) / 32;
  auto issue = [&](int c) {
    if (c < chunks)
#pragma unroll
      for (int t = 0; t < 4; ++t)
        ring_copy(ring + ((c & (kRing - 1)) * 4 + t) * 32 + lane, Ac + (size_t)min(c0 + 32 * c + rp + 8 * t, n - 1) * ld);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < kRing - 1; ++c) issue(c);
  for (int c = 0; c < chunks; ++c) {
    const int R = c0 + 32 * c;
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
    float4 v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = ring[((c & (kRing - 1)) * 4 + t) * 32 + lane];
    issue(c + kRing - 1);
    if (R == c0) {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int r = R + rp + 8 * t, gc = c0 + 4 * cg;
        if (gc >= r) v[t].x = 0.f;
        if (gc + 1 >= r) v[t].y = 0.f;
        if (gc + 2 >= r) v[t].z = 0.f;
        if (gc + 3 >= r) v[t].w = 0.f;
      }
    }
    unsigned long long c01[3], c23[3];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float4 x = ps.row[R + rp + 8 * t];
      const unsigned long long e01 = pack2(v[t].x, v[t].y), e23 = pack2(v[t].z, v[t].w);
      const float xq[3] = {x.x, x.y, x.z};
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const unsigned long long xx = pack2(xq[q], xq[q]);
        c01[q] = t == 0 ? mul2(e01, xx) : fma2(e01, xx, c01[q]);
        c23[q] = t == 0 ? mul2(e23, xx) : fma2(e23, xx, c23[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      float lo, hi;
      unpack2(c01[q], lo, hi);
      cs[0][q] += widen(lo);
      cs[1][q] += widen(hi);
      unpack2(c23[q], lo, hi);
      cs[2][q] += widen(lo);
      cs[3][q] += widen(hi);
    }
  }
  double y[3];
  scatter4<16>(cs, lane, y);
  if ((lane & 4) == 0) {
    double* o = out + (4 * cg + ((lane >> 3) & 3)) * 3;
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = y[q];
  }
}

// Records of the cluster's CTAs summed in order; totals for the whole CTA.
__device__ __forceinline__ void sum_cluster_records(const double* rec, int C, double* out) {
  if (threadIdx.x < kRed) {
    double v = 0.0;
    for (int k = 0; k < C; ++k) v += __ldcg(rec + k * kRed + threadIdx.x);
    out[threadIdx.x] = v;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(CLT, 2) cg_cluster_kernel(CgArgs a, int it0, int it1) {
  namespace cgr = cooperative_groups;
  cgr::cluster_group cl = cgr::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int f = blockIdx.x / C;
  extern __shared__ __align__(16) float4 xs[];
  __shared__ double Rs[CT][3], Zp[4][CT][3], ys[2][2][CT * 3], sm[kRed * 32];
  __shared__ double tot[kRed], s_zr[9], s_m[9];
  __shared__ int s_flag;
  if (stopped(a, f)) return;                     // uniform: the flag is raised behind cluster barriers only
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.n, nt = a.nt, pairs = (nt + 1) / 2;
  const size_t prow = p_shared_rows(nt);
  float* pc = reinterpret_cast<float*>(xs + prow);
  const PShared ps{xs, {pc, pc + prow, pc + 2 * prow}};
  float4* ring = reinterpret_cast<float4*>(pc + 3 * prow) + (tid >> 5) * (kRing * 4 * 32);
  const float* A = a.A32 + (size_t)f * a.a_stride;
  const size_t vo = (size_t)f * a.ystride;
  double* rec1 = a.red + (size_t)f * nt * kRed;
  double* rec2 = a.red2 + (size_t)f * nt * kRed;
  double* st = a.state + f * kCgState;
  if (tid < 9) s_zr[tid] = st[kZR0 + tid];
  const int r = tid / 3, q = tid % 3;            // thread's row and column of a 64-row block (tid < 192)
  for (int i = tid; i < (int)prow; i += CLT) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) {
      const double* p = a.P + vo + (size_t)3 * i;
      x = make_float4((float)p[0], (float)p[1], (float)p[2], 0.f);
    }
    xs[i] = x;
    pc[i] = x.x;
    pc[prow + i] = x.y;
    pc[2 * prow + i] = x.z;
  }
  cl.sync();
  for (int it = it0; it < it1; ++it) {
    // Q = A P on this CTA's blocks; its part of P^T Q
    double vals[kRed];
#pragma unroll
    for (int k = 0; k < kRed; ++k) vals[k] = 0.0;
    for (int p = rank; p < pairs; p += C) {
      for (int e = 0; e < 2; ++e) {
        const int I = e == 0 ? p : nt - 1 - p;
        if (e == 1 && I == p) break;
        const int r0 = I * CT + 16 * (warp & 3);
        if (r0 < n) {
          double* o = ys[e][warp >> 2] + 48 * (warp & 3);
          if (warp < 4) rows_task(A, a.ld, n, ps, r0, lane, ring, o);
          else cols_task(A, a.ld, n, ps, r0, lane, ring, o);
        }
      }
      __syncthreads();
      for (int e = 0; e < 2; ++e) {
        const int I = e == 0 ? p : nt - 1 - p, gr = I * CT + r;
        if (e == 1 && I == p) break;
        if (tid < CT * 3 && gr < n) {
          const size_t o = vo + (size_t)gr * 3;
          const double y = ys[e][0][tid] + ys[e][1][tid];
          a.Q[o + q] = y;
          for (int c = 0; c < 3; ++c) {
            const double t = a.P[o + c] * y;
            if (q == 0) vals[3 * c] += t;
            if (q == 1) vals[3 * c + 1] += t;
            if (q == 2) vals[3 * c + 2] += t;
          }
        }
      }
      __syncthreads();
    }
    cta_record(vals, sm, rec1 + rank * kRed);
    cl.sync();
    // alpha = (P^T Q)^-1 (Z^T R)
    sum_cluster_records(rec1, C, tot);
    if (tid == 0) {
      double pq[9], ipq[9], al[9], zr[9];
      for (int k = 0; k < 9; ++k) {
        pq[k] = tot[k];
        zr[k] = s_zr[k];
        al[k] = 0.0;
      }
      if (inv3(pq, ipq)) mul3(ipq, zr, al);
      for (int k = 0; k < 9; ++k) s_m[k] = al[k];
    } else if (tid == 32) {
      double pq[9];
      for (int k = 0; k < 9; ++k) pq[k] = tot[k];
      s_flag = negative_curvature(pq) ? 1 : 0;
    }
    __syncthreads();
    if (s_flag) {                                // A is not positive definite: ends this frequency's solve
      if (rank == 0 && tid == 0) {
        st[kCgIndefinite] = 1.0;
        st[0] = 3.0;
      }
      return;
    }
#pragma unroll
    for (int k = 0; k < kRed; ++k) vals[k] = 0.0;
    for (int p = rank; p < pairs; p += C)
      for (int e = 0; e < 2; ++e) {
        const int I = e == 0 ? p : nt - 1 - p, gr = I * CT + r;
        if (e == 1 && I == p) break;
        const size_t o = vo + (size_t)gr * 3;
        // M^-1 (symmetric: a thread's row is read down its column) is on its way while R is formed
        const double* M = a.Minv + ((size_t)f * nt + I) * CT * CT;
        const int row = tid & 63, kg = tid >> 6;
        double m[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) m[k] = M[(16 * kg + k) * CT + row];
        double rv = 0.0;
        if (tid < CT * 3) {
          if (gr < n) {
            double x = a.X[o + q];
            rv = a.R[o + q];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              x += a.P[o + c] * s_m[3 * c + q];
              rv -= a.Q[o + c] * s_m[3 * c + q];
            }
            a.X[o + q] = x;
            a.R[o + q] = rv;
          }
          Rs[r][q] = rv;
        }
        __syncthreads();
        {   // Z = M^-1 R: four chains of 16 for each row
          double z0 = 0.0, z1 = 0.0, z2 = 0.0;
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            z0 += m[k] * Rs[16 * kg + k][0];
            z1 += m[k] * Rs[16 * kg + k][1];
            z2 += m[k] * Rs[16 * kg + k][2];
          }
          Zp[kg][row][0] = z0;
          Zp[kg][row][1] = z1;
          Zp[kg][row][2] = z2;
        }
        __syncthreads();
        if (tid < CT * 3) {
          double z[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) z[c] = (Zp[0][r][c] + Zp[1][r][c]) + (Zp[2][r][c] + Zp[3][r][c]);
          if (gr < n) a.Z[o + q] = q == 0 ? z[0] : (q == 1 ? z[1] : z[2]);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double t = z[c] * rv;
            if (q == 0) vals[3 * c] += t;
            if (q == 1) vals[3 * c + 1] += t;
            if (q == 2) vals[3 * c + 2] += t;
          }
          vals[9] += rv * rv;
        }
      }
    __syncthreads();
    cta_record(vals, sm, rec2 + rank * kRed);
    cl.sync();
    // beta = (Z^T R)_old^-1 (Z^T R)_new; convergence test
    sum_cluster_records(rec2, C, tot);
    if (tid == 0) {
      double zo[9], izo[9], zn[9], be[9];
      for (int k = 0; k < 9; ++k) {
        zo[k] = s_zr[k];
        zn[k] = tot[k];
      }
      int done = 0;
      if (tot[9] <= a.tol2) {
        done = 1;
      } else if (!inv3(zo, izo)) {
        done = 2;
      } else {
        mul3(izo, zn, be);
        for (int k = 0; k < 9; ++k) s_m[k] = be[k];
      }
      for (int k = 0; k < 9; ++k) s_zr[k] = zn[k];
      s_flag = done;
      if (rank == 0) {
        st[kRR] = tot[9];
        st[1] = (double)(it + 1);
        if (done) st[0] = (double)done;
      }
    }
    __syncthreads();
    if (s_flag) return;
    for (int p = rank; p < pairs; p += C)
      for (int e = 0; e < 2; ++e) {
        const int I = e == 0 ? p : nt - 1 - p, gr = I * CT + r;
        if (e == 1 && I == p) break;
        const size_t o = vo + (size_t)gr * 3;
        const bool live = tid < CT * 3 && gr < n;
        double v = 0.0;
        if (live) {
          v = a.Z[o + q];
#pragma unroll
          for (int c = 0; c < 3; ++c) v += a.P[o + c] * s_m[3 * c + q];
        }
        __syncthreads();                         // a row's three entries are read by three threads
        if (live) {
          a.P[o + q] = v;
          const float vf = (float)v;             // the entry in every CTA's copies
          for (int k = 0; k < C; ++k) {
            float4* other = cl.map_shared_rank(xs, k);
            reinterpret_cast<float*>(other + gr)[q] = vf;
            reinterpret_cast<float*>(other + prow)[q * prow + gr] = vf;
          }
        }
      }
    cl.sync();
  }
  if (rank == 0 && tid < 9) st[kZR0 + tid] = s_zr[tid];   // for a launch that carries on
}

}  // namespace

size_t cg_minv_doubles(int n, int batch) {
  const int nt = (n + CT - 1) / CT;
  return (size_t)batch * nt * CT * CT;
}

int num_sms() {
  static const int sms = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
  }();
  return sms;
}

template <typename T>
StripArgs<T> strip_args(const CgArgs& a, const T* A, const double* in) {
  return StripArgs<T>{A, a.a_stride, a.ld, a.n, a.nt, a.batch, in, a.ystride, a.partial, a.state};
}

size_t cg_partial_doubles(int n, int batch) {
  const int nt = (n + CT - 1) / CT;
  return (size_t)batch * nt * nt * CT * 3;
}

size_t cg_red_doubles(int n, int batch) {
  const int nt = (n + CT - 1) / CT;
  const int nb = (n / 3 + AT - 1) / AT;
  return (size_t)batch * (nt > nb ? nt : nb) * kRed;
}

cudaError_t init_cg_attributes() {
  cudaError_t e = cudaFuncSetAttribute(cg_tile_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTileInvSmem);
  if (e != cudaSuccess) return e;
  e = init_strip_attributes();
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(cg_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)p_shared_bytes((kCgClusterMaxN + CT - 1) / CT));
}

cudaError_t launch_cg_cluster(const CgArgs& a, int it0, int it1, int share, cudaStream_t s) {
  // A pair of blocks for every CTA, up to the portable cluster size; where
  // `share` geometries run side by side, no more CTAs than the device holds of
  // all of them (a CTA's share of an iteration is then larger than what the
  // iteration's barriers and 3 x 3 steps cost).
  const int room = std::max(2, 2 * num_sms() / (a.batch * std::max(1, share)));
  const int C = std::max(1, std::min({8, room, (a.nt + 1) / 2}));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(a.batch * C);
  cfg.blockDim = dim3(CLT);
  cfg.dynamicSmemBytes = p_shared_bytes(a.nt);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, cg_cluster_kernel, a, it0, it1);
}

void launch_cg_setup(const CgArgs& a, cudaStream_t s) {
  cudaMemsetAsync(a.state, 0, sizeof(double) * kCgState * a.batch, s);
  cg_tile_inv_kernel<<<dim3(a.nt, a.batch), kTileInvThreads, kTileInvSmem, s>>>(a);
  const int ctas = launch_strip(strip_args(a, a.A, a.X), s);
  cg_rows_kernel<double><<<dim3(a.nt, a.batch), 192, 0, s>>>(a, 1, ctas);
  cg_init_tiles_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a);
  cg_init_final_kernel<<<a.batch, 32, 0, s>>>(a, a.nt);
}

void launch_cg_restart(const CgArgs& a, cudaStream_t s) {
  cg_reopen_kernel<<<(a.batch + 31) / 32, 32, 0, s>>>(a);
  const int ctas = launch_strip(strip_args(a, a.A, a.X), s);
  cg_rows_kernel<double><<<dim3(a.nt, a.batch), 192, 0, s>>>(a, 1, ctas);
  cg_init_tiles_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a);
  cg_init_final_kernel<<<a.batch, 32, 0, s>>>(a, a.nt);
}

void launch_cg_iteration(const CgArgs& a, int it, cudaStream_t s, bool fp32) {
  const int nb = (a.N + AT - 1) / AT;
  if (fp32 && a.A32) {
    const int ctas = launch_strip(strip_args(a, a.A32, a.P), s);
    cg_rows_kernel<float><<<dim3(a.nt, a.batch), 192, 0, s>>>(a, 0, ctas);
  } else {
    const int ctas = launch_strip(strip_args(a, a.A, a.P), s);
    cg_rows_kernel<double><<<dim3(a.nt, a.batch), 192, 0, s>>>(a, 0, ctas);
  }
  cg_update_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a, it);
  cg_dir_kernel<<<dim3(nb, a.batch), AT, 0, s>>>(a, it);
}

}  // namespace mbd
