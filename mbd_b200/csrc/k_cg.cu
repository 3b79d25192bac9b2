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
//   cg_strip   partials of A P from the FP32 copy (the lower half serves both
//              triangles); cg_tile from the FP64 matrix
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
#include <type_traits>

#include "chol64.cuh"
#include "kernels.h"

namespace mbd {
namespace {

constexpr int CT = 64;       // tile edge (rows)
constexpr int AT = 64;       // atoms per CTA in the per-atom kernels
constexpr int kRed = 10;     // per-CTA partial sums: a 3x3 matrix and one scalar
// state[f][kCgState]: [0] stop (0 run, 1 converged, 2 breakdown, 3 negative
// curvature), [1] iterations, [2..10] Z^T R (even iterations), [11..19] Z^T R
// (odd), [20] R^T R, [kCgIndefinite] 1 when the relay matrix is shown not to
// be positive definite
constexpr int kZR0 = 2, kRR = 20;

__device__ __forceinline__ void cg_tri(int t, int* ti, int* tj) {
  int i = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((i + 1) * (i + 2) / 2 <= t) ++i;
  while (i * (i + 1) / 2 > t) --i;
  *ti = i;
  *tj = t - i * (i + 1) / 2;
}

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

// partial[f][I][J][64 x 3] = A_IJ v_J, and A_IJ^T v_I into [J][I] (I > J).
// Grid-stride over (tile, frequency) items, so that the launches after every
// frequency has converged cost a few microseconds.  Thread (ty, tx) of 16 x 16
// holds the 16 tile entries of rows ty + 16 i and columns {2 tx, 2 tx + 1,
// 32 + 2 tx, 33 + 2 tx} in registers (16-byte loads, a warp reads two 256-byte
// row segments per instruction), forms their row and column products with v
// (6 FMAs per entry) and the 16 partial sums of every output meet in shared
// memory (fixed order).
constexpr int TT = 256;           // threads of cg_tile
constexpr int RP = CT * 3 + 1;    // row stride of the partial-sum buffer (bank spread)

// A float as a double by integer operations: the conversion instruction has an
// eighth of the ALU's rate, and its queue can set a pass's time.  Zeros
// and denormals come out as some 1e-38, infinities and NaN as some 1e38 (the
// residual gate turns such a solve away).
__device__ __forceinline__ double widen(float x) {
  const int b = __float_as_int(x);
  return __hiloint2double(((b >> 3) & 0x8fffffff) + 0x38000000, b << 29);
}

__global__ void __launch_bounds__(TT, 3) cg_tile_kernel(CgArgs a, const double* in) {
  __shared__ __align__(16) double xI[CT * 3], xJ[CT * 3];
  __shared__ double buf[16 * RP];
  const int ntiles = a.nt * (a.nt + 1) / 2;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int n = a.n;
  const long long items = (long long)ntiles * a.batch;
  for (long long item = blockIdx.x; item < items; item += gridDim.x) {
    const int f = (int)(item / ntiles);
    if (stopped(a, f)) {
      // skip to this CTA's first item of the next frequency (uniform over the CTA)
      const long long next = (long long)(f + 1) * ntiles;
      item += (next - item - 1) / gridDim.x * gridDim.x;
      continue;
    }
    int ti, tj;
    cg_tri((int)(item % ntiles), &ti, &tj);
    const bool diag = ti == tj;
    const double* A = a.A + (size_t)f * a.a_stride;
    const double* x = in + (size_t)f * a.ystride;
    // the 16 entries (pair loads; rows start 16-byte aligned, ld a multiple
    // of 32; an entry beyond n or above the diagonal reads as zero)
    double t[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty + 16 * i, gr = ti * CT + r;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = 2 * tx + 32 * h, gc = tj * CT + c;
        double2 v = make_double2(0.0, 0.0);
        if (gr < n && gc < n && (!diag || c <= r)) v = *reinterpret_cast<const double2*>(A + (size_t)gr * a.ld + gc);
        t[i][2 * h] = v.x;
        t[i][2 * h + 1] = (gc + 1 < n && (!diag || c + 1 <= r)) ? v.y : 0.0;
      }
    }
    __syncthreads();   // the previous item's reads of xI / xJ / buf are done
    for (int idx = tid; idx < CT * 3; idx += TT) {
      const int gi = ti * CT + idx / 3, gj = tj * CT + idx / 3;
      xI[idx] = gi < n ? x[(size_t)ti * CT * 3 + idx] : 0.0;
      xJ[idx] = gj < n ? x[(size_t)tj * CT * 3 + idx] : 0.0;
    }
    __syncthreads();
    double rs[4][3], cs[4][3];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = 0; q < 3; ++q) rs[k][q] = cs[k][q] = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty + 16 * i;
      double xi[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) xi[q] = xI[3 * r + q];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = 2 * tx + 32 * (j >> 1) + (j & 1);
        const double e = t[i][j];
        const double ec = (!diag || c < r) ? e : 0.0;   // the diagonal counts once (row side)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          rs[i][q] += e * xJ[3 * c + q];
          cs[j][q] += ec * xi[q];
        }
      }
    }
    double* pr = a.partial + (size_t)f * a.nt * a.nt * CT * 3;
    // row sums: the 16 column groups of each row
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 3; ++q) buf[tx * RP + 3 * (ty + 16 * i) + q] = rs[i][q];
    __syncthreads();
    double y = 0.0;
    if (tid < CT * 3) {
#pragma unroll
      for (int k = 0; k < 16; ++k) y += buf[k * RP + tid];
    }
    __syncthreads();
    // column sums: the 16 row groups of each column
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = 2 * tx + 32 * (j >> 1) + (j & 1);
#pragma unroll
      for (int q = 0; q < 3; ++q) buf[ty * RP + 3 * c + q] = cs[j][q];
    }
    __syncthreads();
    if (tid < CT * 3) {
      double z = 0.0;
#pragma unroll
      for (int k = 0; k < 16; ++k) z += buf[k * RP + tid];
      if (!diag) {
        pr[((size_t)ti * a.nt + tj) * CT * 3 + tid] = y;
        pr[((size_t)tj * a.nt + ti) * CT * 3 + tid] = z;
      } else {
        pr[((size_t)ti * a.nt + ti) * CT * 3 + tid] = y + z;
      }
    }
  }
}

// ---- FP32 matrix pass ---------------------------------------------------------
// The same partials from the FP32 copy in chunks of 64 x 128 entries, row
// block after row block, frequency after frequency; every CTA (one an SM)
// takes an equal run of chunks.  A warp has 8 rows of a chunk, four entries of
// every row per lane, brought by 16-byte asynchronous copies three chunks
// ahead (512 bytes of a row each; a lane reads what it copied itself).  Row
// sums stay in registers to the end of the row block or the run; column sums
// cross the eight warps in shared memory, added up while the next chunk is
// worked on, with one barrier a chunk.  Four products are summed in FP32, two
// to an instruction (the pass would otherwise stay bound by its 12 FP64 FMAs
// per entry, not by its halved bytes), everything beyond in FP64: the sums
// carry a relative error of a few 1e-7, below what either phase of that solve
// resolves (rms against the FP64 pass 2.6e-8 of the largest entry, as the
// 64 x 64 tile kernel before).
// Slots (the three vectors apart) written in partial[f], row block I: [I][2 c]
// by a run's piece of the row block that begins at chunk c, [I][I] by the last
// piece together with the diagonal block's columns, and [J][I] with the
// columns of the blocks J < I.
// Bound: instruction issue and the FP64 conversions of the sums; the bytes
// alone (half a matrix per frequency) take half the time.  21 matrices of
// n = 6000 (1.5 GB): 0.69 ms by tiles with all sums through shared memory,
// 0.45 now, 0.23 without the arithmetic; an iteration 775 -> 523 us, of
// n = 3000 223 -> 171 us, of n = 2100 126 -> 105 us.
constexpr int RW = 8;                       // rows of a warp
constexpr int ST = 32 * CT / RW;            // threads
constexpr int kStripRing = 4;               // chunks of a CTA in shared memory, one in use
constexpr int kColsElems = 2 * (CT / 4) * 3 * 128;
constexpr int kXElems = 3 * 128 + 3 * CT;   // v on a chunk's columns and rows
constexpr size_t kStripSmem =
    sizeof(float) * (kColsElems + (size_t)kStripRing * CT * 128) + sizeof(double) * kStripRing * kXElems;
constexpr int kMaxActive = 32;              // frequencies of a launch

// Chunks of the row blocks before block I, and the row block of chunk t.
__host__ __device__ inline int chunks_before(int I) { return (I + 1) / 2 * ((I + 2) / 2); }
__device__ __forceinline__ int chunk_row(int t) {
  int m, o;
  cg_tri(t / 2, &m, &o);                    // m (m + 1) <= t < (m + 1) (m + 2)
  return t < (m + 1) * (m + 1) ? 2 * m : 2 * m + 1;
}
// Chunks of a CTA's run when `act` frequencies of nt row blocks take part.
__device__ __forceinline__ int strip_run(int nt, int act, int ctas) { return (chunks_before(nt) * act + ctas - 1) / ctas; }

// The frequencies that still run, as a mask; all threads of a warp.
__device__ __forceinline__ unsigned running(const CgArgs& a) {
  const int lane = threadIdx.x & 31;
  return __ballot_sync(0xffffffffu, lane < a.batch && !stopped(a, lane));
}

// Two floats in one register pair, and the instructions that take them.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ void ring_copy(unsigned dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ring_copy(float4* dst, const float* src) {
  ring_copy((unsigned)__cvta_generic_to_shared(dst), src);
}

__global__ void __launch_bounds__(ST, 1) cg_strip_kernel(CgArgs a, const double* in) {
  __shared__ __align__(16) float xs[2][3][128], xi[2][CT][8];
  __shared__ double ys[2][CT * 3];
  extern __shared__ __align__(16) float dyn[];
  float* cols = dyn;                                   // [2][16][3 x 128]: sums of four rows
  float4* ring = reinterpret_cast<float4*>(dyn + kColsElems) + threadIdx.x;   // [kStripRing][RW][ST], each lane's own
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = a.n, per = chunks_before(a.nt);
  const unsigned act = running(a);
  const int run = strip_run(a.nt, __popc(act), gridDim.x);
  int pos = blockIdx.x * run;
  const int end = min(pos + run, per * __popc(act));
  if (pos >= end) return;
  struct At {                               // chunk c of row block I of frequency f
    int f, I, c;
  };
  auto advance = [&](At& w) {
    if (w.c++ < w.I / 2) return;
    w.c = 0;
    if (++w.I < a.nt) return;
    w.I = 0;
    w.f = __fns(act, w.f + 1, 1);           // -1 behind the last one, not used
  };
  At w;
  w.f = __fns(act, 0, pos / per + 1);
  w.I = chunk_row(pos % per);
  w.c = pos % per - chunks_before(w.I);
  int c0 = w.c;                             // where this run's piece of the row block begins
  At pw = w;
  int ppos = pos, slot = 0;
  const unsigned ring_at = (unsigned)__cvta_generic_to_shared(ring);
  // rows past n and columns past the row's end bring some other entry (masked
  // in a row block's last chunk, times a zero of v, or never read)
  constexpr int XC = (3 * 128 + ST - 1) / ST, XR = (3 * CT + ST - 1) / ST;
  double* xring = reinterpret_cast<double*>(dyn + kColsElems + (size_t)kStripRing * CT * 128) + tid;   // each thread's own
  auto issue_x = [&](double* dst, int f_, int first, int count) {
    const int left = min(count, 3 * n - first) - tid;   // elements at tid, tid + ST, ...
    const double* src = in + (size_t)f_ * a.ystride + (left > 0 ? first + tid : 0);
    for (int u = 0; ST * u < count; ++u)
      if (tid + ST * u < count) {
        const bool ok = ST * u < left;
        const unsigned d = (unsigned)__cvta_generic_to_shared(dst + ST * u);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(ok ? src + ST * u : src), "r"(ok ? 8 : 0) : "memory");
      }
  };
  auto issue = [&](int to) {                // a chunk of the matrix, and v for the one behind it
    if (ppos < end) {
      const float* src = a.A32 + (size_t)pw.f * a.a_stride + (size_t)pw.I * CT * a.ld + min(128 * pw.c + 4 * lane, a.ld - 4);
      const int rmax = n - 1 - pw.I * CT;
      const unsigned d = ring_at + to * (RW * ST * 16);
      if (rmax >= CT - 1) {
        const float* row = src + (size_t)(RW * warp) * a.ld;
#pragma unroll
        for (int r = 0; r < RW; ++r) ring_copy(d + r * (ST * 16), row + (size_t)(unsigned)r * a.ld);
      } else {
#pragma unroll
        for (int r = 0; r < RW; ++r)
          ring_copy(d + r * (ST * 16), src + (size_t)(unsigned)min(RW * warp + r, rmax) * a.ld);
      }
      advance(pw);
      if (++ppos < end) {
        issue_x(xring + to * kXElems, pw.f, 128 * 3 * pw.c, 3 * 128);
        if (pw.c == 0) issue_x(xring + to * kXElems + 3 * 128, pw.f, CT * 3 * pw.I, 3 * CT);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int d = 0; d < kStripRing - 1; ++d) issue(d);
  // v on the chunk's 128 columns and on the row block, the three vectors apart
  // (element e: vector e % 3 of row e / 3)
  auto x_at = [&](int f_, int first, int e, int count) {
    return e < count && first + e < 3 * n ? in[(size_t)f_ * a.ystride + first + e] : 0.0;
  };
  auto put_col = [&](int p, int e, double v) {
    if (e < 3 * 128) xs[p][e % 3][e / 3] = (float)v;
  };
  auto put_row = [&](int p, int e, double v) {
    if (e < 3 * CT) *reinterpret_cast<float2*>(&xi[p][e / 3][2 * (e % 3)]) = make_float2((float)v, (float)v);
  };
#pragma unroll
  for (int u = 0; u < XC; ++u) put_col(0, tid + ST * u, x_at(w.f, 128 * 3 * w.c, tid + ST * u, 3 * 128));
#pragma unroll
  for (int u = 0; u < XR; ++u) put_row(0, tid + ST * u, x_at(w.f, CT * 3 * w.I, tid + ST * u, 3 * CT));
  // the columns of a chunk whose sums all warps have put into cols[p]
  auto columns = [&](const At& o, int p) {
    double* pr = a.partial + (size_t)o.f * a.nt * a.nt * CT * 3;
#pragma unroll
    for (int u = 0; u < XC; ++u) {
      const int e = tid + ST * u, q = e / 128, J = 2 * o.c + e % 128 / CT, k = CT * q + e % CT;
      if (e >= 3 * 128 || J > o.I) continue;
      double z[4] = {J == o.I ? ys[p][k] : 0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int g = 0; g < CT / 4; ++g)   // half of the conversions on either pipe: 2 % of the pass
        z[g % 4] += g % 2 ? widen(cols[(CT / 4 * p + g) * 3 * 128 + e]) : (double)cols[(CT / 4 * p + g) * 3 * 128 + e];
      pr[((size_t)J * a.nt + o.I) * CT * 3 + k] = (z[0] + z[1]) + (z[2] + z[3]);
    }
  };
  __syncthreads();
  double rs[RW][3];
#pragma unroll
  for (int r = 0; r < RW; ++r) rs[r][0] = rs[r][1] = rs[r][2] = 0.0;
  At prev = w;
  for (int p = 0, ip = 0, first = 1;; p ^= 1, first = 0) {
    const bool diag = w.c == w.I / 2, more = ++pos < end, same = more && !diag;
    At nw = w;
    advance(nw);
    asm volatile("cp.async.wait_group %0;" ::"n"(kStripRing - 2) : "memory");
    const float4* mine = ring + slot * RW * ST;
    const double* xmine = xring + slot * kXElems;
    issue(slot == 0 ? kStripRing - 1 : slot - 1);      // the slot of the last chunk
    slot = slot + 1 == kStripRing ? 0 : slot + 1;
    ulonglong2 xj[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) xj[q] = *reinterpret_cast<const ulonglong2*>(&xs[p][q][4 * lane]);
    float* co = cols + (CT / 4 * p + RW / 4 * warp) * 3 * 128 + 4 * lane;
    auto chunk = [&](auto diag_tag) {
      ulonglong2 cs[3];
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        ulonglong2 e = *reinterpret_cast<const ulonglong2*>(mine + r * ST), ec = e;
        if constexpr (decltype(diag_tag)::value) {   // nothing above the diagonal, the diagonal on the row side
          const int d = 128 * w.c + 4 * lane - (w.I * CT + RW * warp + r);
          float e0, e1, e2, e3;
          unpack2(e.x, e0, e1);
          unpack2(e.y, e2, e3);
          e0 = d <= 0 ? e0 : 0.f, e1 = d <= -1 ? e1 : 0.f, e2 = d <= -2 ? e2 : 0.f, e3 = d <= -3 ? e3 : 0.f;
          e = make_ulonglong2(pack2(e0, e1), pack2(e2, e3));
          ec = make_ulonglong2(pack2(d < 0 ? e0 : 0.f, d < -1 ? e1 : 0.f), pack2(d < -2 ? e2 : 0.f, d < -3 ? e3 : 0.f));
        }
        const ulonglong2 x01 = *reinterpret_cast<const ulonglong2*>(&xi[ip][RW * warp + r][0]);
        const unsigned long long x[3] = {x01.x, x01.y, *reinterpret_cast<const unsigned long long*>(&xi[ip][RW * warp + r][4])};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          float v0, v1;
          unpack2(fma2(e.y, xj[q].y, mul2(e.x, xj[q].x)), v0, v1);
          if constexpr (decltype(diag_tag)::value) {   // the diagonal's product is rounded once
            rs[r][q] += (double)v0 + (double)v1;
          } else {
            rs[r][q] += (double)(v0 + v1);
          }
          cs[q].x = r % 4 == 0 ? mul2(ec.x, x[q]) : fma2(ec.x, x[q], cs[q].x);
          cs[q].y = r % 4 == 0 ? mul2(ec.y, x[q]) : fma2(ec.y, x[q], cs[q].y);
          if (r % 4 == 3) *reinterpret_cast<ulonglong2*>(co + (r / 4 * 3 + q) * 128) = cs[q];
        }
      }
    };
    if (diag) {
      chunk(std::true_type());
    } else {
      chunk(std::false_type());
    }
    if (!first) columns(prev, p ^ 1);
    if (!same) {
      // RW rows over 32 lanes: halves exchanged until every lane has one row, then the lanes of a row add up
      double* pr = a.partial + (size_t)w.f * a.nt * a.nt * CT * 3;
      constexpr int L = 32 / RW;            // lanes of a row
      auto fold = [&](auto half) {
        constexpr int h = decltype(half)::value;
        const bool up = lane & (L * h);
#pragma unroll
        for (int r = 0; r < h; ++r)
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const double a0 = rs[r][q], a1 = rs[r + h][q];
            const double got = __shfl_xor_sync(0xffffffffu, up ? a0 : a1, L * h);
            rs[r][q] = (up ? a1 : a0) + got;
          }
      };
      fold(std::integral_constant<int, 4>());
      fold(std::integral_constant<int, 2>());
      fold(std::integral_constant<int, 1>());
      const int row = RW * warp + lane / L;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        double y = rs[0][q];
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (lane % L == 0) {
          if (diag) {
            ys[p][CT * q + row] = y;
          } else {
            pr[((size_t)w.I * a.nt + 2 * c0) * CT * 3 + CT * q + row] = y;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < RW; ++r) rs[r][0] = rs[r][1] = rs[r][2] = 0.0;
      if (more) {
#pragma unroll
        for (int u = 0; u < XR; ++u) if (tid + ST * u < 3 * CT) put_row(ip ^ 1, tid + ST * u, xmine[3 * 128 + ST * u]);
      }
    }
    if (more) {
#pragma unroll
      for (int u = 0; u < XC; ++u) if (tid + ST * u < 3 * 128) put_col(p ^ 1, tid + ST * u, xmine[ST * u]);
    }
    __syncthreads();   // the other copy of each buffer was last read before this barrier
    if (!more) {
      columns(w, p);
      return;
    }
    prev = w;
    if (!same) ip ^= 1, c0 = nw.c;
    w = nw;
  }
}

// Row sums y = (A v) of 64-row block I.  init: R = B - y.  Otherwise Q = y and
// the block's partial of P^T Q goes to red[f][I].  The partials are those of
// cg_strip_kernel or of cg_tile_kernel.
__global__ void __launch_bounds__(192) cg_rows_kernel(CgArgs a, int init, int strips) {
  const int I = blockIdx.x, f = blockIdx.y;
  if (stopped(a, f)) return;
  __shared__ double sm[kRed * 32];
  const int tid = threadIdx.x;
  const int r = tid / 3, q = tid % 3;
  const int gr = I * CT + r;
  const double* pr = a.partial + (size_t)f * a.nt * a.nt * CT * 3 + (size_t)I * a.nt * CT * 3 + (strips ? CT * q + r : tid);
  double y = 0.0;
  if (strips) {   // the CTA count of that launch: the pieces of this row block but the last
    const unsigned act = running(a);
    const int run = strip_run(a.nt, __popc(act), strips);
    const int first = __popc(act & ((1u << f) - 1)) * chunks_before(a.nt) + chunks_before(I), last = first + I / 2;
    for (int x = first, end; (end = (x / run + 1) * run) <= last; x = end) y += pr[(size_t)(2 * (x - first)) * CT * 3];
  } else {
    for (int J = 0; J < I; ++J) y += pr[(size_t)J * CT * 3];
  }
  for (int J = I; J < a.nt; ++J) y += pr[(size_t)J * CT * 3];
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
// cg_strip_kernel: four products in FP32, everything beyond in FP64.
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
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

// CTAs of the grid-stride tile launch: every resident slot of the device.
int cg_tile_grid() {
  static int grid = 0;
  if (grid == 0) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cg_tile_kernel, TT, 0);
    grid = (sms > 0 ? sms : 148) * (per_sm > 0 ? per_sm : 1);
  }
  return grid;
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
  e = cudaFuncSetAttribute(cg_strip_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStripSmem);
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
  const long long items = (long long)a.nt * (a.nt + 1) / 2 * a.batch;
  const int tgrid = (int)std::min<long long>(cg_tile_grid(), items);
  cudaMemsetAsync(a.state, 0, sizeof(double) * kCgState * a.batch, s);
  cg_tile_inv_kernel<<<dim3(a.nt, a.batch), kTileInvThreads, kTileInvSmem, s>>>(a);
  cg_tile_kernel<<<tgrid, TT, 0, s>>>(a, a.X);
  cg_rows_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a, 1, 0);
  cg_init_tiles_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a);
  cg_init_final_kernel<<<a.batch, 32, 0, s>>>(a, a.nt);
}

void launch_cg_restart(const CgArgs& a, cudaStream_t s) {
  const long long items = (long long)a.nt * (a.nt + 1) / 2 * a.batch;
  const int tgrid = (int)std::min<long long>(cg_tile_grid(), items);
  cg_reopen_kernel<<<(a.batch + 31) / 32, 32, 0, s>>>(a);
  cg_tile_kernel<<<tgrid, TT, 0, s>>>(a, a.X);
  cg_rows_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a, 1, 0);
  cg_init_tiles_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a);
  cg_init_final_kernel<<<a.batch, 32, 0, s>>>(a, a.nt);
}

void launch_cg_iteration(const CgArgs& a, int it, cudaStream_t s, bool fp32) {
  const int nb = (a.N + AT - 1) / AT;
  const long long items = (long long)a.nt * (a.nt + 1) / 2 * a.batch;
  const int tgrid = (int)std::min<long long>(cg_tile_grid(), items);
  int strips = 0;
  if (fp32 && a.A32 && a.batch <= kMaxActive) {
    strips = std::min(num_sms(), chunks_before(a.nt) * a.batch);
    cg_strip_kernel<<<strips, ST, kStripSmem, s>>>(a, a.P);
  } else {
    cg_tile_kernel<<<tgrid, TT, 0, s>>>(a, a.P);
  }
  cg_rows_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a, 0, strips);
  cg_update_kernel<<<dim3(a.nt, a.batch), 192, 0, s>>>(a, it);
  cg_dir_kernel<<<dim3(nb, a.batch), AT, 0, s>>>(a, it);
}

}  // namespace mbd
