// FP64 relay solve of the plain path, X = A^-1 [I;I;..;I] (PDPOTRS at
// UTILS.f90:473) from the factors of k_cholflow.cu, and the reductions of
// get_screened_alpha / MBD_at_rsSCS (UTILS.f90:479-495, 272-315, 731-741).
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"

namespace mbd {
namespace {

constexpr int NB = kCholNB;  // 64

// ---------------------------------------------------------------------------
__global__ void init_rhs_kernel(double* Y, size_t ystride, int n, int batch) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t total = (size_t)n * 3 * batch;
  if (idx >= total) return;
  int b = (int)(idx / ((size_t)n * 3));
  int rem = (int)(idx % ((size_t)n * 3));
  int r = rem / 3, c = rem % 3;
  Y[(size_t)b * ystride + (size_t)r * 3 + c] = (r % 3 == c) ? 1.0 : 0.0;
}

// Forward step for block k0: z_k = Linv_k w_k; w[rows below] -= L[rows, k] z_k.
// Every CTA recomputes z_k in shared memory; CTA 0 stores it into Z.  The
// working right-hand side W is only read at block k and only written below
// it, so no CTA reads a value another CTA of the same launch writes.
__global__ void __launch_bounds__(256) trsv_fwd_kernel(BatchMat m, int k0, const double* Linv,
                                                      size_t linv_stride, double* W, double* Z,
                                                      size_t ystride) {
  __shared__ double yk[NB][3];
  __shared__ double bk[NB][3];
  const int b = blockIdx.y;
  const double* A = m.A + (size_t)b * m.stride;
  double* y = W + (size_t)b * ystride;
  double* z = Z + (size_t)b * ystride;
  const double* Li = Linv + (size_t)b * linv_stride + (size_t)(k0 / NB) * NB * NB;
  const int nbk = min(NB, m.n - k0);
  const int tid = threadIdx.x;
  for (int idx = tid; idx < NB * 3; idx += blockDim.x) {
    int r = idx / 3, c = idx % 3;
    bk[r][c] = (r < nbk) ? y[(size_t)(k0 + r) * 3 + c] : 0.0;
  }
  __syncthreads();
  for (int idx = tid; idx < NB * 3; idx += blockDim.x) {
    int r = idx / 3, c = idx % 3;
    double acc = 0.0;
    for (int l = 0; l <= r; ++l) acc += Li[r * NB + l] * bk[l][c];
    yk[r][c] = acc;
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int idx = tid; idx < nbk * 3; idx += blockDim.x) z[(size_t)(k0 + idx / 3) * 3 + idx % 3] = yk[idx / 3][idx % 3];
  // warp per row
  const int warp = tid / 32, lane = tid % 32;
  const int rows_per_cta = 64;
  const int rbase = k0 + nbk + blockIdx.x * rows_per_cta;
  for (int rr = warp; rr < rows_per_cta; rr += blockDim.x / 32) {
    const int r = rbase + rr;
    if (r >= m.n) break;
    double s0 = 0, s1 = 0, s2 = 0;
    for (int l = lane; l < nbk; l += 32) {
      double a = A[(size_t)r * m.ld + k0 + l];
      s0 += a * yk[l][0];
      s1 += a * yk[l][1];
      s2 += a * yk[l][2];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
      y[(size_t)r * 3 + 0] -= s0;
      y[(size_t)r * 3 + 1] -= s1;
      y[(size_t)r * 3 + 2] -= s2;
    }
  }
}

// Backward step for block k0: x_k = Linv_k^T z_k; z[rows above] -= L[k, rows]^T x_k.
__global__ void __launch_bounds__(256) trsv_bwd_kernel(BatchMat m, int k0, const double* Linv,
                                                      size_t linv_stride, double* Zw, double* X,
                                                      size_t ystride) {
  __shared__ double xk[NB][3];
  __shared__ double bk[NB][3];
  const int b = blockIdx.y;
  const double* A = m.A + (size_t)b * m.stride;
  double* y = Zw + (size_t)b * ystride;
  double* xo = X + (size_t)b * ystride;
  const double* Li = Linv + (size_t)b * linv_stride + (size_t)(k0 / NB) * NB * NB;
  const int nbk = min(NB, m.n - k0);
  const int tid = threadIdx.x;
  for (int idx = tid; idx < NB * 3; idx += blockDim.x) {
    int r = idx / 3, c = idx % 3;
    bk[r][c] = (r < nbk) ? y[(size_t)(k0 + r) * 3 + c] : 0.0;
  }
  __syncthreads();
  for (int idx = tid; idx < NB * 3; idx += blockDim.x) {
    int r = idx / 3, c = idx % 3;
    double acc = 0.0;
    for (int l = r; l < NB; ++l) acc += Li[l * NB + r] * bk[l][c];   // (Linv^T)[r][l] = Linv[l][r]
    xk[r][c] = acc;
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int idx = tid; idx < nbk * 3; idx += blockDim.x) xo[(size_t)(k0 + idx / 3) * 3 + idx % 3] = xk[idx / 3][idx % 3];
  // columns j < k0, one thread per j (coalesced along the rows of block k)
  const int j = blockIdx.x * blockDim.x + tid;
  if (j >= k0) return;
  double s0 = 0, s1 = 0, s2 = 0;
  for (int i = 0; i < nbk; ++i) {
    double a = A[(size_t)(k0 + i) * m.ld + j];
    s0 += a * xk[i][0];
    s1 += a * xk[i][1];
    s2 += a * xk[i][2];
  }
  y[(size_t)j * 3 + 0] -= s0;
  y[(size_t)j * 3 + 1] -= s1;
  y[(size_t)j * 3 + 2] -= s2;
}

// ---------------------------------------------------------------------------
// alpha_i = tr X_i / 3 and M = sum_i X_i per frequency (UTILS.f90:487-491).
__global__ void __launch_bounds__(256) relay_reduce_kernel(EpilogueArgs a) {
  const int f = blockIdx.x;
  const double* X = a.X + (size_t)f * a.xstride;
  double m[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = threadIdx.x; i < a.N; i += blockDim.x) {
    const double* x = X + (size_t)(3 * i) * 3;
    a.alpha_iw[(size_t)f * a.N + i] = (x[0] / 3.0 + x[4] / 3.0) + x[8] / 3.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) m[k] += x[k];
  }
  __shared__ double red[9][256];
#pragma unroll
  for (int k = 0; k < 9; ++k) red[k][threadIdx.x] = m[k];
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s)
#pragma unroll
      for (int k = 0; k < 9; ++k) red[k][threadIdx.x] += red[k][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x < 9) a.molpol[f * 9 + threadIdx.x] = red[threadIdx.x][0];
}

// C6_i, alpha_eff, R_vdW_eff, omega (UTILS.f90:302-315, 731-741); block 0
// also forms the system C6 (UTILS.f90:272-288) and sum 3 omega (UTILS.f90:846-848).

__global__ void __launch_bounds__(256) relay_post_kernel(EpilogueArgs a, const double* w) {
  __shared__ double red[256];
  __shared__ int bad[256];
  double s3w = 0.0;
  int nbad = 0;
  for (int i = threadIdx.x; i < a.N; i += blockDim.x) {
    double c6 = 0.0;
    for (int f = 1; f < 21; ++f) {
      double al = a.alpha_iw[(size_t)f * a.N + i];
      c6 = c6 + (w[f] * al * al);
    }
    c6 = c6 * 0.954929658551372;
    const double ae = a.alpha_iw[i];
    a.c6_eff[i] = c6;
    a.alpha_eff[i] = ae;
    a.rvdw_eff[i] = a.r0[i] * pow(ae / a.alpha0[i], 0.33333333333333333333);
    const double om = (4.0 / 3.0) * c6 / (ae * ae);
    a.omega[i] = om;
    s3w += 3.0 * om;
    if (!(ae > 0.0)) ++nbad;
  }
  red[threadIdx.x] = s3w;
  bad[threadIdx.x] = nbad;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) {
      red[threadIdx.x] += red[threadIdx.x + s];
      bad[threadIdx.x] += bad[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double c6m = 0.0;
    for (int f = 1; f < 21; ++f) {
      const double* M = a.molpol + f * 9;
      double iso = (M[0] + M[4] + M[8]) / 3.0;
      c6m = c6m + (w[f] * iso * iso);
    }
    a.scalars[0] = 0.954929658551372 * c6m;
    a.scalars[1] = red[0];
    a.scalars[2] = (double)bad[0];
  }
}

}  // namespace

void launch_init_rhs(double* Y, size_t ystride, int n, int batch, cudaStream_t s) {
  size_t total = (size_t)n * 3 * batch;
  init_rhs_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(Y, ystride, n, batch);
}

void launch_trsv_fwd_step(const BatchMat& m, int k0, const double* Linv, size_t linv_stride, double* W,
                          double* Z, size_t ystride, cudaStream_t s) {
  int nbk = std::min(NB, m.n - k0);
  int rows = m.n - k0 - nbk;
  int ctas = std::max(1, (rows + 63) / 64);
  dim3 grid(ctas, m.batch);
  trsv_fwd_kernel<<<grid, 256, 0, s>>>(m, k0, Linv, linv_stride, W, Z, ystride);
}

void launch_trsv_bwd_step(const BatchMat& m, int k0, const double* Linv, size_t linv_stride, double* Zw,
                          double* X, size_t ystride, cudaStream_t s) {
  int ctas = std::max(1, (k0 + 255) / 256);
  dim3 grid(ctas, m.batch);
  trsv_bwd_kernel<<<grid, 256, 0, s>>>(m, k0, Linv, linv_stride, Zw, X, ystride);
}

void launch_relay_epilogue(const EpilogueArgs& a, cudaStream_t s) {
  relay_reduce_kernel<<<21, 256, 0, s>>>(a);
}

void launch_relay_post(const EpilogueArgs& a, const double* weights_dev, cudaStream_t s) {
  relay_post_kernel<<<1, 256, 0, s>>>(a, weights_dev);
}

}  // namespace mbd
