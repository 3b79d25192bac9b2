// FP64 relay solve of the plain path, X = A^-1 [I;I;..;I] (PDPOTRS at
// UTILS.f90:473) from the factors of k_cholflow.cu, and the reductions of
// get_screened_alpha / MBD_at_rsSCS (UTILS.f90:479-495, 272-315, 731-741).
#include <cooperative_groups.h>
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
// X = (L L^T)^-1 [I; ..; I] in one launch, a thread-block cluster per matrix:
// z_k = Linv_k (b_k - sum_{p<k} L(k,p) z_p) down, x_k = Linv_k^T (z_k -
// sum_{i>k} L(i,k)^T x_i) up.  Block p (i) of a sum belongs to the CTA p mod C;
// a step's partial sums go into every CTA's shared memory before the cluster
// barrier, and every CTA forms the block of the solution itself (the solution
// stays in shared memory).  While the barrier is on its way a CTA sums all but
// the newest block of the next step, so the chain per step is one 64 x 64
// block, the exchange and the product with the inverse.  Bound by that chain
// (2 ceil(n/64) steps) and, for large n, by reading L twice.
constexpr int kTrsvThreads = 256;
constexpr int kTrsvMaxC = 4;

__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

__global__ void __launch_bounds__(kTrsvThreads) trsv_cluster_kernel(BatchMat m, const double* Linv, size_t linv_stride,
                                                                    double* X, size_t ystride) {
  namespace cgr = cooperative_groups;
  cgr::cluster_group cl = cgr::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int b = blockIdx.x / C;
  extern __shared__ __align__(16) double sh[];
  cl.barrier_arrive();                              // the cluster's CTAs have started: waited for before the first push
  const int n = m.n, T = (n + NB - 1) / NB, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* Z = sh;                                   // [T * 64][3]: z, overwritten by x
  double* buf = Z + (size_t)T * NB * 3;             // [2][C][192]: the CTAs' partial sums
  double* w = buf + 2 * kTrsvMaxC * NB * 3;         // [192]
  double* red = w + NB * 3;                         // [8][192]
  const double* A = m.A + (size_t)b * m.stride;
  const double* Li = Linv + (size_t)b * linv_stride;
  auto push = [&](int k, int idx, double v) {       // entry idx of this CTA's partial sum, to all
    for (int c = 0; c < C; ++c) cl.map_shared_rank(buf, c)[((k & 1) * kTrsvMaxC + rank) * NB * 3 + idx] = v;
  };
  // ---- down: thread (row, j) of a block row holds columns 2 j + 8 u, + 1
  const int row = tid >> 2, j = tid & 3;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  auto rows_block = [&](const double2 (&v)[8], int p) {
    const double* zp = Z + (size_t)p * NB * 3;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double* z0 = zp + 3 * (2 * j + 8 * u);
      a0 += v[u].x * z0[0];
      a1 += v[u].x * z0[1];
      a2 += v[u].x * z0[2];
      a0 += v[u].y * z0[3];
      a1 += v[u].y * z0[4];
      a2 += v[u].y * z0[5];
    }
  };
  auto rows_load = [&](double2 (&v)[8], int k, int p) {
    const int gr = k * NB + row;
    const double* src = A + (size_t)min(gr, n - 1) * m.ld + p * NB + 2 * j;
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = *reinterpret_cast<const double2*>(src + 8 * u);
  };
  cl.barrier_wait();
  for (int k = 0; k < T; ++k) {
    a0 = quad_sum(a0);
    a1 = quad_sum(a1);
    a2 = quad_sum(a2);
    if (j < 3) push(k, 3 * row + j, j == 0 ? a0 : (j == 1 ? a1 : a2));
    cl.barrier_arrive();
    a0 = a1 = a2 = 0.0;
    double2 v[8], li[8];
    const bool more = k + 1 < T;
    if (more)
      for (int p = rank; p < k; p += C) {
        rows_load(v, k + 1, p);
        rows_block(v, p);
      }
    const bool mine = more && k % C == rank;
    if (mine) rows_load(v, k + 1, k);
    const double* lk = Li + (size_t)k * NB * NB + row * NB + 2 * j;
#pragma unroll
    for (int u = 0; u < 8; ++u) li[u] = *reinterpret_cast<const double2*>(lk + 8 * u);
    cl.barrier_wait();
    if (tid < NB * 3) {
      const int gr = k * NB + tid / 3;
      double s = (gr < n && gr % 3 == tid % 3) ? 1.0 : 0.0;
      const double* pb = buf + (k & 1) * kTrsvMaxC * NB * 3 + tid;
      for (int c = 0; c < C; ++c) s -= pb[c * NB * 3];
      w[tid] = gr < n ? s : 0.0;
    }
    __syncthreads();
    double z0 = 0.0, z1 = 0.0, z2 = 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double* wp = w + 3 * (2 * j + 8 * u);
      z0 += li[u].x * wp[0] + li[u].y * wp[3];
      z1 += li[u].x * wp[1] + li[u].y * wp[4];
      z2 += li[u].x * wp[2] + li[u].y * wp[5];
    }
    z0 = quad_sum(z0);
    z1 = quad_sum(z1);
    z2 = quad_sum(z2);
    if (j < 3) Z[(size_t)(k * NB + row) * 3 + j] = j == 0 ? z0 : (j == 1 ? z1 : z2);
    __syncthreads();
    if (mine) rows_block(v, k);
  }
  cl.sync();   // the last step's partial sums are read: the way up starts over in the same buffers
  // ---- up: lane holds columns 2 lane, + 1 of a block column, warp its rows 8 warp ..
  double c0[3] = {0.0, 0.0, 0.0}, c1[3] = {0.0, 0.0, 0.0};
  auto cols_load = [&](double2 (&v)[8], int i, int k) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int gr = i * NB + 8 * warp + u;
      v[u] = *reinterpret_cast<const double2*>(A + (size_t)min(gr, n - 1) * m.ld + k * NB + 2 * lane);
    }
  };
  auto cols_block = [&](const double2 (&v)[8], int i) {   // x is zero past n
    const double* xp = Z + (size_t)(i * NB + 8 * warp) * 3;
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        c0[q] += v[u].x * xp[3 * u + q];
        c1[q] += v[u].y * xp[3 * u + q];
      }
  };
  for (int k = T - 1; k >= 0; --k) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      red[warp * NB * 3 + 3 * (2 * lane) + q] = c0[q];
      red[warp * NB * 3 + 3 * (2 * lane + 1) + q] = c1[q];
      c0[q] = c1[q] = 0.0;
    }
    __syncthreads();
    if (tid < NB * 3) {
      double s = 0.0;
#pragma unroll
      for (int v = 0; v < 8; ++v) s += red[v * NB * 3 + tid];
      push(k, tid, s);
    }
    cl.barrier_arrive();
    double2 v[8];
    const bool more = k > 0;
    if (more)
      for (int i = T - 1 - (T - 1 - rank % C + C) % C; i > k; i -= C) {   // blocks i = rank (mod C), from the last
        cols_load(v, i, k - 1);
        cols_block(v, i);
      }
    const bool mine = more && k % C == rank;
    if (mine) cols_load(v, k, k - 1);
    // Linv_k^T: column tid % 64, rows 16 (tid / 64) ..
    double li[16];
    const double* lk = Li + (size_t)k * NB * NB + (size_t)(tid >> 6) * 16 * NB + (tid & 63);
#pragma unroll
    for (int u = 0; u < 16; ++u) li[u] = lk[(size_t)u * NB];
    cl.barrier_wait();
    if (tid < NB * 3) {
      double s = Z[(size_t)k * NB * 3 + tid];
      const double* pb = buf + (k & 1) * kTrsvMaxC * NB * 3 + tid;
      for (int c = 0; c < C; ++c) s -= pb[c * NB * 3];
      w[tid] = k * NB + tid / 3 < n ? s : 0.0;
    }
    __syncthreads();
    {
      const double* wp = w + (size_t)(tid >> 6) * 48;
      double x0 = 0.0, x1 = 0.0, x2 = 0.0;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        x0 += li[u] * wp[3 * u];
        x1 += li[u] * wp[3 * u + 1];
        x2 += li[u] * wp[3 * u + 2];
      }
      double* r = red + (size_t)(tid >> 6) * NB * 3 + 3 * (tid & 63);
      r[0] = x0;
      r[1] = x1;
      r[2] = x2;
    }
    __syncthreads();
    if (tid < NB * 3) {
      const double x = (red[tid] + red[NB * 3 + tid]) + (red[2 * NB * 3 + tid] + red[3 * NB * 3 + tid]);
      const bool in = k * NB + tid / 3 < n;
      Z[(size_t)k * NB * 3 + tid] = in ? x : 0.0;
      if (in && k % C == rank) X[(size_t)b * ystride + (size_t)k * NB * 3 + tid] = x;
    }
    __syncthreads();
    if (mine) cols_block(v, k);
  }
  cl.sync();   // no CTA leaves while another may still write into its shared memory
}

size_t trsv_smem(int n) {
  const size_t T = (n + NB - 1) / NB;
  return sizeof(double) * NB * 3 * (T + 2 * kTrsvMaxC + 1 + 8);
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

cudaError_t init_trsv_attributes() {
  return cudaFuncSetAttribute(trsv_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)trsv_smem(kTrsvMaxN));
}

cudaError_t launch_trsv_cluster(const BatchMat& m, const double* Linv, size_t linv_stride, double* X, size_t ystride,
                                cudaStream_t s) {
  const int T = (m.n + NB - 1) / NB;
  // Solve of one cluster (ms) with 1, 2, 4 and 8 CTAs a frequency: n = 126 0.031,
  // 0.031, 0.031, 0.035; 384 0.055, 0.051, 0.049, 0.059 (two leave more room for
  // other geometries); 999 0.24, 0.17, 0.14, 0.15; 3000 1.96, 1.12, 0.71, 0.72; 6000
  // 6.9, 3.8, 2.2, 2.6 (eight: fewer clusters at once, a longer exchange).
  const int C = T <= 2 ? 1 : (T <= 6 ? 2 : 4);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(m.batch * C);
  cfg.blockDim = dim3(kTrsvThreads);
  cfg.dynamicSmemBytes = trsv_smem(m.n);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, trsv_cluster_kernel, m, Linv, linv_stride, X, ystride);
}

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
