// Batched FP64 Cholesky A + s I = L L^T as ONE persistent launch: the relay
// matrices of the plain mode (PDPOTRF('L') at UTILS.f90:469) and the shifted
// Hamiltonians of the energy's trace form (k_trace.cu).
//
// The lower triangle is cut into 64-wide block columns.  A task is either a
// block column's diagonal block (update, factor, invert) or a tile of up to
// 128 rows below it (update, multiply by the inverse).  Every task is
// left-looking: it accumulates its whole product sum_p L(i,p) L(k,p)^T in
// registers on the FP64 tensor cores and touches its own tile once, so the
// trailing matrix is never read and written again between block columns (the
// former right-looking kernels moved it once per 64 columns and spent three
// launches on each).  CTAs draw tasks from a ticket in (block column, row
// tile, matrix) order and wait, with a limit, on counters of finished block
// columns; a task waits only for tasks with lower tickets, which running
// CTAs hold, so the launch needs no co-residency.
//
// Bound: FP64 tensor-core rate (36.9 TFLOP/s measured for m8n8k4 with all
// operands in registers) while a block column has tiles for the whole chip;
// below that the chain diagonal block -> tile below it -> next diagonal
// block, n / 64 links of ~32 us.  Measured, 21 relay matrices of n rows (right-looking
// kernels before -> now): n = 3000 17.5 -> 7.6 ms (10.8 -> 24.9 TFLOP/s),
// n = 384 0.85 -> 0.20 ms; n = 6000 53 ms (28.4 TFLOP/s).
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "wait_limit.cuh"

namespace mbd {
namespace {

constexpr int NB = kCholNB;      // 64: block-column width
constexpr int RT = 2 * NB;       // rows of a tile task
constexpr int KC = 16;           // columns of one pipeline stage
constexpr int KS = KC + 4;       // shared row stride: a half-warp's 8 x 4 fragment loads hit 16 bank pairs
constexpr int FS = NB + 4;       // row stride of the 64-wide shared blocks, same reason
constexpr int kStages = 3;
constexpr int kStageElems = (RT + NB) * KS;
constexpr int kFlowThreads = 256;
constexpr size_t kTaskElems = (size_t)(RT + NB) * FS;   // tile + inverse; the stages fit in the same space
constexpr size_t kFlowSmem = sizeof(double) * (kTaskElems > (size_t)kStages * kStageElems ? kTaskElems : (size_t)kStages * kStageElems);
constexpr int kErrTimeout = 7;   // MBD_ERR_TIMEOUT

// D = A B + D with A 8x4 (row), B 4x8 (col), D 8x8 in FP64:
// a = A[lane/4][lane%4], b = B[lane%4][lane/4], d = D[lane/4][2*(lane%4) + {0,1}].
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// 16-byte asynchronous copy global -> shared; src_bytes < 16 zero-fills the rest.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Waits until *p >= want; past the limit (or once any wait has run out) it
// records the time-out and returns `want`, so every task still ends.
__device__ int wait_count(const int* p, int want, int* err) {
  int v = ld_acquire(p);
  if (v >= want) return v;
  const long long limit = wait_limit_cycles();
  const long long t0 = clock64();
  while ((v = ld_acquire(p)) < want) {
    if (*(volatile int*)err != 0) return want;
    if (clock64() - t0 > limit) {
      atomicCAS(err, 0, kErrTimeout);
      return want;
    }
    __nanosleep(20);
  }
  return v;
}

// ---- the 64 x 64 diagonal block -------------------------------------------
// S (row stride FS) holds the updated block's lower triangle; X receives
// L^-1 (zeros above the diagonal).  Two 32-column halves: one warp factors a
// 32 x 32 block with a row per lane, each new column broadcast through
// shared memory (its transpose Lt serves the inverse as well), the products
// between the halves run on the tensor cores of all 8 warps.
constexpr int LTS = 34;

__device__ void warp_potrf32(double* S, double* Lt, double* dinv, int lane, int col0, int n_valid, int* bad,
                             double ref, double* logsum) {
  double a[32];
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    const double2 v = *reinterpret_cast<const double2*>(S + lane * FS + j);
    a[j] = v.x;
    a[j + 1] = v.y;
  }
  double mypiv = 1.0;
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    double piv = __shfl_sync(0xffffffffu, a[c], c);
    if (!(piv > 0.0)) {          // not SPD (or NaN): the first failing column, factor on with a unit pivot
      if (*bad == 0 && col0 + c < n_valid) *bad = col0 + c + 1;
      piv = 1.0;
    }
    const double inv = rsqrt(piv);
    if (lane == c) {
      mypiv = piv;
      dinv[c] = inv;
    }
    const double l = lane > c ? a[c] * inv : (lane == c ? piv * inv : 0.0);
    a[c] = l;
    Lt[c * LTS + lane] = l;
    __syncwarp();
    if (c + 1 < 32) {
      if ((c + 1) & 1) a[c + 1] -= l * Lt[c * LTS + c + 1];
#pragma unroll
      for (int j = (c + 2) & ~1; j < 32; j += 2) {
        const double2 q = *reinterpret_cast<const double2*>(Lt + c * LTS + j);
        a[j] -= l * q.x;
        a[j + 1] -= l * q.y;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 32; j += 2)
    *reinterpret_cast<double2*>(S + lane * FS + j) = make_double2(a[j], a[j + 1]);
  if (logsum) {
    double lg = (col0 + lane < n_valid) ? log(mypiv * ref) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lg += __shfl_xor_sync(0xffffffffu, lg, o);
    *logsum = lg;
  }
  __syncwarp();
}

// X (32 x 32, row stride FS) = L^-1, a column per lane; Lt, dinv from warp_potrf32.
__device__ void warp_inv32(const double* Lt, const double* dinv, double* X, int lane) {
  double x[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = (i == lane) ? 1.0 : 0.0;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const double xi = x[i] * dinv[i];
    x[i] = xi;
    if (i + 1 < 32) {
      if ((i + 1) & 1) x[i + 1] -= xi * Lt[i * LTS + i + 1];
#pragma unroll
      for (int j = (i + 2) & ~1; j < 32; j += 2) {
        const double2 q = *reinterpret_cast<const double2*>(Lt + i * LTS + j);
        x[j] -= xi * q.x;
        x[j + 1] -= xi * q.y;
      }
    }
    X[i * FS + lane] = xi;
  }
  __syncwarp();
}

// acc (16 x 8 of a 32 x 32 product, this warp's part) += A B^T (bt) or A B
// over K = 32; A, B in shared memory with row stride FS.
template <bool BT>
__device__ __forceinline__ void mma32(const double* A, const double* B, int warp, int lane, double acc[2][2]) {
  const int g = lane >> 2, q = lane & 3;
  const int r0 = (warp >> 2) * 16, c0 = (warp & 3) * 8;
#pragma unroll
  for (int kk = 0; kk < 32; kk += 4) {
    const double b = BT ? B[(c0 + g) * FS + kk + q] : B[(kk + q) * FS + c0 + g];
#pragma unroll
    for (int i = 0; i < 2; ++i) dmma(acc[i][0], acc[i][1], A[(r0 + 8 * i + g) * FS + kk + q], b);
  }
}

// Factors S (64 x 64) and inverts the factor into X.  All 256 threads.
__device__ void diag_factor(double* S, double* X, double* Lt, double* dinv, int tid, int col0, int n, int* bad,
                            double ref, double* logsum) {
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int r0 = (warp >> 2) * 16, c0 = (warp & 3) * 8;
  double* A21 = S + 32 * FS;
  double* A22 = S + 32 * FS + 32;
  double* X21 = X + 32 * FS;
  double* X22 = X + 32 * FS + 32;
  double lg0 = 0.0, lg1 = 0.0;
  if (warp == 0) {
    warp_potrf32(S, Lt, dinv, lane, col0, n, bad, ref, logsum ? &lg0 : nullptr);
    warp_inv32(Lt, dinv, X, lane);
  } else if (warp == 1) {
    for (int r = 0; r < 32; ++r) X[r * FS + 32 + lane] = 0.0;
  }
  __syncthreads();
  {   // L21 = A21 L11^-T
    double acc[2][2] = {};
    mma32<true>(A21, X, warp, lane, acc);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i)
      *reinterpret_cast<double2*>(A21 + (r0 + 8 * i + g) * FS + c0 + 2 * q) = make_double2(acc[i][0], acc[i][1]);
  }
  __syncthreads();
  {   // A22 -= L21 L21^T
    double acc[2][2] = {};
    mma32<true>(A21, A21, warp, lane, acc);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      double2* p = reinterpret_cast<double2*>(A22 + (r0 + 8 * i + g) * FS + c0 + 2 * q);
      double2 v = *p;
      v.x -= acc[i][0];
      v.y -= acc[i][1];
      *p = v;
    }
  }
  // W = L21 L11^-1, kept in registers while warp 0 factors A22
  double w[2][2] = {};
  mma32<false>(A21, X, warp, lane, w);
  __syncthreads();
  if (warp == 0) {
    warp_potrf32(A22, Lt, dinv, lane, col0 + 32, n, bad, ref, logsum ? &lg1 : nullptr);
    warp_inv32(Lt, dinv, X22, lane);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)   // L21 is no longer needed: W takes its place
    *reinterpret_cast<double2*>(A21 + (r0 + 8 * i + g) * FS + c0 + 2 * q) = make_double2(w[i][0], w[i][1]);
  __syncthreads();
  {   // X21 = -L22^-1 W
    double acc[2][2] = {};
    mma32<false>(X22, A21, warp, lane, acc);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      *reinterpret_cast<double2*>(X21 + (r0 + 8 * i + g) * FS + c0 + 2 * q) = make_double2(-acc[i][0], -acc[i][1]);
  }
  if (logsum && tid == 0) *logsum = lg0 + lg1;
  __syncthreads();
}

// ---- the launch -------------------------------------------------------------
__global__ void __launch_bounds__(kFlowThreads, 2) chol_flow_kernel(CholFlowArgs a) {
  extern __shared__ __align__(16) double dsm[];
  __shared__ double s_dinv[32];
  __shared__ double s_log;
  __shared__ int s_ticket, s_avail, s_bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, q4 = lane & 3;
  const int T = (a.n + NB - 1) / NB;
  const int nb = a.batch_dev ? *a.batch_dev : a.batch;
  int* ticket = a.sync;
  int* done = a.sync + kCholFlowHead;          // [batch][T]: finished block columns of a block row
  int* diag = done + (size_t)a.batch * T;      // [batch]: finished diagonal blocks
  if (nb <= 0) return;
  int k = 0;
  long long base = 0;                          // first ticket of block column k
  for (;;) {
    if (tid == 0) s_ticket = atomicAdd(ticket, 1);
    __syncthreads();
    const int t = s_ticket;
    long long cnt = (long long)nb * (1 + (T - k) / 2);
    while (t >= base + cnt) {
      base += cnt;
      if (++k >= T) return;
      cnt = (long long)nb * (1 + (T - k) / 2);
    }
    const int local = (int)(t - base);
    const int r = local / nb - 1, b = local % nb;   // r = -1: the diagonal block
    const bool is_diag = r < 0;
    const int rb0 = is_diag ? k : k + 1 + 2 * r;    // first block row
    const int row0 = rb0 * NB, col0 = k * NB;
    const bool two = !is_diag && rb0 + 1 < T;
    const double* src = a.src + (size_t)b * a.src_stride;
    double* L = a.L + (size_t)b * a.l_stride;
    int* done_b = done + (size_t)b * T;
    // this warp's 32 x 32 part; the diagonal block's three lower quadrants go
    // to warps 0-3 and 4-7, which take half of the columns of a stage each
    const int wr = is_diag ? ((warp & 3) >> 1) * 32 : (warp >> 1) * 32;
    const int wc = (warp & 1) * 32;
    const int half = is_diag ? (warp >> 2) : 0;
    const bool idle = is_diag && wc > wr;
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j][0] = acc[i][j][1] = 0.0;
        const int rr = row0 + wr + 8 * i + g, cc = col0 + wc + 8 * j + 2 * q4;
        if (half == 0 && !idle && rr < a.n) {
          if (!is_diag || cc + 1 < a.n) {
            const double2 v = *reinterpret_cast<const double2*>(src + (size_t)rr * a.src_ld + cc);
            acc[i][j][0] = -v.x;
            acc[i][j][1] = -v.y;
          } else if (cc < a.n) {
            acc[i][j][0] = -src[(size_t)rr * a.src_ld + cc];
          }
        }
      }
    const int n_chunks = k * (NB / KC);
    int avail = 0;                                   // block columns known to be finished for all operands
    auto await = [&](int want) {                     // block-uniform
      if (tid == 0) {
        int v = wait_count(done_b + k, want, a.err);
        if (!is_diag) v = min(v, wait_count(done_b + rb0, want, a.err));
        if (two) v = min(v, wait_count(done_b + rb0 + 1, want, a.err));
        s_avail = v;
      }
      __syncthreads();
      avail = s_avail;
    };
    auto issue = [&](int c) {
      if (c < n_chunks) {
        double* st = dsm + (c % kStages) * kStageElems;
        const double* Lc = L + c * KC;
        const int rows = is_diag ? NB : RT + NB;
        for (int e = tid; e < rows * (KC / 2); e += kFlowThreads) {
          const int rr = e / (KC / 2), cc = 2 * (e % (KC / 2));
          // operand rows: the tile's 128, then the block column's own 64
          const int gr = rr < RT && !is_diag ? row0 + rr : col0 + (is_diag ? rr : rr - RT);
          const int ok = gr < a.n ? 16 : 0;
          cp_async16(st + rr * KS + cc, Lc + (size_t)(ok ? gr : 0) * a.ld + cc, ok);
        }
      }
      cp_commit();
    };
    if (n_chunks > 0) await(1);
    for (int c = 0; c < kStages - 1; ++c) issue(c);    // n_chunks is 0 or >= 4: both in block column 0
    for (int c = 0; c < n_chunks; ++c) {
      cp_wait<kStages - 2>();
      __syncthreads();
      const int nx = c + kStages - 1, need = nx / (NB / KC) + 1;
      const bool now = nx >= n_chunks || need <= avail;
      if (now) issue(nx);
      if (!idle) {
        const double* As = dsm + (c % kStages) * kStageElems;
        const double* Bs = is_diag ? As : As + RT * KS;
#pragma unroll
        for (int kk = 0; kk < KC; kk += 4) {
          if (is_diag && (kk >= KC / 2) != (half == 1)) continue;
          double af[4], bf[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) af[i] = As[(wr + 8 * i + g) * KS + kk + q4];
#pragma unroll
          for (int j = 0; j < 4; ++j) bf[j] = Bs[(wc + 8 * j + g) * KS + kk + q4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
      }
      if (!now) {
        await(need);
        issue(nx);
      }
    }
    cp_wait<0>();
    __syncthreads();
    double* S = dsm;                                 // tile (128 or 64 rows, stride FS)
    double* X = dsm + (size_t)(is_diag ? NB : RT) * FS;
    if (is_diag) {
      if (half == 1 && !idle) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<double2*>(S + (wr + 8 * i + g) * FS + wc + 8 * j + 2 * q4) =
                make_double2(acc[i][j][0], acc[i][j][1]);
      }
      if (tid == 0) s_bad = 0;
      __syncthreads();
      if (half == 0 && !idle) {
        const double sh = a.shift ? a.shift[b] : 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int rr = wr + 8 * i + g, cc = wc + 8 * j + 2 * q4 + h;
              double v = -(acc[i][j][h] + S[rr * FS + cc]);
              if (rr == cc) v += sh;
              if (col0 + rr >= a.n || col0 + cc >= a.n) v = rr == cc ? 1.0 : 0.0;   // identity padding
              S[rr * FS + cc] = v;
            }
      }
      __syncthreads();
      diag_factor(S, X, X + (size_t)NB * FS, s_dinv, tid, col0, a.n, &s_bad, a.ref ? a.ref[b] : 1.0, a.logdet ? &s_log : nullptr);
      double* Li = a.linv + (size_t)b * a.linv_stride + (size_t)k * NB * NB;
      for (int e = tid; e < NB * NB / 2; e += kFlowThreads) {
        const int rr = e / (NB / 2), cc = 2 * (e % (NB / 2));
        *reinterpret_cast<double2*>(Li + rr * NB + cc) = *reinterpret_cast<const double2*>(X + rr * FS + cc);
      }
      if (tid == 0) {
        if (s_bad) atomicCAS(&a.info[b], 0, s_bad);
        if (a.logdet) a.logdet[(size_t)b * T + k] = s_log;
      }
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        st_release(diag + b, k + 1);
      }
      continue;
    }
    // tile: T = A - sum, then L = T Linv^T with the diagonal block's inverse
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<double2*>(S + (wr + 8 * i + g) * FS + wc + 8 * j + 2 * q4) =
            make_double2(-acc[i][j][0], -acc[i][j][1]);
    if (tid == 0) wait_count(diag + b, k + 1, a.err);
    __syncthreads();
    const double* Li = a.linv + (size_t)b * a.linv_stride + (size_t)k * NB * NB;
    for (int e = tid; e < NB * NB / 2; e += kFlowThreads) {
      const int rr = e / (NB / 2), cc = 2 * (e % (NB / 2));
      cp_async16(X + rr * FS + cc, Li + rr * NB + cc, 16);
    }
    cp_commit();
    cp_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int kmax = wc + 32;                        // the inverse is lower triangular
#pragma unroll 4
    for (int kk = 0; kk < kmax; kk += 4) {
      double af[4], bf[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) af[i] = S[(wr + 8 * i + g) * FS + kk + q4];
#pragma unroll
      for (int j = 0; j < 4; ++j) bf[j] = X[(wc + 8 * j + g) * FS + kk + q4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = row0 + wr + 8 * i + g;
      if (rr < a.n)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<double2*>(L + (size_t)rr * a.ld + col0 + wc + 8 * j + 2 * q4) =
              make_double2(acc[i][j][0], acc[i][j][1]);
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      st_release(done_b + rb0, k + 1);
      if (two) st_release(done_b + rb0 + 1, k + 1);
    }
  }
}

}  // namespace

cudaError_t init_cholflow_attributes() {
  return cudaFuncSetAttribute(chol_flow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlowSmem);
}

size_t chol_flow_sync_ints(int n, int batch) {
  const size_t T = (n + NB - 1) / NB;
  return kCholFlowHead + (size_t)batch * (T + 1);
}

cudaError_t launch_chol_flow(const CholFlowArgs& a, int num_sms, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(a.sync, 0, sizeof(int) * chol_flow_sync_ints(a.n, a.batch), s);
  if (e != cudaSuccess) return e;
  const long long T = (a.n + NB - 1) / NB;
  long long tasks = 0;
  for (long long k = 0; k < T; ++k) tasks += a.batch * (1 + (T - k) / 2);
  const int grid = (int)std::min<long long>(tasks, 2LL * num_sms);
  chol_flow_kernel<<<grid, kFlowThreads, kFlowSmem, s>>>(a);
  return cudaGetLastError();
}

MBD_WAIT_LIMIT_SETTER(set_wait_limit_cholflow)

}  // namespace mbd
