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
// block, n / 64 links of 19 us.  Four warps of 32 x 64 a CTA: 12 fragment
// loads for 32 MMAs, where eight warps of 32 x 32 took 16 and left the MMAs
// waiting; two CTAs an SM, one working while the other changes tiles.
// Measured, batches of matrices of n rows (right-looking kernels; eight warps;
// now): 21 of n = 3000 17.5, 6.5, 5.9 ms (32 TFLOP/s), 14 of n = 6000 -, 31.8,
// 29.4 ms (34.3), 21 of n = 384 0.85, 0.126, 0.126 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <type_traits>

#include "chol64.cuh"
#include "kernels.h"
#include "wait_limit.cuh"

namespace mbd {
namespace {

constexpr int RT = 2 * NB;       // rows of a tile task
constexpr int KC = 16;           // columns of one pipeline stage
constexpr int KS = KC + 4;       // shared row stride: a half-warp's 8 x 4 fragment loads hit 16 bank pairs
constexpr int kStages = 3;
constexpr int kStageElems = (RT + NB) * KS;
constexpr int kFlowThreads = 128;
constexpr int XS = NB + 8;       // row stride of the inverse in a tile task: 16-byte loads of two rows hit all banks
constexpr size_t kFlowSmem = sizeof(double) * kStages * kStageElems;
static_assert(kStageElems >= NB / 2 * XS && kStages * kStageElems >= 2 * NB * FS, "shared memory of a task");
constexpr int kErrTimeout = 7;   // MBD_ERR_TIMEOUT

// 16-byte asynchronous copy global -> shared.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
// The same; src_bytes < 16 zero-fills the rest.
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
// records the time-out and returns `want`, so every task still ends; so it does
// once the launch is called off (*stop).
__device__ int wait_count(const int* p, int want, int* err, const int* stop) {
  int v = ld_acquire(p);
  if (v >= want) return v;
  const long long limit = wait_limit_cycles();
  const long long t0 = clock64();
  while ((v = ld_acquire(p)) < want) {
    if (*(volatile int*)err != 0 || (stop && *(const volatile int*)stop != 0)) return want;
    if (clock64() - t0 > limit) {
      atomicCAS(err, 0, kErrTimeout);
      return want;
    }
    __nanosleep(20);
  }
  return v;
}

// ---- the launch -------------------------------------------------------------
__global__ void __launch_bounds__(kFlowThreads, 2) chol_flow_kernel(CholFlowArgs a) {
  extern __shared__ __align__(16) double dsm[];
  __shared__ double s_dinv[NB], s_diagx[NB];
  __shared__ int s_ticket, s_avail, s_early, s_bad;
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
  auto draw = [&] {                            // none once the launch is called off
    const int t = atomicAdd(ticket, 1);
    return a.stop && *(const volatile int*)a.stop != 0 ? INT_MAX : t;
  };
  if (tid == 0) s_ticket = draw();
  for (;;) {
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
    int avail = 0;                                   // block columns known to be finished for all operands
    auto await = [&](int want) {                     // block-uniform
      if (tid == 0) {
        int v = wait_count(done_b + k, want, a.err, a.stop);
        if (!is_diag) v = min(v, wait_count(done_b + rb0, want, a.err, a.stop));
        if (two) v = min(v, wait_count(done_b + rb0 + 1, want, a.err, a.stop));
        s_avail = v;
      }
      __syncthreads();
      avail = s_avail;
    };
    if (is_diag) {
      // Lower triangle of the 8 x 8 blocks, block rows 7 - w and w on warp w:
      // nine blocks for every sub-partition.  Whole block columns of L in two
      // buffers: behind the last one, which the chain waits for, all of its
      // loads are out at once.
      const int hi = 7 - warp, lo = warp;
      double acc[8][2], acl[4][2];
      auto entry = [&](int bi, int j, double* d) {
        d[0] = d[1] = 0.0;
        const int rr = col0 + 8 * bi + g, cc = col0 + 8 * j + 2 * q4;
        if (j > bi || rr >= a.n) return;
        if (cc + 1 < a.n) {
          const double2 v = *reinterpret_cast<const double2*>(src + (size_t)rr * a.src_ld + cc);
          d[0] = -v.x;
          d[1] = -v.y;
        } else if (cc < a.n) {
          d[0] = -src[(size_t)rr * a.src_ld + cc];
        }
      };
#pragma unroll
      for (int j = 0; j < 8; ++j) entry(hi, j, acc[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) entry(lo, j, acl[j]);
      auto issue = [&](int p) {
        double* buf = dsm + (p & 1) * (NB * FS);
        const double* Lp = L + p * NB;
#pragma unroll
        for (int c = 0; c < NB / KC; ++c) {
          for (int e = tid; e < NB * (KC / 2); e += kFlowThreads) {
            const int rr = e / (KC / 2), cc = KC * c + 2 * (e % (KC / 2));
            const int ok = col0 + rr < a.n ? 16 : 0;
            cp_async16(buf + rr * FS + cc, Lp + (size_t)(ok ? col0 + rr : 0) * a.ld + cc, ok);
          }
          cp_commit();
        }
      };
      if (k > 0) {
        await(1);
        issue(0);
      }
      for (int p = 0; p < k; ++p) {
        const bool next = p + 2 <= avail && p + 1 < k;
        if (next) issue(p + 1);   // its buffer was last read before the barrier that closed block column p - 1
        const double* buf = dsm + (p & 1) * (NB * FS);
#pragma unroll
        for (int c = 0; c < NB / KC; ++c) {
          if (next) {
            if (c == 0) cp_wait<7>();
            if (c == 1) cp_wait<6>();
            if (c == 2) cp_wait<5>();
            if (c == 3) cp_wait<4>();
          } else {
            if (c == 0) cp_wait<3>();
            if (c == 1) cp_wait<2>();
            if (c == 2) cp_wait<1>();
            if (c == 3) cp_wait<0>();
          }
          __syncthreads();
#pragma unroll
          for (int kk = KC * c; kk < KC * (c + 1); kk += 4) {
            const double ah = buf[(8 * hi + g) * FS + kk + q4], al = buf[(8 * lo + g) * FS + kk + q4];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (j > hi) continue;
              const double bf = buf[(8 * j + g) * FS + kk + q4];
              dmma(acc[j][0], acc[j][1], ah, bf);
              if (j < 4 && j <= lo) dmma(acl[j & 3][0], acl[j & 3][1], al, bf);
            }
          }
        }
        __syncthreads();
        if (!next && p + 1 < k) {
          await(p + 2);
          issue(p + 1);
        }
      }
      double* S = dsm;
      double* X = dsm + (size_t)NB * FS;
      if (tid == 0) s_bad = 0;
      auto put = [&](int bi, int j, const double* d) {
        if (j > bi) return;
        const int rr = 8 * bi + g, cc = 8 * j + 2 * q4;
        double2 v = make_double2(-d[0], -d[1]);
        if (col0 + rr >= a.n || col0 + cc >= a.n) v.x = rr == cc ? 1.0 : 0.0;   // identity padding
        if (col0 + rr >= a.n || col0 + cc + 1 >= a.n) v.y = rr == cc + 1 ? 1.0 : 0.0;
        *reinterpret_cast<double2*>(S + rr * FS + cc) = v;
      };
#pragma unroll
      for (int j = 0; j < 8; ++j) put(hi, j, acc[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) put(lo, j, acl[j]);
      __syncthreads();
      DiagShift ds{0.0, 0.0, 0.0};
      if (a.shift) ds = DiagShift{a.shift[b], *a.c2, a.ref[b]};
      diag_factor<kFlowThreads>(S, X, s_dinv, s_diagx, tid, col0, a.n, &s_bad, ds.shift);
      double* Li = a.linv + (size_t)b * a.linv_stride + (size_t)k * NB * NB;
      for (int e = tid; e < NB * NB / 2; e += kFlowThreads) {
        const int rr = e / (NB / 2), cc = 2 * (e % (NB / 2));
        *reinterpret_cast<double2*>(Li + rr * NB + cc) = *reinterpret_cast<const double2*>(X + rr * FS + cc);
      }
      __syncthreads();
      if (tid == 0) {
        if (s_bad) atomicCAS(&a.info[b], 0, s_bad);
        __threadfence();
        st_release(diag + b, k + 1);
      }
      if (a.logdet && warp == 1) {   // off the chain
        double lg = 0.0;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (col0 + lane + 32 * h < a.n) lg += log1p((s_diagx[lane + 32 * h] - ds.c2) * ds.ref);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lg += __shfl_xor_sync(0xffffffffu, lg, o);
        if (lane == 0) a.logdet[(size_t)b * T + k] = lg;
      }
      if (tid == 0) s_ticket = draw();
      continue;
    }
    // tile: T = A - sum, then L = T Linv^T with the diagonal block's inverse.
    // Warp w takes the 8-row blocks w + 4 i, all 64 columns: its part of T is
    // then the second product's operand as it lies in the registers.
    // Operand rows: the tile's 128, then the block column's own 64 (which all
    // exist, as there are rows below them), kRowStep apart for a thread.
    constexpr int kRowStep = kFlowThreads / (KC / 2), kCopies = (RT + NB) / kRowStep;
    const int cr = tid / (KC / 2), cc = 2 * (tid % (KC / 2));
    const double* csrc[kCopies];                       // rows past the last: some row, their results are dropped
#pragma unroll
    for (int u = 0; u < kCopies; ++u) {
      const int gr = u * kRowStep < RT ? min(row0 + cr + u * kRowStep, a.n - 1) : col0 + cr + u * kRowStep - RT;
      csrc[u] = L + (size_t)gr * a.ld + cc;
    }
    double* cdst = dsm + cr * KS + cc;
    auto copy = [&](int c, int u) {
      cp_async16(cdst + (c % kStages) * kStageElems + u * kRowStep * KS, csrc[u] + c * KC);
    };
    const int n_chunks = k * (NB / KC);
    // the inverse, 32 rows to each of the stages that the last chunk leaves
    const double* Li = a.linv + (size_t)b * a.linv_stride + (size_t)k * NB * NB;
    auto copy_inverse = [&](int c) {
      double* X = dsm + (c % kStages) * kStageElems;
      const double* Lh = Li + (size_t)(c - n_chunks) * (NB / 2) * NB;
#pragma unroll
      for (int u = 0; u < NB * NB / 4 / kFlowThreads; ++u) {
        const int e = tid + u * kFlowThreads, rr = e / (NB / 2), c2 = 2 * (e % (NB / 2));
        cp_async16(X + rr * XS + c2, Lh + rr * NB + c2);
      }
    };
    if (n_chunks > 0) {
      await(1);
      for (int c = 0; c < kStages - 1; ++c) {          // n_chunks >= 4: both in block column 0
#pragma unroll
        for (int u = 0; u < kCopies; ++u) copy(c, u);
        cp_commit();
      }
    }
    double acc[4][8][2];                               // sum - A
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int rr = row0 + 8 * (warp + 4 * i) + g;
        double2 v = make_double2(0.0, 0.0);
        if (rr < a.n) v = *reinterpret_cast<const double2*>(src + (size_t)rr * a.src_ld + col0 + 8 * j + 2 * q4);
        acc[i][j][0] = -v.x;
        acc[i][j][1] = -v.y;
      }
    bool early = false;                                // the diagonal block was finished before the last chunk
    auto run = [&](auto rows_tag) {
      constexpr int MI = decltype(rows_tag)::value;    // 4, or 2 where the tile has one block row
      auto step = [&](int c, auto copy_tag) {          // straight-line MMAs and copies: a branch for the copies costs 2 %, one for MI 3 %
        const double* As = dsm + (c % kStages) * kStageElems + (8 * warp + g) * KS + q4;
        const double* Bs = dsm + (c % kStages) * kStageElems + (RT + g) * KS + q4;
#pragma unroll
        for (int kk = 0; kk < KC; kk += 4) {
          double af[MI], bf[8];
#pragma unroll
          for (int i = 0; i < MI; ++i) af[i] = As[32 * i * KS + kk];
#pragma unroll
          for (int j = 0; j < 8; ++j) bf[j] = Bs[8 * j * KS + kk];
          if constexpr (decltype(copy_tag)::value) {
#pragma unroll
            for (int u = 0; u < kCopies / (KC / 4); ++u) copy(c + kStages - 1, kk / 4 * (kCopies / (KC / 4)) + u);
          }
#pragma unroll
          for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
      };
      for (int c = 0; c < n_chunks; ++c) {
        for (const int last = min(n_chunks, avail * (NB / KC)) - (kStages - 1); c < last; ++c) {
          cp_wait<kStages - 2>();
          __syncthreads();
          step(c, std::true_type());
          cp_commit();
        }
        cp_wait<kStages - 2>();
        __syncthreads();
        if (c == n_chunks - 2 && tid == 0) s_early = ld_acquire(diag + b);
        if (c == n_chunks - 1 && s_early > k) {        // both other stages are free
          early = true;
          copy_inverse(n_chunks);
          copy_inverse(n_chunks + 1);
        }
        step(c, std::false_type());
        const int nx = c + kStages - 1;
        if (nx < n_chunks) {
          await(nx / (NB / KC) + 1);
#pragma unroll
          for (int u = 0; u < kCopies; ++u) copy(nx, u);
        }
        cp_commit();
      }
    };
    if (two) {
      run(std::integral_constant<int, 4>());
    } else {
      run(std::integral_constant<int, 2>());
    }
    if (!early) {
      if (tid == 0) wait_count(diag + b, a.stall && k == 0 ? 1 << 30 : k + 1, a.err, a.stop);
      __syncthreads();
      copy_inverse(n_chunks);
      copy_inverse(n_chunks + 1);
      cp_commit();
    }
    cp_wait<0>();
    __syncthreads();
    int next = 0;
    if (tid == 0) next = draw();   // this task waits for nothing any more
    const double* X0 = dsm + (n_chunks % kStages) * kStageElems + g * XS + 2 * q4;
    const double* X1 = dsm + ((n_chunks + 1) % kStages) * kStageElems + g * XS + 2 * q4;
    // 64 rows at a time, so that the block row the next diagonal block waits
    // for is out first; of the inverse's lower triangle the blocks that are
    // not zero.  An 8-column block of T is one operand by its even columns
    // and one by its odd ones.
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && !two) break;
#pragma unroll
      for (int j = 0; j < 8; j += 2) {   // two blocks of columns at a time: four chains of products
        const double* Xj = (j < 4 ? X0 : X1) + 8 * (j & 3) * XS;
        double o[2][2][2] = {};
#pragma unroll
        for (int p = 0; p <= j + 1; ++p) {
          const double2 x1 = *reinterpret_cast<const double2*>(Xj + 8 * XS + 8 * p);
          const double2 x0 = p <= j ? *reinterpret_cast<const double2*>(Xj + 8 * p) : make_double2(0.0, 0.0);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (p <= j) dmma(o[i][0][0], o[i][0][1], acc[2 * h + i][p][0], x0.x);
            dmma(o[i][1][0], o[i][1][1], acc[2 * h + i][p][0], x1.x);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (p <= j) dmma(o[i][0][0], o[i][0][1], acc[2 * h + i][p][1], x0.y);
            dmma(o[i][1][0], o[i][1][1], acc[2 * h + i][p][1], x1.y);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int rr = row0 + 8 * (warp + 4 * (2 * h + i)) + g;
          if (rr < a.n) {
            double* d = L + (size_t)rr * a.ld + col0 + 8 * j + 2 * q4;
            *reinterpret_cast<double2*>(d) = make_double2(-o[i][0][0], -o[i][0][1]);
            *reinterpret_cast<double2*>(d + 8) = make_double2(-o[i][1][0], -o[i][1][1]);
          }
        }
      }
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        st_release(done_b + rb0 + h, k + 1);
      }
    }
    if (tid == 0) s_ticket = next;
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
  // Every slot of the device where the products set the time; where the chain
  // of diagonal blocks does (20 us a link), twice the CTAs it can keep at
  // work, so that the waiting ones leave room for other streams' kernels.
  const double work_us = a.batch * (double)a.n * a.n * a.n / 3.0 / 29e6, chain_us = 20.0 * T;
  const double share = std::min(1.0, std::max(2.0 * work_us / chain_us, 6.0 * a.batch / (2.0 * num_sms)));
  const int grid = (int)std::min<long long>(tasks, (long long)(2.0 * num_sms * share));
  chol_flow_kernel<<<grid, kFlowThreads, kFlowSmem, s>>>(a);
  return cudaGetLastError();
}

MBD_WAIT_LIMIT_SETTER(set_wait_limit_cholflow)

}  // namespace mbd
