// Products of symmetric, lower-stored matrices with three vectors, one pass
// over the lower halves (k_strip.cu), and what its readers need.
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"
#include "../../include/mbd_b200.h"

namespace mbd {

constexpr int kStripRows = 64;      // rows of a row block
constexpr int kStripMaxBatch = 32;  // matrices of a launch (a warp's ballot)
static_assert(MBD_N_FREQ <= kStripMaxBatch, "a matrix per frequency");

template <typename T>
struct StripArgs {
  const T* A;                // [batch] row-major lower, row stride ld (a multiple of 32), 16-byte aligned
  size_t a_stride;
  int ld, n, nt, batch;      // nt = ceil(n / 64)
  const double* in;          // [batch][n][3]
  size_t ystride;
  double* partial;           // [batch][nt][nt][3][64]
  const double* state;       // block-CG state: stopped matrices are left out; or null
};
// Returns the number of CTAs launched, which the reader of the partials needs.
int launch_strip(const StripArgs<float>& a, cudaStream_t s);
int launch_strip(const StripArgs<double>& a, cudaStream_t s);
cudaError_t init_strip_attributes();

namespace {

__device__ __forceinline__ void cg_tri(int t, int* ti, int* tj) {
  int i = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((i + 1) * (i + 2) / 2 <= t) ++i;
  while (i * (i + 1) / 2 > t) --i;
  *ti = i;
  *tj = t - i * (i + 1) / 2;
}

// A float as a double by integer operations: the conversion instruction has an
// eighth of the ALU's rate, and its queue can set a pass's time.  Zeros
// and denormals come out as some 1e-38, infinities and NaN as some 1e38 (the
// residual gate turns such a solve away).
__device__ __forceinline__ double widen(float x) {
  const int b = __float_as_int(x);
  return __hiloint2double(((b >> 3) & 0x8fffffff) + 0x38000000, b << 29);
}

// Columns of a chunk: 32 lanes x 16 bytes.
template <typename T>
constexpr int kStripCols = 512 / (int)sizeof(T);

// Chunks of the row blocks before block I; the last chunk of block I is the
// one with its diagonal, number I (FP64) or I / 2 (FP32).
template <typename T>
__host__ __device__ __forceinline__ int chunks_before(int I) {
  return sizeof(T) == 4 ? (I + 1) / 2 * ((I + 2) / 2) : I * (I + 1) / 2;
}
template <typename T>
__host__ __device__ __forceinline__ int last_chunk(int I) {
  return sizeof(T) == 4 ? I / 2 : I;
}
// Chunks of a CTA's run when `act` matrices of nt row blocks take part.
template <typename T>
__device__ __forceinline__ int strip_run(int nt, int act, int ctas) {
  return (chunks_before<T>(nt) * act + ctas - 1) / ctas;
}

// The matrices that take part (state: slot 0 of each kCgState record is zero; or
// all), as a mask; all threads of a warp.
__device__ __forceinline__ unsigned strip_active(const double* state, int batch) {
  const int lane = threadIdx.x & 31;
  return __ballot_sync(0xffffffffu, lane < batch && (!state || state[lane * kCgState] == 0.0));
}

// (A v) at row r of row block I, vector q, of matrix f from the partials that
// strip_kernel<T> left on `ctas` CTAs.  Whole warps, with f and I uniform.
template <typename T>
__device__ __forceinline__ double strip_row_sum(const double* partial, const double* state, int batch, int nt, int f,
                                                int I, int ctas, int r, int q) {
  const unsigned act = strip_active(state, batch);
  const int run = strip_run<T>(nt, __popc(act), ctas);
  const int first = __popc(act & ((1u << f) - 1)) * chunks_before<T>(nt) + chunks_before<T>(I);
  const int last = first + last_chunk<T>(I);
  const double* pr = partial + ((size_t)f * nt + I) * nt * kStripRows * 3 + kStripRows * q + r;
  double y = 0.0;
  // the pieces of the row block but the last
  for (int x = first, end; (end = (x / run + 1) * run) <= last; x = end)
    y += pr[(size_t)(kStripCols<T> / kStripRows * (x - first)) * kStripRows * 3];
  for (int J = I; J < nt; ++J) y += pr[(size_t)J * kStripRows * 3];
  return y;
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

__device__ __forceinline__ void ring_copy(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ring_copy(float4* dst, const void* src) {
  ring_copy((unsigned)__cvta_generic_to_shared(dst), src);
}

}  // namespace
}  // namespace mbd
