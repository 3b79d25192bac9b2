// Products of symmetric, lower-stored matrices with three vectors in one pass
// over the lower halves: the matrix pass of the block CG (k_cg.cu; from the
// FP32 copy in its iterations) and of the relay residual (k_mixed.cu).
//
// Chunks of 64 rows x 512 bytes (128 floats or 64 doubles), row block after row
// block, matrix after matrix; every CTA (one an SM) takes an equal run of
// chunks.  A warp has 8 rows of a chunk, 16 bytes of every row per lane,
// brought by asynchronous copies two or three chunks ahead (a lane reads what
// it copied itself).  Row sums stay in registers to the end of the row block
// or the run; column sums cross the eight warps in shared memory, added up
// while the next chunk is worked on, with one barrier a chunk.
// FP32: four products are summed in FP32, two to an instruction (the pass
// would otherwise stay bound by its 12 FP64 FMAs per entry, not by its halved
// bytes), everything beyond in FP64: the sums carry a relative error of a few
// 1e-7, below what either phase of that solve resolves (rms against the FP64
// pass 2.6e-8 of the largest entry, as the 64 x 64 tile kernel before).
// FP64: products and sums in FP64.
//
// Slots (64 rows of the three vectors, apart) written in partial[f], row block
// I: [I][first block of chunk c] by a run's piece of the row block that begins
// at chunk c, [I][I] by the last piece together with the diagonal block's
// columns, and [J][I] with the columns of the blocks J < I.
//
// Bound: FP64 by HBM, FP32 by instruction issue and the conversions of its
// sums (the bytes alone take half the time).  21 matrices of n = 6000, by
// 64 x 64 tiles with all sums through shared memory and now: FP64 (3 GB) 0.82
// ms in the block CG, 1.40 ms in the residual, both 0.57 (5.3 TB/s of 6.4); FP32
// (1.5 GB) 0.69 -> 0.45, 0.23 without the arithmetic.  An FP32 iteration of the
// block CG 775 -> 525 us, of n = 3000 223 -> 171 us, of n = 2100 126 -> 105 us.
#include <algorithm>
#include <type_traits>

#include "strip.cuh"

namespace mbd {
namespace {

constexpr int CT = kStripRows;
constexpr int RW = 8;                       // rows of a warp
constexpr int ST = 32 * CT / RW;            // threads
constexpr size_t kChunkBytes = CT * 512;

template <typename T>
struct Dims {
  static constexpr int kRing = sizeof(T) == 4 ? 4 : 3;                 // chunks of a CTA in shared memory, one in use
  static constexpr int kGroups = sizeof(T) == 4 ? CT / 4 : CT / RW;    // row groups whose column sums are kept apart
  static constexpr size_t kColsBytes = sizeof(T) * 2 * kGroups * 3 * kStripCols<T>;
  static constexpr int kX = 3 * kStripCols<T> + 3 * CT;                // v on a chunk's columns and rows
  static constexpr size_t kSmem = kColsBytes + kRing * kChunkBytes + sizeof(double) * kRing * kX;
};

// The row block of chunk t of a matrix.
template <typename T>
__device__ __forceinline__ int chunk_row(int t) {
  int m, o;
  if (sizeof(T) == 8) {
    cg_tri(t, &m, &o);
    return m;
  }
  cg_tri(t / 2, &m, &o);                    // m (m + 1) <= t < (m + 1) (m + 2)
  return t < (m + 1) * (m + 1) ? 2 * m : 2 * m + 1;
}

template <typename T>
__global__ void __launch_bounds__(ST, 1) strip_kernel(StripArgs<T> a) {
  using D = Dims<T>;
  constexpr bool F = sizeof(T) == 4;
  constexpr int CW = kStripCols<T>;
  __shared__ __align__(16) T xs[2][3][CW], xi[2][CT][F ? 8 : 4];   // FP32 row values twice, for two products at once
  __shared__ double ys[2][CT * 3];
  extern __shared__ __align__(16) unsigned char dyn[];
  T* cols = reinterpret_cast<T*>(dyn);                 // [2][kGroups][3][CW]: sums of 4 (FP32) or RW rows
  float4* ring = reinterpret_cast<float4*>(dyn + D::kColsBytes) + threadIdx.x;   // [kRing][RW][ST], each lane's own
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = a.n, per = chunks_before<T>(a.nt);
  const unsigned act = strip_active(a.state, a.batch);
  const int run = strip_run<T>(a.nt, __popc(act), gridDim.x);
  int pos = blockIdx.x * run;
  const int end = min(pos + run, per * __popc(act));
  if (pos >= end) return;
  struct At {                               // chunk c of row block I of frequency f
    int f, I, c;
  };
  auto advance = [&](At& w) {
    if (w.c++ < last_chunk<T>(w.I)) return;
    w.c = 0;
    if (++w.I < a.nt) return;
    w.I = 0;
    w.f = __fns(act, w.f + 1, 1);           // -1 behind the last one, not used
  };
  At w;
  w.f = __fns(act, 0, pos / per + 1);
  w.I = chunk_row<T>(pos % per);
  w.c = pos % per - chunks_before<T>(w.I);
  int c0 = w.c;                             // where this run's piece of the row block begins
  At pw = w;
  int ppos = pos, slot = 0;
  const unsigned ring_at = (unsigned)__cvta_generic_to_shared(ring);
  // rows past n and columns past the row's end bring some other entry (masked
  // in a row block's last chunk, times a zero of v, or never read)
  constexpr int XC = (3 * CW + ST - 1) / ST, XR = (3 * CT + ST - 1) / ST;
  double* xring = reinterpret_cast<double*>(dyn + D::kColsBytes + D::kRing * kChunkBytes) + tid;   // each thread's own
  auto issue_x = [&](double* dst, int f_, int first, int count) {
    const int left = min(count, 3 * n - first) - tid;   // elements at tid, tid + ST, ...
    const double* src = a.in + (size_t)f_ * a.ystride + (left > 0 ? first + tid : 0);
    for (int u = 0; ST * u < count; ++u)
      if (tid + ST * u < count) {
        const bool ok = ST * u < left;
        const unsigned d = (unsigned)__cvta_generic_to_shared(dst + ST * u);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(ok ? src + ST * u : src), "r"(ok ? 8 : 0) : "memory");
      }
  };
  auto issue = [&](int to) {                // a chunk of the matrix, and v for the one behind it
    if (ppos < end) {
      const T* src =
          a.A + (size_t)pw.f * a.a_stride + (size_t)pw.I * CT * a.ld + min(CW * pw.c + CW / 32 * lane, a.ld - CW / 32);
      const int rmax = n - 1 - pw.I * CT;
      const unsigned d = ring_at + to * (RW * ST * 16);
      if (rmax >= CT - 1) {
        const T* row = src + (size_t)(RW * warp) * a.ld;
#pragma unroll
        for (int r = 0; r < RW; ++r) ring_copy(d + r * (ST * 16), row + (size_t)(unsigned)r * a.ld);
      } else {
#pragma unroll
        for (int r = 0; r < RW; ++r)
          ring_copy(d + r * (ST * 16), src + (size_t)(unsigned)min(RW * warp + r, rmax) * a.ld);
      }
      advance(pw);
      if (++ppos < end) {
        issue_x(xring + to * D::kX, pw.f, 3 * CW * pw.c, 3 * CW);
        if (pw.c == 0) issue_x(xring + to * D::kX + 3 * CW, pw.f, CT * 3 * pw.I, 3 * CT);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int d = 0; d < D::kRing - 1; ++d) issue(d);
  // v on the chunk's columns and on the row block, the three vectors apart
  // (element e: vector e % 3 of row e / 3)
  auto x_at = [&](int f_, int first, int e, int count) {
    return e < count && first + e < 3 * n ? a.in[(size_t)f_ * a.ystride + first + e] : 0.0;
  };
  auto put_col = [&](int p, int e, double v) {
    if (e < 3 * CW) xs[p][e % 3][e / 3] = (T)v;
  };
  auto put_row = [&](int p, int e, double v) {
    if (e >= 3 * CT) return;
    if constexpr (F) {
      *reinterpret_cast<float2*>(&xi[p][e / 3][2 * (e % 3)]) = make_float2((float)v, (float)v);
    } else {
      xi[p][e / 3][e % 3] = v;
    }
  };
#pragma unroll
  for (int u = 0; u < XC; ++u) put_col(0, tid + ST * u, x_at(w.f, 3 * CW * w.c, tid + ST * u, 3 * CW));
#pragma unroll
  for (int u = 0; u < XR; ++u) put_row(0, tid + ST * u, x_at(w.f, CT * 3 * w.I, tid + ST * u, 3 * CT));
  // the columns of a chunk whose sums all warps have put into cols[p]
  auto columns = [&](const At& o, int p) {
    double* pr = a.partial + (size_t)o.f * a.nt * a.nt * CT * 3;
#pragma unroll
    for (int u = 0; u < XC; ++u) {
      const int e = tid + ST * u, q = e / CW, J = CW / CT * o.c + e % CW / CT, k = CT * q + e % CT;
      if (e >= 3 * CW || J > o.I) continue;
      double z[4] = {J == o.I ? ys[p][k] : 0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int g = 0; g < D::kGroups; ++g) {   // FP32: half of the conversions on either pipe, 2 % of the pass
        const T v = cols[(D::kGroups * p + g) * 3 * CW + e];
        if constexpr (F) {
          z[g % 4] += g % 2 ? widen(v) : (double)v;
        } else {
          z[g % 4] += v;
        }
      }
      pr[((size_t)J * a.nt + o.I) * CT * 3 + k] = (z[0] + z[1]) + (z[2] + z[3]);
    }
  };
  __syncthreads();
  double rs[RW][3];
#pragma unroll
  for (int r = 0; r < RW; ++r) rs[r][0] = rs[r][1] = rs[r][2] = 0.0;
  At prev = w;
  for (int p = 0, ip = 0, first = 1;; p ^= 1, first = 0) {
    const bool diag = w.c == last_chunk<T>(w.I), more = ++pos < end, same = more && !diag;
    At nw = w;
    advance(nw);
    asm volatile("cp.async.wait_group %0;" ::"n"(D::kRing - 2) : "memory");
    const float4* mine = ring + slot * RW * ST;
    const double* xmine = xring + slot * D::kX;
    issue(slot == 0 ? D::kRing - 1 : slot - 1);      // the slot of the last chunk
    slot = slot + 1 == D::kRing ? 0 : slot + 1;
    using V = std::conditional_t<F, ulonglong2, double2>;   // 16 bytes: four floats in pairs, or two doubles
    V xj[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) xj[q] = *reinterpret_cast<const V*>(&xs[p][q][CW / 32 * lane]);
    T* co = cols + (D::kGroups * p + D::kGroups / (CT / RW) * warp) * 3 * CW + CW / 32 * lane;
    auto chunk = [&](auto diag_tag) {
      V cs[3];
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        V e = *reinterpret_cast<const V*>(mine + r * ST), ec = e;
        [[maybe_unused]] const int d = CW * w.c + CW / 32 * lane - (w.I * CT + RW * warp + r);
        if constexpr (F) {
          if constexpr (decltype(diag_tag)::value) {   // nothing above the diagonal, the diagonal on the row side
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
            if (r % 4 == 3) *reinterpret_cast<ulonglong2*>(co + (r / 4 * 3 + q) * CW) = cs[q];
          }
        } else {
          if constexpr (decltype(diag_tag)::value) {   // nothing above the diagonal, the diagonal on the row side
            e = make_double2(d <= 0 ? e.x : 0.0, d <= -1 ? e.y : 0.0);
            ec = make_double2(d < 0 ? e.x : 0.0, d < -1 ? e.y : 0.0);
          }
          const double2 x01 = *reinterpret_cast<const double2*>(&xi[ip][RW * warp + r][0]);
          const double x[3] = {x01.x, x01.y, xi[ip][RW * warp + r][2]};
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            rs[r][q] = fma(e.y, xj[q].y, fma(e.x, xj[q].x, rs[r][q]));
            cs[q].x = r == 0 ? ec.x * x[q] : fma(ec.x, x[q], cs[q].x);
            cs[q].y = r == 0 ? ec.y * x[q] : fma(ec.y, x[q], cs[q].y);
            if (r == RW - 1) *reinterpret_cast<double2*>(co + q * CW) = cs[q];
          }
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
            pr[((size_t)w.I * a.nt + CW / CT * c0) * CT * 3 + CT * q + row] = y;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < RW; ++r) rs[r][0] = rs[r][1] = rs[r][2] = 0.0;
      if (more) {
#pragma unroll
        for (int u = 0; u < XR; ++u) if (tid + ST * u < 3 * CT) put_row(ip ^ 1, tid + ST * u, xmine[3 * CW + ST * u]);
      }
    }
    if (more) {
#pragma unroll
      for (int u = 0; u < XC; ++u) if (tid + ST * u < 3 * CW) put_col(p ^ 1, tid + ST * u, xmine[ST * u]);
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

template <typename T>
int launch(const StripArgs<T>& a, cudaStream_t s) {
  static const int sms = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
  }();
  const int ctas = std::min(sms, chunks_before<T>(a.nt) * a.batch);
  strip_kernel<T><<<ctas, ST, Dims<T>::kSmem, s>>>(a);
  return ctas;
}

}  // namespace

int launch_strip(const StripArgs<float>& a, cudaStream_t s) { return launch(a, s); }
int launch_strip(const StripArgs<double>& a, cudaStream_t s) { return launch(a, s); }

cudaError_t init_strip_attributes() {
  cudaError_t e = cudaFuncSetAttribute(strip_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)Dims<float>::kSmem);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(strip_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)Dims<double>::kSmem);
}

}  // namespace mbd
