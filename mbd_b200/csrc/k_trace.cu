// The MBD energy from shifted Cholesky factors of the coupled-oscillator
// Hamiltonian H, in place of its eigenvalues (PDSYEV at UTILS.f90:835, the
// sum at UTILS.f90:839-858).  The energy needs sum_i sqrt(lambda_i) and the
// number of negative eigenvalues only.  For c > 0
//
//   sum_i (sqrt(lambda_i) - c) = 1/pi int_0^inf ln det[(H + u^2)/(c^2 + u^2)] du,
//
// whose integrand, as a function of u, has its singularities on
// +-i [sqrt(m), sqrt(M)] (m <= lambda <= M) and at +-ic.  u = sqrt(m) sc(v, k),
// k^2 = 1 - m/M, maps the plane without those slits onto a strip of period
// 2K(k) and half-height K'(k), where the midpoint rule in v converges like
// exp(-2 pi^2 nodes / (ln(M/m) + 4 ln 2)) (the mapping of Hale, Higham and
// Trefethen, SIAM J. Numer. Anal. 46, 2505 (2008), used here on the
// logarithm).  Each node is one Cholesky factorisation of H + u^2 I; all run
// as one batch (k_cholflow.cu).  Against the reduction to tridiagonal form
// (a chain of n columns, then n bulge-chasing sweeps) the nodes cost ~3x the
// operations, all of them in matrix products with the whole chip at work.
//
// M is Gershgorin's bound.  m = min diagonal / 5 (the smallest eigenvalue of
// molecules, clusters, boxes and sheets measured 0.4 to 0.9 of the smallest
// diagonal entry), or for large H 0.7 of the smallest Ritz value of a few
// Lanczos steps (1.0 to 1.25 of the smallest eigenvalue there), which saves two
// nodes; the factorisation of H - m I, one more matrix of the batch, proves
// m <= lambda.  Where it fails (which calls the rest of the batch off), or M/m
// asks for more than kTraceNodes nodes, the result is refused and the caller
// takes the eigenvalues (imaginary modes, near-instabilities).  Calling off: a
// refused chain of 800 Na atoms 36.2 -> 34.6 ms (34.7 by eigenvalues alone), 16
// chains of 40 to 190 14.0 -> 13.8 (13.0); nothing measurable where all succeed.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"

namespace mbd {
namespace {

constexpr int NB = kCholNB;
constexpr double kLowerShare = 0.2;      // m over the smallest diagonal entry
// Lanczos steps for matrices of at least kLanczosMinN rows.  A step reads H once
// (n = 6000: 57 us with its two small launches, 0.9 ms in all, against 5 to 6 ms for
// two nodes; n = 3000 0.3 against 0.7).
constexpr int kLanczosSteps = 16;
constexpr int kLanczosMinN = 2500;
constexpr double kRitzShare = 0.7;       // m over the smallest Ritz value
struct TraceWs {
  double* part;      // [T][T * 64] absolute row sums per block column
  double* rowred;    // [T][3] per block row: largest Gershgorin bound, smallest diagonal, sum of the diagonal
  double* shift;     // [kTraceBatch]
  double* ref;       // [kTraceBatch] 1 / (c^2 + u^2)
  double* weight;    // [kTraceBatch]
  double* c2;        // [1] c^2, the mean of the diagonal
  double* logdet;    // [kTraceBatch][T]
  int* info;         // [kTraceBatch]
  int* count;        // [1] matrices of the batch (0: refused)
  int* sync;
  // Lanczos: u (next vector, not normalised), the last two vectors, y = H v;
  // [steps + 1][T] squared norms of u and [steps][T] dots v^T y by block row
  double *u, *v[2], *y, *norms, *dots;
};

size_t up(size_t b) { return (b + 255) & ~size_t(255); }

size_t carve(void* base, int n, TraceWs* w) {
  const size_t T = (n + NB - 1) / NB;
  char* p = static_cast<char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = p + off;
    off += up(bytes);
    return q;
  };
  w->part = reinterpret_cast<double*>(take(sizeof(double) * T * T * NB));
  w->rowred = reinterpret_cast<double*>(take(sizeof(double) * 3 * T));
  w->shift = reinterpret_cast<double*>(take(sizeof(double) * kTraceBatch));
  w->ref = reinterpret_cast<double*>(take(sizeof(double) * kTraceBatch));
  w->weight = reinterpret_cast<double*>(take(sizeof(double) * kTraceBatch));
  w->c2 = reinterpret_cast<double*>(take(sizeof(double)));
  w->logdet = reinterpret_cast<double*>(take(sizeof(double) * kTraceBatch * T));
  w->info = reinterpret_cast<int*>(take(sizeof(int) * kTraceBatch));
  w->count = reinterpret_cast<int*>(take(sizeof(int)));
  w->sync = reinterpret_cast<int*>(take(sizeof(int) * chol_flow_sync_ints(n, kTraceBatch)));
  const bool lz = n >= kLanczosMinN;
  auto vec = [&](size_t k) { return reinterpret_cast<double*>(take(lz ? sizeof(double) * k : 0)); };
  w->u = vec(T * NB);
  w->v[0] = vec(T * NB);
  w->v[1] = vec(T * NB);
  w->y = vec(T * NB);
  w->norms = vec((kLanczosSteps + 1) * T);
  w->dots = vec(kLanczosSteps * T);
  return off;
}

// Absolute off-diagonal sums of one 64 x 64 lower tile, along its rows and
// (off the diagonal blocks) its columns: part[J][row of I] and
// part[I][row of J].  One read of H; bound by it.
__global__ void __launch_bounds__(256) abs_sums_kernel(const double* H, int n, int ld, int T, double* part) {
  __shared__ double s[NB][NB + 1];
  int I = (int)((sqrt(8.0 * blockIdx.x + 1.0) - 1.0) * 0.5);
  while ((I + 1) * (I + 2) / 2 <= (int)blockIdx.x) ++I;
  while (I * (I + 1) / 2 > (int)blockIdx.x) --I;
  const int J = (int)blockIdx.x - I * (I + 1) / 2;
  for (int e = threadIdx.x; e < NB * NB; e += 256) {
    const int r = e / NB, c = e % NB, gr = I * NB + r, gc = J * NB + c;
    s[r][c] = (gr < n && gc < gr) ? fabs(H[(size_t)gr * ld + gc]) : 0.0;
  }
  __syncthreads();
  const int t = threadIdx.x;
  const size_t width = (size_t)T * NB;
  if (t < NB) {
    double a = 0.0;
    for (int c = 0; c < NB; ++c) a += s[t][c];
    if (I == J)
      for (int r = 0; r < NB; ++r) a += s[r][t];
    part[J * width + I * NB + t] = a;
  } else if (t < 2 * NB && I != J) {
    double a = 0.0;
    for (int r = 0; r < NB; ++r) a += s[r][t - NB];
    part[I * width + J * NB + t - NB] = a;
  }
}

// Per block row: max over rows of d + sum |off|, min d, sum d.
__global__ void __launch_bounds__(NB) row_bounds_kernel(const double* H, int n, int ld, int T, const double* part,
                                                       double* rowred) {
  __shared__ double sm[3][NB];
  const int t = threadIdx.x, r = blockIdx.x * NB + t;
  const size_t width = (size_t)T * NB;
  double off = 0.0;
  for (int J = 0; J < T; ++J) off += part[J * width + r];
  const bool in = r < n;
  const double d = in ? H[(size_t)r * ld + r] : 0.0;
  sm[0][t] = in ? d + off : -1e300;
  sm[1][t] = in ? d : 1e300;
  sm[2][t] = in ? d : 0.0;
  // a NaN anywhere must reach the bounds: it is refused there
  if (in && !(d + off == d + off)) sm[1][t] = -1.0;
  __syncthreads();
  for (int h = NB / 2; h > 0; h >>= 1) {
    if (t < h) {
      sm[0][t] = fmax(sm[0][t], sm[0][t + h]);
      sm[1][t] = fmin(sm[1][t], sm[1][t + h]);
      sm[2][t] += sm[2][t + h];
    }
    __syncthreads();
  }
  if (t < 3) rowred[3 * blockIdx.x + t] = sm[t][0];
}

// ---- Lanczos: the smallest Ritz value ---------------------------------------
// Start vector: signs from a hash of the row, norm 1 (block sums of squares as
// every later u's).
__global__ void __launch_bounds__(NB) lanczos_start_kernel(TraceWs w, int n, int T) {
  const int t = threadIdx.x, r = blockIdx.x * NB + t;
  unsigned h = (unsigned)r * 2654435761u;
  h ^= h >> 15;
  h *= 2246822519u;
  h ^= h >> 13;
  w.u[r] = r < n ? ((h & 1) ? 1.0 : -1.0) : 0.0;
  w.v[1][r] = 0.0;
  if (t == 0) w.norms[blockIdx.x] = (double)min(NB, n - (int)blockIdx.x * NB);
}

// Sum of T partials, the same in every thread of the CTA (fixed order).
__device__ __forceinline__ double sum_partials(const double* p, int T) {
  double s = 0.0;
  for (int k = threadIdx.x & 31; k < T; k += 32) s += p[k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
__device__ __forceinline__ double inv_norm(const double* p, int T) {
  const double s = sum_partials(p, T);
  return s > 0.0 ? 1.0 / sqrt(s) : 0.0;
}

// part[J][row of I], part[I][row of J]: the two products of one lower tile of H
// with v = u / |u|.  Warp: 8 rows, lane: two columns.  Bound by the read of H.
__global__ void __launch_bounds__(256) lanczos_symv_kernel(const double* H, int n, int ld, int T, TraceWs w, int step) {
  __shared__ double xi[NB], xj[NB], cs[8][NB];
  int I = (int)((sqrt(8.0 * blockIdx.x + 1.0) - 1.0) * 0.5);
  while ((I + 1) * (I + 2) / 2 <= (int)blockIdx.x) ++I;
  while (I * (I + 1) / 2 > (int)blockIdx.x) --I;
  const int J = (int)blockIdx.x - I * (I + 1) / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2 a[8];
  const int gc = J * NB + 2 * lane;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int gr = I * NB + 8 * warp + u;
    a[u] = make_double2(0.0, 0.0);
    if (gr < n && gc < n) a[u] = *reinterpret_cast<const double2*>(H + (size_t)gr * ld + gc);
  }
  const double s = inv_norm(w.norms + (size_t)step * T, T);
  if (tid < NB) xi[tid] = w.u[I * NB + tid] * s;
  else if (tid < 2 * NB) xj[tid - NB] = w.u[J * NB + tid - NB] * s;
  __syncthreads();
  double rs[8], c0 = 0.0, c1 = 0.0;
  const double x0 = xj[2 * lane], x1 = xj[2 * lane + 1];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int r = 8 * warp + u;
    double ax = a[u].x, ay = a[u].y, bx = ax, by = ay;
    if (I == J) {   // entries above the diagonal are not the matrix's; the diagonal counts once
      if (2 * lane > r) ax = 0.0;
      if (2 * lane + 1 > r) ay = 0.0;
      if (2 * lane >= r) bx = 0.0;
      if (2 * lane + 1 >= r) by = 0.0;
    } else if (gc + 1 >= n) {
      ay = by = 0.0;
    }
    rs[u] = ax * x0 + ay * x1;
    c0 += bx * xi[r];
    c1 += by * xi[r];
  }
  // rows: reduce-scatter over the lanes, row (lane >> 2) & 7 on four lanes
#pragma unroll
  for (int m = 4, off = 16; m >= 1; m >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int u = 0; u < m; ++u) {
      const double send = up ? rs[u] : rs[u + m], keep = up ? rs[u + m] : rs[u];
      rs[u] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  double y = rs[0] + __shfl_xor_sync(0xffffffffu, rs[0], 2);
  y += __shfl_xor_sync(0xffffffffu, y, 1);
  cs[warp][2 * lane] = c0;
  cs[warp][2 * lane + 1] = c1;
  __shared__ double row[NB];
  if ((lane & 3) == 0) row[8 * warp + (lane >> 2)] = y;
  __syncthreads();
  if (tid < NB) {
    double c = 0.0;
#pragma unroll
    for (int v = 0; v < 8; ++v) c += cs[v][tid];
    const size_t width = (size_t)T * NB;
    w.part[J * width + I * NB + tid] = I == J ? row[tid] + c : row[tid];
    if (I != J) w.part[I * width + J * NB + tid] = c;
  }
}

// y = H v on a block row, v kept, the block's part of v^T y.
__global__ void __launch_bounds__(NB) lanczos_rows_kernel(TraceWs w, int T, int step) {
  __shared__ double sm[NB];
  const int t = threadIdx.x, r = blockIdx.x * NB + t;
  const size_t width = (size_t)T * NB;
  double y = 0.0;
#pragma unroll 8
  for (int J = 0; J < T; ++J) y += w.part[J * width + r];
  const double v = w.u[r] * inv_norm(w.norms + (size_t)step * T, T);
  w.y[r] = y;
  w.v[step & 1][r] = v;
  sm[t] = v * y;
  __syncthreads();
  for (int h = NB / 2; h > 0; h >>= 1) {
    if (t < h) sm[t] += sm[t + h];
    __syncthreads();
  }
  if (t == 0) w.dots[(size_t)step * T + blockIdx.x] = sm[0];
}

// u = y - alpha v - beta v_prev; the block's part of |u|^2.
__global__ void __launch_bounds__(NB) lanczos_next_kernel(TraceWs w, int T, int step) {
  __shared__ double sm[NB];
  const int t = threadIdx.x, r = blockIdx.x * NB + t;
  const double alpha = sum_partials(w.dots + (size_t)step * T, T);
  const double beta = step > 0 ? sqrt(sum_partials(w.norms + (size_t)step * T, T)) : 0.0;
  const double u = w.y[r] - alpha * w.v[step & 1][r] - beta * w.v[(step + 1) & 1][r];
  w.u[r] = u;
  sm[t] = u * u;
  __syncthreads();
  for (int h = NB / 2; h > 0; h >>= 1) {
    if (t < h) sm[t] += sm[t + h];
    __syncthreads();
  }
  if (t == 0) w.norms[(size_t)(step + 1) * T + blockIdx.x] = sm[0];
}

// Smallest eigenvalue of the Lanczos tridiagonal matrix, by Sturm counts at 32
// points of the bracket at a time; one warp.
__device__ double smallest_ritz(const TraceWs& w, int T) {
  const int lane = threadIdx.x & 31;
  double d[kLanczosSteps], e2[kLanczosSteps];
  double lo = 1e300, hi = 1e300, scale = 0.0;
  int k_end = kLanczosSteps;
  for (int k = 0; k < kLanczosSteps; ++k) {
    d[k] = sum_partials(w.dots + (size_t)k * T, T);
    e2[k] = sum_partials(w.norms + (size_t)(k + 1) * T, T);   // beta_{k+1}^2
    scale = fmax(scale, fabs(d[k]));
    if (!(e2[k] > 1e-24 * scale * scale)) {   // an invariant subspace: the values are exact
      k_end = k + 1;
      break;
    }
  }
  for (int k = 0; k < k_end; ++k) {
    const double off = (k > 0 ? sqrt(e2[k - 1]) : 0.0) + (k + 1 < k_end ? sqrt(e2[k]) : 0.0);
    lo = fmin(lo, d[k] - off);
    hi = fmin(hi, d[k]);                       // the smallest value is below every diagonal entry
  }
  for (int it = 0; it < 5; ++it) {
    const double x = lo + (hi - lo) * (lane + 1) / 33.0;
    bool below = false;                        // some eigenvalue < x
    double q = d[0] - x;
    below = q < 0.0;
    for (int k = 1; k < k_end; ++k) {
      q = d[k] - x - e2[k - 1] / (fabs(q) > 1e-300 ? q : 1e-300);
      below = below || q < 0.0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, below);
    const int first = m ? __ffs(m) - 1 : 32;   // first point past the smallest value
    const double w0 = hi - lo, l0 = lo;
    lo = l0 + w0 * first / 33.0;
    hi = l0 + w0 * (first + 1) / 33.0;
  }
  return lo;
}

// Bounds, node count and nodes; one warp.
__global__ void __launch_bounds__(32) nodes_kernel(TraceWs w, int n, int T, double digits) {
  const int lane = threadIdx.x;
  double hi = -1e300, lo = 1e300, tr = 0.0;
  for (int b = lane; b < T; b += 32) {
    hi = fmax(hi, w.rowred[3 * b]);
    lo = fmin(lo, w.rowred[3 * b + 1]);
    tr += w.rowred[3 * b + 2];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    tr += __shfl_xor_sync(0xffffffffu, tr, o);
  }
  double m = kLowerShare * lo;
  const double M = hi;
  if (n >= kLanczosMinN && lo > 0.0) m = kRitzShare * smallest_ritz(w, T);
  int nodes = 0;
  if (lo > 0.0 && m > 0.0 && M >= lo && M < 1e300) {
    const double want = ceil(digits * (log(M / m) + 2.772588722239781) / (2.0 * 9.869604401089358));
    nodes = want <= kTraceNodes ? (int)want : 0;
  }
  if (lane < kTraceBatch) w.info[lane] = 0;
  if (lane == 0) *w.count = nodes > 0 ? nodes + 1 : 0;
  if (nodes == 0) return;
  const double c2 = tr / n;
  // K(k) and sn, cn, dn by the arithmetic-geometric mean (Abramowitz and
  // Stegun 17.6, 16.4), k' = sqrt(m/M)
  double av[10], cv[10];
  const double kp2 = m / M;
  double a = 1.0, b = sqrt(kp2);
  av[0] = 1.0;
  cv[0] = sqrt(1.0 - kp2);
#pragma unroll
  for (int i = 1; i < 10; ++i) {   // kp >= ~1e-3: converged after 7 steps
    cv[i] = 0.5 * (a - b);
    const double g = sqrt(a * b);
    a = 0.5 * (a + b);
    b = g;
    av[i] = a;
  }
  const double K = 1.5707963267948966 / a;
  if (lane < nodes) {
    const double h = K / nodes;
    double phi = 512.0 * a * ((lane + 0.5) * h);   // 2^9 a_9 v
#pragma unroll
    for (int i = 9; i > 0; --i) phi = 0.5 * (phi + asin(fmin(1.0, fmax(-1.0, cv[i] / av[i] * sin(phi)))));
    const double sn = sin(phi), cn = cos(phi);
    const double dn = sqrt(cn * cn + kp2 * sn * sn);
    const double u = sqrt(m) * sn / cn;
    w.shift[lane + 1] = u * u;
    w.ref[lane + 1] = 1.0 / (c2 + u * u);
    w.weight[lane + 1] = h * sqrt(m) * dn / (cn * cn) * 0.3183098861837907;
  }
  if (lane == 0) {
    w.shift[0] = -m;
    w.ref[0] = 1.0 / c2;
    w.weight[0] = 0.0;
    *w.c2 = c2;
  }
}

__device__ __forceinline__ void two_sum(double a, double b, double& s, double& err) {
  s = a + b;
  const double bb = s - a;
  err = (a - (s - bb)) + (b - bb);
}

// sum sqrt(lambda) = n c + sum_j w_j ln det_j; the energy.  One warp, a node
// per lane.
__global__ void __launch_bounds__(32) trace_energy_kernel(TraceWs w, int n, int T, int nsl, const double* scalars,
                                                         double* out) {
  const int lane = threadIdx.x;
  const int nb = *w.count;
  double s = 0.0, comp = 0.0;
  bool bad = nb == 0;
  if (lane < nb) {
    bad = w.info[lane] != 0;
    for (int k = 0; k < T; ++k) {
      double t, e;
      two_sum(s, w.logdet[(size_t)lane * T + k], t, e);
      s = t;
      comp += e;
    }
    s = (s + comp) * w.weight[lane];
    if (!(fabs(s) < 1e300)) bad = true;
  }
  const bool refused = __any_sync(0xffffffffu, bad);
  comp = 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double s2 = __shfl_down_sync(0xffffffffu, s, o), c2 = __shfl_down_sync(0xffffffffu, comp, o);
    double t, e;
    two_sum(s, s2, t, e);
    s = t;
    comp += c2 + e;
  }
  if (lane == 0) {
    // E = sum sqrt / (2 nsl) - sum 3 omega / 2: the two large terms first
    const double c2v = refused ? 0.0 : *w.c2;
    const double c = sqrt(c2v);
    // n sqrt(c2) to twice the precision: c2 = c^2 + r, sqrt(c2) = c + r / 2c
    const double r = refused ? 0.0 : fma(-c, c, c2v) / (2.0 * c);
    const double lead = n * c;
    const double lead_err = fma((double)n, c, -lead) + n * r;
    const double ni = scalars[1] * nsl;
    const double ni_err = fma(scalars[1], (double)nsl, -ni);
    double d, e, t, e2;
    two_sum(lead, -ni, d, e);
    two_sum(d, s, t, e2);
    out[0] = 0.5 * (t + (e + e2 + comp + lead_err - ni_err)) / nsl;
    out[1] = lead + (s + (comp + lead_err));
    out[2] = 0.0;
    out[3] = refused ? kTraceRefused : kTraceOk;
  }
}

}  // namespace

int trace_launches(int n) { return 5 + (n >= kLanczosMinN ? 1 + 3 * kLanczosSteps : 0); }

size_t trace_ws_bytes(int n) {
  TraceWs w;
  return carve(nullptr, n, &w);
}

cudaError_t launch_trace_energy(const TraceArgs& a, int num_sms, cudaStream_t s) {
  TraceWs w;
  carve(a.ws, a.n, &w);
  const int T = (a.n + NB - 1) / NB;
  abs_sums_kernel<<<T * (T + 1) / 2, 256, 0, s>>>(a.H, a.n, a.ld, T, w.part);
  row_bounds_kernel<<<T, NB, 0, s>>>(a.H, a.n, a.ld, T, w.part, w.rowred);
  if (a.n >= kLanczosMinN) {
    lanczos_start_kernel<<<T, NB, 0, s>>>(w, a.n, T);
    for (int k = 0; k < kLanczosSteps; ++k) {
      lanczos_symv_kernel<<<T * (T + 1) / 2, 256, 0, s>>>(a.H, a.n, a.ld, T, w, k);
      lanczos_rows_kernel<<<T, NB, 0, s>>>(w, T, k);
      lanczos_next_kernel<<<T, NB, 0, s>>>(w, T, k);
    }
  }
  nodes_kernel<<<1, 32, 0, s>>>(w, a.n, T, a.digits);
  CholFlowArgs f{};
  f.src = a.H;
  f.src_stride = 0;
  f.src_ld = a.ld;
  f.L = a.L;
  f.l_stride = (size_t)a.n * a.ld;
  f.ld = a.ld;
  f.n = a.n;
  f.batch = kTraceBatch;
  f.batch_dev = w.count;
  f.shift = w.shift;
  f.linv = a.linv;
  f.linv_stride = (size_t)T * NB * NB;
  f.logdet = w.logdet;
  f.ref = w.ref;
  f.c2 = w.c2;
  f.info = w.info;
  f.sync = w.sync;
  f.stop = w.info;   // the certificate's: where it fails, nothing else counts
  f.err = a.err;
  f.stall = a.stall;
  cudaError_t e = launch_chol_flow(f, num_sms, s);
  if (e != cudaSuccess) return e;
  trace_energy_kernel<<<1, 32, 0, s>>>(w, a.n, T, a.nsl, a.scalars, a.out);
  return cudaGetLastError();
}

}  // namespace mbd
