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
// diagonal entry); the factorisation of H - m I, one more matrix of the
// batch, proves m <= lambda.  Where it fails, or M/m asks for more than
// kTraceNodes nodes, the result is refused and the caller takes the
// eigenvalues (imaginary modes, near-instabilities).
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"

namespace mbd {
namespace {

constexpr int NB = kCholNB;
constexpr double kLowerShare = 0.2;      // m over the smallest diagonal entry
// Digits the rule is run to: exp(-33) of the strip estimate, measured
// <= 2e-16 of sum sqrt(lambda) on clusters, molecules, sheets and boxes
// (spectra from LAPACK, M/m from 6 to 160: 8 to 14 nodes).
constexpr double kDigits = 33.0;

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

// Bounds, node count and nodes; one warp.
__global__ void __launch_bounds__(32) nodes_kernel(TraceWs w, int n, int T) {
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
  const double m = kLowerShare * lo, M = hi;
  int nodes = 0;
  if (lo > 0.0 && M >= lo && M < 1e300) {
    const double want = ceil(kDigits * (log(M / m) + 2.772588722239781) / (2.0 * 9.869604401089358));
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
  nodes_kernel<<<1, 32, 0, s>>>(w, a.n, T);
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
  f.err = a.err;
  cudaError_t e = launch_chol_flow(f, num_sms, s);
  if (e != cudaSuccess) return e;
  trace_energy_kernel<<<1, 32, 0, s>>>(w, a.n, T, a.nsl, a.scalars, a.out);
  return cudaGetLastError();
}

}  // namespace mbd
