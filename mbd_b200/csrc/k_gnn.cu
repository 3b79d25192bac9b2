// Message-passing network of the learned relay warm start: forward pass,
// loss, backward pass and Adam, FP32, one graph per geometry with the 21
// imaginary frequencies as 21 copies of the atom graph (node = f * N + i).
//
//   x      = [onehot(H, C, N, O, other), h_i, log alpha_i(iw_f), log(1 + w_f)]
//   h0     = silu(W0 x + b0)
//   layer l = 0..2:  m_i = sum_j (Wf_l e_ij) * h_j;  h_i += silu(Wu_l m_i + bu_l)
//   s_i = ws.h_i + bs,  a_i = wa.h_i + ca,  g_ij = wg.e_ij
//   S_i = (1 + s_i) I + sum_j a_j g_ij (u_ij u_ij^T - I/3),   X_i = alpha_i S_i
// e_ij: 16 Gaussian radial functions of |r_ij| times a cosine cut-off at 5 A;
// u_ij the unit vector from i to j.  Neighbour lists are symmetric (j in
// nbr(i) <=> i in nbr(j) with the same distance), so every backward scatter
// is written as a gather over the receiving node's own list.
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "gnn.h"

namespace mbd {
namespace {

constexpr int H = kGnnHidden;
constexpr int NR = kGnnRbf;
constexpr int NI = kGnnIn;

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }
__device__ __forceinline__ float dsilu(float z) {
  const float s = sigm(z);
  return s * (1.0f + z * (1.0f - s));
}

__global__ void edge_kernel(const float* dvec, int E, float* efeat, float* eproj) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const float dx = dvec[3 * e], dy = dvec[3 * e + 1], dz = dvec[3 * e + 2];
  const float r = sqrtf(dx * dx + dy * dy + dz * dz);
  const float ir = 1.0f / r;
  const float ux = dx * ir, uy = dy * ir, uz = dz * ir;
  const float rc = kGnnCutoffBohr;
  const float w = rc / (NR - 1);
  const float fc = 0.5f * (cosf(3.14159265358979f * r / rc) + 1.0f);
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    const float t = (r - w * k) / w;
    efeat[(size_t)e * NR + k] = __expf(-0.5f * t * t) * fc;
  }
  float* p = eproj + (size_t)e * 6;
  p[0] = ux * ux - 1.0f / 3.0f;
  p[1] = uy * uy - 1.0f / 3.0f;
  p[2] = uz * uz - 1.0f / 3.0f;
  p[3] = ux * uy;
  p[4] = ux * uz;
  p[5] = uy * uz;
}

__global__ void features_kernel(const int* species, const double* hirsh, const double* alpha_w, const double* omega,
                                int N, int F, float* x) {
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= N * F) return;
  const int f = node / N, i = node % N;
  float* xo = x + (size_t)node * NI;
  const int sp = species[i];
#pragma unroll
  for (int k = 0; k < 5; ++k) xo[k] = (k == sp) ? 1.0f : 0.0f;
  xo[5] = (float)hirsh[i];
  xo[6] = (float)log(alpha_w[(size_t)f * N + i]);
  xo[7] = (float)log1p(omega[f]);
}

// filt[l][e][k] = Wf_l[k] . e_e (l = 0..2), g[e] = wg . e_e.  A thread keeps
// the weights of one output in registers and takes the CTA's edges in turn
// (their features broadcast from shared memory); bound by the stores.  With
// the weights and features read from global memory for every output: 74 us at
// 15 000 edges, 8 now.
constexpr int kFilterEdges = 32;
constexpr int kFilterOut = kGnnLayers * H + 1;
__global__ void __launch_bounds__(224) filter_kernel(const float* P, const float* efeat, int E, float* filt, float* g) {
  __shared__ __align__(16) float es[kFilterEdges][NR];
  const int e0 = blockIdx.x * kFilterEdges, ne = min(kFilterEdges, E - e0), c = threadIdx.x;
  for (int t = threadIdx.x; t < ne * NR; t += blockDim.x) es[t / NR][t % NR] = efeat[(size_t)e0 * NR + t];
  const int l = c / H, k = c % H;
  float W[NR];
  if (c < kFilterOut) {
    const float* Wg = c == kGnnLayers * H ? P + kGnnOffWg : P + kGnnOffWf(l) + k * NR;
#pragma unroll
    for (int q = 0; q < NR; ++q) W[q] = Wg[q];
  }
  __syncthreads();
  if (c >= kFilterOut) return;
  float* out = c == kGnnLayers * H ? g + e0 : filt + ((size_t)l * E + e0) * H + k;
  const int stride = c == kGnnLayers * H ? 1 : H;
  for (int e = 0; e < ne; ++e) {
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < NR; ++q) s += W[q] * es[e][q];
    out[(size_t)e * stride] = s;
  }
}

__global__ void embed_kernel(const float* P, const float* x, int M, float* pre0, float* h0) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)M * H) return;
  const int node = (int)(idx / H), k = (int)(idx % H);
  const float* W = P + kGnnOffW0 + k * NI;
  const float* xi = x + (size_t)node * NI;
  float s = P[kGnnOffB0 + k];
#pragma unroll
  for (int q = 0; q < NI; ++q) s += W[q] * xi[q];
  pre0[idx] = s;
  h0[idx] = silu(s);
}

// m[f*N+i][k] = sum_{e in nbr(i)} filt[e][k] h[f*N+nbr[e]][k] (plus start[f*N+i][k]
// where given).  A CTA takes an atom and kConvGroups * kConvF frequencies: a
// filter entry is read once for a thread's kConvF frequencies, and the loads
// of four edges are in flight together.
constexpr int kConvGroups = 4, kConvF = 2;
__device__ __forceinline__ void conv(const float* h, const float* filt, const int* off, const int* nbr, int N, int F,
                                     const float* start, float* m, int i, int fblock) {
  const int k = threadIdx.x % H, fg = threadIdx.x / H;
  const int e0 = off[i], e1 = off[i + 1];
  const int f0 = fblock * kConvGroups * kConvF;
  float s[kConvF];
#pragma unroll
  for (int u = 0; u < kConvF; ++u) {
    const int f = f0 + fg + kConvGroups * u;
    s[u] = start && f < F ? start[((size_t)f * N + i) * H + k] : 0.f;
  }
#pragma unroll 4
  for (int e = e0; e < e1; ++e) {
    const float w = filt[(size_t)e * H + k];
    const float* hj = h + (size_t)nbr[e] * H + k;
#pragma unroll
    for (int u = 0; u < kConvF; ++u) {
      const int f = f0 + fg + kConvGroups * u;
      if (f < F) s[u] += w * hj[(size_t)f * N * H];
    }
  }
#pragma unroll
  for (int u = 0; u < kConvF; ++u) {
    const int f = f0 + fg + kConvGroups * u;
    if (f < F) m[((size_t)f * N + i) * H + k] = s[u];
  }
}

__global__ void __launch_bounds__(64 * kConvGroups) conv_kernel(const float* h, const float* filt, const int* off,
                                                               const int* nbr, int N, int F, float* m) {
  conv(h, filt, off, nbr, N, F, nullptr, m, blockIdx.x, blockIdx.y);
}

// Y[16 nodes][64] = (init +) X W^T-like products from shared memory: thread =
// one node x 4 outputs.  Ws[q][k].
constexpr int kDenseNodes = 16;
__device__ __forceinline__ void dense_tile(const float (*Ws)[H + 4], const float (*Xs)[H + 1], int k4, int node,
                                           float (&acc)[4]) {
#pragma unroll 8
  for (int q = 0; q < H; ++q) {
    const float4 w = *reinterpret_cast<const float4*>(&Ws[q][k4]);
    const float x = Xs[node][q];
    acc[0] += w.x * x;
    acc[1] += w.y * x;
    acc[2] += w.z * x;
    acc[3] += w.w * x;
  }
}

// u = Wu m + bu; h_out = h_in + silu(u)
__global__ void __launch_bounds__(256) dense_kernel(const float* P, int l, const float* m, const float* h_in,
                                                    float* u, float* h_out, int M) {
  __shared__ __align__(16) float Wt[H][H + 4];   // Wt[q][k] = Wu[k][q]
  __shared__ float ms[kDenseNodes][H + 1];
  const float* W = P + kGnnOffWu(l);
  const int n0 = blockIdx.x * kDenseNodes;
  for (int t = threadIdx.x; t < H * H; t += 256) Wt[t % H][t / H] = W[t];
  for (int t = threadIdx.x; t < kDenseNodes * H; t += 256)
    ms[t / H][t % H] = n0 + t / H < M ? m[(size_t)n0 * H + t] : 0.f;
  __syncthreads();
  const int k4 = 4 * (threadIdx.x & 15), node = threadIdx.x >> 4;
  float acc[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) acc[c] = P[kGnnOffBu(l) + k4 + c];
  dense_tile(Wt, ms, k4, node, acc);
  if (n0 + node >= M) return;
  const size_t o = (size_t)(n0 + node) * H + k4;
  const float4 hi = *reinterpret_cast<const float4*>(h_in + o);
  *reinterpret_cast<float4*>(u + o) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  *reinterpret_cast<float4*>(h_out + o) =
      make_float4(hi.x + silu(acc[0]), hi.y + silu(acc[1]), hi.z + silu(acc[2]), hi.w + silu(acc[3]));
}

// s = ws.h + bs, a = wa.h + ca (one warp per node)
__global__ void sa_kernel(const float* P, const float* h, int M, float* s, float* a) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
  if (warp >= M) return;
  const float* hn = h + (size_t)warp * H;
  float vs = P[kGnnOffWs + lane] * hn[lane] + P[kGnnOffWs + lane + 32] * hn[lane + 32];
  float va = P[kGnnOffWa + lane] * hn[lane] + P[kGnnOffWa + lane + 32] * hn[lane + 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vs += __shfl_xor_sync(0xffffffffu, vs, o);
    va += __shfl_xor_sync(0xffffffffu, va, o);
  }
  if (lane == 0) {
    s[warp] = vs + P[kGnnOffBs];
    a[warp] = va + P[kGnnOffCa];
  }
}

// S (row-major 3x3) per node, one of its six sums per lane of eight: every sum
// runs over the edges in their order, so that the prediction keeps its bits
// (eight lanes that split the edges and add up took as long).
__global__ void tensor_kernel(const float* s, const float* a, const float* g, const float* eproj, const int* off,
                              const int* nbr, int N, int F, float* S) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x, node = idx >> 3, c = idx & 7;
  if (node >= N * F || c >= 6) return;
  const int f = node / N, i = node % N;
  float p = 0.f;
#pragma unroll 4
  for (int e = off[i]; e < off[i + 1]; ++e) {
    const float w = a[(size_t)f * N + nbr[e]] * g[e];
    p += w * eproj[(size_t)e * 6 + c];
  }
  float* o = S + (size_t)node * 9;
  if (c < 3) {
    o[4 * c] = (1.0f + s[node]) + p;
  } else {   // xy, xz, yz
    const int k = c == 5 ? 5 : c - 2;
    o[k] = o[c == 3 ? 3 : (c == 4 ? 6 : 7)] = p;
  }
}

// dS = 2 (S - S_true) / M; loss += ||S - S_true||^2 / M
__global__ void loss_kernel(const float* S, const float* St, int M, float* dS, double* loss) {
  __shared__ double red[256];
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  double l = 0.0;
  if (node < M) {
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      const float d = S[(size_t)node * 9 + c] - St[(size_t)node * 9 + c];
      dS[(size_t)node * 9 + c] = 2.0f * d / (float)M;
      l += (double)d * d;
    }
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, red[0] / M);
}

__device__ __forceinline__ float dot_proj(const float* dS, const float* p) {
  return dS[0] * p[0] + dS[4] * p[1] + dS[8] * p[2] + (dS[1] + dS[3]) * p[3] + (dS[2] + dS[6]) * p[4] +
         (dS[5] + dS[7]) * p[5];
}

// ds = tr dS; da_j = sum_{e in nbr(j)} g_e <dS_nbr, P_e>; cw[f][e] = <dS_i, P_e> a_nbr
__global__ void readout_bwd_kernel(const float* dS, const float* a, const float* g, const float* eproj,
                                   const int* off, const int* nbr, int N, int F, int E, float* ds, float* da,
                                   float* cw) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x, node = idx >> 3, sub = idx & 7;   // 8 lanes a node
  const bool live = node < N * F;
  const int f = live ? node / N : 0, i = live ? node % N : 0;
  const float* dSi = dS + (size_t)(live ? node : 0) * 9;
  const int e0 = live ? off[i] : 0, e1 = live ? off[i + 1] : 0;
  const int rounds = __reduce_max_sync(0xffffffffu, (e1 - e0 + 7) / 8);
  float acc = 0.f;
  for (int r = 0; r < rounds; ++r) {
    const int e = e0 + 8 * r + sub;
    float t = 0.f, ge = 0.f;
    if (e < e1) {
      const int j = f * N + nbr[e];
      const float* pe = eproj + (size_t)e * 6;
      ge = g[e];
      t = dot_proj(dS + (size_t)j * 9, pe);
      cw[(size_t)f * E + e] = dot_proj(dSi, pe) * a[j];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)   // in the order of the edges; zeros behind the last
      acc += __shfl_sync(0xffffffffu, ge, u, 8) * __shfl_sync(0xffffffffu, t, u, 8);
  }
  if (!live || sub != 0) return;
  ds[node] = dSi[0] + dSi[4] + dSi[8];
  da[node] = acc;
}

// dh = ds ws + da wa
__global__ void readout_dh_kernel(const float* P, const float* ds, const float* da, int M, float* dh) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)M * H) return;
  const int node = (int)(idx / H), k = (int)(idx % H);
  dh[idx] = ds[node] * P[kGnnOffWs + k] + da[node] * P[kGnnOffWa + k];
}

// du = dh * silu'(u); dm = Wu^T du
__device__ __forceinline__ void dense_bwd(const float* Wg, const float* dh, const float* u, float* du, float* dm, int M,
                                          int block, float* smem) {
  float(*W)[H + 4] = reinterpret_cast<float(*)[H + 4]>(smem);   // W[k][q]
  float(*ds_)[H + 1] = reinterpret_cast<float(*)[H + 1]>(smem + H * (H + 4));
  const int n0 = block * kDenseNodes;
  for (int t = threadIdx.x; t < H * H; t += 256) W[t / H][t % H] = Wg[t];
  for (int t = threadIdx.x; t < kDenseNodes * H; t += 256) {
    float d = 0.f;
    if (n0 + t / H < M) {
      d = dh[(size_t)n0 * H + t] * dsilu(u[(size_t)n0 * H + t]);
      du[(size_t)n0 * H + t] = d;
    }
    ds_[t / H][t % H] = d;
  }
  __syncthreads();
  const int k4 = 4 * (threadIdx.x & 15), node = threadIdx.x >> 4;
  float acc[4] = {};
  dense_tile(W, ds_, k4, node, acc);
  if (n0 + node < M)
    *reinterpret_cast<float4*>(dm + (size_t)(n0 + node) * H + k4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
}

// dfilt[e][k] = sum_f dm[f, src_e][k] h[f, nbr_e][k]
__device__ __forceinline__ void filter_grad(const float* dm, const float* h, const int* src, const int* nbr, int N,
                                            int F, int E, float* dfilt, int block) {
  const long long idx = (long long)block * 256 + threadIdx.x;
  if (idx >= (long long)E * H) return;
  const int e = (int)(idx / H), k = (int)(idx % H);
  const int i = src[e], j = nbr[e];
  float s = 0.f;
  for (int f = 0; f < F; ++f) s += dm[((size_t)f * N + i) * H + k] * h[((size_t)f * N + j) * H + k];
  dfilt[idx] = s;
}

// out[k1][k2] += sum_r A[r][k1] B[r][k2] and, where given, bias[k1] += sum_r
// A[r][k1], for K1 = 64; with pre, A[r][k1] silu'(pre[r][k1]) for A.  A CTA stages 64 rows at a time; a thread keeps a
// TM x 4 block of the outputs, sums 64 rows, adds them to its total and the
// totals atomically at the end.  One output per thread and row read both
// operands from shared memory for every product (17 us a launch, 9 now).
constexpr int kOuterRows = 64;
template <int K2>
__device__ __forceinline__ void outer(const float* A, const float* pre, const float* B, int rows, float* out, float* bias,
                                      int block, int nblocks, float* smem) {
  constexpr int TX = K2 / 4, TM = K2 >= 16 ? H * TX / 256 : 1;
  float(*As)[H + 1] = reinterpret_cast<float(*)[H + 1]>(smem);
  float(*Bs)[K2 + 4] = reinterpret_cast<float(*)[K2 + 4]>(smem + kOuterRows * (H + 1));   // 16-byte aligned
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;   // outputs k1 = TM ty .., k2 = 4 tx ..
  const bool work = TM * ty < H;
  float acc[TM][4], ab[TM];
#pragma unroll
  for (int t = 0; t < TM; ++t) {
    ab[t] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[t][c] = 0.f;
  }
  for (int r0 = block * kOuterRows; r0 < rows; r0 += nblocks * kOuterRows) {
    __syncthreads();
    const int nr = min(kOuterRows, rows - r0);
    for (int t = threadIdx.x; t < kOuterRows * H; t += 256)
      As[t / H][t % H] =
          t < nr * H ? (pre ? A[(size_t)r0 * H + t] * dsilu(pre[(size_t)r0 * H + t]) : A[(size_t)r0 * H + t]) : 0.f;
    for (int t = threadIdx.x; t < kOuterRows * K2; t += 256)
      Bs[t / K2][t % K2] = t < nr * K2 ? B[(size_t)r0 * K2 + t] : 0.f;
    __syncthreads();
    if (!work) continue;
    float s[TM][4], sb[TM];
#pragma unroll
    for (int t = 0; t < TM; ++t) {
      sb[t] = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) s[t][c] = 0.f;
    }
#pragma unroll 8
    for (int rr = 0; rr < kOuterRows; ++rr) {
      const float4 b = *reinterpret_cast<const float4*>(&Bs[rr][4 * tx]);
#pragma unroll
      for (int t = 0; t < TM; ++t) {
        const float x = As[rr][TM * ty + t];
        sb[t] += x;
        s[t][0] += x * b.x;
        s[t][1] += x * b.y;
        s[t][2] += x * b.z;
        s[t][3] += x * b.w;
      }
    }
#pragma unroll
    for (int t = 0; t < TM; ++t) {
      ab[t] += sb[t];
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[t][c] += s[t][c];
    }
  }
  if (!work) return;
#pragma unroll
  for (int t = 0; t < TM; ++t) {
    const int k1 = TM * ty + t;
#pragma unroll
    for (int c = 0; c < 4; ++c) atomicAdd(out + k1 * K2 + 4 * tx + c, acc[t][c]);
    if (bias && tx == 0) atomicAdd(bias + k1, ab[t]);
  }
}

// The readout's gradients: ws += ds^T h, wa += da^T h, bs += sum ds, ca += sum da.
__device__ __forceinline__ void readout_grad(const float* ds, const float* da, const float* h, int M, float* ws,
                                             float* wa, float* bs, float* ca, int block, int nblocks, float* smem) {
  float(*red)[2][H] = reinterpret_cast<float(*)[2][H]>(smem);
  float(*one)[2] = reinterpret_cast<float(*)[2]>(smem + 4 * 2 * H);
  const int k = threadIdx.x % H, sub = threadIdx.x / H;
  float s = 0.f, a = 0.f, s1 = 0.f, a1 = 0.f;
  for (int r0 = block * kOuterRows; r0 < M; r0 += nblocks * kOuterRows) {
    float cs = 0.f, cw = 0.f, c1 = 0.f, c2 = 0.f;
#pragma unroll 4
    for (int r = r0 + sub; r < min(M, r0 + kOuterRows); r += 4) {
      const float x = h[(size_t)r * H + k], u = ds[r], v = da[r];
      cs += u * x;
      cw += v * x;
      c1 += u;
      c2 += v;
    }
    s += cs;
    a += cw;
    s1 += c1;
    a1 += c2;
  }
  red[sub][0][k] = s;
  red[sub][1][k] = a;
  if (k == 0) {
    one[sub][0] = s1;
    one[sub][1] = a1;
  }
  __syncthreads();
  if (threadIdx.x < 2 * H) {
    const int w = threadIdx.x / H;
    atomicAdd((w ? wa : ws) + k, (red[0][w][k] + red[1][w][k]) + (red[2][w][k] + red[3][w][k]));
    if (k == 0) atomicAdd(w ? ca : bs, (one[0][w] + one[1][w]) + (one[2][w] + one[3][w]));
  }
}

// wg += sum over frequencies and edges of cw[f][e] efeat[e]
__device__ __forceinline__ void edge_grad(const float* cw, const float* efeat, int F, int E, float* wg, int block,
                                          int nblocks, float* smem) {
  float(*red)[NR] = reinterpret_cast<float(*)[NR]>(smem);
  const int q = threadIdx.x % NR, sub = threadIdx.x / NR;
  float t = 0.f;
  for (int e = block * 16 + sub; e < E; e += nblocks * 16) {
    float c = 0.f;
    for (int f = 0; f < F; ++f) c += cw[(size_t)f * E + e];
    t += c * efeat[(size_t)e * NR + q];
  }
  red[sub][q] = t;
  __syncthreads();
  if (threadIdx.x < NR) {
    float v = 0.f;
    for (int u = 0; u < 16; ++u) v += red[u][q];
    atomicAdd(wg + q, v);
  }
}

// The backward pass in launches of independent parts, a range of blocks each:
// a part alone leaves most of the device idle (some 20 M = 5000 nodes or
// 10 000 edges, 10-15 us of latency whatever its size).  A layer is
//   bwd_kernel       du, dm of the layer; behind them the weight gradients that
//                    the layer above left (from its du and dfilt), or those of
//                    the readout
//   bwd_conv_kernel  dh of the layer below and dfilt, both from dm
// Training of 16 clusters of 54 to 356 atoms, two epochs: 16.7 -> 14.2 ms against a
// launch for every part (22 launches a backward pass, 10 now).
struct BwdJobs {
  // blocks of each part, in this order
  int dense, embed, unit, filt, readout, edge;
  const float *Wu, *dh, *u;                 // dense: du = dh silu'(u), dm = Wu^T du
  float *du, *dm;
  const float *pre0, *x;                    // embed: W0, b0 from dh silu'(pre0) and x
  float *g_w0, *g_b0;
  const float *du_above, *m_above;          // unit: Wu, bu of the layer above
  float *g_wu, *g_bu;
  const float *dfilt, *efeat;               // filt: Wf of the layer above
  float* g_wf;
  const float *ds, *da, *h, *cw;            // readout and edge
  float *g_ws, *g_wa, *g_bs, *g_ca, *g_wg;
  int M, E, F;
};
__global__ void __launch_bounds__(256) bwd_kernel(BwdJobs j) {
  __shared__ __align__(16) float smem[kOuterRows * (H + 1) + kOuterRows * (H + 4)];
  int b = blockIdx.x;
  if (b < j.dense) return dense_bwd(j.Wu, j.dh, j.u, j.du, j.dm, j.M, b, smem);
  b -= j.dense;
  if (b < j.embed) return outer<kGnnIn>(j.dh, j.pre0, j.x, j.M, j.g_w0, j.g_b0, b, j.embed, smem);
  b -= j.embed;
  if (b < j.unit) return outer<H>(j.du_above, nullptr, j.m_above, j.M, j.g_wu, j.g_bu, b, j.unit, smem);
  b -= j.unit;
  if (b < j.filt) return outer<kGnnRbf>(j.dfilt, nullptr, j.efeat, j.E, j.g_wf, nullptr, b, j.filt, smem);
  b -= j.filt;
  if (b < j.readout)
    return readout_grad(j.ds, j.da, j.h, j.M, j.g_ws, j.g_wa, j.g_bs, j.g_ca, b, j.readout, smem);
  b -= j.readout;
  edge_grad(j.cw, j.efeat, j.F, j.E, j.g_wg, b, j.edge, smem);
}

// dh_out[j] = dh[j] + sum_{e in nbr(j)} filt[e] dm[nbr_e] (the lists are
// symmetric) on the first conv_blocks blocks, dfilt on the rest.
__global__ void __launch_bounds__(256) bwd_conv_kernel(const float* dm, const float* filt, const float* h, const int* off,
                                                       const int* nbr, const int* src, int N, int F, int E,
                                                       const float* dh, float* dh_out, float* dfilt, int conv_blocks) {
  if ((int)blockIdx.x < conv_blocks) return conv(dm, filt, off, nbr, N, F, dh, dh_out, blockIdx.x % N, blockIdx.x / N);
  filter_grad(dm, h, src, nbr, N, F, E, dfilt, blockIdx.x - conv_blocks);
}

__global__ void adam_kernel(float* P, float* G, float* m1, float* m2, int n, float lr, float b1, float b2, float eps,
                            float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = G[i];
  const float a = b1 * m1[i] + (1.f - b1) * g;
  const float b = b2 * m2[i] + (1.f - b2) * g * g;
  m1[i] = a;
  m2[i] = b;
  P[i] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
  G[i] = 0.f;
}

// X0[f][3i+r][c] = alpha_w[f][i] S[f*N+i][r][c]
__global__ void warmstart_kernel(const float* S, const double* alpha_w, int N, int F, double* X, size_t ystride) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)N * F * 9) return;
  const int node = (int)(idx / 9), c = (int)(idx % 9);
  const int f = node / N, i = node % N;
  X[(size_t)f * ystride + (size_t)9 * i + c] = alpha_w[(size_t)f * N + i] * (double)S[idx];
}

// S_true[f*N+i][r][c] = X[f][3i+r][c] / alpha_w[f][i]
__global__ void targets_kernel(const double* X, size_t ystride, const double* alpha_w, int N, int F, float* St) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)N * F * 9) return;
  const int node = (int)(idx / 9), c = (int)(idx % 9);
  const int f = node / N, i = node % N;
  St[idx] = (float)(X[(size_t)f * ystride + (size_t)9 * i + c] / alpha_w[(size_t)f * N + i]);
}

// ---- the network's neighbour lists (radius graph), built on the device ----
// Every (atom i, image t, atom j) is tested with one warp per atom i, lanes
// over j; a ballot orders each warp's edges by (image, j), so the lists come
// out deterministic.  Coordinates are in bohr; the translations and distances
// use explicitly rounded FP64 operations (no contraction), so the count pass
// and the fill pass take the same decisions.

__device__ __forceinline__ void image_shift(const GraphBox& b, int n0, int n1, int n2, double* t) {
#pragma unroll
  for (int c = 0; c < 3; ++c)
    t[c] = __dadd_rn(__dadd_rn(__dmul_rn((double)n0, b.lat[c]), __dmul_rn((double)n1, b.lat[3 + c])),
                     __dmul_rn((double)n2, b.lat[6 + c]));
}

// false when no atom of image t can lie within the cut-off of xi (xi outside
// the image's bounding box widened by the cut-off and a rounding margin)
__device__ __forceinline__ bool image_near(const GraphBox& b, const double* xi, const double* t) {
  bool near = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) near = near && xi[c] >= b.lo[c] + t[c] - b.pad && xi[c] <= b.hi[c] + t[c] + b.pad;
  return near;
}

template <bool FILL>
__global__ void __launch_bounds__(256) graph_kernel(const double* __restrict__ x, int N, GraphBox b,
                                                    const int* __restrict__ off_in, int* cnt_or_off,
                                                    int* __restrict__ nbr, int* __restrict__ src,
                                                    float* __restrict__ dvec) {
  const int lane = threadIdx.x & 31;
  const int i = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
  if (i >= N) return;   // whole warps
  const double xi[3] = {x[3 * i], x[3 * i + 1], x[3 * i + 2]};
  int pos = FILL ? off_in[i] : 0;
  if (FILL && lane == 0) {
    cnt_or_off[i] = pos;
    if (i == N - 1) cnt_or_off[N] = off_in[N];
  }
  for (int n0 = -b.rng[0]; n0 <= b.rng[0]; ++n0)
    for (int n1 = -b.rng[1]; n1 <= b.rng[1]; ++n1)
      for (int n2 = -b.rng[2]; n2 <= b.rng[2]; ++n2) {
        double t[3];
        image_shift(b, n0, n1, n2, t);
        if (!image_near(b, xi, t)) continue;   // uniform over the warp
        for (int j0 = 0; j0 < N; j0 += 32) {
          const int j = j0 + lane;
          bool ok = false;
          double d[3] = {0.0, 0.0, 0.0};
          if (j < N) {
#pragma unroll
            for (int c = 0; c < 3; ++c) d[c] = __dsub_rn(__dadd_rn(x[3 * j + c], t[c]), xi[c]);
            const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2]));
            ok = r2 < b.rc2 && r2 >= 1e-12;   // the atom itself (zero shift) has r = 0
          }
          const unsigned m = __ballot_sync(0xffffffffu, ok);
          if (FILL && ok) {
            const int e = pos + __popc(m & ((1u << lane) - 1u));
            nbr[e] = j;
            src[e] = i;
            dvec[3 * (size_t)e] = (float)d[0];
            dvec[3 * (size_t)e + 1] = (float)d[1];
            dvec[3 * (size_t)e + 2] = (float)d[2];
          }
          pos += __popc(m);
        }
      }
  if (!FILL && lane == 0) cnt_or_off[i] = pos;
}

// In-place exclusive scan of a[0..N) by one CTA; a[N] = *E = the total.
__global__ void __launch_bounds__(1024) graph_scan_kernel(int* a, int N, int* E) {
  __shared__ int wsum[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int chunk = (N + 1023) / 1024;
  const int b0 = min(N, t * chunk), b1 = min(N, b0 + chunk);
  int mine = 0;
  for (int k = b0; k < b1; ++k) mine += a[k];
  int v = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) wsum[w] = v;
  __syncthreads();
  if (w == 0) {
    int q = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, q, o);
      if (lane >= o) q += u;
    }
    wsum[lane] = q;
  }
  __syncthreads();
  int run = v - mine + (w > 0 ? wsum[w - 1] : 0);
  for (int k = b0; k < b1; ++k) {
    const int c = a[k];
    a[k] = run;
    run += c;
  }
  if (t == 0) {
    a[N] = wsum[31];
    *E = wsum[31];
  }
}

inline unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

dim3 conv_grid(const GnnGraph& g) {
  return dim3(g.N, (g.F + kConvGroups * kConvF - 1) / (kConvGroups * kConvF));
}

// Blocks of a part that sums over rows.
int sum_blocks(int rows, int per, int most) { return std::min((rows + per - 1) / per, most); }

}  // namespace

size_t gnn_work_floats(int N, int F, int E, bool train) {
  const size_t M = (size_t)N * F;
  size_t f = M * H * (1 + 4 + 3 + 3)          // pre0, h0..h3, m0..m2, u0..u2
             + (size_t)kGnnLayers * E * H + E // filt, g
             + 2 * M + 9 * M;                 // s, a, S
  if (train) f += 9 * M + 5 * M * H + 2 * M + (size_t)E * H + (size_t)F * E + 9 * M;   // dS, dh*, ds/da, dfilt, cw, S_true
  return f + 512;   // 8-float alignment of every array of the layout
}

GnnWork gnn_work_layout(float* base, int N, int F, int E, bool train) {
  const size_t M = (size_t)N * F;
  GnnWork w{};
  float* p = base;
  auto take = [&](size_t n) {
    float* q = p;
    p += (n + 7) & ~size_t(7);
    return q;
  };
  w.pre0 = take(M * H);
  for (int l = 0; l <= kGnnLayers; ++l) w.h[l] = take(M * H);
  for (int l = 0; l < kGnnLayers; ++l) w.m[l] = take(M * H);
  for (int l = 0; l < kGnnLayers; ++l) w.u[l] = take(M * H);
  w.filt = take((size_t)kGnnLayers * E * H);
  w.g = take(E);
  w.s = take(M);
  w.a = take(M);
  w.S = take(9 * M);
  if (train) {
    w.dS = take(9 * M);
    w.dh = take(M * H);
    w.dh2 = take(M * H);
    w.du = take(M * H);
    w.du2 = take(M * H);
    w.dm = take(M * H);
    w.ds = take(M);
    w.da = take(M);
    w.dfilt = take((size_t)E * H);
    w.cw = take((size_t)F * E);
    w.S_true = take(9 * M);
  }
  return w;
}

void gnn_graph_count(const double* x, int N, const GraphBox& b, int* cnt, cudaStream_t s) {
  graph_kernel<false><<<blocks(32LL * N, 256), 256, 0, s>>>(x, N, b, nullptr, cnt, nullptr, nullptr, nullptr);
}

void gnn_graph_scan(int* cnt_off, int N, int* E, cudaStream_t s) {
  graph_scan_kernel<<<1, 1024, 0, s>>>(cnt_off, N, E);
}

void gnn_graph_fill(const double* x, int N, const GraphBox& b, const int* off_in, int* off, int* nbr, int* src,
                    float* dvec, cudaStream_t s) {
  graph_kernel<true><<<blocks(32LL * N, 256), 256, 0, s>>>(x, N, b, off_in, off, nbr, src, dvec);
}

void gnn_edges(const float* dvec, int E, float* efeat, float* eproj, cudaStream_t s) {
  if (E > 0) edge_kernel<<<blocks(E, 256), 256, 0, s>>>(dvec, E, efeat, eproj);
}

void gnn_features(const int* species, const double* hirsh, const double* alpha_w, const double* omega, int N, int F,
                  float* x, cudaStream_t s) {
  features_kernel<<<blocks((long long)N * F, 256), 256, 0, s>>>(species, hirsh, alpha_w, omega, N, F, x);
}

int gnn_forward(const float* P, const GnnGraph& g, const GnnWork& w, cudaStream_t s) {
  const int M = g.N * g.F;
  if (g.E > 0)
    filter_kernel<<<blocks(g.E, kFilterEdges), 224, 0, s>>>(P, g.efeat, g.E, w.filt, w.g);
  embed_kernel<<<blocks((long long)M * H, 256), 256, 0, s>>>(P, g.x, M, w.pre0, w.h[0]);
  for (int l = 0; l < kGnnLayers; ++l) {
    conv_kernel<<<conv_grid(g), 64 * kConvGroups, 0, s>>>(w.h[l], w.filt + (size_t)l * g.E * H, g.off, g.nbr, g.N, g.F,
                                                          w.m[l]);
    dense_kernel<<<blocks(M, kDenseNodes), 256, 0, s>>>(P, l, w.m[l], w.h[l], w.u[l], w.h[l + 1], M);
  }
  sa_kernel<<<blocks((long long)M * 32, 256), 256, 0, s>>>(P, w.h[kGnnLayers], M, w.s, w.a);
  tensor_kernel<<<blocks(8LL * M, 128), 128, 0, s>>>(w.s, w.a, w.g, g.eproj, g.off, g.nbr, g.N, g.F, w.S);
  return 3 + 2 * kGnnLayers + (g.E > 0 ? 1 : 0);
}

int gnn_loss_backward(const float* P, const GnnGraph& g, const GnnWork& w, float* G, double* loss, cudaStream_t s) {
  const int M = g.N * g.F;
  int launches = 0;
  loss_kernel<<<blocks(M, 256), 256, 0, s>>>(w.S, w.S_true, M, w.dS, loss);
  readout_bwd_kernel<<<blocks(8LL * M, 128), 128, 0, s>>>(w.dS, w.a, w.g, g.eproj, g.off, g.nbr, g.N, g.F, g.E, w.ds, w.da,
                                                     w.cw);
  readout_dh_kernel<<<blocks((long long)M * H, 256), 256, 0, s>>>(P, w.ds, w.da, M, w.dh);
  launches += 3;
  const int outer_blocks = sum_blocks(M, kOuterRows, 592), filt_blocks = sum_blocks(g.E, kOuterRows, 592);
  const dim3 cg = conv_grid(g);
  float* dh = w.dh;
  float* dh_alt = w.dh2;
  BwdJobs j{};
  j.M = M;
  j.E = g.E;
  j.F = g.F;
  j.dfilt = w.dfilt;
  j.efeat = g.efeat;
  j.dm = w.dm;
  for (int l = kGnnLayers; l >= 0; --l) {
    // launch l: layer l - 1 (the embedding below layer 0) and the gradients layer l left
    j.dense = l > 0 ? (int)blocks(M, kDenseNodes) : 0;
    j.embed = l > 0 ? 0 : outer_blocks;
    j.unit = l < kGnnLayers ? outer_blocks : 0;
    j.filt = l < kGnnLayers ? filt_blocks : 0;
    j.readout = l < kGnnLayers ? 0 : outer_blocks;
    j.edge = l < kGnnLayers ? 0 : sum_blocks(g.E, 16, 296);
    j.dh = dh;
    if (l < kGnnLayers) {
      j.du_above = j.du;
      j.m_above = w.m[l];
      j.g_wu = G + kGnnOffWu(l);
      j.g_bu = G + kGnnOffBu(l);
      j.g_wf = G + kGnnOffWf(l);
    } else {
      j.ds = w.ds;
      j.da = w.da;
      j.h = w.h[kGnnLayers];
      j.cw = w.cw;
      j.g_ws = G + kGnnOffWs;
      j.g_wa = G + kGnnOffWa;
      j.g_bs = G + kGnnOffBs;
      j.g_ca = G + kGnnOffCa;
      j.g_wg = G + kGnnOffWg;
    }
    if (l > 0) {
      j.Wu = P + kGnnOffWu(l - 1);
      j.u = w.u[l - 1];
      j.du = l % 2 ? w.du : w.du2;
    } else {
      j.pre0 = w.pre0;
      j.x = g.x;
      j.g_w0 = G + kGnnOffW0;
      j.g_b0 = G + kGnnOffB0;
    }
    bwd_kernel<<<j.dense + j.embed + j.unit + j.filt + j.readout + j.edge, 256, 0, s>>>(j);
    ++launches;
    if (l == 0) break;
    const int conv_blocks = (int)(cg.x * cg.y);
    bwd_conv_kernel<<<conv_blocks + blocks((long long)g.E * H, 256), 256, 0, s>>>(
        w.dm, w.filt + (size_t)(l - 1) * g.E * H, w.h[l - 1], g.off, g.nbr, g.src, g.N, g.F, g.E, dh, dh_alt, w.dfilt,
        conv_blocks);
    ++launches;
    std::swap(dh, dh_alt);
  }
  return launches;
}

void gnn_adam(float* P, float* G, float* m1, float* m2, int step, float lr, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  adam_kernel<<<blocks(kGnnParams, 256), 256, 0, s>>>(P, G, m1, m2, kGnnParams, lr, b1, b2, 1e-8f, c1, c2);
}

void gnn_warmstart(const float* S, const double* alpha_w, int N, int F, double* X, size_t ystride, cudaStream_t s) {
  warmstart_kernel<<<blocks((long long)N * F * 9, 256), 256, 0, s>>>(S, alpha_w, N, F, X, ystride);
}

void gnn_targets(const double* X, size_t ystride, const double* alpha_w, int N, int F, float* St, cudaStream_t s) {
  targets_kernel<<<blocks((long long)N * F * 9, 256), 256, 0, s>>>(X, ystride, alpha_w, N, F, St);
}

}  // namespace mbd
