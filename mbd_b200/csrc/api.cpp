// C ABI of the engine (include/mbd_b200.h): context, upload / compute /
// download, and the orchestration of the kernels for one batch of
// geometries.  Replaces MBD_at_rsSCS (UTILS.f90:153-349) and the BLACS /
// MPI plumbing around it (UTILS.f90:97-149, 499-529) with one GPU.
//
// A batch runs in two parts.  The relay and CFDM stages of each geometry
// (UTILS.f90:239-315 and 745-807) run on one of up to kMaxSlots relay slots,
// each a CUDA stream with its own workspace, so the stages of different
// geometries overlap on the GPU.  Every geometry keeps its own CFDM
// Hamiltonian.  Then one cooperative launch reduces all Hamiltonians to
// tridiagonal form with CTA groups planned on the host (plan_tridiag), and
// one launch each computes all eigenvalues and all energies.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <memory>
#include <numeric>
#include <type_traits>
#include <vector>

#include "kernels.h"
#include "mbd_internal.h"
#include "tc3.h"

#include "context.h"


namespace mbd {
namespace {

// Symmetric 3x3 eigenvalues from the upper triangle (DSYEV('V','U'), UTILS.f90:273),
// cyclic Jacobi in FP64, ascending.  From the fifth sweep on, an off-diagonal
// entry that adds nothing to either diagonal one at a hundredfold counts as
// zero (Rutishauser's criterion): waiting for exact zeros took up to 50
// sweeps, 106 us for a geometry's 21 tensors (27 ms for a batch of 256).
void sym3_eigenvalues_upper(const double* M, double out[3]) {
  double a[3][3];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) a[r][c] = (r <= c) ? M[3 * r + c] : M[3 * c + r];
  for (int sweep = 0; sweep < 50; ++sweep) {
    double off = std::fabs(a[0][1]) + std::fabs(a[0][2]) + std::fabs(a[1][2]);
    if (off == 0.0) break;
    for (int p = 0; p < 2; ++p)
      for (int q = p + 1; q < 3; ++q) {
        if (a[p][q] == 0.0) continue;
        const double g = 100.0 * std::fabs(a[p][q]);
        if (sweep >= 4 && std::fabs(a[p][p]) + g == std::fabs(a[p][p]) &&
            std::fabs(a[q][q]) + g == std::fabs(a[q][q])) {
          a[p][q] = a[q][p] = 0.0;
          continue;
        }
        double theta = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
        double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < 3; ++k) {
          double akp = a[k][p], akq = a[k][q];
          a[k][p] = c * akp - s * akq;
          a[k][q] = s * akp + c * akq;
        }
        for (int k = 0; k < 3; ++k) {
          double apk = a[p][k], aqk = a[q][k];
          a[p][k] = c * apk - s * aqk;
          a[q][k] = s * apk + c * aqk;
        }
      }
  }
  out[0] = a[0][0];
  out[1] = a[1][1];
  out[2] = a[2][2];
  std::sort(out, out + 3);
}

// Sections of a buffer, each 256-byte aligned.
struct Sections {
  size_t size = 0;
  size_t add(size_t bytes) {
    const size_t at = size;
    size += (bytes + 255) & ~size_t(255);
    return at;
  }
};

// One geometry's device arrays: its inputs, the results the host reads back
// and the rest, as sections of the batch's three regions.  fill(dst, src,
// bytes) copies an input into the staging memory.
template <class Place, class Fill>
void lay_out(GeomDev* gd, Sections& in, Sections& out, Sections& work, Place place, Fill fill) {
  const GeomPlan& p = gd->plan;
  const size_t N = p.N;
  auto input = [&](auto*& dev, const auto& v) {
    const size_t bytes = sizeof(v[0]) * v.size(), at = in.add(bytes);
    place(0, at, dev);
    fill(at, v.data(), bytes);
  };
  input(gd->coords, p.coords);
  input(gd->alpha0, p.alpha0);
  input(gd->c6free, p.c6free);
  input(gd->r0, p.r0);
  input(gd->hirsh, p.hirsh);
  input(gd->scs_shifts, p.scs_shifts);
  input(gd->cfdm_shifts, p.cfdm_shifts);
  input(gd->diff_shift, p.diff_shift);
  input(gd->diff_is_zero, p.diff_is_zero);
  input(gd->place_offset, p.place_offset);
  input(gd->place_rc, p.place_rc);
  input(gd->place_cc, p.place_cc);
  gd->out_at = out.size;
  auto result = [&](auto*& dev, size_t n) { place(1, out.add(sizeof(*dev) * n), dev); };
  result(gd->alpha_iw, 21 * N);
  result(gd->molpol, 21 * 9);
  result(gd->c6_eff, N);
  result(gd->alpha_eff, N);
  result(gd->scalars, 8);
  result(gd->energy, 8);
  result(gd->info, 32);
  result(gd->rnorm2, 32);                         // squared relay residual per frequency
  result(gd->cgstate, (size_t)kNFreq * kCgState);
  gd->out_bytes = out.size - gd->out_at;
  auto scratch = [&](double*& dev, size_t n) { place(2, work.add(sizeof(double) * n), dev); };
  scratch(gd->alpha_w, 21 * N);
  scratch(gd->sgm, 21 * N);
  scratch(gd->rvdw_iso, N);
  scratch(gd->omega, N);
  scratch(gd->rvdw_eff, N);
  scratch(gd->d, p.nH);
  scratch(gd->e, p.nH);
  scratch(gd->ev, 2 * (size_t)p.nH);              // + e^2 scratch of the bisection
  gd->n_edges = -1;   // the learned-mode graph of the new geometry is built on first use
}

// Plans and uploads every geometry: one staging copy, one clearing.
int upload_geometries(mbd_ctx* ctx, int n_geom, const mbd_geom* geoms) {
  Sections in, out, work;
  auto nowhere = [](int, size_t, auto*&) {};
  auto nothing = [](size_t, const void*, size_t) {};
  for (int g = 0; g < n_geom; ++g) {
    GeomDev* gd = ctx->geoms[g].get();
    gd->status_host = build_plan(geoms[g], &gd->plan);
    if (gd->status_host == MBD_OK) lay_out(gd, in, out, work, nowhere, nothing);
  }
  if (in.size == 0) return MBD_OK;
  MBD_CUDA(ctx->inputs.reserve(in.size));
  MBD_CUDA(ctx->results.reserve(out.size + work.size));
  MBD_CUDA(ctx->in_staging.reserve(in.size));
  char* const region[3] = {ctx->inputs.as<char>(), ctx->results.as<char>(), ctx->results.as<char>() + out.size};
  char* const host = ctx->in_staging.as<char>();
  auto place = [&](int r, size_t at, auto*& dev) {
    dev = reinterpret_cast<std::remove_reference_t<decltype(dev)>>(region[r] + at);
  };
  auto fill = [&](size_t at, const void* src, size_t bytes) { std::memcpy(host + at, src, bytes); };
  const size_t in_bytes = in.size;
  ctx->out_bytes = out.size;
  in = out = Sections{};
  const size_t work_bytes = work.size;
  work = Sections{};
  for (int g = 0; g < n_geom; ++g)
    if (ctx->geoms[g]->status_host == MBD_OK) lay_out(ctx->geoms[g].get(), in, out, work, place, fill);
  MBD_CUDA(cudaMemcpyAsync(ctx->inputs.p, host, in_bytes, cudaMemcpyHostToDevice, ctx->stream));
  MBD_CUDA(cudaMemsetAsync(ctx->results.p, 0, ctx->out_bytes + work_bytes, ctx->stream));
  ctx->h2d_bytes += (double)in_bytes;
  return MBD_OK;
}

int tridiag_group_ctas(const mbd_ctx* ctx, int n) {
  const int nt = (n + kTrdTile - 1) / kTrdTile;
  const int tiles = nt * (nt + 1) / 2;
  return std::max(1, std::min(std::min(ctx->num_sms * ctx->trd_ctas_per_sm, tiles), kTridiagMaxGroup));
}

// ---- plan of the grouped tridiagonal reduction ----------------------------
// Time model of reducing one n x n matrix with a group of G CTAs, in
// microseconds per column: a fixed part (reflector, cross-CTA sums, and two
// group barriers when G > 1) plus the SYMV over the trailing triangle, whose
// average size per column is n^2/6 elements, shared by min(G, tiles) CTAs.
// Coefficients fitted to B200 runs of the kernel at n = 1500, 3000, 6000.
double trd_col_us(int n, int G) {
  const int nt = (n + kTrdTile - 1) / kTrdTile;
  const int ge = std::max(1, std::min(G, nt * (nt + 1) / 2));
  return (G == 1 ? 7.0 : 12.0) + 9.1e-5 * (double)n * (double)n / ge;
}
double trd_us(int n, int G) { return n < 2 ? 1.0 : (double)n * trd_col_us(n, G); }

struct TrdPlan {
  std::vector<std::vector<int>> bins;   // job indices per group, descending n
  std::vector<int> G;
  double makespan_us = 0.0;
};

// Partitions `ctas` co-resident CTAs into groups and the jobs (matrix sizes)
// among them to minimise the modelled makespan: for B = min(jobs, ctas),
// B/2, ..., 1 groups, longest-first assignment of the jobs at one CTA per
// group, then the spare CTAs go one at a time to the slowest group while that
// shortens it.  The best B wins.
TrdPlan plan_tridiag(const std::vector<int>& sizes, int ctas) {
  TrdPlan best;
  const int J = (int)sizes.size();
  if (J == 0 || ctas < 1) return best;
  std::vector<int> idx(J);
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return sizes[a] > sizes[b]; });
  best.makespan_us = 1e300;
  for (int B = std::min(J, ctas); B >= 1; B = (B == 1) ? 0 : std::max(1, B / 2)) {
    TrdPlan p;
    p.bins.assign(B, {});
    p.G.assign(B, 1);
    std::vector<double> load(B, 0.0);
    for (int j : idx) {
      const int b = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      p.bins[b].push_back(j);
      load[b] += trd_us(sizes[j], 1);
    }
    auto bin_time = [&](int b, int g) {
      double t = 0.0;
      for (int j : p.bins[b]) t += trd_us(sizes[j], g);
      return t;
    };
    int spare = ctas - B;
    while (spare > 0) {
      const int b = (int)(std::max_element(load.begin(), load.end()) - load.begin());
      if (p.G[b] >= kTridiagMaxGroup) break;
      const double t2 = bin_time(b, p.G[b] + 1);
      if (!(t2 < load[b])) break;
      p.G[b] += 1;
      load[b] = t2;
      --spare;
    }
    p.makespan_us = *std::max_element(load.begin(), load.end());
    if (p.makespan_us < best.makespan_us) best = p;
  }
  return best;
}

// ---- relay stages of one geometry (on its slot's stream) ------------------

// Direct FP64 relay solve: the factors of the matrices in sl.relay64 into L
// (which may be the matrices themselves), the solution into sl.rhs.
int relay_direct(mbd_ctx* ctx, GeomDev* gd, RelaySlot& sl, double* L, cudaEvent_t ev_factor, double** X_out) {
  const GeomPlan& p = gd->plan;
  cudaStream_t s = sl.stream;
  const int n = p.n;
  const size_t mstride = (size_t)n * p.ld, ystride = (size_t)n * 3;
  const int nblk = (n + kCholNB - 1) / kCholNB;
  const size_t lstride = (size_t)nblk * kCholNB * kCholNB;
  BatchMat bm{L, mstride, p.ld, n, kNFreq};
  double* Linv = sl.linv.as<double>();
  CholFlowArgs cf{};
  cf.src = sl.relay64.as<double>();
  cf.L = L;
  cf.src_stride = cf.l_stride = mstride;
  cf.src_ld = cf.ld = p.ld;
  cf.n = n;
  cf.batch = kNFreq;
  cf.linv = Linv;
  cf.linv_stride = lstride;
  cf.info = gd->info;
  cf.sync = sl.chol_sync.as<int>();
  cf.err = ctx->err_flag;
  cf.stall = ctx->test_stall_wait == kStallFactor;
  MBD_CUDA(launch_chol_flow(cf, ctx->num_sms, s));
  ctx->launches += 1;
  record_timing(ctx, ev_factor, s);
  double* Wv = sl.rhs.as<double>();
  double* Zv = Wv + kNFreq * ystride;
  double* Xv = Zv + kNFreq * ystride;
  *X_out = Xv;
  if (n <= kTrsvMaxN) {
    MBD_CUDA(launch_trsv_cluster(bm, Linv, lstride, Xv, ystride, s));
    ctx->launches += 1;
    return MBD_OK;
  }
  launch_init_rhs(Wv, ystride, n, kNFreq, s);
  for (int k0 = 0; k0 < n; k0 += kCholNB) launch_trsv_fwd_step(bm, k0, Linv, lstride, Wv, Zv, ystride, s);
  for (int k0 = (nblk - 1) * kCholNB; k0 >= 0; k0 -= kCholNB)
    launch_trsv_bwd_step(bm, k0, Linv, lstride, Zv, Xv, ystride, s);
  ctx->launches += 1 + 2 * nblk;
  return MBD_OK;
}

// Mixed relay solve of a matrix small enough for the direct FP64 solve to be
// the faster one (kMixedDirectMaxN): its factors beside the matrices, and the
// residual the gate reads.
int relay_mixed_direct(mbd_ctx* ctx, GeomDev* gd, RelaySlot& sl, cudaEvent_t ev_factor, double** X_out) {
  const GeomPlan& p = gd->plan;
  int st = relay_direct(ctx, gd, sl, sl.relay32.as<double>(), ev_factor, X_out);
  if (st != MBD_OK) return st;
  launch_relay_residual(sl.relay64.as<double>(), (size_t)p.n * p.ld, p.ld, p.n, kNFreq, *X_out, nullptr,
                        sl.rhs.as<double>(), (size_t)p.n * 3, sl.res_ws.as<double>(), gd->rnorm2, sl.stream);
  ctx->launches += 3;
  return MBD_OK;
}

// Mixed relay solve: FP32 copy factorised with 3xTF32 tcgen05 GEMMs (128-wide
// panels), FP64 iterative refinement against the FP64 matrices.  Leaves the
// refined solution X (n x 3 per frequency) at the start of slot.mixv.
int relay_mixed(mbd_ctx* ctx, GeomDev* gd, RelaySlot& sl, size_t mstride, cudaEvent_t ev_factor) {
  const GeomPlan& p = gd->plan;
  cudaStream_t s = sl.stream;
  const int n = p.n;
  const int npad = round_up(n, kMixNB);
  BatchMat32 m32{sl.relay32.as<float>(), mstride, p.ld, n, kNFreq};
  float* phi = sl.p_hi.as<float>();
  float* plo = sl.p_lo.as<float>();
  float* lhi = sl.l_hi.as<float>();
  float* llo = sl.l_lo.as<float>();
  const size_t pb = (size_t)npad * kMixNB;   // elements per matrix of the panel / Linv buffers
  Tc3Maps trsm_maps, syrk_maps;
  // panel operands/outputs cover rows [0, n) (TMA zero-fills beyond), the
  // diagonal inverses [0, npad), the output matrix is the n x n FP32 relay copy
  bool ok = make_tc3_map(&trsm_maps.a_hi, phi, n, kMixNB, kMixNB, pb, kNFreq) &&
            make_tc3_map(&trsm_maps.a_lo, plo, n, kMixNB, kMixNB, pb, kNFreq) &&
            make_tc3_map(&trsm_maps.b_hi, lhi, npad, kMixNB, kMixNB, pb, kNFreq) &&
            make_tc3_map(&trsm_maps.b_lo, llo, npad, kMixNB, kMixNB, pb, kNFreq) &&
            make_tc3_map(&trsm_maps.c, m32.A, n, n, p.ld, mstride, kNFreq);
  if (!ok) return MBD_ERR_DEVICE;
  trsm_maps.c_hi = trsm_maps.a_hi;
  trsm_maps.c_lo = trsm_maps.a_lo;
  syrk_maps.a_hi = trsm_maps.a_hi;
  syrk_maps.a_lo = trsm_maps.a_lo;
  syrk_maps.b_hi = trsm_maps.a_hi;
  syrk_maps.b_lo = trsm_maps.a_lo;
  syrk_maps.c = trsm_maps.c;
  syrk_maps.c_hi = trsm_maps.a_hi;
  syrk_maps.c_lo = trsm_maps.a_lo;
  for (int k0 = 0; k0 < n; k0 += kMixNB) {
    launch_potrf_diag_f32(m32, k0, lhi, llo, pb, gd->info, s);
    ctx->launches += 1;
    const int rows = n - k0 - kMixNB;
    if (rows <= 0) continue;
    launch_split(m32.A, mstride, p.ld, k0 + kMixNB, k0, rows, kMixNB, phi, plo, pb, kMixNB, kNFreq, s);
    const int mt = (rows + 127) / 128;
    Tc3Params tp{};
    tp.mode = TC3_STORE_SPLIT;
    tp.batch = kNFreq;
    tp.a_row0 = k0 + kMixNB;
    tp.b_row0 = k0;
    tp.m_rows = rows;
    tp.n_cols = kMixNB;
    tp.k = kMixNB;
    tp.n_tiles_n = 1;
    tp.C = m32.A;
    tp.c_bstride = mstride;
    tp.c_ld = p.ld;
    tp.c_row0 = k0 + kMixNB;
    tp.c_col0 = k0;
    tp.out_hi = phi;
    tp.out_lo = plo;
    tp.o_bstride = pb;
    tp.o_ld = kMixNB;
    tp.err = ctx->err_flag;
    launch_tc3_gemm(trsm_maps, tp, mt, s);
    Tc3Params sp = tp;
    sp.mode = TC3_SYRK_LOWER;
    sp.b_row0 = k0 + kMixNB;
    sp.n_cols = rows;
    sp.c_col0 = k0 + kMixNB;
    sp.out_hi = sp.out_lo = nullptr;
    launch_tc3_gemm(syrk_maps, sp, mt * (mt + 1) / 2, s);
    ctx->launches += 3;
  }
  record_timing(ctx, ev_factor, s);
  // FP64 iterative refinement: X = 0, R = B; repeat D = (LL^T)^-1 R, X += D, R = B - A X
  const size_t ystride = (size_t)n * 3;
  double* X = sl.mixv.as<double>();
  double* R = X + kNFreq * ystride;
  double* Z = R + kNFreq * ystride;
  double* D = Z + kNFreq * ystride;
  MBD_CUDA(cudaMemsetAsync(X, 0, sizeof(double) * kNFreq * ystride, s));
  launch_init_rhs(R, ystride, n, kNFreq, s);
  ctx->launches += 1;
  const int nblk = (n + kMixNB - 1) / kMixNB;
  for (int it = 0; it < kRefineIters; ++it) {
    launch_solve_f32(m32, lhi, llo, pb, R, Z, D, ystride, sl.solve_sync.as<int>(), ++sl.solve_epoch,
                     ctx->err_flag, s);
    launch_relay_residual(sl.relay64.as<double>(), mstride, p.ld, n, kNFreq, X, D, R, ystride,
                          sl.res_ws.as<double>(), gd->rnorm2, s);
    ctx->launches += 2 * nblk + 4;
  }
  return MBD_OK;
}

}  // namespace

// Stage timings of the last downloaded compute, from its events (some 3 us an
// interval on the host, so not on every download): relay/CFDM stages summed
// over geometries (they overlap on the slots' streams), the batch-wide stages
// and the total from batch events.
void resolve_timings(mbd_ctx* ctx) {
  if (!ctx->timed.pending) return;
  ctx->timed.pending = false;
  for (int k = 0; k < Stage::kCount; ++k) ctx->last_ms[k] = 0.0;
  auto elapsed = [](cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, a, b) == cudaSuccess) return (double)ms;
    cudaGetLastError();
    return 0.0;
  };
  const cudaEvent_t* bev = ctx->bev[ctx->timed.set];
  ctx->last_ms[Stage::kTotal] = elapsed(bev[0], bev[3]);
  ctx->last_ms[Stage::kTridiag] = elapsed(bev[1], bev[2]);
  ctx->last_band_ms = ctx->last_trace_ms = 0.0;
  ctx->last_chase_ms = ctx->last_ms[Stage::kTridiag];
  ctx->last_onestage_ms = elapsed(bev[1], bev[4]);
  ctx->last_sb2st_ms = elapsed(bev[4], bev[2]);
  ctx->last_ms[Stage::kEig] = elapsed(bev[2], bev[3]);
  for (const auto& [g, trace] : ctx->timed.geoms) {
    const cudaEvent_t* evs = ctx->events[ctx->timed.set].data() + (size_t)g * kGeomEvents;
    for (int k = 1; k + 1 < kGeomEvents; ++k) ctx->last_ms[k] += elapsed(evs[k - 1], evs[k]);
    const double last = elapsed(evs[kGeomEvents - 2], evs[kGeomEvents - 1]);
    ctx->last_ms[trace ? Stage::kEig : Stage::kTridiag] += last;
    (trace ? ctx->last_trace_ms : ctx->last_band_ms) += last;
  }
}

void drop_graphs(mbd_ctx* ctx, bool keep_first) {
  for (int m = 0; m < 3; ++m) {
    cudaGraphExec_t& g = ctx->graph[m];
    cudaGraphExec_t& prev = ctx->graph_prev[m];
    if (g && keep_first && ctx->graph_first[m]) {
      if (prev) cudaGraphExecDestroy(prev);
      prev = g;
    } else if (g) {
      cudaGraphExecDestroy(g);
    }
    g = nullptr;
    ctx->graph_first[m] = false;
    if (!keep_first && prev) {
      cudaGraphExecDestroy(prev);
      prev = nullptr;
      ctx->graph_sig[m].clear();
    }
  }
  // the next compute of each mode launches directly again (and reads back
  // the CG iterations), the one after it captures
  for (auto& gd : ctx->geoms) gd->cg_iters_seen = gd->cg_iters_seen1 = 0;
  for (int& k : ctx->mode_runs) k = 0;
}

int band_to_tridiag_single(mbd_ctx* ctx, double* Br, int n, double* d, double* e, DevBuf& scratch, cudaStream_t s) {
  const int C = (ctx->cluster_chase && ctx->test_stall_wait != kStallChase && n <= sb2st_cluster_max_n() &&
                 tuned_chase_c(ctx, n) != kChaseFlag)
                    ? sb2st_cluster_size(n, 1, ctx->num_sms, tuned_chase_c(ctx, n)) : 0;
  if (C > 0) {
    const BandJob job{Br, n, d, e};
    MBD_CUDA(scratch.reserve(bytes_of<BandJob>(1)));
    MBD_CUDA(cudaMemcpyAsync(scratch.p, &job, sizeof(job), cudaMemcpyHostToDevice, s));
    MBD_CUDA(cudaStreamSynchronize(s));   // the pageable source must outlive the copy
    MBD_CUDA(launch_sb2st_cluster(scratch.as<BandJob>(), 1, n, C, s));
    ctx->launches += 1;
    return MBD_OK;
  }
  std::vector<SweepItem> items;
  for (int i = 0; i + 3 <= n; ++i) items.push_back(SweepItem{0, i, i - 1, 0});
  const BandJob job{Br, n, d, e};
  const size_t b_job = bytes_of<BandJob>(1), b_it = bytes_of<SweepItem>(std::max<size_t>(items.size(), 1));
  const size_t b_pr = bytes_of<int>(2 * std::max<size_t>(items.size(), 1));
  MBD_CUDA(scratch.reserve(b_job + b_it + b_pr));
  char* base = scratch.as<char>();
  std::vector<char> host(b_job + b_it, 0);
  std::memcpy(host.data(), &job, sizeof(job));
  std::memcpy(host.data() + b_job, items.data(), sizeof(SweepItem) * items.size());
  MBD_CUDA(cudaMemcpyAsync(base, host.data(), host.size(), cudaMemcpyHostToDevice, s));
  MBD_CUDA(cudaStreamSynchronize(s));   // the pageable source must outlive the copy
  MBD_CUDA(launch_sb2st(reinterpret_cast<BandJob*>(base), 1, reinterpret_cast<SweepItem*>(base + b_job),
                        (int)items.size(), reinterpret_cast<int*>(base + b_job + b_it), ctx->err_flag,
                        ctx->num_sms, n, n / (2 * kBand) + 1, -1, s));
  ctx->launches += 3;
  return MBD_OK;
}

// Relay and CFDM stages of geometry gi on its slot's stream: per-atom
// frequency table, relay tensors, relay factorisation and solve (plain or
// mixed), screened polarizabilities and C6, CFDM Hamiltonian into gd->hmat.
int run_front(mbd_ctx* ctx, GeomDev* gd, int gi, int mode, bool relay_only) {
  NvtxRange nvtx("mbd_b200 enqueue geometry");
  const GeomPlan& p = gd->plan;
  RelaySlot& sl = *ctx->slots[gd->slot];
  cudaStream_t s = sl.stream;
  const int N = p.N, n = p.n;
  cudaEvent_t* ev = ctx->events[ctx->event_set].data() + (size_t)gi * kGeomEvents;
  auto mark = [&](int k) { record_timing(ctx, ev[k], s); };
  const bool mixed = mode == MBD_MODE_MIXED;
  const bool direct = mixed && mixed_direct(*gd, sl);
  const bool learned = mode == MBD_MODE_MIXED_LEARNED;
  mark(0);
  // 1. per-atom frequency table
  AtomDev ad{gd->coords, gd->alpha0, gd->c6free, gd->r0, gd->hirsh, gd->alpha_w, gd->sgm, gd->rvdw_iso};
  launch_atom_freq(ad, N, s);
  ctx->launches += 1;
  MBD_CUDA(cudaMemsetAsync(gd->info, 0, sizeof(int) * 32, s));
  mark(1);
  // 2. relay matrices (21, FP64; plus an FP32 copy in mixed mode)
  const size_t mstride = (size_t)n * p.ld;
  RelayBuildArgs rb{N, p.ld, mstride, gd->coords, gd->alpha_w, gd->sgm, gd->rvdw_iso, gd->scs_shifts,
                    (int)p.scs_shifts.size() / 3, p.beta, p.scs_eval_cut, sl.relay64.as<double>(),
                    ((mixed && !direct) || (learned && ctx->cg_fp32)) ? sl.relay32.as<float>() : nullptr};
  rb.f32_math = (mixed || learned) && ctx->f32_tensor_build;
  launch_relay_build(rb, s);
  ctx->launches += 1;
  mark(2);
  const size_t ystride = (size_t)n * 3;
  double* Xv = nullptr;
  if (direct) {
    int st = relay_mixed_direct(ctx, gd, sl, ev[3], &Xv);
    if (st != MBD_OK) return st;
  } else if (mixed) {
    int st = relay_mixed(ctx, gd, sl, mstride, ev[3]);
    if (st != MBD_OK) return st;
    Xv = sl.mixv.as<double>();
  } else if (learned) {
    // network warm start (stage 3), block-CG (stage 4)
    int st = relay_learned(ctx, gd, sl, mstride, ev[3], &Xv);
    if (st != MBD_OK) return st;
  } else {
    // 3. Cholesky of the 21 frequency matrices in place, 4. X = A^-1 [I;..;I]
    int st = relay_direct(ctx, gd, sl, sl.relay64.as<double>(), ev[3], &Xv);
    if (st != MBD_OK) return st;
  }
  EpilogueArgs ea{N, Xv, ystride, gd->alpha_iw, gd->molpol, gd->alpha0, gd->c6free, gd->r0,
                  gd->c6_eff, gd->alpha_eff, gd->omega, gd->rvdw_eff, gd->scalars};
  launch_relay_epilogue(ea, s);
  launch_relay_post(ea, ctx->weights_dev, s);
  ctx->launches += 2;
  mark(4);
  if (relay_only) {
    mark(5);
    mark(6);
    return cuda_status(cudaGetLastError());
  }
  // 5. CFDM Hamiltonian (lower blocks; the rest of the matrix is never read)
  CfdmBuildArgs cb{N, p.nsl, p.ldH, gd->coords, gd->omega, gd->alpha_eff, gd->rvdw_eff, gd->cfdm_shifts,
                   (int)p.cfdm_shifts.size() / 3, gd->diff_shift, gd->diff_is_zero, gd->place_offset,
                   gd->place_rc, gd->place_cc, (int)p.diff_is_zero.size(), p.beta, p.cfdm_cut,
                   gd->hmat};
  launch_cfdm_build(cb, s);
  ctx->launches += 1;
  mark(5);
  // 6. the energy from shifted Cholesky factors, or dense -> band (stage 1 of
  // the two-stage tridiagonalisation)
  if (gd->trace) {
    TraceArgs ta{gd->hmat, p.nH, p.ldH, p.nsl, learned ? kTraceDigitsIterative : kTraceDigits,
                 sl.relay64.as<double>(), sl.linv.as<double>(),
                 sl.trace_ws.p, gd->scalars, gd->energy, ctx->err_flag, ctx->test_stall_wait == kStallFactor};
    MBD_CUDA(launch_trace_energy(ta, ctx->num_sms, s));
    ctx->launches += trace_launches(p.nH);
  } else if (two_stage(ctx, p.nH)) {
    MBD_CUDA(launch_sy2sb(gd->hmat, p.ldH, p.nH, sl.trd_ws.as<double>(), gd->band.as<double>(),
                          ctx->num_sms, s, tuned_rows(ctx, p.nH), tuned_panel_qr(ctx, p.nH),
                          lookahead_for(ctx, sl.la)));
    ctx->launches += sy2sb_launches(p.nH);
  }
  mark(6);
  return cuda_status(cudaGetLastError());
}

namespace {

// ---- workspaces and the batch plan ----------------------------------------

size_t plain_bytes(const GeomPlan& p, size_t* relay, size_t* linv, size_t* rhs, size_t* sync) {
  const int nblk = (p.n + kCholNB - 1) / kCholNB;
  *relay = sizeof(double) * (size_t)kNFreq * p.n * p.ld;
  *linv = sizeof(double) * (size_t)kNFreq * nblk * kCholNB * kCholNB;
  *rhs = sizeof(double) * 3 * (size_t)kNFreq * p.n * 3;
  *sync = sizeof(int) * chol_flow_sync_ints(p.n, kNFreq);
  return *relay + *linv + *rhs + *sync;
}

// The trace form's factors and inverses (they take the relay's buffers, used
// up by then) and its own workspace.
size_t trace_bytes(const GeomPlan& p, size_t* factors, size_t* linv, size_t* ws) {
  const int nblk = (p.nH + kCholNB - 1) / kCholNB;
  *factors = sizeof(double) * (size_t)kTraceBatch * p.nH * p.ldH;
  *linv = sizeof(double) * (size_t)kTraceBatch * nblk * kCholNB * kCholNB;
  *ws = trace_ws_bytes(p.nH);
  return *factors + *linv + *ws;
}

// direct: the FP64 factors in the place of the FP32 copy and its panels.
size_t mixed_bytes(const GeomPlan& p, size_t* r32, size_t* pan, size_t* vec, size_t* res, size_t* sync, bool direct) {
  if (direct) {
    *r32 = sizeof(double) * (size_t)kNFreq * p.n * p.ld;
    *pan = *vec = *sync = 0;
    *res = sizeof(double) * relay_residual_ws_doubles(p.n, kNFreq);
    return *r32 + *res;
  }
  *r32 = sizeof(float) * (size_t)kNFreq * p.n * p.ld;
  *pan = sizeof(float) * (size_t)kNFreq * round_up(p.n, kMixNB) * kMixNB;
  *vec = sizeof(double) * 4 * (size_t)kNFreq * p.n * 3;
  *res = sizeof(double) * relay_residual_ws_doubles(p.n, kNFreq);
  *sync = sizeof(int) * solve_sync_ints(p.n, kNFreq);
  return *r32 + 4 * *pan + *vec + *res + *sync;
}

// Assigns the geometries to relay slots (longest first onto the least loaded
// slot, load = (3N)^3), with as many slots as fit in the device memory share.
int plan_slots(mbd_ctx* ctx, bool eigen) {
  const int ng = (int)ctx->order.size();
  int S = std::max(1, std::min(kMaxSlots, ng));
  std::vector<int> slot_of(ctx->geoms.size(), 0);
  auto deal = [&](int slots) {
    std::vector<double> load(slots, 0.0);
    for (int g : ctx->order) {
      const int s = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      slot_of[g] = s;
      load[s] += std::pow((double)ctx->geoms[g]->plan.n, 3.0);
    }
  };
  // Energies as traces: not while an eigenvalue kernel is asked for (its
  // environment switches, the stalled chase of the failure tests)
  for (auto& gd : ctx->geoms) gd->trace = false;
  if (eigen && ctx->trace_form && ctx->test_stall_wait != kStallChase)
    for (int g : ctx->order) ctx->geoms[g]->trace = ctx->geoms[g]->plan.nH <= kTraceMaxN;
  // A batch whose buffers are all there already (a program's second call of a
  // size) does not ask how much memory is free: that query goes through the
  // driver's kernel part, 0.05 to 2 ms depending on what else the host runs.
  deal(S);
  bool held = (int)ctx->slots.size() >= S;
  for (int g : ctx->order) {
    if (!held) break;
    const GeomDev& gd = *ctx->geoms[g];
    const RelaySlot& sl = *ctx->slots[slot_of[g]];
    size_t a, b, c, d;
    plain_bytes(gd.plan, &a, &b, &c, &d);
    held = a <= sl.relay64.bytes && b <= sl.linv.bytes && c <= sl.rhs.bytes && d <= sl.chol_sync.bytes;
    if (!held || !gd.trace) continue;
    trace_bytes(gd.plan, &a, &b, &c);
    held = a <= sl.relay64.bytes && b <= sl.linv.bytes && c <= sl.trace_ws.bytes;
  }
  if (!held) {
    size_t free_b = 0, total_b = 0;
    MBD_CUDA(cudaMemGetInfo(&free_b, &total_b));
    size_t own = 0;
    for (auto& s : ctx->slots) own += s->held();
    const double budget = kSlotMemoryShare * (double)(free_b + own);
    // no trace form for Hamiltonians whose factors would not fit a share of the memory
    for (int g : ctx->order) {
      size_t a, b, c;
      GeomDev& gd = *ctx->geoms[g];
      gd.trace = gd.trace && (double)trace_bytes(gd.plan, &a, &b, &c) <= 0.5 * budget;
    }
    for (; S >= 1; --S) {
      std::vector<size_t> need(S, 0);
      deal(S);
      for (int g : ctx->order) {
        const GeomPlan& p = ctx->geoms[g]->plan;
        size_t a, b, c, d, e, f, h;
        size_t bytes = plain_bytes(p, &a, &b, &c, &h) +
                       mixed_bytes(p, &d, &e, &f, &h, &a, ctx->mixed_direct && p.n <= kMixedDirectMaxN);
        // the trace form's factors past what the relay's matrices leave
        if (ctx->geoms[g]->trace) {
          plain_bytes(p, &a, &b, &c, &h);
          bytes += trace_bytes(p, &d, &e, &f);
          bytes -= std::min(a, d) + std::min(b, e);
        }
        need[slot_of[g]] = std::max(need[slot_of[g]], bytes);
      }
      double total = 0.0;
      for (size_t x : need) total += (double)x;
      if (total <= budget || S == 1) break;
    }
  }
  ctx->slots_unasked = held;
  for (int g : ctx->order) ctx->geoms[g]->slot = slot_of[g];
  while ((int)ctx->slots.size() < S) {
    std::unique_ptr<RelaySlot> sl(new RelaySlot());
    // slot 0 takes the batch's largest geometry (longest first), whose
    // stages set the batch's length: its stream runs at the device's highest
    // priority, so the block scheduler serves its kernels before the other
    // slots' (MBD_B200_PRIORITY=0: all at the default priority)
    int least = 0, greatest = 0;
    MBD_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    const int prio = (ctx->priorities && ctx->slots.empty()) ? greatest : least;
    MBD_CUDA(cudaStreamCreateWithPriority(&sl->stream, cudaStreamNonBlocking, prio));
    MBD_CUDA(cudaEventCreateWithFlags(&sl->done, cudaEventDisableTiming));
    MBD_CUDA(create_lookahead(&sl->la));
    ctx->slots.push_back(std::move(sl));
  }
  for (auto& sl : ctx->slots) sl->mixed_direct = ctx->mixed_direct;
  ctx->n_slots = S;
  return MBD_OK;
}

// The plan of the eigenvalue stages of the geometries in `list` (descending
// size): the one-stage grouped launch, the bands' chase and the eigenvalue and
// energy launches, with their device tables.
int plan_eigen(mbd_ctx* ctx, const std::vector<int>& list, EigenPlan* ep) {
  auto banded = [&](int g) { return two_stage(ctx, ctx->geoms[g]->plan.nH); };
  // one-stage tridiagonal plan for the matrices too large for the two-stage path
  std::vector<int> sizes, one_stage;
  for (int g : list)
    if (!banded(g)) {
      sizes.push_back(ctx->geoms[g]->plan.nH);
      one_stage.push_back(g);
    }
  const TrdPlan tp = plan_tridiag(sizes, ctx->num_sms * ctx->trd_ctas_per_sm);
  std::vector<TridiagJob> jobs;
  std::vector<TridiagGroup> groups;
  size_t ws_off = 0;
  int cta = 0;
  for (size_t b = 0; b < tp.bins.size(); ++b) {
    TridiagGroup gr{};
    gr.first_cta = cta;
    gr.G = tp.G[b];
    gr.job_begin = (int)jobs.size();
    gr.nmax = 1;
    for (int j : tp.bins[b]) {
      GeomDev* gd = ctx->geoms[one_stage[j]].get();
      const GeomPlan& p = gd->plan;
      jobs.push_back(TridiagJob{gd->hmat, p.nH, p.ldH, gd->d, gd->e});
      gr.nmax = std::max(gr.nmax, p.nH);
    }
    gr.job_end = (int)jobs.size();
    gr.ws_offset = ws_off;
    ws_off += (tridiag_workspace_bytes(gr.nmax, gr.G) + 255) & ~size_t(255);
    cta += gr.G;
    groups.push_back(gr);
  }
  ep->n_trd_groups = (int)groups.size();
  ep->trd_total_ctas = cta;
  MBD_CUDA(ep->tridiag_ws.reserve(ws_off));
  // eigenvalue jobs: the batched launch first, then matrices too large for it
  std::vector<EigJob> eig;
  ep->eig_single.clear();
  ep->eig_batch_max_n = 0;
  for (int pass = 0; pass < 2; ++pass)
    for (int g : list) {
      GeomDev* gd = ctx->geoms[g].get();
      const GeomPlan& p = gd->plan;
      const bool fits = p.nH <= kEigBatchMaxN;
      if (fits != (pass == 0)) continue;
      eig.push_back(EigJob{gd->d, gd->e, gd->ev, gd->scalars, gd->energy, p.nH, p.nsl});
      if (fits) ep->eig_batch_max_n = std::max(ep->eig_batch_max_n, p.nH);
      else ep->eig_single.push_back(g);
    }
  ep->n_eig_jobs = (int)eig.size();
  ep->n_eig_batch = ep->n_eig_jobs - (int)ep->eig_single.size();
  // band -> tridiagonal: one job per two-stage matrix, (job, sweep) items
  // ordered by sweep then job, each pointing at its job's previous sweep
  // (the bands that fit a cluster's shared memory first, largest first; the
  // flag-synchronised chase takes the rest, and all of them while the
  // failure-detection stall is on: its waits are the ones that can run out)
  std::vector<BandJob> bjobs, fjobs;
  // one chase kernel per batch (the two launches would run one after the
  // other): the one tuned for the batch's largest band, whose chase sets the
  // launch's length
  int big = 0;
  for (int g : list)
    if (banded(g)) big = std::max(big, ctx->geoms[g]->plan.nH);
  const bool cluster_ok = ctx->cluster_chase && ctx->test_stall_wait != kStallChase && big > 0 &&
                          big <= sb2st_cluster_max_n() && tuned_chase_c(ctx, big) != kChaseFlag;
  const int cap = cluster_ok ? sb2st_cluster_max_n() : 0;
  ep->band_max_n = ep->band_cluster_max_n = 0;
  for (int g : list) {
    GeomDev* gd = ctx->geoms[g].get();
    if (!banded(g)) continue;
    const BandJob bj{gd->band.as<double>(), gd->plan.nH, gd->d, gd->e};
    if (bj.n <= cap) {
      bjobs.push_back(bj);
      ep->band_cluster_max_n = std::max(ep->band_cluster_max_n, bj.n);
    } else {
      fjobs.push_back(bj);
      ep->band_max_n = std::max(ep->band_max_n, bj.n);
    }
  }
  std::stable_sort(bjobs.begin(), bjobs.end(), [](const BandJob& a, const BandJob& b) { return a.n > b.n; });
  ep->n_band_cluster = (int)bjobs.size();
  ep->band_cluster_C = sb2st_cluster_size(ep->band_cluster_max_n, ep->n_band_cluster, ctx->num_sms,
                                           tuned_chase_c(ctx, ep->band_cluster_max_n));
  if (ep->n_band_cluster > 0 && ep->band_cluster_C < 1) {   // no cluster fits after all
    fjobs.insert(fjobs.begin(), bjobs.begin(), bjobs.end());
    for (const BandJob& bj : bjobs) ep->band_max_n = std::max(ep->band_max_n, bj.n);
    bjobs.clear();
    ep->n_band_cluster = 0;
  }
  std::vector<SweepItem> items;
  {
    std::vector<int> last(fjobs.size(), -1);
    for (int i = 0; i + 3 <= ep->band_max_n; ++i)
      for (size_t j = 0; j < fjobs.size(); ++j) {
        if (i + 3 > fjobs[j].n) continue;
        items.push_back(SweepItem{(int)j, i, last[j], 0});
        last[j] = (int)items.size() - 1;
      }
  }
  bjobs.insert(bjobs.end(), fjobs.begin(), fjobs.end());
  ep->n_band_jobs = (int)bjobs.size();
  ep->sweeps_in_flight = 0;
  for (const BandJob& bj : fjobs) ep->sweeps_in_flight += bj.n / (2 * kBand) + 1;
  ep->n_sweep_items = (int)items.size();
  MBD_CUDA(ep->sweep_progress.reserve(2 * sizeof(int) * std::max<size_t>(items.size(), 1)));
  const size_t b_jobs = bytes_of<TridiagJob>(jobs.size());
  const size_t b_groups = bytes_of<TridiagGroup>(groups.size());
  const size_t b_eig = bytes_of<EigJob>(eig.size());
  const size_t b_bj = bytes_of<BandJob>(bjobs.size());
  const size_t b_it = bytes_of<SweepItem>(items.size());
  MBD_CUDA(ep->tables.reserve(b_jobs + b_groups + b_eig + b_bj + b_it));
  char* base = ep->tables.as<char>();
  ep->trd_jobs = reinterpret_cast<TridiagJob*>(base);
  ep->trd_groups = reinterpret_cast<TridiagGroup*>(base + b_jobs);
  ep->eig_jobs = reinterpret_cast<EigJob*>(base + b_jobs + b_groups);
  ep->band_jobs = reinterpret_cast<BandJob*>(base + b_jobs + b_groups + b_eig);
  ep->sweep_items = reinterpret_cast<SweepItem*>(base + b_jobs + b_groups + b_eig + b_bj);
  std::vector<char> host(b_jobs + b_groups + b_eig + b_bj + b_it, 0);
  std::memcpy(host.data(), jobs.data(), sizeof(TridiagJob) * jobs.size());
  std::memcpy(host.data() + b_jobs, groups.data(), sizeof(TridiagGroup) * groups.size());
  std::memcpy(host.data() + b_jobs + b_groups, eig.data(), sizeof(EigJob) * eig.size());
  std::memcpy(host.data() + b_jobs + b_groups + b_eig, bjobs.data(), sizeof(BandJob) * bjobs.size());
  std::memcpy(host.data() + b_jobs + b_groups + b_eig + b_bj, items.data(), sizeof(SweepItem) * items.size());
  if (!host.empty()) MBD_CUDA(h2d_ordered(ctx, base, host.data(), host.size()));
  ctx->h2d_bytes += (double)host.size();
  return MBD_OK;
}

// Plain-path slot buffers, per-geometry Hamiltonians, the tridiagonal plan and
// the device job tables of the uploaded batch.
// tight: memory ran out; the slots of earlier batches give theirs back and are
// planned anew (the device is idle).
int prepare_batch(mbd_ctx* ctx, bool eigen, bool tight = false) {
  drop_graphs(ctx, true);
  if (tight) {
    cudaGetLastError();
    ctx->n_slots = 0;
    ctx->slots.clear();
  }
  ctx->replan = false;
  ctx->order.clear();
  for (size_t g = 0; g < ctx->geoms.size(); ++g)
    if (ctx->geoms[g]->status_host == MBD_OK) ctx->order.push_back((int)g);
  // Tridiagonalisation path.  Measured on B200 (mixed mode, one geometry,
  // reduction + eigenvalues, one-stage vs two-stage): n = 300: 7.6 vs 3.7 ms,
  // n = 1050: 15.0 vs 14.2, n = 1500: 22.4 vs 20.9, n = 3000: 54.8 vs 47.3;
  // a batch of 8 geometries n = 270 .. 1800: step 50.3 vs 38.6 ms.  So every
  // matrix the two-stage reduction can take goes through it; larger ones
  // (n above the panel cluster's rows) take the one-stage grouped launch.
  ctx->two_stage_batch = ctx->two_stage_force != 0;
  std::stable_sort(ctx->order.begin(), ctx->order.end(),
                   [&](int a, int b) { return ctx->geoms[a]->plan.n > ctx->geoms[b]->plan.n; });
  if (eigen) {
    Sections h;
    std::vector<size_t> at;
    for (int g : ctx->order) {
      const GeomPlan& p = ctx->geoms[g]->plan;
      at.push_back(h.add(sizeof(double) * (size_t)p.nH * p.ldH));
    }
    MBD_CUDA(ctx->hmats.reserve(h.size));
    for (size_t k = 0; k < at.size(); ++k)
      ctx->geoms[ctx->order[k]]->hmat = reinterpret_cast<double*>(ctx->hmats.as<char>() + at[k]);
  }
  const size_t nev = ctx->geoms.size() * kGeomEvents;
  for (auto& set : ctx->events)
    while (set.size() < nev) {
      cudaEvent_t e;
      MBD_CUDA(cudaEventCreate(&e));
      set.push_back(e);
    }
  if (ctx->order.empty()) {
    ctx->n_slots = 0;
    return plan_eigen(ctx, {}, &ctx->eigen);
  }
  int st = plan_slots(ctx, eigen);
  if (st != MBD_OK) return st;
  // geometries whose energy comes from eigenvalues, by the two-stage reduction
  auto banded = [&](int g) {
    const GeomDev& gd = *ctx->geoms[g];
    return !gd.trace && two_stage(ctx, gd.plan.nH);
  };
  if (eigen)
    for (int g : ctx->order)
      if (banded(g))
        MBD_CUDA(ctx->geoms[g]->band.reserve(sizeof(double) * (size_t)ctx->geoms[g]->plan.nH * kBandLd));
  for (int s = 0; s < ctx->n_slots; ++s) {
    size_t relay = 0, linv = 0, rhs = 0, sync = 0, trace = 0;
    for (int g : ctx->order) {
      const GeomDev& gd = *ctx->geoms[g];
      if (gd.slot != s) continue;
      size_t a, b, c, d;
      plain_bytes(gd.plan, &a, &b, &c, &d);
      relay = std::max(relay, a);
      linv = std::max(linv, b);
      rhs = std::max(rhs, c);
      sync = std::max(sync, d);
      if (!gd.trace) continue;
      trace_bytes(gd.plan, &a, &b, &c);
      relay = std::max(relay, a);
      linv = std::max(linv, b);
      trace = std::max(trace, c);
    }
    RelaySlot& sl = *ctx->slots[s];
    MBD_CUDA(sl.relay64.reserve(relay));
    MBD_CUDA(sl.linv.reserve(linv));
    MBD_CUDA(sl.rhs.reserve(rhs));
    MBD_CUDA(sl.chol_sync.reserve(sync));
    MBD_CUDA(sl.trace_ws.reserve(trace));
    if (eigen) {
      size_t tw = 0;
      for (int g : ctx->order)
        if (ctx->geoms[g]->slot == s && banded(g))
          tw = std::max(tw, sizeof(double) * sy2sb_workspace_doubles(ctx->geoms[g]->plan.nH));
      MBD_CUDA(sl.trd_ws.reserve(tw));
    }
  }
  if (!eigen) {
    return plan_eigen(ctx, {}, &ctx->eigen);
  }
  std::vector<int> list;
  for (int g : ctx->order)
    if (!ctx->geoms[g]->trace) list.push_back(g);
  return plan_eigen(ctx, list, &ctx->eigen);
}

// Buffers only the mixed mode uses (allocated on first use).  Where the FP64
// factors of a slot's small geometries do not fit, they go the way of the
// large ones.
int reserve_mixed(mbd_ctx* ctx) {
  for (int s = 0; s < ctx->n_slots; ++s) {
    RelaySlot& sl = *ctx->slots[s];
    bool moved = false;
    auto grow = [&](DevBuf& b, size_t bytes) {
      const bool re = bytes > b.bytes;
      moved = moved || re;
      return b.reserve(bytes);
    };
    auto reserve = [&]() -> cudaError_t {
      size_t r32 = 0, pan = 0, vec = 0, res = 0, sync = 0;
      for (int g : ctx->order) {
        const GeomDev& gd = *ctx->geoms[g];
        if (gd.slot != s) continue;
        size_t a, b, c, d, e;
        mixed_bytes(gd.plan, &a, &b, &c, &d, &e, mixed_direct(gd, sl));
        r32 = std::max(r32, a);
        pan = std::max(pan, b);
        vec = std::max(vec, c);
        res = std::max(res, d);
        sync = std::max(sync, e);
      }
      cudaError_t e = grow(sl.relay32, r32);
      for (DevBuf* b : {&sl.p_hi, &sl.p_lo, &sl.l_hi, &sl.l_lo})
        if (e == cudaSuccess) e = grow(*b, pan);
      if (e == cudaSuccess) e = grow(sl.mixv, vec);
      if (e == cudaSuccess) e = grow(sl.res_ws, res);
      if (e == cudaSuccess) e = grow(sl.solve_sync, sync);
      return e;
    };
    cudaError_t e = reserve();
    if (e == cudaErrorMemoryAllocation && sl.mixed_direct) {   // stays so until the slots are planned again
      cudaGetLastError();
      sl.mixed_direct = false;
      e = reserve();
    }
    if (moved) drop_graphs(ctx, true);
    MBD_CUDA(e);
  }
  return MBD_OK;
}

// Enqueues a plan's stages behind the bands and Hamiltonians of its geometries;
// bev (or null): the batch's timing events.
int enqueue_eigen(mbd_ctx* ctx, const EigenPlan& ep, cudaStream_t s, const cudaEvent_t* bev) {
  // bands -> tridiagonal in one persistent launch; matrices too large for the
  // two-stage path in one grouped one-stage launch
  if (ep.n_trd_groups > 0) {
    MBD_CUDA(launch_tridiag_groups(ep.trd_jobs, ep.trd_groups, ep.n_trd_groups, ep.trd_total_ctas,
                                   ep.tridiag_ws.p, ctx->err_flag, s));
    ctx->launches += 2;
  }
  if (bev) record_timing(ctx, bev[4], s);
  if (ep.n_band_cluster > 0) {
    MBD_CUDA(launch_sb2st_cluster(ep.band_jobs, ep.n_band_cluster, ep.band_cluster_max_n,
                                  ep.band_cluster_C, s));
    ctx->launches += 1;
  }
  if (ep.n_band_jobs > ep.n_band_cluster) {
    MBD_CUDA(launch_sb2st(ep.band_jobs + ep.n_band_cluster, ep.n_band_jobs - ep.n_band_cluster,
                          ep.sweep_items, ep.n_sweep_items, ep.sweep_progress.as<int>(), ctx->err_flag,
                          ctx->num_sms, ep.band_max_n, ep.sweeps_in_flight, ctx->test_stall_wait == kStallChase ? 0 : -1, s));
    ctx->launches += 3;
  }
  if (bev) record_timing(ctx, bev[2], s);
  // eigenvalues and energies
  launch_eigen_batch(ep.eig_jobs, ep.n_eig_batch, ep.eig_batch_max_n, s);
  ctx->launches += ep.n_eig_batch > 0 ? 1 : 0;
  for (int g : ep.eig_single) {
    GeomDev* gd = ctx->geoms[g].get();
    launch_tridiag_eigenvalues(gd->d, gd->e, gd->plan.nH, gd->ev, s);
    ctx->launches += 2;
  }
  launch_energy_batch(ep.eig_jobs, ep.n_eig_jobs, s);
  ctx->launches += ep.n_eig_jobs > 0 ? 1 : 0;
  return cuda_status(cudaGetLastError());
}

// Lets stream s wait for everything enqueued on the slots' streams.
int join_slots(mbd_ctx* ctx, cudaStream_t s) {
  for (int k = 0; k < ctx->n_slots; ++k) {
    MBD_CUDA(cudaEventRecord(ctx->slots[k]->done, ctx->slots[k]->stream));
    MBD_CUDA(cudaStreamWaitEvent(s, ctx->slots[k]->done, 0));
  }
  return MBD_OK;
}

// The energies of `list` (descending size) from eigenvalues, after a compute:
// geometries whose trace form was refused (their Hamiltonians are whole), and
// re-runs of the residual gate (reduced to their bands by run_front already,
// unless they too were traced).  The reductions run side by side on the slots'
// streams, then one launch a stage serves all, as in the batch: 40 chains of 10
// to 88 Na atoms 65 ms one after the other, 10.5 so.
int run_tail(mbd_ctx* ctx, const std::vector<int>& list) {
  for (int g : list) {
    GeomDev* gd = ctx->geoms[g].get();
    if (!gd->trace || !two_stage(ctx, gd->plan.nH)) continue;
    MBD_CUDA(gd->band.reserve(sizeof(double) * (size_t)gd->plan.nH * kBandLd));
    MBD_CUDA(ctx->slots[gd->slot]->tail_trd_ws.reserve(sizeof(double) * sy2sb_workspace_doubles(gd->plan.nH)));
  }
  int st = plan_eigen(ctx, list, &ctx->tail);
  if (st != MBD_OK) return st;
  for (int g : list) {
    GeomDev* gd = ctx->geoms[g].get();
    const GeomPlan& p = gd->plan;
    if (!gd->trace || !two_stage(ctx, p.nH)) continue;
    RelaySlot& sl = *ctx->slots[gd->slot];
    MBD_CUDA(launch_sy2sb(gd->hmat, p.ldH, p.nH, sl.tail_trd_ws.as<double>(), gd->band.as<double>(), ctx->num_sms,
                          sl.stream, tuned_rows(ctx, p.nH), tuned_panel_qr(ctx, p.nH), lookahead_for(ctx, sl.la)));
    ctx->launches += sy2sb_launches(p.nH);
  }
  st = join_slots(ctx, ctx->stream);
  if (st != MBD_OK) return st;
  return enqueue_eigen(ctx, ctx->tail, ctx->stream, nullptr);
}

// Enqueues the whole batch (relay stages on the slots' streams, then the
// batch-wide eigen stages on the context stream).  Stream-capture safe: no
// allocation, no host-side copies, and the mixed solve's progress flags are
// cleared and its epochs restarted on every run.
int enqueue_batch(mbd_ctx* ctx, int mode) {
  cudaStream_t s = ctx->stream;
  const cudaEvent_t* bev = ctx->bev[ctx->event_set];
  ctx->launches = 0;
  MBD_CUDA(cudaMemsetAsync(ctx->err_flag, 0, sizeof(int), s));
  record_timing(ctx, bev[0], s);
  if (ctx->order.empty()) {
    for (int k = 1; k < 5; ++k) record_timing(ctx, bev[k], s);
    return cuda_status(cudaGetLastError());
  }
  // relay and CFDM stages, geometries spread over the slots' streams
  MBD_CUDA(cudaEventRecord(ctx->fork_ev, s));
  for (int k = 0; k < ctx->n_slots; ++k) {
    RelaySlot& sl = *ctx->slots[k];
    MBD_CUDA(cudaStreamWaitEvent(sl.stream, ctx->fork_ev, 0));
    if (mode == MBD_MODE_MIXED && sl.solve_sync.p) {
      MBD_CUDA(cudaMemsetAsync(sl.solve_sync.p, 0, sl.solve_sync.bytes, sl.stream));
      sl.solve_epoch = 0;
    }
  }
  for (int g : ctx->order) {
    int st = run_front(ctx, ctx->geoms[g].get(), g, mode);
    if (st != MBD_OK) return st;
  }
  int st = join_slots(ctx, s);
  if (st != MBD_OK) return st;
  record_timing(ctx, bev[1], s);
  st = enqueue_eigen(ctx, ctx->eigen, s, bev);
  if (st != MBD_OK) return st;
  record_timing(ctx, bev[3], s);
  return cuda_status(cudaGetLastError());
}

// Captures enqueue_batch into a graph for `mode`; false when capture is not
// possible (the caller then enqueues directly).  first: the batch's first
// compute in the mode (the full CG schedule); its graph updates the one kept
// from an earlier batch when the launch sequences match (same kernels and
// dependencies: cudaGraphExecUpdate then rewrites only the launch arguments,
// far cheaper than instantiating), else it is instantiated.
bool capture_batch(mbd_ctx* ctx, int mode, bool first) {
  NvtxRange nvtx(first ? "mbd_b200 capture first compute" : "mbd_b200 capture");
  cudaGraph_t graph = nullptr;
  if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  ctx->capturing = true;
  const int st = enqueue_batch(ctx, mode);
  ctx->capturing = false;
  const cudaError_t ec = cudaStreamEndCapture(ctx->stream, &graph);
  cudaGraphExec_t exec = nullptr;
  bool ok = st == MBD_OK && ec == cudaSuccess && graph;
  if (ok && first && ctx->graph_prev[mode]) {
    cudaGraphExecUpdateResultInfo info{};
    const cudaError_t eu = cudaGraphExecUpdate(ctx->graph_prev[mode], graph, &info);
    ctx->graph_update_result = (int)info.result;
    ctx->graph_update_node = -1;
    cudaGraphNodeType nt;
    if (info.errorNode && cudaGraphNodeGetType(info.errorNode, &nt) == cudaSuccess) ctx->graph_update_node = (int)nt;
    if (eu == cudaSuccess) {
      exec = ctx->graph_prev[mode];
      ctx->graph_updates += 1;
    } else {
      cudaGetLastError();
      cudaGraphExecDestroy(ctx->graph_prev[mode]);
    }
    ctx->graph_prev[mode] = nullptr;
  }
  if (ok && !exec)
    ok = cudaGraphInstantiate(&exec, graph, ctx->priorities ? cudaGraphInstantiateFlagUseNodePriority : 0) ==
         cudaSuccess;
  if (graph) cudaGraphDestroy(graph);
  if (!ok) {
    if (exec) cudaGraphExecDestroy(exec);
    cudaGetLastError();
    return false;
  }
  ctx->graph[mode] = exec;
  ctx->graph_events[mode] = ctx->event_set;
  ctx->graph_first[mode] = first;
  ctx->graph_launches[mode] = ctx->launches;
  return true;
}

// What fixes a batch's launch sequence in `mode`, as far as the host knows
// it before enqueueing: the geometries' sizes, image counts, slots and
// reduction paths.  A first compute is captured only when this matches the
// batch whose graph is kept (or the batch before it), so batches of changing
// shape keep launching kernel by kernel instead of instantiating every time.
std::vector<long long> batch_signature(const mbd_ctx* ctx, int mode) {
  std::vector<long long> sig{mode, ctx->n_slots, (long long)ctx->order.size(), ctx->two_stage_batch ? 1 : 0};
  for (int g : ctx->order) {
    const GeomDev& gd = *ctx->geoms[g];
    const GeomPlan& p = gd.plan;
    sig.insert(sig.end(), {p.N, p.nsl, p.nH, gd.slot, (long long)p.scs_shifts.size(),
                           (long long)p.cfdm_shifts.size(), (long long)p.diff_shift.size(),
                           gd.trace ? 2 : (two_stage(ctx, p.nH) ? 1 : 0)});
  }
  return sig;
}

}  // namespace
}  // namespace mbd

using namespace mbd;

extern "C" {

int mbd_rsscs_create(mbd_ctx** out, int device) {
  if (!out) return MBD_ERR_ARG;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return MBD_ERR_DEVICE;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return MBD_ERR_DEVICE;
  if (prop.major != 10) return MBD_ERR_DEVICE;   // sm_100a only
  if (!prop.cooperativeLaunch) return MBD_ERR_DEVICE;
  std::unique_ptr<mbd_ctx> ctx(new mbd_ctx());
  ctx->device = device;
  MBD_CUDA(cudaSetDevice(device));
  ctx->num_sms = prop.multiProcessorCount;
  MBD_CUDA(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
  for (auto& set : ctx->bev)
    for (auto& e : set) MBD_CUDA(cudaEventCreate(&e));
  MBD_CUDA(cudaEventCreateWithFlags(&ctx->fork_ev, cudaEventDisableTiming));
  MBD_CUDA(create_lookahead(&ctx->la_ctx));
  {
    const char* ng = std::getenv("MBD_B200_NO_GRAPHS");
    ctx->use_graphs = !(ng && ng[0] && ng[0] != '0');
    const char* gu = std::getenv("MBD_B200_GRAPH_UPDATE");
    ctx->graph_update = gu && gu[0] == '1';
    // the band -> tridiagonal chase of size classes the autotuner has not
    // timed: flag-synchronised (measured faster at every size on B200);
    // MBD_B200_CLUSTER_CHASE=1 makes it the cluster-resident one, =0 rules
    // the cluster-resident chase out even where the autotuner picks it
    // the learned mode's block-CG runs its matrix passes on an FP32 copy of
    // the relay matrices in two phases with an FP64 restart between them
    // (measured on B200 for the 2000-atom cluster: relay solve 15.7 ms
    // against 17.4 ms for the one-phase FP64 passes) wherever the copy (50 %
    // more relay memory) fits in half the free device memory;
    // MBD_B200_CG_FP32=1 always, =0 never
    const char* cf = std::getenv("MBD_B200_CG_FP32");
    ctx->cg_fp32_mode = (cf && cf[0] == '1') ? 1 : ((cf && cf[0] == '0') ? 0 : -1);
    const char* cc = std::getenv("MBD_B200_CLUSTER_CHASE");
    ctx->cluster_chase = !(cc && cc[0] == '0');
    if (cc && cc[0] == '1')
      for (TuneChoice& t : ctx->tune) t.chase_c = 0;
    const char* pq = std::getenv("MBD_B200_PANEL_QR");
    ctx->panel_qr_default = (pq && std::strcmp(pq, "tsqr") == 0) ? 1 : 0;
    // the dense -> band reduction's look-ahead: each panel's QR beside the
    // previous panel's trailing update (MBD_B200_LOOKAHEAD=0: one stream)
    const char* la = std::getenv("MBD_B200_LOOKAHEAD");
    ctx->lookahead = !(la && la[0] == '0');
    // the mixed mode's FP64 factors of small relay matrices
    // (MBD_B200_MIXED_DIRECT=0: 3xTF32 factors and refinement at every size)
    const char* md = std::getenv("MBD_B200_MIXED_DIRECT");
    ctx->mixed_direct = !(md && md[0] == '0');
    // stream priorities (the largest geometry's slot, the look-ahead QR),
    // kept by captured graphs (MBD_B200_PRIORITY=0: default priority everywhere)
    const char* pr = std::getenv("MBD_B200_PRIORITY");
    ctx->priorities = !(pr && pr[0] == '0');
  }
  MBD_CUDA(init_device_constants());
  MBD_CUDA(init_cholflow_attributes());
  MBD_CUDA(init_trsv_attributes());
  MBD_CUDA(init_eigvec_attributes());
  MBD_CUDA(init_cg_attributes());
  MBD_CUDA(init_eigval_attributes());
  MBD_CUDA(init_tc3_attributes());
  MBD_CUDA(init_mixed_attributes());
  MBD_CUDA(init_sy2sb_attributes());
  {
    // reduction path (prepare_batch): MBD_B200_TWO_STAGE=0 forces the
    // one-stage path; otherwise two-stage wherever it applies
    const char* ts = std::getenv("MBD_B200_TWO_STAGE");
    ctx->two_stage_max_n = sy2sb_max_n();
    ctx->two_stage_force = (ts && ts[0] == '1') ? 1 : ((ts && ts[0] == '0') ? 0 : -1);
    // MBD_B200_TRACE=0: every energy from eigenvalues; a switch that picks
    // one of their kernels asks for them too
    const char* tf = std::getenv("MBD_B200_TRACE");
    ctx->trace_form = tf ? tf[0] != '0'
                         : !(ts || std::getenv("MBD_B200_CLUSTER_CHASE") || std::getenv("MBD_B200_PANEL_QR"));
  }
  MBD_CUDA(init_sb2st_attributes());
  ctx->trd_ctas_per_sm = std::max(1, tridiag_max_ctas_per_sm());
  MBD_CUDA(ctx->misc.reserve(4096));
  char* m = ctx->misc.as<char>();
  ctx->weights_dev = reinterpret_cast<double*>(m);
  ctx->err_flag = reinterpret_cast<int*>(m + 256);
  ctx->job_dev = reinterpret_cast<TridiagJob*>(m + 512);
  ctx->omega_dev = reinterpret_cast<double*>(m + 1024);
  ctx->loss_dev = reinterpret_cast<double*>(m + 1280);
  MBD_CUDA(h2d_ordered(ctx.get(), ctx->omega_dev, kCasimirOmega, sizeof(double) * kNFreq));
  MBD_CUDA(h2d_ordered(ctx.get(), ctx->weights_dev, kCasimirWeight, sizeof(double) * kNFreq));
  MBD_CUDA(zero_ordered(ctx.get(), ctx->err_flag, sizeof(int)));
  *out = ctx.release();
  return MBD_OK;
}

void mbd_rsscs_destroy(mbd_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  cudaDeviceSynchronize();
  for (auto& set : ctx->events)
    for (auto e : set) cudaEventDestroy(e);
  drop_graphs(ctx);
  for (auto& set : ctx->bev)
    for (auto e : set)
      if (e) cudaEventDestroy(e);
  if (ctx->fork_ev) cudaEventDestroy(ctx->fork_ev);
  if (ctx->la_ctx.ready) cudaEventDestroy(ctx->la_ctx.ready);
  if (ctx->la_ctx.done) cudaEventDestroy(ctx->la_ctx.done);
  if (ctx->la_ctx.aux) cudaStreamDestroy(ctx->la_ctx.aux);
  ctx->geoms.clear();
  ctx->slots.clear();
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
}

int mbd_rsscs_upload(mbd_ctx* ctx, int n_geom, const mbd_geom* geoms) {
  NvtxRange nvtx("mbd_b200 upload");
  if (!ctx || n_geom < 1 || !geoms) return MBD_ERR_ARG;
  return upload_batch(ctx, n_geom, geoms, true);
}

}  // extern "C"

namespace mbd {

// Uploads a batch; eigen = false prepares only the relay stages (training
// batches: no CFDM Hamiltonians, no eigen plan, not computable).
int upload_batch(mbd_ctx* ctx, int n_geom, const mbd_geom* geoms, bool eigen) {
  MBD_CUDA(cudaSetDevice(ctx->device));
  // buffers of the previous batch may still be in use by its kernels
  MBD_CUDA(cudaDeviceSynchronize());
  ctx->have_batch = false;
  ctx->h2d_bytes = 0;
  while ((int)ctx->geoms.size() < n_geom) ctx->geoms.emplace_back(new GeomDev());
  ctx->geoms.resize(n_geom);
  if (!eigen) resolve_timings(ctx);   // a training batch's stages record the same events
  int st = upload_geometries(ctx, n_geom, geoms);
  if (st != MBD_OK) return st;
  int first = MBD_OK;
  for (int g = 0; g < n_geom && first == MBD_OK; ++g) first = ctx->geoms[g]->status_host;
  const bool had_slots = !ctx->slots.empty();
  st = prepare_batch(ctx, eigen);
  if (st == MBD_ERR_OUT_OF_MEMORY && had_slots) st = prepare_batch(ctx, eigen, true);
  if (st != MBD_OK) return st;
  ctx->have_batch = eigen;
  return first;
}

}  // namespace mbd

extern "C" {

int mbd_rsscs_compute(mbd_ctx* ctx, int mode) {
  static const char* const kRange[3] = {"mbd_b200 compute plain", "mbd_b200 compute mixed",
                                        "mbd_b200 compute mixed_learned"};
  NvtxRange nvtx(mode >= 0 && mode < 3 ? kRange[mode] : "mbd_b200 compute");
  if (!ctx || !ctx->have_batch) return MBD_ERR_ARG;
  if (mode != MBD_MODE_PLAIN_FP64 && mode != MBD_MODE_MIXED && mode != MBD_MODE_MIXED_LEARNED) return MBD_ERR_ARG;
  if (mode == MBD_MODE_MIXED_LEARNED && ctx->use_net && !ctx->have_net) return MBD_ERR_NO_NETWORK;
  MBD_CUDA(cudaSetDevice(ctx->device));
  if (ctx->replan) {   // an option that the plan depends on has changed since the upload
    MBD_CUDA(cudaDeviceSynchronize());
    int st = prepare_batch(ctx, true);
    if (st != MBD_OK) return st;
  }
  auto reserve = [&] {
    return mode == MBD_MODE_MIXED ? reserve_mixed(ctx) : (mode == MBD_MODE_MIXED_LEARNED ? reserve_learned(ctx) : MBD_OK);
  };
  int st = reserve();
  if (st == MBD_ERR_OUT_OF_MEMORY && ctx->slots_unasked) {   // fewer slots, for what memory there is
    MBD_CUDA(cudaDeviceSynchronize());
    st = prepare_batch(ctx, true, true);
    if (st == MBD_OK) st = reserve();
  }
  if (st != MBD_OK) return st;
  ctx->last_mode = mode;
  // From the second compute of a batch in a mode on, capture the batch into a
  // CUDA graph once and replay it; a batch computed once (energy_batch, an
  // upload per call) is launched directly and does not pay for the capture.
  //   A context that uploads batch after batch of one shape (a trajectory,
  // the same structures re-submitted) runs each batch's first compute as a
  // graph as well: captured, then written into the graph kept from the
  // previous batch with cudaGraphExecUpdate, which costs a fraction of the
  // gaps between kernels launched one by one.  The learned mode's graph of
  // a first compute runs the full CG schedule; its second compute captures
  // the iterations seen instead and the first graph is kept for the next
  // batch.
  const bool repeat = ctx->mode_runs[mode]++ > 0;
  // this compute's timing events: a replay's are those of its capture; else
  // the set that the last compute did not use
  const int events = ctx->use_graphs && repeat && ctx->graph[mode] ? ctx->graph_events[mode] : 1 - ctx->event_set;
  if (ctx->timed.pending && ctx->timed.set == events) resolve_timings(ctx);
  ctx->event_set = events;
  if (ctx->use_graphs && repeat && ctx->graph[mode] && ctx->graph_first[mode] &&
      mode == MBD_MODE_MIXED_LEARNED) {
    if (ctx->graph_prev[mode]) cudaGraphExecDestroy(ctx->graph_prev[mode]);
    ctx->graph_prev[mode] = ctx->graph[mode];
    ctx->graph[mode] = nullptr;
    ctx->graph_first[mode] = false;
  }
  if (ctx->use_graphs && !ctx->graph[mode]) {
    if (repeat) {
      if (!capture_batch(ctx, mode, false)) ctx->use_graphs = false;
    } else if (ctx->graph_update) {
      std::vector<long long> sig = batch_signature(ctx, mode);
      const bool same = sig == ctx->graph_sig[mode] || sig == ctx->last_sig[mode];
      ctx->last_sig[mode] = sig;
      // a failed capture launches directly below
      if (same && capture_batch(ctx, mode, true)) ctx->graph_sig[mode] = std::move(sig);
    }
  }
  if (ctx->use_graphs && ctx->graph[mode]) {
    ctx->launches = ctx->graph_launches[mode];
    ctx->graph_kind = repeat ? 1 : 2;
    return cuda_status(cudaGraphLaunch(ctx->graph[mode], ctx->stream));
  }
  ctx->graph_kind = 0;
  return enqueue_batch(ctx, mode);
}

int mbd_rsscs_download(mbd_ctx* ctx, mbd_result* out) {
  NvtxRange nvtx("mbd_b200 download");
  if (!ctx || !ctx->have_batch || !out) return MBD_ERR_ARG;
  MBD_CUDA(cudaSetDevice(ctx->device));
  // Every geometry's results in one copy into page-locked memory, queued
  // behind the batch on the context stream, one synchronisation.
  constexpr size_t kHead = 256;   // the error flag
  MBD_CUDA(ctx->staging.reserve(kHead + ctx->out_bytes));
  char* hs = ctx->staging.as<char>();
  const char* dev_out = ctx->results.as<char>();
  MBD_CUDA(cudaMemcpyAsync(hs, ctx->err_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  ctx->d2h_bytes = sizeof(int);
  auto fetch = [&](size_t at, size_t bytes) -> cudaError_t {
    ctx->d2h_bytes += (double)bytes;
    return cudaMemcpyAsync(hs + kHead + at, dev_out + at, bytes, cudaMemcpyDeviceToHost, ctx->stream);
  };
  if (!ctx->order.empty()) MBD_CUDA(fetch(0, ctx->out_bytes));
  MBD_CUDA(cudaStreamSynchronize(ctx->stream));
  int err = 0;
  std::memcpy(&err, hs, sizeof(int));
  // what a re-run of some geometries left in the place of their staged
  // results; its device waits may have run out
  auto fetch_again = [&](const std::vector<int>& list) -> int {
    MBD_CUDA(cudaMemcpyAsync(hs, ctx->err_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    for (int g : list) MBD_CUDA(fetch(ctx->geoms[g]->out_at, ctx->geoms[g]->out_bytes));
    MBD_CUDA(cudaStreamSynchronize(ctx->stream));
    std::memcpy(&err, hs, sizeof(int));
    return MBD_OK;
  };
  auto host = [&](const void* dev) -> const char* { return hs + kHead + (static_cast<const char*>(dev) - dev_out); };
  // the stage timings are read from their events when someone asks for them
  ctx->timed.pending = true;
  ctx->timed.set = ctx->event_set;
  ctx->timed.geoms.clear();
  for (int g : ctx->order) ctx->timed.geoms.emplace_back(g, ctx->geoms[g]->trace);
  for (size_t g = 0; g < ctx->geoms.size(); ++g) {
    mbd_result& r = out[g];
    r.status = ctx->geoms[g]->status_host;
    for (int k = 0; k < 3; ++k) r.supercell[k] = ctx->geoms[g]->plan.sl[k];
    r.refine_iters = 0;
    for (int k = 0; k < 3; ++k) r.err_est[k] = 0.0;
  }
  // residual gate of the mixed relay solves; a miss re-runs the geometry with
  // the direct FP64 solve (the plain path) before its results are read
  std::vector<int> rerun, tail;
  if (ctx->last_mode != MBD_MODE_PLAIN_FP64)
    for (int g : ctx->order) {
      GeomDev* gd = ctx->geoms[g].get();
      mbd_result& r = out[g];
      const double* rn = reinterpret_cast<const double*>(host(gd->rnorm2));
      double worst = 0.0;
      for (int f = 0; f < 21; ++f) {
        const double v = std::sqrt(rn[f] / (3.0 * gd->plan.N));
        worst = std::isfinite(v) ? std::max(worst, v) : std::numeric_limits<double>::infinity();
      }
      r.err_est[0] = r.err_est[1] = r.err_est[2] = worst;
      r.refine_iters = mixed_direct(*gd, *ctx->slots[gd->slot]) ? 1 : kRefineIters;
      if (ctx->last_mode == MBD_MODE_MIXED_LEARNED) {
        const double* cs = reinterpret_cast<const double*>(host(gd->cgstate));
        double most = 0.0, most1 = 0.0;
        bool indefinite = false;
        for (int f = 0; f < kNFreq; ++f) {
          most = std::max(most, cs[(size_t)f * kCgState + 1]);
          if (ctx->cg_fp32) most1 = std::max(most1, cs[(size_t)f * kCgState + kCgPhase1Iters]);
          indefinite = indefinite || cs[(size_t)f * kCgState + kCgIndefinite] != 0.0;
        }
        // iterations of both phases (the mixed-precision form) or of the one
        r.refine_iters = (int)(most1 + most);
        // a negative curvature proves the relay matrix indefinite: the direct
        // solve below then reports it (MBD_ERR_RELAY_NOT_SPD)
        if (indefinite) worst = std::numeric_limits<double>::infinity();
        const bool ok = worst <= ctx->residual_gate;
        gd->cg_iters_seen = ok ? (int)most : 0;
        gd->cg_iters_seen1 = ok ? (int)most1 : 0;
      }
      if (worst <= ctx->residual_gate) continue;
      rerun.push_back(g);
      r.refine_iters = -1;
    }
  if (!rerun.empty()) {
    for (int g : rerun) {
      int st = run_front(ctx, ctx->geoms[g].get(), g, MBD_MODE_PLAIN_FP64);
      if (st != MBD_OK) return st;
      if (!ctx->geoms[g]->trace) tail.push_back(g);
    }
    int st = join_slots(ctx, ctx->stream);
    if (st == MBD_OK) st = fetch_again(rerun);
    if (st != MBD_OK) return st;
  }
  // refused trace forms (an imaginary mode, or a Hamiltonian too near one): the
  // eigenvalues, where the relay gave a Hamiltonian at all
  for (int g : ctx->order) {
    const GeomDev* gd = ctx->geoms[g].get();
    if (!gd->trace || reinterpret_cast<const double*>(host(gd->energy))[3] == kTraceOk) continue;
    const int* info = reinterpret_cast<const int*>(host(gd->info));
    const bool relay_ok = std::all_of(info, info + 21, [](int i) { return i == 0; });
    if (relay_ok && reinterpret_cast<const double*>(host(gd->scalars))[2] == 0.0) tail.push_back(g);
  }
  if (!tail.empty() && err == 0) {
    std::stable_sort(tail.begin(), tail.end(),
                     [&](int a, int b) { return ctx->geoms[a]->plan.n > ctx->geoms[b]->plan.n; });
    int st = run_tail(ctx, tail);
    if (st == MBD_OK) st = fetch_again(tail);
    if (st != MBD_OK) return st;
  }
  int first = MBD_OK;
  for (size_t g = 0; g < ctx->geoms.size(); ++g) {
    GeomDev* gd = ctx->geoms[g].get();
    mbd_result& r = out[g];
    if (gd->status_host != MBD_OK) {
      r.energy_Ha = std::nan("");
      r.c6_mol = std::nan("");
      r.nimag = 0;
      if (first == MBD_OK) first = r.status;
      continue;
    }
    const int N = gd->plan.N;
    const double* aiw = reinterpret_cast<const double*>(host(gd->alpha_iw));
    const double* molpol = reinterpret_cast<const double*>(host(gd->molpol));
    const double* scal = reinterpret_cast<const double*>(host(gd->scalars));
    const double* en = reinterpret_cast<const double*>(host(gd->energy));
    const int* info = reinterpret_cast<const int*>(host(gd->info));
    int status = err;   // first: what unfinished factors say of the matrix means nothing
    for (int f = 0; f < 21; ++f)
      if (status == MBD_OK && info[f] != 0) status = MBD_ERR_RELAY_NOT_SPD;
    if (status == MBD_OK && scal[2] > 0.0) status = MBD_ERR_NONPOSITIVE_ALPHA;
    r.status = status;
    r.c6_mol = scal[0];
    if (status == MBD_OK) {
      r.energy_Ha = en[0];
      r.nimag = (int)en[2];
    } else {
      r.energy_Ha = std::nan("");
      r.nimag = 0;
    }
    // per-atom results back in the caller's atom order
    const std::vector<int>& pm = gd->plan.perm;
    if (r.alpha_iw)   // column-major alpha(f, i): element (f, i) at f + 21 i
      for (int q = 0; q < N; ++q)
        for (int f = 0; f < 21; ++f) r.alpha_iw[f + 21 * (size_t)pm[q]] = aiw[(size_t)f * N + q];
    if (r.alpha_eff) {
      const double* a = reinterpret_cast<const double*>(host(gd->alpha_eff));
      for (int q = 0; q < N; ++q) r.alpha_eff[pm[q]] = a[q];
    }
    if (r.c6_eff) {
      const double* c = reinterpret_cast<const double*>(host(gd->c6_eff));
      for (int q = 0; q < N; ++q) r.c6_eff[pm[q]] = c[q];
    }
    if (r.molpol_eig)
      for (int f = 0; f < 21; ++f) {
        double e3[3];
        sym3_eigenvalues_upper(molpol + 9 * f, e3);
        for (int k = 0; k < 3; ++k) r.molpol_eig[f + 21 * k] = e3[k];
      }
    if (status != MBD_OK && first == MBD_OK) first = status;
  }
  return first;
}

int mbd_rsscs_energy_batch(mbd_ctx* ctx, int n_geom, const mbd_geom* geoms, int mode, mbd_result* out) {
  if (!ctx || !geoms || !out || n_geom < 1) return MBD_ERR_ARG;
  int st = mbd_rsscs_upload(ctx, n_geom, geoms);
  if (st == MBD_ERR_OUT_OF_MEMORY || st == MBD_ERR_DEVICE || st == MBD_ERR_ARG) {
    for (int g = 0; g < n_geom; ++g) out[g].status = st;
    return st;
  }
  int cs = mbd_rsscs_compute(ctx, mode);
  if (cs != MBD_OK) {
    for (int g = 0; g < n_geom; ++g) out[g].status = cs;
    return cs;
  }
  return mbd_rsscs_download(ctx, out);
}

int mbd_rsscs_energy(mbd_ctx* ctx, const mbd_geom* geom, int mode, mbd_result* out) {
  if (!out) return MBD_ERR_ARG;
  int st = mbd_rsscs_energy_batch(ctx, 1, geom, mode, out);
  out->status = out->status ? out->status : st;
  return out->status;
}

int mbd_rsscs_eigvalsh(mbd_ctx* ctx, const double* H, int n, int ld, double* w) {
  NvtxRange nvtx("mbd_b200 eigvalsh");
  if (!ctx || !H || !w || n < 1 || ld < n) return MBD_ERR_ARG;
  MBD_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  const int ldp = round_up(n, 32);
  MBD_CUDA(ctx->eig_a.reserve(sizeof(double) * (size_t)n * ldp));
  MBD_CUDA(ctx->eig_vec.reserve(sizeof(double) * 4 * (size_t)n));   // d, e, ev (2n)
  double* A = ctx->eig_a.as<double>();
  double* d = ctx->eig_vec.as<double>();
  double* e = d + n;
  double* ev = e + n;
  MBD_CUDA(cudaMemcpy2DAsync(A, sizeof(double) * ldp, H, sizeof(double) * ld, sizeof(double) * n, n,
                             cudaMemcpyHostToDevice, s));
  MBD_CUDA(cudaMemsetAsync(ctx->err_flag, 0, sizeof(int), s));
  if (n <= ctx->two_stage_max_n) {
    const size_t wsd = sy2sb_workspace_doubles(n);
    MBD_CUDA(ctx->eig_ws.reserve(sizeof(double) * (wsd + (size_t)n * kBandLd)));
    double* ws = ctx->eig_ws.as<double>();
    double* band = ws + wsd;
    MBD_CUDA(launch_sy2sb(A, ldp, n, ws, band, ctx->num_sms, s, tuned_rows(ctx, n), tuned_panel_qr(ctx, n),
                          lookahead_for(ctx, ctx->la_ctx)));
    int st = band_to_tridiag_single(ctx, band, n, d, e, ctx->fb_ws, s);
    if (st != MBD_OK) return st;
  } else {
    const int G = tridiag_group_ctas(ctx, n);
    const size_t wsb = tridiag_workspace_bytes(n, G);
    MBD_CUDA(ctx->eig_ws.reserve(wsb));
    TridiagJob job{A, n, ldp, d, e};
    MBD_CUDA(cudaMemcpyAsync(ctx->job_dev, &job, sizeof(job), cudaMemcpyHostToDevice, s));
    MBD_CUDA(launch_tridiag(ctx->job_dev, 1, 1, G, ctx->eig_ws.p, wsb, n, ctx->err_flag, s));
  }
  launch_tridiag_eigenvalues(d, e, n, ev, s);
  MBD_CUDA(cudaMemcpyAsync(w, ev, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
  MBD_CUDA(cudaStreamSynchronize(s));
  int err = 0;
  MBD_CUDA(cudaMemcpy(&err, ctx->err_flag, sizeof(int), cudaMemcpyDeviceToHost));
  return err ? err : MBD_OK;
}

int mbd_rsscs_eigh(mbd_ctx* ctx, const double* H, int n, int ld, double* w, double* Z, int ldz) {
  NvtxRange nvtx("mbd_b200 eigh");
  if (!ctx || !H || !w || !Z || n < 1 || ld < n || ldz < n) return MBD_ERR_ARG;
  MBD_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  constexpr int NBW = kWyNB;   // reflectors per compact-WY block of the back-transformation
  const size_t nwy = (n + NBW - 1) / NBW;
  const size_t ldp = round_up(n, 32);
  const size_t nn = (size_t)n * ldp;
  const int G = tridiag_group_ctas(ctx, n);
  const size_t wsb = tridiag_workspace_bytes(n, G);
  MBD_CUDA(ctx->eig_ws.reserve(wsb));
  // A, V (reflectors), X, X2 (vectors), Gram; scratch; W, W2 (NBW x n);
  // S, T (NBW x NBW a block); tau, d, e, ev (2n); the deviation word
  size_t off = 0;
  std::vector<size_t> o;
  auto add = [&](size_t doubles) { o.push_back(off); off += (doubles + 31) & ~size_t(31); };
  add(nn);
  add(nn);
  add(nn);
  add(nn);
  add((size_t)n * n);
  add(eigh_scratch_doubles(n));
  add((size_t)NBW * n);
  add((size_t)NBW * n);
  add(nwy * NBW * NBW);
  add(nwy * NBW * NBW);
  add(n);
  add(n);
  add(n);
  add(2 * (size_t)n);
  add(4);
  MBD_CUDA(ctx->eigh_buf.reserve(sizeof(double) * off));
  double* base = ctx->eigh_buf.as<double>();
  double* A = base + o[0];
  double* V = base + o[1];
  double* X = base + o[2];
  double* X2 = base + o[3];
  double* Gm = base + o[4];
  double* scratch = base + o[5];
  double* W = base + o[6];
  double* W2 = base + o[7];
  double* Sg = base + o[8];
  double* Tb = base + o[9];
  double* tau = base + o[10];
  double* d = base + o[11];
  double* e = base + o[12];
  double* ev = base + o[13];
  unsigned long long* dev = reinterpret_cast<unsigned long long*>(base + o[14]);
  MBD_CUDA(cudaMemcpy2DAsync(A, sizeof(double) * ldp, H, sizeof(double) * ld, sizeof(double) * n, n,
                             cudaMemcpyHostToDevice, s));
  MBD_CUDA(cudaMemsetAsync(V, 0, sizeof(double) * nn, s));
  MBD_CUDA(cudaMemsetAsync(tau, 0, sizeof(double) * n, s));
  MBD_CUDA(cudaMemsetAsync(e, 0, sizeof(double) * n, s));
  MBD_CUDA(cudaMemsetAsync(ctx->err_flag, 0, sizeof(int), s));
  // A = Q T Q^T, the reflectors of Q kept
  TridiagJob job{A, n, (int)ldp, d, e};
  job.vsave = V;
  job.tau = tau;
  job.ldv = ldp;
  MBD_CUDA(cudaMemcpyAsync(ctx->job_dev, &job, sizeof(job), cudaMemcpyHostToDevice, s));
  MBD_CUDA(launch_tridiag(ctx->job_dev, 1, 1, G, ctx->eig_ws.p, wsb, n, ctx->err_flag, s));
  launch_tridiag_eigenvalues(d, e, n, ev, s);
  double ends[2];
  MBD_CUDA(cudaMemcpyAsync(&ends[0], ev, sizeof(double), cudaMemcpyDeviceToHost, s));
  MBD_CUDA(cudaMemcpyAsync(&ends[1], ev + n - 1, sizeof(double), cudaMemcpyDeviceToHost, s));
  MBD_CUDA(cudaStreamSynchronize(s));
  int err = 0;
  MBD_CUDA(cudaMemcpy(&err, ctx->err_flag, sizeof(int), cudaMemcpyDeviceToHost));
  if (err) return err;
  const double tnorm = std::max(std::fabs(ends[0]), std::fabs(ends[1]));
  // the tridiagonal's eigenvectors, then Newton-Schulz to orthonormality
  launch_tri_vectors(d, e, ev, n, tnorm, X, ldp, scratch, s);
  // a step maps a deviation dv of X^T X from I to about 3/4 dv^2: after one
  // from dv <= ns_one the product is not formed again to check it
  const double ns_tol = 1e-15 * std::max(10.0, 4.0 * std::sqrt((double)n));
  const double ns_one = std::sqrt(ns_tol);
  for (int step = 0; step < 4; ++step) {
    dgemm_rm(true, false, n, n, n, 1.0, X, ldp, X, ldp, 0.0, Gm, n, s);   // X^T X
    MBD_CUDA(cudaMemsetAsync(dev, 0, sizeof(unsigned long long), s));
    launch_ns_prepare(Gm, n, dev, s);
    unsigned long long bits = 0;
    MBD_CUDA(cudaMemcpyAsync(&bits, dev, sizeof(bits), cudaMemcpyDeviceToHost, s));
    MBD_CUDA(cudaStreamSynchronize(s));
    double dv;
    std::memcpy(&dv, &bits, sizeof(dv));
    if (!(dv > ns_tol)) break;
    dgemm_rm(false, false, n, n, n, 1.0, X, ldp, Gm, n, 0.0, X2, ldp, s);   // X (3I - X^T X) / 2
    std::swap(X, X2);
    if (dv <= ns_one) break;
  }
  // X <- Q X: blocks of reflectors c0 .. c0 + kb - 1 (rows c0 + 1 .. n - 1),
  // the last block first; V^T of a block is row-major (kb x m) at
  // V + c0 * ldp + c0 + 1
  const int nr = n - 1;
  for (int c0 = 0; c0 < nr; c0 += NBW) {   // S = V^T V of every block, then every T
    const int kb = std::min(NBW, nr - c0);
    const double* Vt = V + (size_t)c0 * ldp + c0 + 1;
    dgemm_rm(false, true, kb, kb, n - c0 - 1, 1.0, Vt, ldp, Vt, ldp, 0.0, Sg + (size_t)(c0 / NBW) * NBW * NBW, NBW, s);
  }
  launch_wy_t(Sg, tau, nr, Tb, s);
  for (int c0 = nr > 0 ? ((nr - 1) / NBW) * NBW : -1; c0 >= 0; c0 -= NBW) {
    const int kb = std::min(NBW, nr - c0);
    const int m = n - c0 - 1;
    const double* Vt = V + (size_t)c0 * ldp + c0 + 1;
    double* Xs = X + (size_t)(c0 + 1) * ldp;
    dgemm_rm(false, false, kb, n, m, 1.0, Vt, ldp, Xs, ldp, 0.0, W, n, s);       // W = V^T X
    dgemm_rm(false, false, kb, n, kb, 1.0, Tb + (size_t)(c0 / NBW) * NBW * NBW, NBW, W, n, 0.0, W2, n, s);   // W2 = T W
    dgemm_rm(true, false, m, n, kb, -1.0, Vt, ldp, W2, n, 1.0, Xs, ldp, s);      // X -= V W2
  }
  MBD_CUDA(cudaGetLastError());
  MBD_CUDA(cudaMemcpyAsync(w, ev, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
  MBD_CUDA(cudaMemcpy2DAsync(Z, sizeof(double) * ldz, X, sizeof(double) * ldp, sizeof(double) * n, n,
                             cudaMemcpyDeviceToHost, s));
  MBD_CUDA(cudaStreamSynchronize(s));
  return MBD_OK;
}

int mbd_rsscs_element_z(const char* symbol) { return element_z(symbol); }

int mbd_rsscs_frequency_grid(double* omega, double* weight, int n) {
  if (!omega || n < kNFreq) return MBD_ERR_ARG;
  for (int f = 0; f < kNFreq; ++f) {
    omega[f] = kCasimirOmega[f];
    if (weight) weight[f] = kCasimirWeight[f];
  }
  return MBD_OK;
}

int mbd_rsscs_vdw_params(int z, double* alpha0, double* c6, double* r0) {
  VdwParam v;
  if (!vdw_param(z, &v)) return MBD_ERR_UNKNOWN_ELEMENT;
  if (alpha0) *alpha0 = v.alpha0;
  if (c6) *c6 = v.c6;
  if (r0) *r0 = v.r0;
  return MBD_OK;
}

const char* mbd_rsscs_strerror(int code) {
  switch (code) {
    case MBD_OK: return "ok";
    case MBD_ERR_ARG: return "invalid argument";
    case MBD_ERR_UNKNOWN_ELEMENT: return "VdW parameters not defined for atom";
    case MBD_ERR_RELAY_NOT_SPD: return "relay matrix is not positive definite (Cholesky failed)";
    case MBD_ERR_NONPOSITIVE_ALPHA: return "screened polarizability alpha_eff <= 0; R_vdW_eff undefined";
    case MBD_ERR_EIGENSOLVER: return "diagonalization of CFDM hamiltonian failed";
    case MBD_ERR_DEVICE: return "CUDA device error or no sm_100 device";
    case MBD_ERR_TIMEOUT: return "a bounded device-side wait timed out";
    case MBD_ERR_OUT_OF_MEMORY: return "out of device memory";
    case MBD_ERR_REFINEMENT: return "mixed-precision refinement missed the residual gate; FP64 fallback used";
    case MBD_ERR_NOT_BUILT: return "mode not available in this build";
    case MBD_ERR_TOO_LARGE: return "matrix larger than the fixed scratch of the allocation-free entry point";
    case MBD_ERR_NO_NETWORK: return "MIXED_LEARNED needs a trained or loaded network (or the network switched off)";
    default: return "unknown error";
  }
}

int mbd_rsscs_last_stats(mbd_ctx* ctx, double* out, int n) {
  if (!ctx || !out || n < 3) return MBD_ERR_ARG;
  out[0] = ctx->launches;
  out[1] = ctx->h2d_bytes;
  out[2] = ctx->d2h_bytes;
  if (n >= 4) out[3] = ctx->graph_kind;
  if (n >= 5) {
    double edges = 0.0;
    for (const auto& gd : ctx->geoms) edges += std::max(gd->n_edges, 0);
    out[4] = edges;
  }
  if (n >= 6) out[5] = ctx->graph_updates;
  if (n >= 7) out[6] = ctx->graph_update_result;
  if (n >= 8) out[7] = ctx->graph_update_node;
  return MBD_OK;
}

void* mbd_rsscs_stream(mbd_ctx* ctx) { return ctx ? (void*)ctx->stream : nullptr; }

int mbd_rsscs_set_option(mbd_ctx* ctx, int option, double value) {
  if (!ctx) return MBD_ERR_ARG;
  switch (option) {
    case MBD_OPT_RESIDUAL_GATE:
      if (!(value >= 0.0)) return MBD_ERR_ARG;
      ctx->residual_gate = value;
      return MBD_OK;
    case MBD_OPT_WAIT_LIMIT_S: {
      if (!(value > 0.0 && value <= 60.0)) return MBD_ERR_ARG;
      // clock64 counts SM cycles: seconds x the device's maximum SM clock
      int khz = 0;
      MBD_CUDA(cudaSetDevice(ctx->device));
      MBD_CUDA(cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, ctx->device));
      const long long cycles = std::max(1LL, (long long)(value * 1e3 * (double)khz));
      MBD_CUDA(cudaDeviceSynchronize());   // no launch of this device reads the limit meanwhile
      MBD_CUDA(set_wait_limit_sb2st(cycles));
      MBD_CUDA(set_wait_limit_tridiag(cycles));
      MBD_CUDA(set_wait_limit_mixed(cycles));
      MBD_CUDA(set_wait_limit_tc3(cycles));
      MBD_CUDA(set_wait_limit_cholflow(cycles));
      ctx->wait_limit_s = value;
      return MBD_OK;
    }
    case MBD_OPT_FP32_TENSOR_BUILD: {
      const int on = value != 0.0;
      if (on != ctx->f32_tensor_build) {
        MBD_CUDA(cudaSetDevice(ctx->device));
        MBD_CUDA(cudaDeviceSynchronize());
        drop_graphs(ctx);   // the captured launches carry the old setting
      }
      ctx->f32_tensor_build = on;
      return MBD_OK;
    }
    case MBD_OPT_TEST_STALL_WAIT: {
      const int on = value == kStallFactor ? kStallFactor : (value != 0.0 ? kStallChase : 0);
      if (on != ctx->test_stall_wait) {
        MBD_CUDA(cudaSetDevice(ctx->device));
        MBD_CUDA(cudaDeviceSynchronize());
        drop_graphs(ctx);   // the captured launches carry the old setting
        // the chase's stall needs the eigenvalue path (plan_slots)
        if (on == kStallChase || ctx->test_stall_wait == kStallChase) ctx->replan = true;
      }
      ctx->test_stall_wait = on;
      return MBD_OK;
    }
    default:
      return MBD_ERR_ARG;
  }
}

int mbd_rsscs_autotune(mbd_ctx* ctx, int max_n) {
  NvtxRange nvtx("mbd_b200 autotune");
  if (!ctx || max_n < 1) return MBD_ERR_ARG;
  MBD_CUDA(cudaSetDevice(ctx->device));
  MBD_CUDA(cudaDeviceSynchronize());
  return autotune(ctx, max_n);
}

int mbd_rsscs_tuning(mbd_ctx* ctx, double* out, int n) {
  if (!ctx || !out || n < 8 * kTuneClasses) return MBD_ERR_ARG;
  int filled = 0;
  for (int k = 0; k < kTuneClasses; ++k) {
    const TuneChoice& t = ctx->tune[k];
    double* o = out + 8 * k;
    o[0] = t.n;
    o[1] = t.rows;
    o[2] = t.chase_c;
    o[3] = t.sy2sb_ms;
    o[4] = t.chase_ms;
    o[5] = t.panel_qr;
    o[6] = t.flag_chase_ms;
    o[7] = t.cluster_chase_ms;
    if (t.n > 0) filled = k + 1;
  }
  return filled;
}

int mbd_rsscs_get_option(mbd_ctx* ctx, int option, double* value) {
  if (!ctx || !value) return MBD_ERR_ARG;
  switch (option) {
    case MBD_OPT_RESIDUAL_GATE: *value = ctx->residual_gate; return MBD_OK;
    case MBD_OPT_WAIT_LIMIT_S: *value = ctx->wait_limit_s; return MBD_OK;
    case MBD_OPT_TEST_STALL_WAIT: *value = ctx->test_stall_wait; return MBD_OK;
    case MBD_OPT_FP32_TENSOR_BUILD: *value = ctx->f32_tensor_build; return MBD_OK;
    default: return MBD_ERR_ARG;
  }
}

int mbd_rsscs_last_timings(mbd_ctx* ctx, double* ms, int n) {
  if (!ctx || !ms || n < Stage::kCount) return MBD_ERR_ARG;
  resolve_timings(ctx);
  for (int k = 0; k < Stage::kCount; ++k) ms[k] = ctx->last_ms[k];
  if (n >= Stage::kCount + 2) {
    ms[Stage::kCount] = ctx->last_band_ms;        // dense -> band, summed over geometries
    ms[Stage::kCount + 1] = ctx->last_chase_ms;   // band (or dense, one-stage) -> tridiagonal, batch-wide
  }
  if (n >= Stage::kCount + 4) {
    ms[Stage::kCount + 2] = ctx->last_onestage_ms;   // the grouped one-stage launch alone
    ms[Stage::kCount + 3] = ctx->last_sb2st_ms;      // the bulge-chasing launch alone
  }
  if (n >= Stage::kCount + 5) ms[Stage::kCount + 4] = ctx->last_trace_ms;   // the trace forms, summed over geometries
  return MBD_OK;
}

}  // extern "C"
