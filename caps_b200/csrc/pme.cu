// Host side of PME: plans, twiddle tables and line blocking per grid, and the spread / transform / solve / gather
// launch sequence.
#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <cmath>
#include <cstring>
#include <functional>
#include <vector>

#include "engine.h"
#include "pme.cuh"

namespace capsb {

namespace {

// The passes of a length: as few radices as can be (at most 16 each), and among those with odd ones first, whose first
// pass writes shared memory at an odd stride. Grid lengths are 2^a 3^b 5^c 7^d.
void plan_radices(int n, int* rad, int& nst) {
  static const int radices[] = {16, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  std::vector<int> best(size_t(n) + 1, kMaxRadices + 1), from(size_t(n) + 1, 0);
  best[1] = 0;
  for (int m = 2; m <= n; ++m)
    for (int r : radices)
      if (m % r == 0 && best[size_t(m / r)] + 1 < best[size_t(m)]) best[size_t(m)] = best[size_t(m / r)] + 1, from[size_t(m)] = r;
  if (best[size_t(n)] > kMaxRadices) throw ModelError(CAPS_GPU_EINVAL, "PME grid length " + std::to_string(n) + " cannot be factored for the line FFT");
  nst = 0;
  for (int m = n; m > 1; m /= from[size_t(m)]) rad[nst++] = from[size_t(m)];
  std::sort(rad, rad + nst, [](int a, int b) { return (a & 1) != (b & 1) ? (a & 1) > (b & 1) : a < b; });
}

int log2_floor(int v) {
  int s = 0;
  while ((2 << s) <= v) ++s;
  return s;
}

}  // namespace

// The active path's spread grid, zero when it is made: every transform of it leaves it zero (k_fft_x_fwd).
void Engine::ensure_grid() {
  const size_t want = size_t(pk_[0]) * pk_[1] * pk_[2];
  if (mixed_ && (!d_gridq_.p || d_gridq_.n < want)) {
    d_gridq_.alloc(want);
    d_gridq_.zero(stream_);
  } else if (!mixed_ && (!d_grid_.p || d_grid_.n < want)) {
    d_grid_.alloc(want);
    d_grid_.zero(stream_);
  }
}

template <class R>
void Engine::pme_setup(PmePath<R>& P) {
  using T = typename Cpx<R>::T;
  const size_t half = size_t(ph1_) * pk_[1] * pk_[2];
  P.h.alloc(half);
  P.gr.alloc(size_t(pk_[0]) * pk_[1] * pk_[2]);
  P.gt.alloc(half);
  P.wt.alloc(6 * half);
  ensure_grid();
  for (int d = 0; d < 3; ++d) {
    const int nn = pk_[d];
    std::vector<T> tw(static_cast<size_t>(nn));
    for (int k = 0; k < nn; ++k) {
      const double ang = 2 * kPi * k / nn;
      tw[size_t(k)] = T{R(std::cos(ang)), R(-std::sin(ang))};
    }
    P.tw[d].upload(tw, stream_);
    FftPlan<R>& pl = P.plan[d];
    pl.n = nn;
    plan_radices(nn, pl.rad, pl.nst);
    int ns = 1;
    for (int p = 0; p < pl.nst; ++p) {
      pl.nb[p] = nn / pl.rad[p];
      pl.ns[p] = ns;
      pl.m_nb[p] = div_magic(unsigned(pl.nb[p]));
      pl.m_ns[p] = div_magic(unsigned(ns));
      ns *= pl.rad[p];
    }
    pl.tw = P.tw[d].p;
  }
  // Lines per block. x: pairs of contiguous lines, enough blocks for four per SM, two buffers within 40 KB of shared
  // memory. y, z: consecutive a per block (a power of two of them) so that each row read is 128 bytes.
  const int cap = int(40 * 1024 / (2 * sizeof(T)));
  const int nlx = (pk_[1] * pk_[2] + 1) / 2;
  P.lines[0] = std::max(1, std::min({cap / pk_[0], 16, (nlx + 4 * dev_sms_ - 1) / (4 * dev_sms_)}));
  const int la = int(128 / sizeof(T));
  P.lines[1] = std::max(1, std::min({la, cap / pk_[1], ph1_}));
  P.lines[2] = std::max(1, std::min({la, cap / pk_[2], ph1_}));
  if (tuning_pinned_)
    for (int d = 0; d < 3; ++d) P.lines[d] = pinned_lines_[d];
  else
    pme_tune(P);
  for (int d = 0; d < 3; ++d) P.k[d] = pk_[d];
  green_valid_ = false;
  CK(cudaStreamSynchronize(stream_));
}

void Engine::tuning(int32_t v[7]) const {
  const int* l = pme_lines();
  const int32_t t[7] = {batch_, pair_cut_, pme_cap_, bonded_cap_, l[0], l[1], l[2]};
  std::memcpy(v, t, sizeof t);
}

void Engine::pin_tuning(const int32_t v[7]) {
  if (v[0] < 1 || v[0] > kBatch || v[1] < 0 || v[2] < 0 || v[3] < 0 || v[4] < 1 || v[5] < 1 || v[6] < 1)
    throw ModelError(CAPS_GPU_EINVAL, "tuning values out of range");
  batch_ = geom_.batch = v[0];
  pair_cut_ = v[1];
  pme_cap_ = v[2];
  bonded_cap_ = v[3];
  for (int d = 0; d < 3; ++d) pinned_lines_[d] = v[4 + d];
  auto& lines = mixed_ ? pf_.lines : pd_.lines;
  for (int d = 0; d < 3; ++d) lines[d] = v[4 + d];
  tuning_pinned_ = true;
  shapes_tuned_ = true;
  list_valid_ = false;
  drop_run_state();
}

// The mixed path transforms in FP32 (pf_), the FP64 path in FP64 (pd_); each path is set up for the current grid on
// first use.
void Engine::ensure_pme() {
  if (!pme_ || pk_[0] == 0) return;
  auto same = [&](const int* k) { return k[0] == pk_[0] && k[1] == pk_[1] && k[2] == pk_[2]; };
  if (mixed_) {
    if (!same(pf_.k)) pme_setup(pf_);
    ensure_grid();
  } else if (!same(pd_.k)) {
    pme_setup(pd_);
  } else {
    ensure_grid();
  }
}

// The five line-transform passes of one PME evaluation (forward x, y; z with the solve; inverse y, x).
template <class R>
void Engine::fft_passes(PmePath<R>& P, bool ener, bool vir) {
  using T = typename Cpx<R>::T;
  PmeArgs A{pk_[0], pk_[1], pk_[2], ph1_, dcell_, nullptr, d_q_.p, n_};
  // shared memory: twiddle table + two line buffers (y, z: 1 << ly, lz lines, the powers of two in P.lines)
  const int ly = log2_floor(P.lines[1]), lz = log2_floor(P.lines[2]);
  const size_t sx = (size_t(P.lines[0]) * 2 * (pk_[0] | 1) + pk_[0]) * sizeof(T), sy = ((size_t(2) << ly) + 1) * pk_[1] * sizeof(T),
               sz = ((size_t(2) << lz) + 1) * pk_[2] * sizeof(T);
  const int nlx = (pk_[1] * pk_[2] + 1) / 2;
  // the kernels stride over their line groups: a grid cap (the tuner's pme_cap_, 0 for none) leaves SM slots to the
  // pair kernel that runs beside them
  auto capped = [&](int g) { return pme_cap_ > 0 ? std::min(g, pme_cap_) : g; };
  auto allow = [&](auto* kernel, size_t smem) {   // long lines need more than the default 48 KB
    if (smem > 48 * 1024) CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    return kernel;
  };
  const int gx = capped(blocks_for(size_t(nlx), P.lines[0]));
  launch_k(allow(k_fft_x_fwd<R>, sx), gx, kFftThreads, sx, stream_, A, mixed_ ? nullptr : d_grid_.p, mixed_ ? d_gridq_.p : nullptr, P.h.p, P.plan[0], P.lines[0]);
  const int gy = capped(blocks_for(size_t(ph1_), 1 << ly) * pk_[2]);
  launch_k(allow(k_fft_y<R, false>, sy), gy, kFftThreads, sy, stream_, A, P.h.p, P.plan[1], ly);
  const int gz = capped(blocks_for(size_t(ph1_), 1 << lz) * pk_[1]);
  EnergySink en{d_efix_.p, d_edbl_.p};
  auto* solve = ener ? (vir ? k_fft_z_solve<R, true, true> : k_fft_z_solve<R, true, false>) : (vir ? k_fft_z_solve<R, false, true> : k_fft_z_solve<R, false, false>);
  launch_k(allow(solve, sz), gz, kFftThreads, sz, stream_, A, P.h.p, P.gt.p, P.wt.p, P.plan[2], lz, en, mixed_);
  launch_k(allow(k_fft_y<R, true>, sy), gy, kFftThreads, sy, stream_, A, P.h.p, P.plan[1], ly);
  launch_k(allow(k_fft_x_inv<R>, sx), gx, kFftThreads, sx, stream_, A, P.h.p, P.gr.p, P.plan[0], P.lines[0]);
}

// Autotuner for the line transforms: every block shape that fits (x: 1-8 pairs of lines per block; y, z: 1-16 consecutive
// a per block) is timed on this grid (the transforms' time does not depend on the values), and the fastest kept. Results are
// cached per grid, precision and SM count for the process.
template <class R>
void Engine::pme_tune(PmePath<R>& P) {
  using T = typename Cpx<R>::T;
  static std::mutex mu;
  static std::map<std::array<int, 5>, std::array<int, 3>> cache;
  const std::array<int, 5> key{pk_[0], pk_[1], pk_[2], int(sizeof(R)), dev_sms_};
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      P.lines[0] = it->second[0], P.lines[1] = it->second[1], P.lines[2] = it->second[2];
      return;
    }
  }
  if (before_timing_) before_timing_();
  const size_t half = size_t(ph1_) * pk_[1] * pk_[2];
  CK(cudaMemsetAsync(P.gt.p, 0, half * sizeof(R), stream_));
  CK(cudaMemsetAsync(P.wt.p, 0, 6 * half * sizeof(R), stream_));
  CK(cudaMemsetAsync(P.h.p, 0, half * sizeof(T), stream_));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  const size_t smax = 48 * 1024;
  float best = 1e30f;
  std::array<int, 3> pick{P.lines[0], P.lines[1], P.lines[2]};
  for (int lx : {1, 2, 4, 8})
    for (int la : {1, 2, 4, 8, 16}) {
      if (((size_t(lx) * 2) * (pk_[0] | 1) + pk_[0]) * sizeof(T) > smax) continue;
      if ((size_t(la) * 2 + 1) * std::max(pk_[1], pk_[2]) * sizeof(T) > smax) continue;
      P.lines[0] = lx, P.lines[1] = la, P.lines[2] = la;
      fft_passes(P, false, false);   // warm
      CK(cudaEventRecord(e0, stream_));
      for (int rep = 0; rep < 3; ++rep) fft_passes(P, false, false);
      CK(cudaEventRecord(e1, stream_));
      CK(cudaEventSynchronize(e1));
      float ms = 0;
      CK(cudaEventElapsedTime(&ms, e0, e1));
      if (ms < best) best = ms, pick = {lx, la, la};
    }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  P.lines[0] = pick[0], P.lines[1] = pick[1], P.lines[2] = pick[2];
  std::lock_guard<std::mutex> lock(mu);
  cache[key] = pick;
}

template <class R>
void Engine::pme_run(PmePath<R>& P, const double* d_x, bool ener, bool vir) {
  using T = typename Cpx<R>::T;
  PmeArgs A{pk_[0], pk_[1], pk_[2], ph1_, dcell_, d_x, d_q_.p, n_};
  if (!green_valid_ || std::memcmp(green_cell_, cell_h_, sizeof cell_h_) != 0) {
    const size_t half = size_t(ph1_) * pk_[1] * pk_[2];
    launch_k(k_pme_green<R>, blocks_for(half, 256), 256, 0, stream_, A, d_bsp_[0].p, d_bsp_[1].p, d_bsp_[2].p, beta_, kCoulomb, P.gt.p, P.wt.p);
    std::memcpy(green_cell_, cell_h_, sizeof cell_h_);
    green_valid_ = true;
  }
  // enough blocks of the spread for two per SM where atoms are few
  const int pb = std::clamp(n_ / (2 * dev_sms_), 8, kPmeAtoms), nb = blocks_for(size_t(n_), pb);
  const bool big = grid_needs_64(pk_[0], pk_[1], pk_[2]);
#define SPREAD(P_)                                                                            \
  do {                                                                                        \
    auto* kernel = mixed_ ? (big ? k_spread<float, P_, size_t> : k_spread<float, P_, int>)    \
                          : (big ? k_spread<double, P_, size_t> : k_spread<double, P_, int>); \
    launch_k(kernel, nb, kPmeThreads, 0, stream_, A, pb, d_grid_.p, d_gridq_.p);              \
  } while (0)
  switch (order_) {
    case 3: SPREAD(3); break;
    case 4: SPREAD(4); break;
    case 5: SPREAD(5); break;
    case 6: SPREAD(6); break;
    case 7: SPREAD(7); break;
    default: SPREAD(8); break;
  }
#undef SPREAD
  fft_passes(P, ener, vir);
  const ForceSink<float> Ff{d_F_.p, d_F_.p + n_, d_F_.p + 2 * size_t(n_), d_counters_.p + kCntErr};
  const ForceSink<double> Fd{d_Fd_.p, d_Fd_.p + n_, d_Fd_.p + 2 * size_t(n_)};
  // four lanes per atom up to four waves of threads, 75,000 atoms: there the gather waits for its loads, beyond it the
  // splines' repetition costs more
  const bool split = n_ <= 512 * dev_sms_;
  const int gb = blocks_for(size_t(n_) * (split ? 4 : 1), 128);
#define GATHER(P_)                                                                            \
  do {                                                                                        \
    if (mixed_) launch_k(split ? k_gather<float, R, P_, 4> : k_gather<float, R, P_, 1>, gb, 128, 0, stream_, A, P.gr.p, Ff);   \
    else launch_k(split ? k_gather<double, R, P_, 4> : k_gather<double, R, P_, 1>, gb, 128, 0, stream_, A, P.gr.p, Fd);       \
  } while (0)
  switch (order_) {
    case 3: GATHER(3); break;
    case 4: GATHER(4); break;
    case 5: GATHER(5); break;
    case 6: GATHER(6); break;
    case 7: GATHER(7); break;
    default: GATHER(8); break;
  }
#undef GATHER
  CK(cudaGetLastError());
}

void Engine::pme_forces(const double* d_x, bool ener, bool vir) {
  if (mixed_) pme_run(pf_, d_x, ener, vir);
  else pme_run(pd_, d_x, ener, vir);
}


template void Engine::pme_setup<double>(PmePath<double>&);
template void Engine::pme_run<double>(PmePath<double>&, const double*, bool, bool);
template void Engine::fft_passes<double>(PmePath<double>&, bool, bool);
template void Engine::pme_tune<double>(PmePath<double>&);
template void Engine::pme_setup<float>(PmePath<float>&);
template void Engine::pme_run<float>(PmePath<float>&, const double*, bool, bool);
template void Engine::fft_passes<float>(PmePath<float>&, bool, bool);
template void Engine::pme_tune<float>(PmePath<float>&);

}  // namespace capsb
