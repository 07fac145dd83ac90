// K-LIST: everything between a step's drift and its pair kernel in one launch: the gated list build (bin, scan, scatter,
// column sort, super-clusters, search), the packed positions and the gated dynamic prune.
//
// A step without a build or a prune (about three in four at 500 K) only packs: the blocks stride over the slots and
// leave. On the others the work is cut into units, numbered in the order of the stages, and every block takes the next
// number from a device counter; a unit whose stage reads another's results waits until that stage's finished-unit count is
// complete. A block only ever waits for lower numbers, and those are held by blocks that run (a block takes a number when
// it is running and finishes it before it takes another), so the wait ends whatever else is on the GPU and however few of
// the blocks are resident; no launch has to hold the whole grid at once.
//
// What this is bound by: latency. As six launches (bin, scatter, sort, search, pack, prune, each returning at once unless
// flagged) a plain step of the 32,000-atom melt spent 28 us between its drift and its pair kernel, 594 atoms 11 us: the
// launches, not their work.
#pragma once
#include "pair.cuh"

namespace capsb {

enum ListStage { kStBin = 0, kStScan, kStScatter, kStSort, kStSuper, kStSearch, kStPack, kStNum };
static_assert(kStNum == kCntNum - kCntStage, "a counter per stage");

struct ListArgs {
  int n, nslots;
  const double* x;
  DevCell cell;
  ListGeom g;
  ListBufs b;
  const uint32_t* excl_off;
  const uint32_t* excl_list;
  int force;      // 1: build whatever the flag says
  int pack_only;  // 1: a frozen list (no build, no prune)
  int polls;      // of a wait before it gives up (Engine::list_polls_)
  // pack
  const double* q;
  const int* type;
  int pad_type;
  float4* xq;     // FP32 path: per slot the position relative to the super-cluster's origin, and the charge
  double4* xqd;   // FP64 path: the wrapped absolute position, and the charge
  int* tslot;
  double* x0;     // positions of the last build
  double* xp;     // positions of the last prune
  long long* fs;  // slot-order sums (FP32 path; FP64: fsd), cleared for the pair kernel
  double* fsd;
  // prune
  double rprune2;
};

// Packs slot s. A padding slot sits far from everything, each of its super-cluster at its own place.
template <bool DBL>
__device__ __forceinline__ void pack_slot(const ListArgs& L, int s, int nsc, bool built) {
  if (s >= L.nslots) return;
  for (int r = 0; r < 3; ++r) {
    if (DBL) L.fsd[size_t(r) * L.nslots + s] = 0;
    else L.fs[size_t(r) * L.nslots + s] = 0;
  }
  if (s >= 64 * nsc) return;
  const int a = L.b.perm[s];
  if (a < 0) {
    if (DBL) L.xqd[s] = make_double4(1e7, 1e7, 1e7 + 16.0 * (s & 63), 0.0);
    else L.xq[s] = make_float4(0.f, 0.f, kPadFar, 0.f);
    L.tslot[s] = L.pad_type;
    return;
  }
  const int o0 = L.b.ioff[3 * a], o1 = L.b.ioff[3 * a + 1], o2 = L.b.ioff[3 * a + 2];
  double p[3];
  for (int r = 0; r < 3; ++r) {
    const double xr = L.x[3 * a + r];
    if (built) L.x0[3 * a + r] = xr;
    p[r] = xr + (L.cell.h[r][0] * o0 + L.cell.h[r][1] * o1 + L.cell.h[r][2] * o2);
  }
  if (DBL) {
    L.xqd[s] = make_double4(p[0], p[1], p[2], L.q[a]);
  } else {
    const int sc = s >> 6;
    L.xq[s] = make_float4(float(p[0] - L.b.sc_org[3 * sc]), float(p[1] - L.b.sc_org[3 * sc + 1]), float(p[2] - L.b.sc_org[3 * sc + 2]), float(L.q[a]));
  }
  L.tslot[s] = L.type[a];
}

struct PruneShared {   // per warp: its entries' j atoms (x, y, z, (|x|^2 - r_prune^2) / 2) from the work item's origin
  float4 xj[kListThreads / 32][kBatch * 8];
  float4 sh[kListThreads / 32][kBatch];   // the entries' shifts, and their j clusters
};

// Dynamic pruning (as core/src/nbnxm.cpp:328-363 does on the CPU), a warp per work item w: each entry's mask is rewritten
// to the (i cluster, j half) pairs with at least one atom pair inside r_prune = r_c + b at the present positions; the pair
// kernels read that mask. The j halves are the cluster's lower-x and upper-x four atoms (the cluster split orders its
// atoms along x), so a half mask drops the far half of a j cluster that reaches an i cluster with its near half only.
// Pruned again once an atom has moved b/2 since the last prune, so no pair inside r_c is lost.
//
// Bound by issue. A lane keeps its eight i atoms in registers and tests them against its two j atoms of an entry without a
// branch, as x_i x_j - |x_i|^2 / 2 > (|x_j|^2 - r^2) / 2, positions from the work item's origin (three multiply-adds and a
// compare per pair; the squares a millionth low and r^2 0.02 Å^2 high, so that rounding only ever keeps a pair); one
// reduction over the warp per entry. Branches and two votes per
// i cluster took 54 us for 45 million listed pairs, a box test before them 57.
template <bool DBL>
__device__ void prune_item(const ListArgs& L, int w, PruneShared& S) {
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i8 = lane & 7, jq = lane >> 3;
  const float rp2 = float(L.rprune2) + 0.02f;
  const int4 wk = L.b.work[w];
  const int sc = wk.x;
  const int ne = min(wk.z, kBatch);
  uint4 en = make_uint4(0u, 0u, 0u, 0u);
  if (lane < ne) en = L.b.ent[wk.y + lane];
  // positions from the super-cluster's origin (FP32 path: packed so) or first atom (FP64 path: slot 0 is always real)
  double4 o = make_double4(0, 0, 0, 0);
  if (DBL) o = L.xqd[64 * sc];
  auto at = [&](int s) {
    float4 v;
    if (DBL) {
      const double4 d = L.xqd[s];
      v = make_float4(float(d.x - o.x), float(d.y - o.y), float(d.z - o.z), 0.f);
    } else {
      v = L.xq[s];
    }
    return v;
  };
  if (lane < ne) {
    float4 sh;
    if (DBL) {
      int qa, qb, qc;
      unpack_image(en.y >> 8, qa, qb, qc);
      sh = make_float4(float(L.cell.h[0][0] * qa + L.cell.h[0][1] * qb + L.cell.h[0][2] * qc), float(L.cell.h[1][0] * qa + L.cell.h[1][1] * qb + L.cell.h[1][2] * qc),
                       float(L.cell.h[2][0] * qa + L.cell.h[2][1] * qb + L.cell.h[2][2] * qc), 0.f);
    } else {
      sh = L.b.ent_shift[wk.y + lane];
    }
    sh.w = __int_as_float(int(en.x));
    S.sh[wib][lane] = sh;
  }
  float xi[8], yi[8], zi[8], hi[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int s = 64 * sc + 8 * c + i8;
    const float4 v = at(s);
    xi[c] = v.x, yi[c] = v.y, zi[c] = v.z;
    hi[c] = L.tslot[s] != L.pad_type ? -0.4999995f * (v.x * v.x + v.y * v.y + v.z * v.z) : -1e30f;   // padding is never near
  }
  __syncwarp();
  for (int t = lane; t < 8 * ne; t += 32) {   // entry t / 8, j atom t % 8
    const float4 sh = S.sh[wib][t >> 3];
    const int s = 8 * __float_as_int(sh.w) + (t & 7);
    float4 v = at(s);
    v.x += sh.x, v.y += sh.y, v.z += sh.z;
    v.w = L.tslot[s] != L.pad_type ? 0.4999995f * (v.x * v.x + v.y * v.y + v.z * v.z) - 0.5f * rp2 : 1e30f;
    S.xj[wib][t] = v;
  }
  __syncwarp();
  unsigned mine = 0;   // lane e: entry e's new mask
  for (int el = 0; el < ne; ++el) {
    const float4 a0 = S.xj[wib][8 * el + jq], a1 = S.xj[wib][8 * el + jq + 4];
    unsigned keep = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float d0 = fmaf(xi[c], a0.x, fmaf(yi[c], a0.y, fmaf(zi[c], a0.z, hi[c])));
      const float d1 = fmaf(xi[c], a1.x, fmaf(yi[c], a1.y, fmaf(zi[c], a1.z, hi[c])));
      if (d0 > a0.w) keep |= 1u << c;
      if (d1 > a1.w) keep |= 256u << c;
    }
    keep = __reduce_or_sync(0xffffffffu, keep);
    if (lane == el) mine = keep;
  }
  if (lane < ne) {
    en.w = mine & ((en.y & 255u) * 0x101u);
    L.b.ent[wk.y + lane] = en;
  }
  __syncwarp();
}

union ListShared {
  unsigned char sort[kSortSmem];
  SearchShared search;
  PruneShared prune;
};

// Waits (every thread of the block calls it) until `want` units of a stage are finished; false after L.polls looks.
__device__ __forceinline__ bool list_wait(const ListArgs& L, int stage, int want, int* s_ok) {
  int* counters = L.b.counters;
  if (threadIdx.x == 0) {
    volatile const int* done = counters + kCntStage + stage;
    int k = 0;
    while (*done < want && k < L.polls) {
      __nanosleep(64);
      ++k;
    }
    *s_ok = *done >= want;
    if (!*s_ok) raise_error(counters, kErrListWait);
    __threadfence();   // the stage's results, written before its count went up, are read after this
  }
  __syncthreads();
  const bool ok = *s_ok != 0;
  __syncthreads();   // every thread has read it before a later wait writes it
  return ok;
}
// A unit of a stage is finished: its block's writes become visible before the count goes up. Returns the units finished
// before it (thread 0; the others 0).
__device__ __forceinline__ int list_done(int* counters, int stage) {
  __syncthreads();
  if (threadIdx.x != 0) return 0;
  __threadfence();
  return atomicAdd(counters + kCntStage + stage, 1);
}

template <bool DBL>
static __global__ void __launch_bounds__(kListThreads, 4) k_list(ListArgs L) {
  extern __shared__ __align__(16) unsigned char list_smem[];
  ListShared& S = *reinterpret_cast<ListShared*>(list_smem);
  __shared__ int s_t, s_ok;
  int* cnt = L.b.counters;
  // the flags are set by earlier kernels and lowered by the pair kernel: the same for every block of this launch
  const bool built = !L.pack_only && (L.force || *(volatile const int*)(cnt + kCntRebuild) != 0);
  const bool pruned = built || (!L.pack_only && *(volatile const int*)(cnt + kCntPrune) != 0);   // a fresh list is pruned at once
  const int npack = (L.nslots + kListThreads - 1) / kListThreads;
  if (!pruned) {
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[kCntPairNext] = 0;   // the pair kernel's work-item counter
    const int nsc = min(cnt[kCntNsc], L.b.nsc_cap);
    for (int u = blockIdx.x; u < npack; u += gridDim.x) pack_slot<DBL>(L, u * kListThreads + threadIdx.x, nsc, false);
    return;
  }
  // units of each stage; the prune's are the grid's blocks, striding over the work items
  const int nbin = built ? (L.n + kListThreads - 1) / kListThreads : 0;
  const int nsort = built ? L.g.ncol : 0, nsuper = built ? (L.b.nsc_cap + kScWarps - 1) / kScWarps : 0, nsearch = built ? L.b.nsc_cap : 0;
  const int e_bin = nbin, e_scat = e_bin + nbin, e_sort = e_scat + nsort, e_super = e_sort + nsuper, e_search = e_super + nsearch, e_pack = e_search + npack;
  const int total = e_pack + int(gridDim.x);
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_t = atomicAdd(cnt + kCntTicket, 1);
    __syncthreads();
    const int t = s_t;
    if (t >= total) break;
    if (t < e_bin) {
      bin_atom(L.n, t * kListThreads + threadIdx.x, L.x, L.cell, L.g, L.b);
      const int before = list_done(cnt, kStBin);
      if (threadIdx.x == 0) s_ok = before == nbin - 1;
      __syncthreads();
      if (s_ok) {   // the last block scans the columns
        __threadfence();
        scan_columns<kListThreads>(L.g, L.b);
        list_done(cnt, kStScan);
      }
    } else if (t < e_scat) {
      if (!list_wait(L, kStScan, 1, &s_ok)) break;
      scatter_atom(L.n, (t - e_bin) * kListThreads + threadIdx.x, L.b);
      list_done(cnt, kStScatter);
    } else if (t < e_sort) {
      if (!list_wait(L, kStScatter, nbin, &s_ok)) break;
      sort_column(t - e_scat, L.b, S.sort);
      list_done(cnt, kStSort);
    } else if (t < e_super) {
      if (!list_wait(L, kStSort, nsort, &s_ok)) break;
      super_unit(t - e_sort, L.cell, L.b);
      list_done(cnt, kStSuper);
    } else if (t < e_search) {
      if (!list_wait(L, kStSuper, nsuper, &s_ok)) break;
      const int sc = t - e_super;
      if (sc < min(L.b.counters[kCntNsc], L.b.nsc_cap)) search_supercluster(sc, L.cell, L.g, L.excl_off, L.excl_list, L.b, S.search);
      list_done(cnt, kStSearch);
    } else if (t < e_pack) {
      // the pack reads the slots that the super-clusters' stage made; it runs beside the last of the search
      if (built && !list_wait(L, kStSuper, nsuper, &s_ok)) break;
      const int u = t - e_search;
      if (u == 0 && threadIdx.x == 0) {
        cnt[kCntPairNext] = 0;
        if (built) cnt[kCntBuilds] += 1;
        cnt[kCntPrunes] += 1;
      }
      pack_slot<DBL>(L, u * kListThreads + threadIdx.x, min(L.b.counters[kCntNsc], L.b.nsc_cap), built);
      list_done(cnt, kStPack);
    } else {
      if (!list_wait(L, kStPack, npack, &s_ok) || (built && !list_wait(L, kStSearch, nsearch, &s_ok))) break;
      const int u = t - e_pack;
      // the positions of this prune, for the next displacement check
      for (int i = u * kListThreads + threadIdx.x; i < 3 * L.n; i += gridDim.x * kListThreads) L.xp[i] = L.x[i];
      if (cnt[kCntErr] & kErrListBad) continue;
      const int nwork = min(L.b.counters[kCntWork], L.b.work_cap);
      constexpr int W = kListThreads / 32;
      for (int w = u * W + int(threadIdx.x >> 5); w < nwork; w += gridDim.x * W) prune_item<DBL>(L, w, S.prune);
    }
  }
  // the last block to leave clears the counters for the next launch
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(cnt + kCntLeft, 1) == int(gridDim.x) - 1) {
    cnt[kCntTicket] = 0;
    cnt[kCntLeft] = 0;
    for (int k = 0; k < kStNum; ++k) cnt[kCntStage + k] = 0;
  }
}

}  // namespace capsb
