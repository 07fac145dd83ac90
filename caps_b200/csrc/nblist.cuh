// The cluster pair list on the device (the reference builds it on the CPU: core/src/nbnxm.cpp:22-326, and its FP64
// atom-pair list, core/src/field.cpp:892-1101).
//
// Layout. Atoms are binned into columns over the (a, b) fractional plane, sorted along c inside each column and cut
// into super-clusters of 64 consecutive atoms; each super-cluster is split 2 x 2 x 2 (z halves, then y, then x) into
// eight clusters of 8 atoms. Slot s = 64 sc + 8 k + l holds atom perm[s] (-1 padding). A list entry pairs one
// super-cluster (the i side, 64 atoms, held by one warp) with one j cluster (8 atoms) under one periodic image, with an
// 8-bit mask of the super-cluster's clusters whose bounding boxes come within the list radius, and an optional index to
// eight 64-bit atom masks (exclusions at their nearest image, each pair of one cluster once). The half list keeps each
// cluster pair from one side, chosen by the parity of ci + cj as the reference does (nbnxm.cpp:201-206), and a cluster
// with its own images once per +- shift. Entries are produced in batches of up to 32 per super-cluster: each batch is
// one work item of the pair kernel.
#pragma once
#include "list_types.cuh"

namespace capsb {

// ---------------------------------------------------------------------------------------------------------------
// K-CHECK: the displacement check as a kernel of its own, for force evaluations outside a step that folds it in.
static __global__ void k_check_step(int n, const double* __restrict__ x, ListCheck L) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool mb = false, mp = false;
  if (i < n) list_check_atom(L, i, x, mb, mp);
  list_check_flags(L, mb, mp);
}

// Scan stage (one block, NT threads): column starts, super-cluster starts (64 atoms each, the last one of a column
// partial), and the column of every super-cluster. Also resets the list counters for the search. The column counts are
// read through L2 (the other blocks of the binning made them with atomics).
template <int NT>
__device__ void scan_columns(const ListGeom& g, const ListBufs& b) {
  __shared__ int s_a[NT / 32], s_s[NT / 32];
  __shared__ int s_max;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int carry_a = 0, carry_s = 0;
  if (threadIdx.x == 0) s_max = 0;
  __syncthreads();
  for (int base = 0; base < g.ncol; base += NT) {
    const int c = base + threadIdx.x;
    const int cnt = c < g.ncol ? __ldcg(b.col_count + c) : 0;
    if (c < g.ncol) b.col_count[c] = 0;   // cleared for the next build's binning
    if (cnt) atomicMax(&s_max, cnt);
    int a = cnt, sc = (cnt + kScAtoms - 1) / kScAtoms;   // inclusive scans of both, by warp and then over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ta = __shfl_up_sync(0xffffffffu, a, o), ts = __shfl_up_sync(0xffffffffu, sc, o);
      if (lane >= o) a += ta, sc += ts;
    }
    if (lane == 31) s_a[warp] = a, s_s[warp] = sc;
    __syncthreads();
    int tot_a = 0, tot_s = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
      if (w < warp) a += s_a[w], sc += s_s[w];
      tot_a += s_a[w], tot_s += s_s[w];
    }
    if (c < g.ncol) {
      b.col_start[c + 1] = carry_a + a;
      b.col_sc[c + 1] = carry_s + sc;
      b.col_fill[c] = 0;
    }
    carry_a += tot_a, carry_s += tot_s;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    b.col_start[0] = 0;
    b.col_sc[0] = 0;
    b.counters[kCntNsc] = carry_s;
    b.counters[kCntMaxCol] = s_max;
    b.counters[kCntEnt] = 0;
    b.counters[kCntWork] = 0;
    b.counters[kCntMask] = 0;
    if (carry_s > b.nsc_cap) raise_error(b.counters, kErrScOverflow);
    if (s_max > kSortMax) raise_error(b.counters, kErrColumnTooBig);
  }
  __syncthreads();
  const int nsc = min(carry_s, b.nsc_cap);
  for (int c = threadIdx.x; c < g.ncol; c += NT)
    for (int s = b.col_sc[c]; s < b.col_sc[c + 1] && s < nsc; ++s) b.sc_col[s] = c;
}

// Bin stage: wrapped fractional coordinates, lattice offsets and the column of atom i; column counts.
constexpr int kListThreads = 256;   // block size of k_list (list.cuh), whose stages these are
__device__ __forceinline__ void bin_atom(int n, int i, const double* __restrict__ x, const DevCell& cell, const ListGeom& g, const ListBufs& b) {
  if (i >= n) return;
  const double xi[3] = {x[3 * i], x[3 * i + 1], x[3 * i + 2]};
  double f[3];
  frac_of(cell, xi, f);
  for (int k = 0; k < 3; ++k) {
    const double fl = floor(f[k]);
    f[k] = fmin(fmax(f[k] - fl, 0.0), 1.0 - 1e-12);
    b.frac[3 * i + k] = f[k];
    b.ioff[3 * i + k] = -int(fl);
  }
  const int cu = min(g.nu - 1, int(f[0] * g.nu)), cv = min(g.nv - 1, int(f[1] * g.nv));
  const int c = cu * g.nv + cv;
  b.col[i] = c;
  // one atomic per distinct column in the warp (a column holds hundreds of atoms: the adds would contend)
  const unsigned act = __activemask();
  const unsigned same = __match_any_sync(act, c);
  if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(b.col_count + c, __popc(same));
}

// Scatter stage: atom i into its column's range (unordered; the sort that follows fixes the order).
__device__ __forceinline__ void scatter_atom(int n, int i, const ListBufs& b) {
  if (i >= n) return;
  const int c = b.col[i];
  // warp-aggregated: the lowest lane of each column group reserves the group's places
  const unsigned act = __activemask();
  const unsigned same = __match_any_sync(act, c);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(b.col_fill + c, __popc(same));
  base = __shfl_sync(same, base, leader);
  b.order[b.col_start[c] + base + __popc(same & ((1u << lane) - 1))] = i;
}

// One compare-exchange of a bitonic network over the lanes: the pair (lane, lane ^ j) ascending where up.
__device__ __forceinline__ void lane_exchange(unsigned& key, int& id, int j, bool up) {
  const unsigned k = __shfl_xor_sync(0xffffffffu, key, j);
  const int i = __shfl_xor_sync(0xffffffffu, id, j);
  const bool low = (threadIdx.x & j) == 0;   // the pair's lower lane keeps the smaller key
  if (low == up ? k < key : k > key) key = k, id = i;
}
// Sorts key (and id) over groups of N lanes, ascending. Deterministic: the network's exchanges depend on the keys alone.
template <int N>
__device__ __forceinline__ void lane_sort(unsigned& key, int& id) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int kk = 2; kk <= N; kk <<= 1)
#pragma unroll
    for (int j = kk >> 1; j > 0; j >>= 1) lane_exchange(key, id, j, kk == N || (lane & kk) == 0);
}

// K-SUPER (a warp per super-cluster): the 2 x 2 x 2 split into clusters, perm / iperm, cluster boxes and real-atom masks,
// the super-cluster's origin and its c range. Lane l holds atoms l (lower c half) and l + 32 (upper c half), sorted along b
// over the warp and then along a over each half of it (keys in units of 2^-32 of the cell), which leaves slot 32 h + l in
// lane l; padding sorts last. (Ranks by
// comparing with every other atom took some 2,600 instructions of one warp: 17 us a build at any size.)
__device__ void form_supercluster(const DevCell& cell, const ListBufs& b, int sc, int c, int lane) {
  const int k = sc - b.col_sc[c];
  const int s0 = b.col_start[c] + kScAtoms * k;
  const int m = min(kScAtoms, b.col_start[c + 1] - s0);
  if (m <= 0) {   // not made by the scan (every super-cluster holds at least one atom); kept empty
    b.perm[64 * sc + lane] = b.perm[64 * sc + lane + 32] = -1;
    return;
  }
  const int first = b.order[s0], last = b.order[s0 + m - 1];
  int id[2];
  unsigned key[2];
  auto key_of = [&](int a, int axis) { return a >= 0 ? unsigned(b.frac[3 * a + axis] * 4294967295.0) : ~0u; };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = lane + 32 * h;
    id[h] = t < m ? b.order[s0 + t] : -1;
    key[h] = key_of(id[h], 1);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) lane_sort<32>(key[h], id[h]);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    key[h] = key_of(id[h], 0);
    lane_sort<16>(key[h], id[h]);
  }
  // cluster boxes and real masks: slot lane + 32 h belongs to cluster (lane >> 3) + 4 h. The origin, which the packed
  // positions are rounded from, is the middle of the atoms' own extent, in double.
  double slo[3] = {1e300, 1e300, 1e300}, shi[3] = {-1e300, -1e300, -1e300};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int a = id[h];
    b.perm[64 * sc + lane + 32 * h] = a;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    if (a >= 0) {
      b.iperm[a] = 64 * sc + lane + 32 * h;
      const double f0 = b.frac[3 * a], f1 = b.frac[3 * a + 1], f2 = b.frac[3 * a + 2];
      for (int r = 0; r < 3; ++r) lo[r] = hi[r] = cell.o[r] + cell.h[r][0] * f0 + cell.h[r][1] * f1 + cell.h[r][2] * f2;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
      for (int r = 0; r < 3; ++r) {
        lo[r] = fmin(lo[r], __shfl_xor_sync(0xffffffffu, lo[r], o));
        hi[r] = fmax(hi[r], __shfl_xor_sync(0xffffffffu, hi[r], o));
      }
    const unsigned real = __ballot_sync(0xffffffffu, a >= 0);
    if ((lane & 7) == 0) {
      const int cg = 8 * sc + (lane >> 3) + 4 * h;
      for (int r = 0; r < 3; ++r) b.cl_box[6 * cg + r] = lo[r], b.cl_box[6 * cg + 3 + r] = hi[r];
      b.cl_boxf[2 * cg] = make_float4(float(lo[0]), float(lo[1]), float(lo[2]), 0.f);   // an empty cluster: +inf and -inf
      b.cl_boxf[2 * cg + 1] = make_float4(float(hi[0]), float(hi[1]), float(hi[2]), 0.f);
      b.cl_real[cg] = (unsigned char)((real >> (lane & 24)) & 255u);
    }
    for (int r = 0; r < 3; ++r) slo[r] = fmin(slo[r], lo[r]), shi[r] = fmax(shi[r], hi[r]);
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1)
    for (int r = 0; r < 3; ++r) {
      slo[r] = fmin(slo[r], __shfl_xor_sync(0xffffffffu, slo[r], o));
      shi[r] = fmax(shi[r], __shfl_xor_sync(0xffffffffu, shi[r], o));
    }
  if (lane == 0) {
    for (int r = 0; r < 3; ++r) b.sc_org[3 * sc + r] = 0.5 * (slo[r] + shi[r]);
    b.sc_z[2 * sc] = b.frac[3 * first + 2];
    b.sc_z[2 * sc + 1] = b.frac[3 * last + 2];
  }
}

// Sort stage (a block per column): atoms by fractional c, ties by index, as one 64-bit key each (c in units of 2^-32 of the
// cell, the index). Runs of 32 are sorted by the lanes of a warp, then runs are merged in pairs: every key finds its place
// among the sibling run's by binary search. Columns past kSortMax / 2, whose second buffer has no room, take a bitonic
// network in place (55 rounds with a barrier each took 40 us for columns of 650 atoms).
constexpr size_t kSortSmem = size_t(kSortMax) * sizeof(unsigned long long);
__device__ void sort_column(int c, const ListBufs& b, unsigned char* smem_raw) {
  using Key = unsigned long long;
  Key* A = reinterpret_cast<Key*>(smem_raw);
  const int s0 = b.col_start[c], n = min(b.col_start[c + 1] - s0, kSortMax);
  auto key_of = [&](int k) {
    const int a = b.order[s0 + k];
    return (Key(unsigned(b.frac[3 * a + 2] * 4294967296.0)) << 32) | unsigned(a);   // fractional coordinates are below 1 - 1e-12
  };
  if (n <= kSortMax / 2) {
    Key* B = A + kSortMax / 2;
    const int lane = threadIdx.x & 31;
    for (int k0 = (threadIdx.x >> 5) * 32; k0 < n; k0 += kListThreads) {
      Key key = k0 + lane < n ? key_of(k0 + lane) : ~0ull;
#pragma unroll
      for (int kk = 2; kk <= 32; kk <<= 1)
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
          const Key o = __shfl_xor_sync(0xffffffffu, key, j);
          const bool low = (lane & j) == 0, up = kk == 32 || (lane & kk) == 0;
          if (low == up ? o < key : o > key) key = o;
        }
      if (k0 + lane < n) A[k0 + lane] = key;
    }
    __syncthreads();
    for (int ws = 5; (1 << ws) < n; ++ws) {
      const int width = 1 << ws;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const Key key = A[i];
        const int run = i >> ws, sib = (run ^ 1) << ws;
        int lo = sib, hi = min(sib + width, n);   // the sibling's first key above this one (keys are distinct)
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (A[mid] < key) lo = mid + 1;
          else hi = mid;
        }
        B[((run & ~1) << ws) + (i & (width - 1)) + max(0, lo - sib)] = key;
      }
      __syncthreads();
      Key* t = A;
      A = B;
      B = t;
    }
  } else {
    int np = 1;
    while (np < n) np <<= 1;
    for (int k = threadIdx.x; k < np; k += blockDim.x) A[k] = k < n ? key_of(k) : ~0ull;
    __syncthreads();
    for (int kk = 2; kk <= np; kk <<= 1)
      for (int j = kk >> 1; j > 0; j >>= 1) {
        for (int t = threadIdx.x; t < (np >> 1); t += blockDim.x) {
          const int lo = 2 * (t & ~(j - 1)) + (t & (j - 1)), hi = lo + j;
          const Key ka = A[lo], kb = A[hi];
          if ((ka > kb) == ((lo & kk) == 0)) A[lo] = kb, A[hi] = ka;
        }
        __syncthreads();
      }
  }
  for (int k = threadIdx.x; k < n; k += blockDim.x) b.order[s0 + k] = int(unsigned(A[k]));
}

// Super-cluster stage: kScWarps of them to a unit, a warp each.
constexpr int kScWarps = kListThreads / 32;
__device__ __forceinline__ void super_unit(int unit, const DevCell& cell, const ListBufs& b) {
  const int sc = unit * kScWarps + int(threadIdx.x >> 5);
  if (sc < min(b.counters[kCntNsc], b.nsc_cap)) form_supercluster(cell, b, sc, b.sc_col[sc], threadIdx.x & 31);
}

// ---------------------------------------------------------------------------------------------------------------
constexpr int kSearchWarps = 8;       // warps per super-cluster in the search

// One warp's batch of entries in the making.
struct SearchBatch {
  uint4 ent[2 * kBatch];
  float4 sh[2 * kBatch];
  int nent;
};

struct SearchShared {
  int xfirst[65];                         // exclusions of the super-cluster's atoms: where each atom's begin
  int xatom[64];                          // the atoms
  unsigned xoff[64];                      // and their places in the exclusion list
  uint2 rec[kExclRecMax];                 // x: j cluster, y: i local (6 bits) | j in cluster (3) << 6 | image << 9
  unsigned long long key[kExclHash];      // distinct (j cluster, image) of the records; ~0 empty
  unsigned short krank[kExclHash];        // rank of each occupied key slot: its masks are number mbase + rank
  int mbase;
  double ibox[8][6];            // the i clusters' boxes
  float ilo[8][3], ihi[8][3];   // the same in float, from the super-cluster's origin
  double org_i[3];
  int nrec;
  SearchBatch batch[kSearchWarps];
};

__device__ __forceinline__ unsigned long long excl_key(unsigned cj, unsigned img) { return (unsigned long long)cj | ((unsigned long long)img << 32); }

// The slot of a key in the open-addressing table, or -1.
static __device__ int key_slot(const SearchShared& S, unsigned long long key) {
  unsigned h = (unsigned)(key * 0x9E3779B97F4A7C15ull >> 56) & (kExclHash - 1);
  for (int p = 0; p < kExclHash; ++p) {
    const unsigned long long v = S.key[h];
    if (v == key) return int(h);
    if (v == ~0ull) return -1;
    h = (h + 1) & (kExclHash - 1);
  }
  return -1;
}

static __device__ int key_insert(SearchShared& S, unsigned long long key, int* counters) {
  unsigned h = (unsigned)(key * 0x9E3779B97F4A7C15ull >> 56) & (kExclHash - 1);
  for (int p = 0; p < kExclHash; ++p) {
    const unsigned long long old = atomicCAS(&S.key[h], ~0ull, key);
    if (old == ~0ull || old == key) return int(h);
    h = (h + 1) & (kExclHash - 1);
  }
  raise_error(counters, kErrExclOverflow);
  return -1;
}
// Writes the entries [0, cnt) of B as work items of up to `depth` entries. One atomic reserves them all: the entry and work
// counters are the two halves of one 64-bit word (entries low, work items high), shared by every warp of the build.
static __device__ void flush_entries(SearchBatch& B, int sc, int cnt, int depth, int lane, const ListBufs& b) {
  if (cnt <= 0) return;
  static_assert(kCntEnt == 0 && kCntWork == 1, "entry and work counters form one 64-bit word");
  const int items = (cnt + depth - 1) / depth;
  int base = 0, wi = 0;
  if (lane == 0) {
    const unsigned long long old =
        atomicAdd(reinterpret_cast<unsigned long long*>(b.counters + kCntEnt), ((unsigned long long)(unsigned)items << 32) | unsigned(cnt));
    base = int(unsigned(old & 0xffffffffull));
    wi = int(unsigned(old >> 32));
  }
  base = __shfl_sync(0xffffffffu, base, 0);
  wi = __shfl_sync(0xffffffffu, wi, 0);
  if (base + cnt > b.ent_cap || wi + items > b.work_cap) {
    if (lane == 0) raise_error(b.counters, kErrListOverflow);
    return;
  }
  for (int e = lane; e < cnt; e += 32) {
    uint4 en = B.ent[e];
    en.w = (en.y & 255u) * 0x101u;   // unpruned until the first prune: both halves of every listed i cluster
    b.ent[base + e] = en;
    b.ent_shift[base + e] = B.sh[e];
  }
  for (int k = lane; k < items; k += 32) b.work[wi + k] = make_int4(sc, base + k * depth, min(depth, cnt - k * depth), 0);
}

// Search stage: one block of kSearchWarps warps per super-cluster. The block records the super-cluster's excluded pairs and
// builds the atom masks of every (j cluster, image) they touch; then each warp takes a contiguous share of the
// neighbouring columns (with their images) and batches its own entries. Exclusions (ForceField::excluded) hold at their
// nearest image only (core/src/nbnxm.cpp:229-252): each of the super-cluster's excluded atom pairs is recorded with the
// image that is nearest at the build, and the entry for that j cluster under that image carries masks with those pairs
// cleared. The super-cluster's own clusters under the zero image always carry masks (each pair of a cluster with
// itself once).
static_assert(kListThreads == 32 * kSearchWarps, "the search runs in k_list's blocks");
__device__ void search_supercluster(int sc, const DevCell& cell, const ListGeom& g, const uint32_t* __restrict__ excl_off,
                                    const uint32_t* __restrict__ excl_list, const ListBufs& b, SearchShared& S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  SearchBatch& B = S.batch[warp];
  const int nsc = min(b.counters[kCntNsc], b.nsc_cap);
  {
    // --- the super-cluster's boxes and exclusion records (the whole block)
    for (int t = threadIdx.x; t < kExclHash; t += blockDim.x) S.key[t] = ~0ull;
    if (threadIdx.x < 24) {
      const int c = threadIdx.x / 3, r = threadIdx.x % 3;
      const double* box = b.cl_box + 6 * (8 * sc + c);
      const double o = b.sc_org[3 * sc + r];
      S.ibox[c][r] = box[r], S.ibox[c][3 + r] = box[3 + r];
      S.ilo[c][r] = float(box[r] - o), S.ihi[c][r] = float(box[3 + r] - o);
      if (c == 0) S.org_i[r] = o;
    }
    if (threadIdx.x == 0) S.nrec = 0;
    if (lane == 0) B.nent = 0;
    __syncthreads();
    if (threadIdx.x < 8) key_insert(S, excl_key(unsigned(8 * sc + threadIdx.x), pack_image(0, 0, 0)), b.counters);
    // the super-cluster's exclusions, one to a thread: their counts per atom, the running sums, then each (atom, partner)
    if (threadIdx.x < 64) {
      const int a = b.perm[64 * sc + threadIdx.x];
      const unsigned o = a >= 0 ? excl_off[a] : 0u;
      S.xatom[threadIdx.x] = a;
      S.xoff[threadIdx.x] = o;
      int sum = a >= 0 ? int(excl_off[a + 1] - o) : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += y;
      }
      S.xfirst[threadIdx.x + 1] = sum;   // within each half; the upper half's offset is added below
    }
    if (threadIdx.x == 0) S.xfirst[0] = 0;
    __syncthreads();
    const int xhalf = S.xfirst[32], nexcl = xhalf + S.xfirst[64];
    for (int q = threadIdx.x; q < nexcl; q += blockDim.x) {
      // the atom of exclusion q: the last whose first is at most q
      const int up = q >= xhalf ? 32 : 0, qq = q - (up ? xhalf : 0);
      int t = 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
        if ((t + d ? S.xfirst[up + t + d] : 0) <= qq) t += d;
      const int firstq = t ? S.xfirst[up + t] : 0;
      t += up;
      const int a = S.xatom[t];
      const int bb = int(excl_list[S.xoff[t] + unsigned(qq - firstq)]);
      const int sb = b.iperm[bb];
      const double* fa = b.frac + 3 * a;
      const double* fb = b.frac + 3 * bb;
      // nearest image of bb seen from a: bb + q, q = -round(fb - fa)
      const int qa = -int(rint(fb[0] - fa[0])), qb = -int(rint(fb[1] - fa[1])), qc = -int(rint(fb[2] - fa[2]));
      if (qa < -63 || qa > 63 || qb < -63 || qb > 63 || qc < -63 || qc > 63) { raise_error(b.counters, kErrImageRange); continue; }
      const unsigned img = pack_image(qa, qb, qc);
      const int r = atomicAdd(&S.nrec, 1);
      if (r >= kExclRecMax) { raise_error(b.counters, kErrExclOverflow); continue; }
      S.rec[r] = make_uint2(unsigned(sb >> 3), unsigned(t) | (unsigned(sb & 7) << 6) | (img << 9));
      key_insert(S, excl_key(unsigned(sb >> 3), img), b.counters);
    }
    __syncthreads();
    if (threadIdx.x == 0 && S.nrec > kExclRecMax) S.nrec = kExclRecMax;
    // masks: one set of 8 rows (i cluster r against the key's j cluster) per occupied key slot, numbered by the slot's
    // rank from a base reserved with one atomic; rows start as all pairs (each pair once for a cluster with itself under
    // the zero image), then every record clears its pair
    if (warp == 0) {
      constexpr int per = kExclHash / 32;
      unsigned occ = 0;
#pragma unroll
      for (int q = 0; q < per; ++q) occ |= unsigned(S.key[lane * per + q] != ~0ull) << q;
      const unsigned tot = __popc(occ);
      unsigned run = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += y;
      }
      unsigned start = run - tot;
#pragma unroll
      for (int q = 0; q < per; ++q) {
        S.krank[lane * per + q] = (unsigned short)start;
        start += (occ >> q) & 1u;
      }
      const unsigned nkeys = __shfl_sync(0xffffffffu, run, 31);
      if (lane == 0) {
        const int m0 = atomicAdd(b.counters + kCntMask, int(nkeys));
        if (m0 + int(nkeys) > b.mask_cap) raise_error(b.counters, kErrMaskOverflow);
        S.mbase = m0;
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 8 * kExclHash; t += blockDim.x) {
      const int h = t >> 3, r = t & 7;
      const unsigned long long key = S.key[h];
      if (key == ~0ull) continue;
      const int mi = S.mbase + S.krank[h];
      if (mi >= b.mask_cap) continue;
      unsigned long long mm = ~0ull;
      if (key == excl_key(unsigned(8 * sc + r), pack_image(0, 0, 0))) {
        mm = 0;
        for (int i = 0; i < 8; ++i)
          for (int j = i + 1; j < 8; ++j) mm |= 1ull << (8 * i + j);
      }
      b.masks[8 * size_t(mi) + r] = mm;
    }
    __syncthreads();   // the rows are written before any record clears a bit of them
    for (int r = threadIdx.x; r < S.nrec; r += blockDim.x) {
      const uint2 rc = S.rec[r];
      const int h = key_slot(S, excl_key(rc.x, rc.y >> 9));
      if (h < 0) continue;
      const int mi = S.mbase + S.krank[h];
      if (mi >= b.mask_cap) continue;
      const unsigned il = rc.y & 63u, jl = (rc.y >> 6) & 7u;
      atomicAnd(b.masks + 8 * size_t(mi) + (il >> 3), ~(1ull << (8 * (il & 7) + jl)));
    }
    // --- candidates: neighbouring columns (with their images), super-clusters in c range, their 8 clusters. Each warp
    // takes a contiguous block of the columns: its entries (and the pair kernel's work items made of them) stay spatially
    // together, which measured faster in the pair kernel than an interleaved split. The split is fixed, so every build
    // groups the same entries into the same work items (the pair kernel's float partial sums, and so the forces, do not
    // depend on timing).
    const int col = b.sc_col[sc];
    const int cu = col / g.nv, cv = col % g.nv;
    const double zlo = b.sc_z[2 * sc], zhi = b.sc_z[2 * sc + 1];
    const int nvw = 2 * g.rv + 1, ncols = (2 * g.ru + 1) * nvw;
    const int kper = (ncols + kSearchWarps - 1) / kSearchWarps;
    for (int k = warp * kper; k < min(ncols, (warp + 1) * kper); ++k) {
      const int du = k / nvw - g.ru, dv = k % nvw - g.rv;
      int U = cu + du;
      const int qa = (int)floor(double(U) / g.nu);
      U -= qa * g.nu;
      int V = cv + dv;
      const int qb = (int)floor(double(V) / g.nv);
      V -= qb * g.nv;
      const int cc = U * g.nv + V;
      const int qc0 = max(-g.rq, (int)floor(zlo - g.dw)), qc1 = min(g.rq, (int)floor(zhi + g.dw));
      for (int qc = qc0; qc <= qc1; ++qc) {
        const double S0 = cell.h[0][0] * qa + cell.h[0][1] * qb + cell.h[0][2] * qc;
        const double S1 = cell.h[1][0] * qa + cell.h[1][1] * qb + cell.h[1][2] * qc;
        const double S2 = cell.h[2][0] * qa + cell.h[2][1] * qb + cell.h[2][2] * qc;
        const bool zero = qa == 0 && qb == 0 && qc == 0;
        const bool positive = qa > 0 || (qa == 0 && (qb > 0 || (qb == 0 && qc > 0)));
        const unsigned img = pack_image(qa, qb, qc);
        const double lo = zlo - g.dw - qc, hi = zhi + g.dw - qc;
        // the image's shift as seen from the super-cluster's origin
        const float F0 = float(S0 - S.org_i[0]), F1 = float(S1 - S.org_i[1]), F2 = float(S2 - S.org_i[2]);
        // super-clusters of column cc whose c range meets [lo, hi]: their ranges rise along the column, 32 looked at at once
        const int sj0 = b.col_sc[cc], sje = min(b.col_sc[cc + 1], nsc);
        for (int sjb = sj0; sjb < sje; sjb += 32) {
          unsigned in = 0;
          {
            const int t = sjb + lane;
            const double2 z = t < sje ? *reinterpret_cast<const double2*>(b.sc_z + 2 * t) : make_double2(3e300, -3e300);
            in = __ballot_sync(0xffffffffu, z.y >= lo && z.x <= hi);
          }
          if (!in) continue;
          const int sj1 = sjb + __ffs(in) - 1, sj2 = sjb + 32 - __clz(in);
          for (int sj = sj1; sj < sj2; sj += 4) {
            // four candidate super-clusters per pass: lane = 8 * which + j cluster
            const int sjl = sj + (lane >> 3);
            bool have = false;
            unsigned imask = 0, sure = 0;
            int cj = -1;
            if (sjl < sj2) {
              cj = 8 * sjl + (lane & 7);
              const float4 bl = b.cl_boxf[2 * cj], bh = b.cl_boxf[2 * cj + 1];
              const float l0 = bl.x + F0, l1 = bl.y + F1, l2 = bl.z + F2, h0 = bh.x + F0, h1 = bh.y + F1, h2 = bh.z + F2;
  #pragma unroll
              for (int c = 0; c < 8; ++c) {
                const float g0 = fmaxf(fmaxf(l0 - S.ihi[c][0], S.ilo[c][0] - h0), 0.f), g1 = fmaxf(fmaxf(l1 - S.ihi[c][1], S.ilo[c][1] - h1), 0.f),
                            g2 = fmaxf(fmaxf(l2 - S.ihi[c][2], S.ilo[c][2] - h2), 0.f);
                const float d2 = g0 * g0 + g1 * g1 + g2 * g2;
                imask |= unsigned(d2 < g.far2) << c;
                sure |= unsigned(d2 < g.near2) << c;
              }
              // half list: one side of each cluster pair by parity; a cluster with itself under zero or + images
              const unsigned even = 0x55u << (cj & 1);   // the i clusters ci with ci + cj even (8 sc is)
              if (sjl != sc) imask &= sjl > sc ? even : ~even;
              else {
                const int k = lane & 7;
                const unsigned below = (1u << k) - 1;
                imask &= (even & below) | (~even & ~below & ~(1u << k)) | (zero || positive ? 1u << k : 0u);
              }
              // the few that float cannot decide
              for (unsigned open = imask & ~sure; open; open &= open - 1) {
                const int c = __ffs(open) - 1;
                const double* bj = b.cl_box + 6 * cj;
                const double jlo[3] = {bj[0] + S0, bj[1] + S1, bj[2] + S2}, jhi[3] = {bj[3] + S0, bj[4] + S1, bj[5] + S2};
                double d2 = 0;
                for (int r = 0; r < 3; ++r) {
                  const double g1 = jlo[r] - S.ibox[c][3 + r], g2 = S.ibox[c][r] - jhi[r];
                  const double gg = g1 > 0 ? g1 : (g2 > 0 ? g2 : 0.0);
                  d2 += gg * gg;
                }
                if (!(d2 < g.rlist2)) imask &= ~(1u << c);
              }
              have = imask != 0;
            }
            const unsigned ball = __ballot_sync(0xffffffffu, have);
            if (have) {
              const int pos = B.nent + __popc(ball & ((1u << lane) - 1));   // < batch + 32 <= 2 kBatch (flushed below)
              const int sjc = cj >> 3;
              const int h = key_slot(S, excl_key(unsigned(cj), img));
              const int mi = h >= 0 ? S.mbase + S.krank[h] : -1;
              B.ent[pos] = make_uint4(unsigned(cj), imask | (img << 8), mi >= 0 && mi < b.mask_cap ? unsigned(mi + 1) : 0u, 0u);
              B.sh[pos] = make_float4(float(b.sc_org[3 * sjc] + S0 - S.org_i[0]), float(b.sc_org[3 * sjc + 1] + S1 - S.org_i[1]),
                                      float(b.sc_org[3 * sjc + 2] + S2 - S.org_i[2]), 0.f);
            }
            __syncwarp();
            if (lane == 0) B.nent += __popc(ball);
            __syncwarp();
            if (B.nent >= g.batch) {   // a pass adds up to 32 entries: all full work items go together
              const int full = B.nent / g.batch * g.batch, rest = B.nent - full;
              flush_entries(B, sc, full, g.batch, lane, b);
              __syncwarp();
              // the rest (fewer than a work item's, at most 31) moves down: read, then write (the ranges can overlap)
              uint4 te;
              float4 ts;
              if (lane < rest) te = B.ent[full + lane], ts = B.sh[full + lane];
              __syncwarp();
              if (lane < rest) B.ent[lane] = te, B.sh[lane] = ts;
              if (lane == 0) B.nent = rest;
              __syncwarp();
            }
          }
        }
      }
    }
    flush_entries(B, sc, B.nent, g.batch, lane, b);
    __syncthreads();   // S is rewritten for the next super-cluster
  }
}

}  // namespace capsb
