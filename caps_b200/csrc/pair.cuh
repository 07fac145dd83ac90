// K-PAIR: the LJ 12-6 plus real-space Coulomb pair kernels over the cluster pair list.
//
// Reference: the FP64 atom-pair loop (core/src/field.cpp:1604-1686: 12-6 LJ with the cut-off shift, Ewald real space
// from the cubic-Hermite table of erf(kappa sqrt s)/sqrt s, field.cpp:1126-1157 and 1593-1602, DSF) and the FP32
// cluster kernel (core/src/nbnxm.cpp:408-567). Excluded pairs are left out of the list (their Ewald / DSF corrections
// are the bonded-phase kernel's, as the reference's FP64 path does at field.cpp:2206-2266).
//
// One warp per work item: a super-cluster of 64 i atoms (8 clusters, kept in shared memory) against up to 32 j
// clusters. Lane l takes i atom l & 7 of every i cluster and j atoms (l >> 3) and (l >> 3) + 4 of each j cluster, so a
// j cluster costs one 128-byte line and its forces are reduced over 8 lanes once per entry, after all 8 i clusters.
// FP32 path: float arithmetic, positions relative to super-cluster origins (the shift of an entry carries the origins'
// difference, so single precision keeps its digits), forces and energies summed as 64-bit fixed point.
// FP64 path: double arithmetic on wrapped absolute positions, the reference's Hermite table for the Ewald term.
#pragma once
#include "common.cuh"
#include "nblist.cuh"
#include "ewald_fit.cuh"

namespace capsb {

constexpr float kPadFar = 1.0e5f;   // padding slots sit this far from their super-cluster's origin (never within reach)

struct PairArgs {
  const int4* work;
  const uint4* ent;
  const float4* ent_shift;
  const unsigned long long* masks;
  const unsigned long long* frozen;   // a frozen pair set: 8 per entry (one per i cluster), the pairs that interact
  const int* counters;
  const int* tslot;
  const float4* xq;      // FP32 path
  const double4* xqd;    // FP64 path
  const float4* tab;     // FP32: per type pair (c6, c12, energy shift, 0)
  const float2* ljf;     // FP32 with geometric mixing: per type (sqrt c6, sqrt c12)
  int batch;             // entries per work item of the list (<= kBatch): the FP32 kernel's staging per warp
  const double4* tabd;   // FP64: per type pair (c6, c12, energy shift, 0)
  const double4* tabcap; // FP64 with a force cap: per type pair (r_cap^2, E at r_cap, |F| at r_cap, 0)
  const double4* tabg;   // FP64 generic forms (tabd.w the form): per type pair (a, b, c, the pair's own cut-off^2)
  const double4* tabg2;  // and the lj/gromacs switch coefficients
  double lj_inner;
  int lj_fsw;            // FP64: CHARMM's force switch on the 12-6 pairs
  PairTables tables;
  const double4* gcoef;  // FP64 Ewald table: per node the polynomial of its interval (EwaldTab)
  int ntab;              // types incl. the padding type
  int gnodes;            // table nodes
  double ghi;            // 1 / node spacing
  DevCell cell;
  double rc2, rc, beta, kc, kcoul, dsf_e0, dsf_f0;
  long long* fsx;        // slot-order force sums (FP32 path: fixed point)
  long long* fsy;
  long long* fsz;
  double* fdx;           // slot-order force sums (FP64 path)
  double* fdy;
  double* fdz;
  EnergySink en;
  int work_cap;
  int* err;              // the error word (range errors of the fixed-point sums)
};

// Work items are taken dynamically: each warp fetches the next unclaimed item from a device counter (reset by k_list
// before every force evaluation). Items differ in size, so a static split leaves SMs idle at the end of the launch.
// (Asked for before the present item's entries instead, and looked at after them: 113 us against 104 at 32,000 atoms.)
__device__ __forceinline__ int next_work_item(const int* counters, int lane) {
  int w = 0;
  if (lane == 0) w = atomicAdd(const_cast<int*>(counters) + kCntPairNext, 1);
  return __shfl_sync(0xffffffffu, w, 0);
}

// Sums the j forces (a: j atom q, b: j atom q + 4) over the 8 lanes of an i8 group (lanes xor 1, 2, 4): the first level
// swaps halves so that each lane keeps one j atom's three components, the other two are a butterfly. 9 shuffles; lanes
// with i8 < 4 end with a's sums, lanes with i8 >= 4 with b's.
template <class T>
__device__ __forceinline__ void reduce_j(int i8, T ax, T ay, T az, T bx, T by, T bz, T& kx, T& ky, T& kz) {
  const bool hi = (i8 & 4) != 0;
  kx = hi ? bx : ax, ky = hi ? by : ay, kz = hi ? bz : az;
  const T sx = hi ? ax : bx, sy = hi ? ay : by, sz = hi ? az : bz;
  kx += __shfl_xor_sync(0xffffffffu, sx, 4);
  ky += __shfl_xor_sync(0xffffffffu, sy, 4);
  kz += __shfl_xor_sync(0xffffffffu, sz, 4);
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    kx += __shfl_xor_sync(0xffffffffu, kx, o);
    ky += __shfl_xor_sync(0xffffffffu, ky, o);
    kz += __shfl_xor_sync(0xffffffffu, kz, o);
  }
}

// Sums the i forces of the 8 clusters over the 4 lanes of each i atom (lanes xor 8, 16) by halving: 18 shuffles. Lane
// jq ends with clusters jq and jq + 4: out[0..2] = cluster jq (x, y, z), out[3..5] = cluster jq + 4.
template <class T>
__device__ __forceinline__ void reduce_i(int jq, const T fx[8], const T fy[8], const T fz[8], T out[6]) {
  // level xor 16: keep the clusters c with (c & 2) == (jq & 2): c0 in {0, 1, 4, 5} or c0 ^ 2
  const bool b1 = (jq & 2) != 0, b0 = (jq & 1) != 0;
  T h[4][3];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c0 = (k & 1) | ((k & 2) << 1);   // 0, 1, 4, 5
    const int c2 = c0 ^ 2;
    const T kx = b1 ? fx[c2] : fx[c0], ky = b1 ? fy[c2] : fy[c0], kz = b1 ? fz[c2] : fz[c0];
    const T sx = b1 ? fx[c0] : fx[c2], sy = b1 ? fy[c0] : fy[c2], sz = b1 ? fz[c0] : fz[c2];
    h[k][0] = kx + __shfl_xor_sync(0xffffffffu, sx, 16);
    h[k][1] = ky + __shfl_xor_sync(0xffffffffu, sy, 16);
    h[k][2] = kz + __shfl_xor_sync(0xffffffffu, sz, 16);
  }
  // level xor 8: of h[k] (k = 0, 1: clusters (jq & 2) + 0/1; k = 2, 3: the same + 4) keep (c & 1) == (jq & 1)
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int k0 = 2 * m, k1 = 2 * m + 1;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const T kv = b0 ? h[k1][r] : h[k0][r];
      const T sv = b0 ? h[k0][r] : h[k1][r];
      out[3 * m + r] = kv + __shfl_xor_sync(0xffffffffu, sv, 8);
    }
  }
}

// --- FP32 path ---------------------------------------------------------------------------------------------------
// Packed FP32 arithmetic (sm_100 f32x2): a lane's two j atoms of an entry (quarters jq and jq + 4) are the two lanes of
// every add, multiply and multiply-add, so one instruction evaluates both of its pairs with an i atom.
__device__ __forceinline__ float2 p_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 p_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 p_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 p_dup(float v) { return make_float2(v, v); }
// the SFU's approximate 1/sqrt with denormals flushed (squared distances of listed pairs are > 0.01, or 1 for a pair
// left out)
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// COUL: 0 none; 1 Ewald real space (PME) and 2 damped shifted force through the rational fits of ewald_fit.cuh
// (kappa r_c <= 4); 3 and 4 the same through erfcf and expf (any kappa). COMB: the LJ coefficients of a type pair are
// products of per-type factors (geometric mixing: c6_ab = sqrt(c6_aa c6_bb), the same for c12), taken from a
// per-type table instead of the per-pair one. Force-only evaluations only: the products of rounded factors carry a
// bias of a few 1e-7 per type pair, which the cancelling sums of LJ energies would magnify, so energy steps take the
// per-pair table.
template <int COUL, bool ENER, bool VIR, bool LJ96 = false, bool COMB = false>
static __global__ void __launch_bounds__(128, (ENER || VIR) ? 4 : 5) k_pair_f32(PairArgs A) {
  static_assert(!(COMB && ENER), "energy evaluations use the per-pair table");
  extern __shared__ float4 smem_f4[];
  float4* tab = smem_f4;                                  // ntab * ntab (per-pair table; COMB: ntab float2 factors)
  float2* ljf = reinterpret_cast<float2*>(smem_f4);
  // per warp and i atom: (-x, -x, -y, -y), (-z, -z, q, q) and, COMB, (-6 f6, -6 f6, 12 f12, 12 f12); else the type
  float4* s_xi = smem_f4 + A.ntab * A.ntab;               // 4 warps x 64 x 3
  int* s_ti = reinterpret_cast<int*>(s_xi + 4 * 64 * 3);  // 4 warps x 64
  // a work item's entries, their j atoms and their exclusion masks, staged per warp in one batch of independent loads
  // (sized for the list's entries per work item, A.batch <= kBatch)
  const int nb = A.batch;
  uint4* s_en_all = reinterpret_cast<uint4*>(s_ti + 4 * 64);   // 4 warps x nb entries
  float4* s_sh_all = reinterpret_cast<float4*>(s_en_all + 4 * nb);
  // the j atoms of an entry, shifted by its image and packed per lane quarter jq as the lane's operands:
  // (x_jq, x_jq+4, y_jq, y_jq+4), (z_jq, z_jq+4, q_jq, q_jq+4)
  float4* s_xj_all = s_sh_all + 4 * nb;                         // 4 warps x nb entries x 8 float4
  // COMB: the j atoms' LJ factors per quarter, (f6_jq, f6_jq+4, f12_jq, f12_jq+4); else the j atoms' types
  float4* s_gj_all = s_xj_all + 4 * nb * 8;                     // 4 warps x nb entries x 4 float4 (or 8 int)
  unsigned long long* s_mk_all = reinterpret_cast<unsigned long long*>(s_gj_all + 4 * nb * 4);
  if (COMB) {
    for (int t = threadIdx.x; t < A.ntab; t += blockDim.x) ljf[t] = A.ljf[t];
  } else {
    for (int t = threadIdx.x; t < A.ntab * A.ntab; t += blockDim.x) tab[t] = A.tab[t];
  }
  __syncthreads();
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i8 = lane & 7, jq = lane >> 3;
  float4* xi_s = s_xi + 3 * 64 * wib;
  int* ti_s = s_ti + 64 * wib;
  if (blockIdx.x == 0 && threadIdx.x == 0) {   // the step's list work is done: lower the rebuild and prune flags
    int* c = const_cast<int*>(A.counters);
    c[kCntRebuild] = 0;
    c[kCntPrune] = 0;
  }
  // a list build that ran out of room leaves stale work items: skip the pass, the host reports the error
  if (A.counters[kCntErr] & kErrListBad) return;
  const int nwork = min(A.counters[kCntWork], A.work_cap);
  const int pad = A.ntab - 1;
  const float rc2 = float(A.rc2), beta = float(A.beta), kc = float(A.kc), kcoul = float(A.kcoul);
  const float2 ku = p_dup(float(A.beta * A.beta / kEwUMax)), nkap3 = p_dup(-float(A.beta * A.beta * A.beta));
  const float e0 = float(A.dsf_e0), f0 = float(A.dsf_f0), rcf = float(A.rc);
  // energies and virial: every pair's terms rounded to fixed point on their own (2^24 per kcal/mol), so that the totals do
  // not depend on the list's grouping of pairs. The virial's six products and twelve conversions to 64-bit integers per
  // pair of pairs take a seventh of this variant's time (32,000 atoms: 223 us; 194 with a lane's pairs of an entry summed in
  // float first, which drops bits; 214 summed in double, 239 in two floats: no closer to 64 bits, 4.9e-7 of the trace
  // against 4.8e-7 at 33,000 atoms). From the atoms' force sums instead (sum x F, as the FP64 kernel) it is off twice as
  // far: those sums' rounding times positions of 20 Å.
  long long acc_v = 0, acc_c = 0, acc_w[6] = {0, 0, 0, 0, 0, 0};
  double acc_np = 0, acc_nl = 0;
  constexpr float kq = 16777216.f;
  for (int w = next_work_item(A.counters, lane); w < nwork; w = next_work_item(A.counters, lane)) {
    const int4 wk = A.work[w];
    const int sc = wk.x;
    for (int t = lane; t < 64; t += 32) {
      const float4 v = A.xq[64 * sc + t];
      const int ty = A.tslot[64 * sc + t];
      const float q = v.w * kcoul;
      xi_s[3 * t] = make_float4(-v.x, -v.x, -v.y, -v.y);
      xi_s[3 * t + 1] = make_float4(-v.z, -v.z, q, q);
      if (COMB) {
        const float2 g = ljf[ty];
        xi_s[3 * t + 2] = make_float4(-6.f * g.x, -6.f * g.x, 12.f * g.y, 12.f * g.y);
      }
      ti_s[t] = ty;
    }
    __syncwarp();
    // real i atoms of the lane, per i cluster c, in the layout of an entry's prune mask (bit c: the pair with j atom
    // jq, bit c + 8: with jq + 4)
    unsigned ireal = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) ireal |= unsigned(ti_s[8 * c + i8] != pad) << c;
    ireal |= ireal << 8;
    float fix[8], fiy[8], fiz[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) fix[c] = fiy[c] = fiz[c] = 0.f;
    float npair = 0.f, nlist = 0.f;
    uint4* s_en = s_en_all + nb * wib;
    float4* s_sh = s_sh_all + nb * wib;
    float4* s_xj = s_xj_all + nb * 8 * wib;
    float4* s_gj = s_gj_all + nb * 4 * wib;
    int* s_tj = reinterpret_cast<int*>(s_gj);
    unsigned long long* s_mk = s_mk_all + nb * 8 * wib;
    const int ne = min(wk.z, nb);
    if (lane < ne) {
      s_en[lane] = A.ent[wk.y + lane];
      s_sh[lane] = A.ent_shift[wk.y + lane];
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int t = lane + 32 * k;   // entry t / 8, j atom t % 8
      if (t < 8 * ne) {
        const int e = t >> 3, j = t & 7, q4 = j & 3, h = j >> 2;
        const uint4 e4 = s_en[e];
        const float4 sh = s_sh[e];
        const int ja = 8 * int(e4.x) + j;
        const float4 v = A.xq[ja];
        float* px = reinterpret_cast<float*>(s_xj + 8 * e + 2 * q4);
        px[h] = v.x + sh.x;
        px[2 + h] = v.y + sh.y;
        px[4 + h] = v.z + sh.z;
        px[6 + h] = v.w;
        const int ty = A.tslot[ja];
        if (COMB) {
          const float2 g = ljf[ty];
          float* pg = reinterpret_cast<float*>(s_gj + 4 * e + q4);
          pg[h] = g.x;
          pg[2 + h] = g.y;
        } else {
          s_tj[t] = ty;
        }
        s_mk[t] = e4.z ? A.masks[8 * size_t(e4.z - 1) + j] : ~0ull;   // entry t / 8, i cluster t % 8
      }
    }
    __syncwarp();
    for (int el = 0; el < ne; ++el) {
      const uint4 en = s_en[el];
      const unsigned hmask = en.w & 0xffffu;
      if (!hmask) continue;
      const int cj = int(en.x);
      // by a vote, which the compiler knows to be the same in every lane: branches on it need no reconvergence
      const unsigned imask = __ballot_sync(0xffffffffu, ((hmask | (hmask >> 8)) >> (lane & 7)) & 1u) & 255u;
      // the lane's listed pairs of the entry: a j half within the prune radius, a real i atom and, where the entry
      // has exclusion masks, bits jq and jq + 4 of the i atom's row of its cluster's mask
      unsigned lv = hmask & ireal;
      if (en.z) {
        unsigned xm = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const unsigned b = unsigned(s_mk[8 * el + c] >> (8 * i8 + jq));
          xm |= ((b & 1u) << c) | (((b >> 4) & 1u) << (c + 8));
        }
        lv &= xm;
      }
      const int j0 = 8 * cj + jq, j1 = j0 + 4;
      const float4 xa = s_xj[8 * el + 2 * jq], xb = s_xj[8 * el + 2 * jq + 1];
      const float2 xj = make_float2(xa.x, xa.y), yj = make_float2(xa.z, xa.w), zj = make_float2(xb.x, xb.y), qj = make_float2(xb.z, xb.w);
      float2 g6j = p_dup(0.f), g12j = p_dup(0.f);
      int t0 = 0, t1 = 0;
      if (COMB) {
        const float4 gg = s_gj[4 * el + jq];
        g6j = make_float2(gg.x, gg.y);
        g12j = make_float2(gg.z, gg.w);
      } else {
        t0 = s_tj[8 * el + jq];
        t1 = s_tj[8 * el + jq + 4];
      }
      float2 fjx = p_dup(0.f), fjy = p_dup(0.f), fjz = p_dup(0.f);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (!((imask >> c) & 1u)) continue;
        const float4 pa = xi_s[3 * (8 * c + i8)], pb = xi_s[3 * (8 * c + i8) + 1];
        const bool l0 = (lv >> c) & 1u, l1 = (lv >> (c + 8)) & 1u;
        const float2 dx = p_add(xj, make_float2(pa.x, pa.y)), dy = p_add(yj, make_float2(pa.z, pa.w)), dz = p_add(zj, make_float2(pb.x, pb.y));
        const float2 r2 = p_fma(dx, dx, p_fma(dy, dy, p_mul(dz, dz)));
        const bool ok0 = l0 && (r2.x < rc2), ok1 = l1 && (r2.y < rc2);
        if (ENER) {
          npair += float(ok0) + float(ok1);
          nlist += float(l0) + float(l1);
        }
        const float2 r2s = make_float2(ok0 ? r2.x : 1.f, ok1 ? r2.y : 1.f);
        const float2 rinv = make_float2(rsqrt_ftz(r2s.x), rsqrt_ftz(r2s.y));
        const float2 r2i = p_mul(rinv, rinv);
        const float2 r6i = p_mul(p_mul(r2i, r2i), r2i);
        float2 fr, elj;
        if (COMB) {
          const float4 pl = xi_s[3 * (8 * c + i8) + 2];
          const float2 nC6 = p_mul(make_float2(pl.x, pl.y), g6j), C12 = p_mul(make_float2(pl.z, pl.w), g12j);
          fr = p_mul(p_mul(r6i, p_fma(C12, r6i, nC6)), r2i);   // (12 c12 r^-12 - 6 c6 r^-6) / r^2
        } else {
          const int ti = ti_s[8 * c + i8];
          const float4 cc0 = tab[ti * A.ntab + t0], cc1 = tab[ti * A.ntab + t1];
          const float2 c6 = make_float2(cc0.x, cc1.x), c12 = make_float2(cc0.y, cc1.y);
          // 12-6: a = c12 r^-6; 9-6: a = c9 r^-3 (the table's second slot holds c12 or c9): E = r^-6 (a - c6) - shift
          const float2 a12 = p_mul(c12, LJ96 ? p_mul(r2i, rinv) : r6i);
          fr = p_mul(p_mul(r6i, p_fma(p_dup(LJ96 ? 9.f : 12.f), a12, p_mul(p_dup(-6.f), c6))), r2i);
          if (ENER) elj = p_fma(r6i, p_add(a12, p_mul(p_dup(-1.f), c6)), make_float2(-cc0.z, -cc1.z));
        }
        if (ENER) acc_v += (ok0 ? __float2ll_rn(elj.x * kq) : 0ll) + (ok1 ? __float2ll_rn(elj.y * kq) : 0ll);
        if (COUL == 1 || COUL == 2) {
          // E = qq (1/r - kappa g(u)), F = qq (1/r^3 - kappa^3 h(u)), u = (kappa r)^2: FMAs and one division per pair
          const float2 qq = p_mul(make_float2(pb.z, pb.w), qj);
          const float2 t = p_mul(r2s, ku);
          float2 fc = p_mul(qq, p_fma(nkap3, ew_h2(t), p_mul(rinv, r2i)));
          if (COUL == 2) fc = p_fma(p_mul(qq, p_dup(-f0)), rinv, fc);
          fr = p_add(fr, fc);
          if (ENER) {
            float2 ecp = p_mul(qq, p_fma(p_dup(-beta), ew_g2(t), rinv));
            if (COUL == 2) ecp = p_fma(qq, p_fma(p_dup(f0), p_add(p_mul(r2s, rinv), p_dup(-rcf)), p_dup(-e0)), ecp);
            acc_c += (ok0 ? __float2ll_rn(ecp.x * kq) : 0ll) + (ok1 ? __float2ll_rn(ecp.y * kq) : 0ll);
          }
        }
        if (COUL == 3 || COUL == 4) {
          const float2 qq = p_mul(make_float2(pb.z, pb.w), qj);
          const float2 r = p_mul(r2s, rinv);
          float fcs[2], ecs[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float rh = h ? r.y : r.x, ih = h ? rinv.y : rinv.x, qh = h ? qq.y : qq.x;
            const float br = beta * rh;
            const float erfcv = erfcf(br);
            const float ex = __expf(-br * br);
            fcs[h] = qh * fmaf(erfcv, ih, kc * ex) * (ih * ih);
            if (COUL == 4) fcs[h] -= qh * f0 * ih;
            ecs[h] = qh * erfcv * ih;
            if (COUL == 4) ecs[h] += qh * (f0 * (rh - rcf) - e0);
          }
          fr = p_add(fr, make_float2(fcs[0], fcs[1]));
          if (ENER) acc_c += (ok0 ? __float2ll_rn(ecs[0] * kq) : 0ll) + (ok1 ? __float2ll_rn(ecs[1] * kq) : 0ll);
        }
        fr = make_float2(ok0 ? fr.x : 0.f, ok1 ? fr.y : 0.f);
        const float2 fx = p_mul(fr, dx), fy = p_mul(fr, dy), fz = p_mul(fr, dz);
        fjx = p_add(fjx, fx);
        fjy = p_add(fjy, fy);
        fjz = p_add(fjz, fz);
        fix[c] -= fx.x + fx.y;
        fiy[c] -= fy.x + fy.y;
        fiz[c] -= fz.x + fz.y;
        if (VIR) {   // fr is 0 for the pairs left out
          const float2 w6[6] = {p_mul(fx, dx), p_mul(fy, dy), p_mul(fz, dz), p_mul(fx, dy), p_mul(fx, dz), p_mul(fy, dz)};
#pragma unroll
          for (int k = 0; k < 6; ++k) acc_w[k] += __float2ll_rn(w6[k].x * kq) + __float2ll_rn(w6[k].y * kq);
        }
      }
      // j forces: summed over the 8 lanes holding the same j atoms, then one fixed-point add per component
      {
        float kx, ky, kz;
        reduce_j(i8, fjx.x, fjy.x, fjz.x, fjx.y, fjy.y, fjz.y, kx, ky, kz);
        const int comp = i8 & 3;
        if (comp < 3) {
          const float v = comp == 0 ? kx : comp == 1 ? ky : kz;
          long long* dst = comp == 0 ? A.fsx : comp == 1 ? A.fsy : A.fsz;
          if (v != 0.f) fix_add_f(dst + ((i8 & 4) ? j1 : j0), v, A.err);
        }
      }
    }
    // i forces: summed over the 4 lanes of each i atom; lane jq adds clusters jq and jq + 4
    {
      float fo[6];
      reduce_i(jq, fix, fiy, fiz, fo);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int c = jq + 4 * m;
        if (!((ireal >> c) & 1u)) continue;
        const int s = 64 * sc + 8 * c + i8;
        if (fo[3 * m] != 0.f) fix_add_f(A.fsx + s, fo[3 * m], A.err);
        if (fo[3 * m + 1] != 0.f) fix_add_f(A.fsy + s, fo[3 * m + 1], A.err);
        if (fo[3 * m + 2] != 0.f) fix_add_f(A.fsz + s, fo[3 * m + 2], A.err);
      }
    }
    if (ENER) {
      acc_np += double(warp_sum(npair));   // whole numbers: exact in any order
      acc_nl += double(warp_sum(nlist));
    }
    __syncwarp();
  }
  if (ENER) {
    acc_v = warp_sum(acc_v);
    acc_c = warp_sum(acc_c);
  }
  if (VIR)
    for (int k = 0; k < 6; ++k) acc_w[k] = warp_sum(acc_w[k]);
  if (lane == 0) {
    if (ENER) {
      atomic_add_fix(A.en.fix + kEVdw, acc_v);
      atomic_add_fix(A.en.fix + kECoul, acc_c);
      A.en.add(kEPairs, acc_np, true);
      A.en.add(kEListed, acc_nl, true);
    }
    if (VIR)
      for (int k = 0; k < 6; ++k) atomic_add_fix(A.en.fix + kEW0 + k, acc_w[k]);
  }
}

// --- FP64 path ---------------------------------------------------------------------------------------------------

// The reference's ewald_ef (field.cpp:1593-1602): E = 1/r - G(s), F = 1/r^3 + 2 dG/ds by cubic Hermite interpolation of G
// over nodes of spacing h. The interpolant is held as its polynomial in t = s/h - k, c[k] = (a1, a2, a3, G_k) with
// 2 dG/ds = a1 + t (a2 + t a3): a force takes three loads and two multiply-adds.
struct EwaldTab {
  const double4* c;
  double ghi, hh;   // 1 / h, h / 2
};
__device__ __forceinline__ int ewald_node(double u, double& t) {   // node and offset of u = s / h in [0, 2^31)
  const double m = (u - 0.5) + 6755399441055744.0;   // 1.5 2^52: the sum's low word is u - 1/2 rounded to an integer
  t = u - (m - 6755399441055744.0);                  // in [0, 1] (a tie may take either end)
  return __double2loint(m);
}
template <bool ENER>
__device__ __forceinline__ double ewald_f(const EwaldTab& T, double s, double& G) {
  double t;
  const double4* c = T.c + ewald_node(s * T.ghi, t);
  const double2 a = *reinterpret_cast<const double2*>(c);
  if (ENER) {
    const double2 g = *(reinterpret_cast<const double2*>(c) + 1);
    G = g.y + t * T.hh * (a.x + t * (0.5 * a.y + t * (g.x * (1.0 / 3.0))));
    return a.x + t * (a.y + t * g.x);
  }
  return a.x + t * (a.y + t * c->z);
}

// 1/sqrt(x) and 1/x in double from the hardware's 20-bit estimate y: with e = 1 - x y^2, y (1 + e/2 + 3 e^2/8) is off by
// 5 e^3 / 16 < 2^-58, and its square is corrected once. x is a squared distance, neither 0 nor denormal.
__device__ __forceinline__ double rsqrt_sq(double x, double& inv) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  y = fma(y * e, fma(e, 0.375, 0.5), y);
  inv = y * y;
  inv = fma(inv, fma(-x, inv, 1.0), inv);
  return y;
}

// erfc(x) and exp(-x^2) by Abramowitz & Stegun 7.1.26, the reference's erfc_exp (field.cpp:585-590): the closed form a
// frozen pair takes beyond the cut-off, where the Ewald table ends.
__device__ __forceinline__ double erfc_exp_as(double x, double& ex2) {
  const double P = 0.3275911, A1 = 0.254829592, A2 = -0.284496736, A3 = 1.421413741, A4 = -1.453152027, A5 = 1.061405429;
  ex2 = exp(-x * x);
  const double t = 1.0 / (1.0 + P * x);
  return t * (A1 + t * (A2 + t * (A3 + t * (A4 + t * A5)))) * ex2;
}

// One pair at squared distance r2 of types (ti, tj): |F| / r, energies added to ev and ec.
// FROZEN: a pair of the frozen set beyond the cut-off takes the closed-form Coulomb term (field.cpp:1759-1768).
// CAP: the rare forms' variant (the push-off force cap, the generic pair forms, CHARMM's force switch), taken with energies
// and virial on; the plain variants carry none of their branches.
template <int COUL, bool ENER, bool CAP, bool LJ96, bool FROZEN>
__device__ __forceinline__ double pair_f64(const PairArgs& A, const EwaldTab& T, const double4* tab, int tt, double r2, double qq, double& ev, double& ec) {
  double r2i;
  const double rinv = rsqrt_sq(r2, r2i);
  const double r6i = r2i * r2i * r2i;
  const double2 c = *reinterpret_cast<const double2*>(tab + tt);
  double fr;
  const double4 cc = (ENER || CAP || FROZEN) ? tab[tt] : make_double4(c.x, c.y, 0, 0);
  const double4 cp = CAP ? A.tabcap[tt] : make_double4(0, 0, 0, 0);
  if (CAP && r2 < cp.x) {
    // the push-off cap (field.cpp:1534-1538): LJ continued linearly inside the radius where |F| reaches the cap
    fr = cp.z * rinv;   // F / r with |F| = the cap
    if (ENER) ev += cp.y + cp.z * (sqrt(cp.x) - r2 * rinv) - cc.z;
  } else if ((CAP || FROZEN) && cc.w != 0) {
    // a generic form (field.cpp:1381-1396), nothing beyond the pair's own cut-off (and no shift there)
    const double4 g = A.tabg[tt];
    double e = 0;
    fr = (g.w > 0 && r2 > g.w) ? 0.0 : generic_pair(int(cc.w), g, A.tabg2[tt], A.lj_inner, A.tables, r2, e);
    if (ENER && !(g.w > 0 && r2 > g.w)) ev += e - cc.z;
  } else if (LJ96) {   // field.cpp:1658-1661
    const double r9i = r6i * r2i * rinv;
    fr = (9 * cc.y * r9i - 6 * cc.x * r6i) * r2i;
    if (ENER) ev += cc.y * r9i - cc.x * r6i - cc.z;
  } else if ((CAP || FROZEN) && A.lj_fsw) {
    fr = charmm_fsw(cc.y, cc.x, A.lj_inner, A.rc, r2, ev, ENER);
  } else {
    fr = r6i * (12 * cc.y * r6i - 6 * cc.x) * r2i;
    if (ENER) ev += r6i * (cc.y * r6i - cc.x) - cc.z;
  }
  if (COUL != 0 && FROZEN && !(r2 < A.rc2)) {
    const double r = sqrt(r2);
    double ex2;
    const double er = erfc_exp_as(A.beta * r, ex2);   // beta: the Ewald or DSF coefficient; kc = 2 beta / sqrt(pi)
    if (COUL == 1) {
      if (ENER) ec += qq * er / r;
      fr += qq * (er / r2 + A.kc * ex2 / r) / r;
    } else {
      if (ENER) ec += qq * (er / r - A.dsf_e0 + A.dsf_f0 * (r - A.rc));
      fr += qq * (er / r2 + A.kc * ex2 / r - A.dsf_f0) / r;
    }
  } else if (COUL != 0) {
    double G = 0;
    const double Fc = fma(rinv, r2i, ewald_f<ENER>(T, r2, G));
    if (COUL == 1) {
      if (ENER) ec += qq * (rinv - G);
      fr += qq * Fc;
    } else {
      if (ENER) ec += qq * (rinv - G - A.dsf_e0 + A.dsf_f0 * (r2 * rinv - A.rc));
      fr += qq * (Fc - A.dsf_f0 * rinv);
    }
  }
  return fr;
}

// The FP64 pair kernel, staged as the FP32 one: a work item's i atoms, entries, shifted j atoms and exclusion masks by one
// batch of loads into shared memory, a lane's pairs of an entry in one 16-bit word, and both of the lane's j atoms of an
// entry evaluated side by side, so that two independent chains of FP64 operations fill the pipe's latency. FROZEN: the
// pairs are those of the frozen set (A.frozen), whatever their distance now (field.cpp:1700).
// Bound by its dependent chains: 46 double operations per pair (a division and a square root made it 75) with three blocks,
// 11 warps, per SM keep the FP64 pipe 37 % busy and 47 % of the issue slots (32,000 atoms, 176 us); the stalls are fixed-latency
// waits, shared memory and the work items' loads. The rare variants keep the loop over the i clusters rolled: sixteen copies of
// their pair code missed the instruction cache (a force cap at 32,000 atoms 518 us a launch unrolled, 297 rolled, i forces in
// local memory and all; frozen pairs 595 and 269). GSM: the Ewald table in shared memory (else read through L1, for tables too large for it).
template <int COUL, bool ENER, bool VIR, bool CAP = false, bool LJ96 = false, bool FROZEN = false, bool GSM = true>
static __global__ void __launch_bounds__(128, 3) k_pair_f64(PairArgs A) {
  extern __shared__ double4 smem_d4[];
  const int nb = A.batch;
  double4* tab = smem_d4;                                            // ntab * ntab
  double4* gt = tab + A.ntab * A.ntab;                               // gnodes with Coulomb, none without (as the launch sizes it)
  double4* s_xi_all = gt + (COUL != 0 && GSM ? A.gnodes : 0);        // 4 warps x 64
  double4* s_xj_all = s_xi_all + 4 * 64;                             // 4 warps x nb entries x 8, shifted by the entry's image
  unsigned long long* s_mk_all = reinterpret_cast<unsigned long long*>(s_xj_all + 4 * nb * 8);   // 4 warps x nb x 8
  uint4* s_en_all = reinterpret_cast<uint4*>(s_mk_all + 4 * nb * 8); // 4 warps x nb entries
  int* s_ti_all = reinterpret_cast<int*>(s_en_all + 4 * nb);         // 4 warps x 64, a type's row in tab
  int* s_tj_all = s_ti_all + 4 * 64;                                 // 4 warps x nb x 8
  for (int t = threadIdx.x; t < A.ntab * A.ntab; t += blockDim.x) tab[t] = A.tabd[t];
  if (COUL != 0 && GSM)
    for (int t = threadIdx.x; t < A.gnodes; t += blockDim.x) gt[t] = A.gcoef[t];
  __syncthreads();
  const EwaldTab T{COUL != 0 && GSM ? gt : A.gcoef, A.ghi, 0.5 / A.ghi};
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i8 = lane & 7, jq = lane >> 3;
  double4* xi_s = s_xi_all + 64 * wib;
  double4* xj_s = s_xj_all + 8 * nb * wib;
  unsigned long long* mk_s = s_mk_all + 8 * nb * wib;
  uint4* en_s = s_en_all + nb * wib;
  int* ti_s = s_ti_all + 64 * wib;
  int* tj_s = s_tj_all + 8 * nb * wib;
  if (blockIdx.x == 0 && threadIdx.x == 0) {   // the step's list work is done: lower the rebuild and prune flags
    int* c = const_cast<int*>(A.counters);
    c[kCntRebuild] = 0;
    c[kCntPrune] = 0;
  }
  if (A.counters[kCntErr] & kErrListBad) return;
  const int nwork = min(A.counters[kCntWork], A.work_cap);
  const int pad = A.ntab - 1;
  // energies; virial: sum of d F over a work item's pairs, d = x_j - x_i, as sum x_j F_j + sum x_i F_i over its atoms with
  // the force sums the kernel has anyway (positions from the first i atom)
  double acc_v = 0, acc_c = 0, acc_w[6] = {0, 0, 0, 0, 0, 0}, acc_wj[2] = {0, 0};
  for (int w = next_work_item(A.counters, lane); w < nwork; w = next_work_item(A.counters, lane)) {
    const int4 wk = A.work[w];
    const int sc = wk.x;
    const int ne = min(wk.z, nb);
    if (lane < ne) en_s[lane] = A.ent[wk.y + lane];
    for (int t = lane; t < 64; t += 32) {
      double4 v = A.xqd[64 * sc + t];
      v.w *= A.kcoul;
      xi_s[t] = v;
      ti_s[t] = A.tslot[64 * sc + t] * A.ntab;
    }
    __syncwarp();
    for (int t = lane; t < 8 * ne; t += 32) {   // entry t / 8, j atom (and i cluster of the mask) t % 8
      const uint4 en = en_s[t >> 3];
      int qa, qb, qc;
      unpack_image(en.y >> 8, qa, qb, qc);
      const int ja = 8 * int(en.x) + (t & 7);
      double4 v = A.xqd[ja];
      v.x += A.cell.h[0][0] * qa + A.cell.h[0][1] * qb + A.cell.h[0][2] * qc;
      v.y += A.cell.h[1][0] * qa + A.cell.h[1][1] * qb + A.cell.h[1][2] * qc;
      v.z += A.cell.h[2][0] * qa + A.cell.h[2][1] * qb + A.cell.h[2][2] * qc;
      xj_s[t] = v;
      tj_s[t] = A.tslot[ja];
      mk_s[t] = FROZEN ? A.frozen[8 * size_t(wk.y) + t] : en.z ? A.masks[8 * size_t(en.z - 1) + (t & 7)] : ~0ull;
    }
    unsigned ireal = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) ireal |= unsigned(ti_s[8 * c + i8] != pad * A.ntab) << c;
    ireal |= ireal << 8;
    double fix[8], fiy[8], fiz[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) fix[c] = fiy[c] = fiz[c] = 0.0;
    double ev = 0, ec = 0;
    __syncwarp();
    for (int el = 0; el < ne; ++el) {
      const uint4 en = en_s[el];
      const unsigned hmask = en.w & 0xffffu;
      if (!hmask) continue;
      const unsigned imask = __ballot_sync(0xffffffffu, ((hmask | (hmask >> 8)) >> (lane & 7)) & 1u) & 255u;   // uniform branches
      // the lane's listed pairs of the entry (as the FP32 kernel)
      unsigned lv = hmask & ireal;
      if (FROZEN || en.z) {
        unsigned xm = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const unsigned b = unsigned(mk_s[8 * el + c] >> (8 * i8 + jq));
          xm |= ((b & 1u) << c) | (((b >> 4) & 1u) << (c + 8));
        }
        lv &= xm;
      }
      const double4 a0 = xj_s[8 * el + jq], a1 = xj_s[8 * el + jq + 4];
      const int t0 = tj_s[8 * el + jq], t1 = tj_s[8 * el + jq + 4];
      double f0x = 0, f0y = 0, f0z = 0, f1x = 0, f1y = 0, f1z = 0;
      // i clusters in a turn (two loops, not an unroll count on one: with that the plain variants took 177.6 us, not 175.6)
      constexpr int kTurn = CAP || FROZEN ? 1 : 8;
#pragma unroll 1
      for (int c0 = 0; c0 < 8; c0 += kTurn)
#pragma unroll
      for (int c = c0; c < c0 + kTurn; ++c) {
        if (!((imask >> c) & 1u)) continue;
        const double4 xi = xi_s[8 * c + i8];
        const int ti = ti_s[8 * c + i8];
        const double dx0 = a0.x - xi.x, dy0 = a0.y - xi.y, dz0 = a0.z - xi.z;
        const double dx1 = a1.x - xi.x, dy1 = a1.y - xi.y, dz1 = a1.z - xi.z;
        const double r20 = dx0 * dx0 + dy0 * dy0 + dz0 * dz0, r21 = dx1 * dx1 + dy1 * dy1 + dz1 * dz1;
        const bool ok0 = ((lv >> c) & 1u) && (FROZEN || r20 < A.rc2), ok1 = ((lv >> (c + 8)) & 1u) && (FROZEN || r21 < A.rc2);
        if (!__any_sync(0xffffffffu, ok0 || ok1)) continue;
        double e0 = 0, e1 = 0, q0 = 0, q1 = 0;
        double fr0 = 0, fr1 = 0;
        if (CAP || FROZEN) {   // the rare variants branch within a pair: a pair at a time
          if (ok0) fr0 = pair_f64<COUL, ENER, CAP, LJ96, FROZEN>(A, T, tab, ti + t0, r20, xi.w * a0.w, e0, q0);
          if (ok1) fr1 = pair_f64<COUL, ENER, CAP, LJ96, FROZEN>(A, T, tab, ti + t1, r21, xi.w * a1.w, e1, q1);
        } else {               // a pair left out is evaluated at a distance inside the table and dropped
          fr0 = pair_f64<COUL, ENER, CAP, LJ96, FROZEN>(A, T, tab, ti + t0, ok0 ? r20 : 0.5 * A.rc2, xi.w * a0.w, e0, q0);
          fr1 = pair_f64<COUL, ENER, CAP, LJ96, FROZEN>(A, T, tab, ti + t1, ok1 ? r21 : 0.5 * A.rc2, xi.w * a1.w, e1, q1);
          fr0 = ok0 ? fr0 : 0.0, fr1 = ok1 ? fr1 : 0.0;
        }
        if (ENER) {
          ev += (ok0 ? e0 : 0.0) + (ok1 ? e1 : 0.0);
          ec += (ok0 ? q0 : 0.0) + (ok1 ? q1 : 0.0);
        }
        // a padding slot's separation may overflow a product, never reach a sum
        const double fx0 = ok0 ? fr0 * dx0 : 0.0, fy0 = ok0 ? fr0 * dy0 : 0.0, fz0 = ok0 ? fr0 * dz0 : 0.0;
        const double fx1 = ok1 ? fr1 * dx1 : 0.0, fy1 = ok1 ? fr1 * dy1 : 0.0, fz1 = ok1 ? fr1 * dz1 : 0.0;
        f0x += fx0, f0y += fy0, f0z += fz0;
        f1x += fx1, f1y += fy1, f1z += fz1;
        fix[c] -= fx0 + fx1;
        fiy[c] -= fy0 + fy1;
        fiz[c] -= fz0 + fz1;
      }
      {
        double kx, ky, kz;
        reduce_j(i8, f0x, f0y, f0z, f1x, f1y, f1z, kx, ky, kz);
        const int comp = i8 & 3;
        if (comp < 3) {
          const double v = comp == 0 ? kx : comp == 1 ? ky : kz;
          double* dst = comp == 0 ? A.fdx : comp == 1 ? A.fdy : A.fdz;
          if (v != 0.0) atomicAdd(dst + 8 * int(en.x) + jq + (i8 & 4), v);
          if (VIR) {   // not for v alone: the lane's second product is another component's, and v may be exactly zero
            const double4 a = xj_s[8 * el + jq + (i8 & 4)], r = xi_s[0];
            acc_wj[0] += (comp == 0 ? a.x - r.x : comp == 1 ? a.y - r.y : a.z - r.z) * v;
            acc_wj[1] += (comp == 1 ? a.y - r.y : a.x - r.x) * (comp == 0 ? ky : kz);
          }
        }
      }
    }
    {
      double fo[6];
      reduce_i(jq, fix, fiy, fiz, fo);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int c = jq + 4 * m;
        if (!((ireal >> c) & 1u)) continue;
        const int s = 64 * sc + 8 * c + i8;
        if (fo[3 * m] != 0.0) atomicAdd(A.fdx + s, fo[3 * m]);
        if (fo[3 * m + 1] != 0.0) atomicAdd(A.fdy + s, fo[3 * m + 1]);
        if (fo[3 * m + 2] != 0.0) atomicAdd(A.fdz + s, fo[3 * m + 2]);
        if (VIR) {
          const double4 x = xi_s[8 * c + i8], r = xi_s[0];
          const double px = x.x - r.x, py = x.y - r.y, pz = x.z - r.z;
          acc_w[0] += px * fo[3 * m];
          acc_w[1] += py * fo[3 * m + 1];
          acc_w[2] += pz * fo[3 * m + 2];
          acc_w[3] += px * fo[3 * m + 1];
          acc_w[4] += px * fo[3 * m + 2];
          acc_w[5] += py * fo[3 * m + 2];
        }
      }
    }
    acc_v += ev;
    acc_c += ec;
    __syncwarp();
  }
  if (ENER) {
    acc_v = warp_sum(acc_v);
    acc_c = warp_sum(acc_c);
  }
  if (VIR) {
    const int comp = i8 & 3;
    if (comp < 3) {
      acc_w[0] += comp == 0 ? acc_wj[0] : 0, acc_w[1] += comp == 1 ? acc_wj[0] : 0, acc_w[2] += comp == 2 ? acc_wj[0] : 0;
      acc_w[3] += comp == 0 ? acc_wj[1] : 0, acc_w[5] += comp == 1 ? acc_wj[1] : 0, acc_w[4] += comp == 2 ? acc_wj[1] : 0;
    }
    for (int k = 0; k < 6; ++k) acc_w[k] = warp_sum(acc_w[k]);
  }
  if (lane == 0) {
    if (ENER) {
      A.en.add(kEVdw, acc_v, false);
      A.en.add(kECoul, acc_c, false);
    }
    if (VIR)
      for (int k = 0; k < 6; ++k) A.en.add(kEW0 + k, acc_w[k], false);
  }
}

// K-FREEZE: the frozen pair set of Evaluator::freeze_pairs (field.cpp:2541-2559) on the FP64 path: per entry and i
// cluster the 64 atom pairs that are listed, real, not excluded and inside r_c at the packed positions; the entry's
// half mask becomes their union, so that the pair kernel visits exactly those halves. One thread per entry.
static __global__ void __launch_bounds__(128) k_freeze(PairArgs A, uint4* __restrict__ ent, unsigned long long* __restrict__ frozen) {
  if (A.counters[kCntErr] & kErrListBad) return;
  const int nwork = min(A.counters[kCntWork], A.work_cap);
  const int pad = A.ntab - 1;
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nwork; w += nwarps) {
    const int4 wk = A.work[w];
    for (int e = wk.y + lane; e < wk.y + wk.z; e += 32) {
      uint4 en = ent[e];
      int qa, qb, qc;
      unpack_image(en.y >> 8, qa, qb, qc);
      const double Sx = A.cell.h[0][0] * qa + A.cell.h[0][1] * qb + A.cell.h[0][2] * qc;
      const double Sy = A.cell.h[1][0] * qa + A.cell.h[1][1] * qb + A.cell.h[1][2] * qc;
      const double Sz = A.cell.h[2][0] * qa + A.cell.h[2][1] * qb + A.cell.h[2][2] * qc;
      const unsigned built = en.y & 255u;
      unsigned keep = 0;
      for (int c = 0; c < 8; ++c) {
        unsigned long long m = 0;
        if ((built >> c) & 1u) {
          const unsigned long long mm = en.z ? A.masks[8 * size_t(en.z - 1) + c] : ~0ull;
          for (int i8 = 0; i8 < 8; ++i8) {
            const int si = 64 * wk.x + 8 * c + i8;
            if (A.tslot[si] == pad) continue;
            const double4 xi = A.xqd[si];
            const double xs = xi.x - Sx, ys = xi.y - Sy, zs = xi.z - Sz;
            for (int jl = 0; jl < 8; ++jl) {
              const int bit = 8 * i8 + jl;
              const int sj = 8 * int(en.x) + jl;
              if (!((mm >> bit) & 1ull) || A.tslot[sj] == pad) continue;
              const double4 aj = A.xqd[sj];
              const double dx = aj.x - xs, dy = aj.y - ys, dz = aj.z - zs;
              if (dx * dx + dy * dy + dz * dz < A.rc2) m |= 1ull << bit;
            }
          }
        }
        frozen[8 * size_t(e) + c] = m;
        if (m & 0x0f0f0f0f0f0f0f0full) keep |= 1u << c;         // j atoms 0-3: the lower half
        if (m & 0xf0f0f0f0f0f0f0f0ull) keep |= 1u << (c + 8);   // j atoms 4-7: the upper half
      }
      en.w = keep;
      ent[e] = en;
    }
  }
}

// K-COUNT-PAIRS: the atom pairs of the list within r_list = r_c + skin at the positions of its build (x0), real and not
// excluded, each unordered pair once: Evaluator::pairs() of the reference's FP64 atom-pair list (field.cpp:1030-1049).
static __global__ void __launch_bounds__(128) k_count_pairs(PairArgs A, const uint4* __restrict__ ent, const int* __restrict__ perm,
                                                           const double* __restrict__ x0, const int* __restrict__ ioff, double rl2,
                                                           unsigned long long* __restrict__ out) {
  if (A.counters[kCntErr] & kErrListBad) return;
  const int nwork = min(A.counters[kCntWork], A.work_cap);
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long cnt = 0;
  auto pos = [&](int a, double p[3]) {
    const int o0 = ioff[3 * a], o1 = ioff[3 * a + 1], o2 = ioff[3 * a + 2];
    for (int r = 0; r < 3; ++r) p[r] = x0[3 * a + r] + (A.cell.h[r][0] * o0 + A.cell.h[r][1] * o1 + A.cell.h[r][2] * o2);
  };
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nwork; w += nwarps) {
    const int4 wk = A.work[w];
    for (int e = wk.y + lane; e < wk.y + wk.z; e += 32) {
      const uint4 en = ent[e];
      int qa, qb, qc;
      unpack_image(en.y >> 8, qa, qb, qc);
      const double S[3] = {A.cell.h[0][0] * qa + A.cell.h[0][1] * qb + A.cell.h[0][2] * qc, A.cell.h[1][0] * qa + A.cell.h[1][1] * qb + A.cell.h[1][2] * qc,
                           A.cell.h[2][0] * qa + A.cell.h[2][1] * qb + A.cell.h[2][2] * qc};
      const unsigned built = en.y & 255u;
      for (int c = 0; c < 8; ++c) {
        if (!((built >> c) & 1u)) continue;
        const unsigned long long mm = en.z ? A.masks[8 * size_t(en.z - 1) + c] : ~0ull;
        for (int i8 = 0; i8 < 8; ++i8) {
          const int ai = perm[64 * wk.x + 8 * c + i8];
          if (ai < 0) continue;
          double pi[3];
          pos(ai, pi);
          for (int jl = 0; jl < 8; ++jl) {
            const int aj = perm[8 * int(en.x) + jl];
            if (aj < 0 || !((mm >> (8 * i8 + jl)) & 1ull)) continue;
            double pj[3];
            pos(aj, pj);
            const double dx = pj[0] - (pi[0] - S[0]), dy = pj[1] - (pi[1] - S[1]), dz = pj[2] - (pi[2] - S[2]);
            cnt += dx * dx + dy * dy + dz * dz < rl2 ? 1 : 0;
          }
        }
      }
    }
  }
  if (cnt) atomicAdd(out, cnt);
}

}  // namespace capsb
