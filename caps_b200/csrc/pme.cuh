// PME on the device: order-p cardinal B-spline spreading, the 3-D FFT of the real charge grid (half spectrum along
// the first axis), the influence function with energy and virial, the inverse transform and the force gather.
// Reference: core/src/kspace.cpp:80-175 (the stage pipeline) over core/fortran/caps_kspace.f90: bspline :568-598,
// splines and grid indices :776-796, spreading :800-822, the half-spectrum influence function with Nyquist averaging
// (green :518-564, applied with e_m doubled for interior m1 at :943-962), gather :965-992. The grid layout and index
// convention are the reference's: g(a, b, c) at a + K1 (b + K2 c), and theta(a) weighs grid point floor(u) - p + a.
//
// Precision: the FP64 path is double throughout. The mixed path spreads in FP32 arithmetic into an exact fixed-point
// grid, transforms, solves and gathers in FP32 arithmetic (twiddles and butterfly constants computed in double and rounded
// once).
//
// Kernels: K-SPREAD (an atom's splines by one thread, its grid points by a group of lanes along x), K-GATHER, K-FFT-X
// (pairs of real lines as one complex line, to half spectra), K-FFT-Y, K-FFT-Z+SOLVE (forward z transform, G multiply with
// energy/virial, inverse z transform, fused in one pass over the grid), K-FFT-Y inverse, K-FFT-X inverse (half spectra to
// pairs of real lines). Each line transform is a Stockham autosort FFT of two or three passes: butterflies of radix up to
// 16 in registers, the first pass straight from global memory, one exchange through shared memory per pass. These kernels
// are bound by latency (a 70^3 grid is 1.4 MB of half spectrum), so fewer passes and exchanges per line, not fewer bytes,
// are what counts.
#pragma once
#include "pme_types.cuh"

namespace capsb {

// cos and sin of 2 pi e / n in double, at compile time (Taylor series after reduction to [-pi, pi]).
constexpr double tw_series(double x, bool sine) {
  double term = sine ? x : 1.0, sum = term;
  for (int k = 1; k < 24; ++k) {
    term *= -x * x / (sine ? (2.0 * k) * (2.0 * k + 1.0) : (2.0 * k - 1.0) * (2.0 * k));
    sum += term;
  }
  return sum;
}
constexpr double tw_angle(int e, int n) {
  const int r = ((e % n) + n) % n;
  return 2.0 * kPi * double(2 * r > n ? r - n : r) / double(n);
}
template <class R, int N, int E>
struct TwConst {   // exp(-2 pi i E / N)
  static constexpr double c = tw_series(tw_angle(E, N), false), s = -tw_series(tw_angle(E, N), true);
};

// The forward DFT of N values in registers: o_m = sum_k v_k exp(-2 pi i m k / N).
template <class T, int N>
struct Dft;
template <class T>
struct Dft<T, 1> {
  static __device__ __forceinline__ void run(T*) {}
};
template <class T>
struct Dft<T, 2> {
  static __device__ __forceinline__ void run(T* v) {
    const T a = v[0], b = v[1];
    v[0] = cadd(a, b), v[1] = csub(a, b);
  }
};
template <class T>
struct Dft<T, 4> {
  static __device__ __forceinline__ void run(T* v) {
    const T s0 = cadd(v[0], v[2]), s1 = csub(v[0], v[2]), s2 = cadd(v[1], v[3]), s3 = csub(v[1], v[3]);
    const T is3 = {s3.y, -s3.x};   // -i s3
    v[0] = cadd(s0, s2), v[2] = csub(s0, s2);
    v[1] = cadd(s1, is3), v[3] = csub(s1, is3);
  }
};
// odd prime lengths: the sums and differences of v_k and v_(N-k) against real constants
template <class T, int N, int M, int K>
struct OddTerm {
  static __device__ __forceinline__ void run(const T* s, const T* d, T& re, T& im) {
    using R = decltype(T::x);
    constexpr R c = R(TwConst<R, N, M * K>::c), q = R(TwConst<R, N, M * K>::s);
    re.x += c * s[K].x, re.y += c * s[K].y;
    im.x -= q * d[K].y, im.y += q * d[K].x;   // i q d
    if constexpr (K < (N - 1) / 2) OddTerm<T, N, M, K + 1>::run(s, d, re, im);
  }
};
template <class T, int N, int M>
struct OddOut {
  static __device__ __forceinline__ void run(const T* s, const T* d, T v0, T* o) {
    T re = v0, im = {0, 0};
    OddTerm<T, N, M, 1>::run(s, d, re, im);
    o[M] = cadd(re, im);
    o[N - M] = csub(re, im);
    if constexpr (M < (N - 1) / 2) OddOut<T, N, M + 1>::run(s, d, v0, o);
  }
};
template <class T, int N>
struct DftOdd {
  static __device__ __forceinline__ void run(T* v) {
    constexpr int H = (N - 1) / 2;
    T s[H + 1], d[H + 1], o[N], sum = v[0];
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      s[k] = cadd(v[k], v[N - k]), d[k] = csub(v[k], v[N - k]);
      sum = cadd(sum, s[k]);
    }
    o[0] = sum;
    OddOut<T, N, 1>::run(s, d, v[0], o);
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = o[k];
  }
};
template <class T> struct Dft<T, 3> : DftOdd<T, 3> {};
template <class T> struct Dft<T, 5> : DftOdd<T, 5> {};
template <class T> struct Dft<T, 7> : DftOdd<T, 7> {};
// N = A B: B transforms of length A over the stride B, twiddles, A transforms of length B
template <class T, int N, int A, int B, int I, int J>
struct SplitTw {
  static __device__ __forceinline__ void run(T (&u)[B][A]) {
    using R = decltype(T::x);
    if constexpr (I * J != 0) {
      constexpr R c = R(TwConst<R, N, I * J>::c), q = R(TwConst<R, N, I * J>::s);
      u[J][I] = cmul(u[J][I], T{c, q});
    }
    if constexpr (I + 1 < A) SplitTw<T, N, A, B, I + 1, J>::run(u);
    else if constexpr (J + 1 < B) SplitTw<T, N, A, B, 0, J + 1>::run(u);
  }
};
template <class T, int A, int B>
struct DftSplit {
  static __device__ __forceinline__ void run(T* v) {
    T u[B][A];
#pragma unroll
    for (int b = 0; b < B; ++b) {
#pragma unroll
      for (int a = 0; a < A; ++a) u[b][a] = v[B * a + b];
      Dft<T, A>::run(u[b]);
    }
    SplitTw<T, A * B, A, B, 0, 0>::run(u);
#pragma unroll
    for (int a = 0; a < A; ++a) {
      T w[B];
#pragma unroll
      for (int b = 0; b < B; ++b) w[b] = u[b][a];
      Dft<T, B>::run(w);
#pragma unroll
      for (int b = 0; b < B; ++b) v[a + A * b] = w[b];
    }
  }
};
template <class T> struct Dft<T, 6> : DftSplit<T, 3, 2> {};
template <class T> struct Dft<T, 8> : DftSplit<T, 4, 2> {};
template <class T> struct Dft<T, 9> : DftSplit<T, 3, 3> {};
template <class T> struct Dft<T, 10> : DftSplit<T, 5, 2> {};
template <class T> struct Dft<T, 12> : DftSplit<T, 4, 3> {};
template <class T> struct Dft<T, 16> : DftSplit<T, 4, 4> {};

// A block's lines in shared memory: element i of line l at l ls + i is. LFAST: consecutive threads take consecutive lines
// (y and z, whose rows in global memory run across the lines), 1 << lsh lines to the block; else consecutive elements (x).
struct LineBuf {
  int nl, ls, is, lsh;
};

// One radix-RAD Stockham pass (pass p of plan P): butterfly j of line l takes elements j + r nb, from `load(l, i)`, and
// leaves element (j - k) RAD + k + r ns, k = j mod ns, in `out`.
template <class T, int RAD, bool LFAST, class R, class LOAD>
__device__ __forceinline__ void fft_pass(const LOAD& load, T* __restrict__ out, const T* __restrict__ tw, const FftPlan<R>& P, int p, const LineBuf& B) {
  const int nb = P.nb[p], ns = P.ns[p], stride = nb / ns;   // n / (ns RAD)
  const int total = LFAST ? nb << B.lsh : nb * B.nl;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    int l, j;
    if (LFAST) {
      l = t & ((1 << B.lsh) - 1), j = t >> B.lsh;
      if (l >= B.nl) continue;
    } else {
      l = div_by(t, P.m_nb[p]);
      j = t - l * nb;
    }
    const int k = j - div_by(j, P.m_ns[p]) * ns;
    T v[RAD];
#pragma unroll
    for (int r = 0; r < RAD; ++r) v[r] = load(l, j + r * nb);
    if (ns > 1) {
#pragma unroll
      for (int r = 1; r < RAD; ++r) v[r] = cmul(v[r], tw[r * k * stride]);
    }
    Dft<T, RAD>::run(v);
    T* dst = out + l * B.ls + ((j - k) * RAD + k) * B.is;
#pragma unroll
    for (int r = 0; r < RAD; ++r) dst[r * ns * B.is] = v[r];
  }
}
template <class T, bool LFAST, class R, class LOAD>
__device__ __forceinline__ void fft_pass_any(const LOAD& load, T* out, const T* tw, const FftPlan<R>& P, int p, const LineBuf& B) {
  switch (P.rad[p]) {
    case 2: fft_pass<T, 2, LFAST>(load, out, tw, P, p, B); break;
    case 3: fft_pass<T, 3, LFAST>(load, out, tw, P, p, B); break;
    case 4: fft_pass<T, 4, LFAST>(load, out, tw, P, p, B); break;
    case 5: fft_pass<T, 5, LFAST>(load, out, tw, P, p, B); break;
    case 6: fft_pass<T, 6, LFAST>(load, out, tw, P, p, B); break;
    case 7: fft_pass<T, 7, LFAST>(load, out, tw, P, p, B); break;
    case 8: fft_pass<T, 8, LFAST>(load, out, tw, P, p, B); break;
    case 9: fft_pass<T, 9, LFAST>(load, out, tw, P, p, B); break;
    case 10: fft_pass<T, 10, LFAST>(load, out, tw, P, p, B); break;
    case 12: fft_pass<T, 12, LFAST>(load, out, tw, P, p, B); break;
    default: fft_pass<T, 16, LFAST>(load, out, tw, P, p, B); break;
  }
}
// The forward transform of a block's lines from `load` (first pass) into shared memory; a and b are the buffers, and the
// one that holds the result is returned (every thread may read it). tw in shared memory; the caller has synchronised after
// staging it and after the last use of the buffers.
template <bool LFAST, class R, class LOAD>
__device__ __forceinline__ typename Cpx<R>::T* fft_lines(const LOAD& load, typename Cpx<R>::T* a, typename Cpx<R>::T* b, const typename Cpx<R>::T* tw,
                                                         const FftPlan<R>& P, const LineBuf& B) {
  using T = typename Cpx<R>::T;
  fft_pass_any<T, LFAST>(load, a, tw, P, 0, B);
  __syncthreads();
  for (int p = 1; p < P.nst; ++p) {
    const T* in = a;
    fft_pass_any<T, LFAST>([&](int l, int i) { return in[l * B.ls + i * B.is]; }, b, tw, P, p, B);
    __syncthreads();
    T* t = a;
    a = b;
    b = t;
  }
  return a;
}
// The inverse transform is the forward one of the values with real and imaginary parts exchanged, exchanged back.
template <class T>
__device__ __forceinline__ T swap_ri(T v) { return {v.y, v.x}; }

template <class T>
__device__ __forceinline__ void stage_twiddles(T* dst, const T* __restrict__ src, int n) {
  for (int t = threadIdx.x; t < n; t += blockDim.x) dst[t] = src[t];
}

// Cardinal B-spline weights of order P at fractional offset w (caps_kspace.f90:568-598), 0-based: th[j] weighs grid
// point floor(u) - P + 1 + j.
template <class R, int P>
__device__ __forceinline__ void bspline(R w, R th[P], R dth[P]) {
#pragma unroll
  for (int j = 0; j < P; ++j) th[j] = 0;
  th[1] = w;
  th[0] = 1 - w;
#pragma unroll
  for (int k = 3; k <= P - 1; ++k) {
    const R div = R(1) / R(k - 1);
    th[k - 1] = div * w * th[k - 2];
#pragma unroll
    for (int j = 1; j <= k - 2; ++j) th[k - j - 1] = div * ((w + R(j)) * th[k - j - 2] + (R(k - j) - w) * th[k - j - 1]);
    th[0] = div * (1 - w) * th[0];
  }
  dth[0] = -th[0];
#pragma unroll
  for (int j = 2; j <= P; ++j) dth[j - 1] = th[j - 2] - th[j - 1];
  const R div = R(1) / R(P - 1);
  th[P - 1] = div * w * th[P - 2];
#pragma unroll
  for (int j = 1; j <= P - 2; ++j) th[P - j - 1] = div * ((w + R(j)) * th[P - j - 2] + (R(P - j) - w) * th[P - j - 1]);
  th[0] = div * (1 - w) * th[0];
}

struct PmeArgs {
  int k1, k2, k3, h1;
  DevCell cell;
  const double* x;
  const double* q;
  int n;
};

// fractional coordinates as the Fortran takes them: s = h^-1 x (no origin), u = frac(s) K, w = frac(u)
template <class R, int P>
__device__ __forceinline__ void atom_splines(const PmeArgs& A, int i, R th[3][P], R dth[3][P], int base[3]) {
  const double xi[3] = {A.x[3 * i], A.x[3 * i + 1], A.x[3 * i + 2]};
  const int K[3] = {A.k1, A.k2, A.k3};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double s = A.cell.hi[d][0] * xi[0] + A.cell.hi[d][1] * xi[1] + A.cell.hi[d][2] * xi[2];
    const double u = (s - floor(s)) * K[d];
    const double fu = floor(u);
    bspline<R, P>(R(u - fu), th[d], dth[d]);
    base[d] = int(fu) - P + 1;
  }
}

__device__ __forceinline__ int wrapk(int v, int K) {
  v %= K;
  return v < 0 ? v + K : v;
}

// An atom's grid points are worked on by a group of lanes: P^2 lanes of P = 3 and 4 (two atoms and more to a warp), a warp
// for the higher orders; a lane's points follow one another G lanes apart, x fastest.
template <int P>
constexpr int pme_group() { return P == 3 ? 9 : P == 4 ? 16 : 32; }
constexpr int kPmeThreads = 128;
constexpr int kPmeAtoms = 64;   // atoms per block at most
// What coordinate k along axis d adds to a point's place in the grid, a + K1 (b + K2 c). The places of grids past 2^31 points
// (1,291^3) take 64 bits (Off = size_t), by grid_needs_64; the others stay in 32, with which the FP64 path's step is 1.3 %
// faster at 32,000 atoms (250 us against 253: the kernel then takes 34 registers, not 32, and leaves the pair kernel more).
template <class Off>
__host__ __device__ __forceinline__ Off grid_place(int k, int d, int k1, int k2) { return d == 0 ? Off(k) : d == 1 ? Off(k) * Off(k1) : Off(k) * Off(k1) * Off(k2); }
__host__ __device__ __forceinline__ bool grid_needs_64(int k1, int k2, int k3) { return size_t(k1) * size_t(k2) * size_t(k3) > size_t(0x7fffffff); }
template <class R, int P, class Off>
struct PmeAtom {
  R th[3][P];
  Off at[3][P];   // the places of the P points along each axis
  R q;
};

// K-SPREAD. FP64: double atomics into g. FP32: fixed point (2^40 per e) into gq, exact and order-free. A row of P points
// along x is P neighbouring lanes', so that it reaches L2 as one or two sectors of adds instead of P: the kernel is bound
// by its atomics there (64 per atom at order 4).
template <class R, int P, class Off>
static __global__ void __launch_bounds__(kPmeThreads) k_spread(PmeArgs A, int per_block, double* __restrict__ g, long long* __restrict__ gq) {
  __shared__ PmeAtom<R, P, Off> S[kPmeAtoms];
  const int i0 = blockIdx.x * per_block, n = min(per_block, A.n - i0);
  for (int t = threadIdx.x; t < n; t += kPmeThreads) {
    R th[3][P], dth[3][P];
    int base[3];
    atom_splines<R, P>(A, i0 + t, th, dth, base);
    const int K[3] = {A.k1, A.k2, A.k3};
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int k = 0; k < P; ++k) S[t].th[d][k] = th[d][k], S[t].at[d][k] = grid_place<Off>(wrapk(base[d] + k, K[d]), d, A.k1, A.k2);
    S[t].q = R(A.q[i0 + t]);
  }
  __syncthreads();
  constexpr int G = pme_group<P>(), NG = kPmeThreads / G;
  const int grp = threadIdx.x / G, lane = threadIdx.x % G;
  if (grp >= NG) return;
  for (int t = grp; t < n; t += NG) {
    const PmeAtom<R, P, Off>& a = S[t];
    if (a.q == 0) continue;
#pragma unroll
    for (int k = 0; k < (P * P * P + G - 1) / G; ++k) {
      const int pt = lane + k * G;
      if (P * P * P % G != 0 && pt >= P * P * P) break;
      const int ia = pt % P, ib = pt / P % P, ic = pt / (P * P);
      const R st = a.q * a.th[1][ib] * a.th[2][ic];
      const Off at = a.at[0][ia] + a.at[1][ib] + a.at[2][ic];
      const R v = st * a.th[0][ia];
      if (sizeof(R) == 8) atomicAdd(g + at, double(v));
      else atomic_add_fix(gq + at, __float2ll_rn(float(v) * float(kFixQ)));   // the scale is a power of two: no rounding
    }
  }
}

// Block size of the line transforms. At 64 registers (FP32) two blocks fit an SM beside a pair grid one block short of full.
constexpr int kFftThreads = 128;
// Shared memory of the line-transform kernels: the twiddle table, then two buffers of the block's lines.
// K-FFT-X forward: real lines (b, c) of length K1 to half spectra h(a, b, c), a <= K1/2; lines 2 m and 2 m + 1 are the real
// and imaginary parts of one complex line, parted again in the spectrum by its symmetry. Input: g (FP64 path) or gq (mixed path, fixed),
// cleared as it is read: the grid is zero for the next spread, with no launch of its own for it (as a memset node of the
// step's graph it started up to 10 us after the step's drift, and the spread behind it). lpb: pairs of lines per block.
template <class R>
static __global__ void __launch_bounds__(kFftThreads) k_fft_x_fwd(PmeArgs A, double* __restrict__ g, long long* __restrict__ gq,
                                                          typename Cpx<R>::T* __restrict__ h, FftPlan<R> P, int lpb) {
  using T = typename Cpx<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ls = A.k1 | 1;
  T* tw = reinterpret_cast<T*>(smem_raw);
  T* s0 = tw + A.k1;
  T* s1 = s0 + lpb * ls;
  const int nlines = A.k2 * A.k3, npairs = (nlines + 1) / 2;
  stage_twiddles(tw, P.tw, A.k1);
  // no branch around a load, so that a butterfly's loads go out together (a line past the last reads the last, times 0)
  auto take = [&](int line, int i) {
    const size_t at = size_t(min(line, nlines - 1)) * A.k1 + i;   // lines are contiguous in the real grid
    R v;
    if constexpr (sizeof(R) == 4) v = R(double(gq[at]) * kInvFixQ);
    else v = g[at];
    return line < nlines ? v : R(0);
  };
  const unsigned m_h1 = div_magic(unsigned(A.h1));
  // groups of lpb pairs, strided over the grid (the grid may be smaller than the group count)
  for (int l0 = blockIdx.x * lpb; l0 < npairs; l0 += gridDim.x * lpb) {
    const LineBuf B{min(lpb, npairs - l0), ls, 1, 0};
    __syncthreads();
    const T* z = fft_lines<false, R>([&](int l, int i) { return T{take(2 * (l0 + l), i), take(2 * (l0 + l) + 1, i)}; }, s0, s1, tw, P, B);
    // every value is read: cleared together, so that no store stands between two loads
    const size_t first = size_t(2 * l0) * A.k1, cells = size_t(min(2 * B.nl, nlines - 2 * l0)) * A.k1;
    for (size_t t = threadIdx.x; t < cells; t += blockDim.x) {
      if constexpr (sizeof(R) == 4) gq[first + t] = 0;
      else g[first + t] = 0;
    }
    for (int t = threadIdx.x; t < 2 * B.nl * A.h1; t += blockDim.x) {
      const int l = div_by(t, m_h1), a = t - l * A.h1;
      if (2 * l0 + l >= nlines) continue;
      const T u = z[(l >> 1) * ls + a], w = z[(l >> 1) * ls + (a ? A.k1 - a : 0)];   // Z(a), Z(-a)
      h[size_t(2 * l0 + l) * A.h1 + a] = (l & 1) ? T{R(0.5) * (u.y + w.y), R(0.5) * (w.x - u.x)} : T{R(0.5) * (u.x + w.x), R(0.5) * (u.y - w.y)};
    }
  }
}

// K-FFT-X inverse: half spectra back to real lines, two at a time (the missing halves by Hermitian symmetry).
template <class R>
static __global__ void __launch_bounds__(kFftThreads) k_fft_x_inv(PmeArgs A, const typename Cpx<R>::T* __restrict__ h, R* __restrict__ gr, FftPlan<R> P, int lpb) {
  using T = typename Cpx<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ls = A.k1 | 1;
  T* tw = reinterpret_cast<T*>(smem_raw);
  T* s0 = tw + A.k1;
  T* s1 = s0 + lpb * ls;
  const int nlines = A.k2 * A.k3, npairs = (nlines + 1) / 2;
  stage_twiddles(tw, P.tw, A.k1);
  const unsigned m_k1 = div_magic(unsigned(A.k1));
  for (int l0 = blockIdx.x * lpb; l0 < npairs; l0 += gridDim.x * lpb) {
    const LineBuf B{min(lpb, npairs - l0), ls, 1, 0};
    __syncthreads();
    const T* z = fft_lines<false, R>(
        [&](int l, int m) {
          const int line = 2 * (l0 + l), a = 2 * m <= A.k1 ? m : A.k1 - m;
          const R sg = 2 * m <= A.k1 ? R(1) : R(-1);
          const T u = h[size_t(line) * A.h1 + a];
          T w = h[size_t(min(line + 1, nlines - 1)) * A.h1 + a];
          if (line + 1 >= nlines) w = {R(0), R(0)};
          // Z = U + i W with conjugates past the middle, real and imaginary parts exchanged
          return T{sg * u.y + w.x, u.x - sg * w.y};
        },
        s0, s1, tw, P, B);
    for (int t = threadIdx.x; t < 2 * B.nl * A.k1; t += blockDim.x) {
      const int l = div_by(t, m_k1), i = t - l * A.k1;
      if (2 * l0 + l >= nlines) continue;
      const T v = z[(l >> 1) * ls + i];
      gr[size_t(2 * l0 + l) * A.k1 + i] = (l & 1) ? v.x : v.y;
    }
  }
}

// K-FFT-Y: lines along b for fixed (a, c); a block takes 1 << lsh consecutive a (coalesced rows) of one c.
template <class R, bool INV>
static __global__ void __launch_bounds__(kFftThreads) k_fft_y(PmeArgs A, typename Cpx<R>::T* __restrict__ h, FftPlan<R> P, int lsh) {
  using T = typename Cpx<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int la = 1 << lsh;
  T* tw = reinterpret_cast<T*>(smem_raw);
  T* s0 = tw + A.k2;
  T* s1 = s0 + la * A.k2;
  const int ngrp = (A.h1 + la - 1) >> lsh;
  stage_twiddles(tw, P.tw, A.k2);
  for (int grp = blockIdx.x; grp < ngrp * A.k3; grp += gridDim.x) {
    const int c = grp / ngrp, a0 = (grp - c * ngrp) << lsh;
    const LineBuf B{min(la, A.h1 - a0), 1, la, lsh};
    T* row = h + size_t(a0) + size_t(A.h1) * size_t(A.k2) * c;
    __syncthreads();
    const T* res = fft_lines<true, R>(
        [&](int l, int i) {
          const T v = row[l + size_t(A.h1) * i];
          return INV ? swap_ri(v) : v;
        },
        s0, s1, tw, P, B);
    for (int t = threadIdx.x; t < A.k2 << lsh; t += blockDim.x) {
      const int l = t & (la - 1), i = t >> lsh;
      if (l < B.nl) row[l + size_t(A.h1) * i] = INV ? swap_ri(res[t]) : res[t];
    }
  }
}

// K-FFT-Z+SOLVE: lines along c for fixed (a, b): forward transform, energy and virial of the half spectrum (e_m doubled
// for 0 < a < K1/2), multiply by G, inverse transform, in one pass.
template <class R, bool ENER, bool VIR>
static __global__ void __launch_bounds__(kFftThreads) k_fft_z_solve(PmeArgs A, typename Cpx<R>::T* __restrict__ h, const R* __restrict__ gt,
                                                            const R* __restrict__ wt, FftPlan<R> P, int lsh, EnergySink en, int fixed) {
  using T = typename Cpx<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int la = 1 << lsh;
  T* tw = reinterpret_cast<T*>(smem_raw);
  T* s0 = tw + A.k3;
  T* s1 = s0 + la * A.k3;
  const int ngrp = (A.h1 + la - 1) >> lsh;
  const size_t plane = size_t(A.h1) * A.k2;
  stage_twiddles(tw, P.tw, A.k3);
  double e = 0, w[6] = {0, 0, 0, 0, 0, 0};
  long long ef = 0, wf[6] = {0, 0, 0, 0, 0, 0};
  for (int grp = blockIdx.x; grp < ngrp * A.k2; grp += gridDim.x) {
    const int b = grp / ngrp, a0 = (grp - b * ngrp) << lsh;
    const LineBuf B{min(la, A.h1 - a0), 1, la, lsh};
    const size_t first = size_t(a0) + size_t(A.h1) * b;
    T* row = h + first;
    __syncthreads();
    T* res = fft_lines<true, R>([&](int l, int i) { return row[l + plane * i]; }, s0, s1, tw, P, B);
    // the inverse transform's first pass reads the spectrum times G (parts exchanged); every point is read once
    const T* back = fft_lines<true, R>(
        [&](int l, int i) {
          const T v = res[l + (i << lsh)];
          const size_t gi = first + l + plane * i;
          const R G = gt[gi];
          if (ENER || VIR) {
            const int a = a0 + l;
            double em = 0.5 * (double(v.x) * v.x + double(v.y) * v.y);
            if (a > 0 && 2 * a != A.k1) em *= 2;
            // mixed path: every term rounded to fixed point on its own, so the sum does not depend on which block took
            // which line group
            if (ENER) {
              if (fixed) ef += to_fix(em * double(G), kFixE);
              else e += em * double(G);
            }
            if (VIR)
              for (int k = 0; k < 6; ++k) {
                if (fixed) wf[k] += to_fix(em * double(wt[6 * gi + k]), kFixE);
                else w[k] += em * double(wt[6 * gi + k]);
              }
          }
          return T{v.y * G, v.x * G};
        },
        res == s0 ? s1 : s0, res, tw, P, B);
    for (int t = threadIdx.x; t < A.k3 << lsh; t += blockDim.x) {
      const int l = t & (la - 1), i = t >> lsh;
      if (l < B.nl) row[l + plane * i] = swap_ri(back[t]);
    }
  }
  if ((ENER || VIR) && fixed) {
    __shared__ long long scratch_q[32];
    if (ENER) {
      const long long s = block_sum(ef, scratch_q);
      if (threadIdx.x == 0) atomic_add_fix(en.fix + kECoul, s), atomic_add_fix(en.fix + kEPmeRecip, s);
    }
    if (VIR)
      for (int k = 0; k < 6; ++k) {
        const long long s = block_sum(wf[k], scratch_q);
        if (threadIdx.x == 0) atomic_add_fix(en.fix + kEW0 + k, s);
      }
  } else if (ENER || VIR) {
    __shared__ double scratch[32];
    if (ENER) {
      const double s = block_sum(e, scratch);
      if (threadIdx.x == 0) en.add(kECoul, s, false);
      if (threadIdx.x == 0) en.add(kEPmeRecip, s, false);
    }
    if (VIR)
      for (int k = 0; k < 6; ++k) {
        const double s = block_sum(w[k], scratch);
        if (threadIdx.x == 0) en.add(kEW0 + k, s, false);
      }
  }
}

// The influence function and its virial weights on the half spectrum (caps_kspace.f90:518-564, 916-940), in double,
// stored as R. Rebuilt when the cell, grid, order or beta change.
template <class R>
static __global__ void k_pme_green(PmeArgs A, const double* __restrict__ b1, const double* __restrict__ b2, const double* __restrict__ b3, double beta,
                            double kcoul, R* __restrict__ gt, R* __restrict__ wt) {
  const size_t total = size_t(A.h1) * A.k2 * A.k3;
  const double fac = kPi * kPi / (beta * beta);
  const int K[3] = {A.k1, A.k2, A.k3};
  for (size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += size_t(gridDim.x) * blockDim.x) {
    const int a = int(t % A.h1), b = int((t / A.h1) % A.k2), c = int(t / (size_t(A.h1) * A.k2));
    if (a == 0 && b == 0 && c == 0) {
      gt[t] = 0;
      for (int k = 0; k < 6; ++k) wt[6 * t + k] = 0;
      continue;
    }
    const int idx[3] = {a, b, c};
    int m[3];
    bool nyq[3];
    int nn = 0;
    for (int d = 0; d < 3; ++d) {
      m[d] = idx[d];
      if (m[d] >= (K[d] + 1) / 2) m[d] -= K[d];
      nyq[d] = K[d] % 2 == 0 && 2 * idx[d] == K[d];
      nn += nyq[d];
    }
    const double bm = b1[a] * b2[b] * b3[c];
    const int ns = 1 << nn;
    double g = 0, w[6] = {0, 0, 0, 0, 0, 0};
    for (int s = 0; s < ns; ++s) {
      int sel = 0;
      double mv[3] = {0, 0, 0};
      for (int d = 0; d < 3; ++d) {
        double sg = 1;
        if (nyq[d]) {
          if ((s >> sel) & 1) sg = -1;
          ++sel;
        }
        for (int r = 0; r < 3; ++r) mv[r] += sg * m[d] * A.cell.hi[d][r];
      }
      const double m2 = mv[0] * mv[0] + mv[1] * mv[1] + mv[2] * mv[2];
      const double e = kcoul * exp(-fac * m2) / (kPi * A.cell.vol * m2 * bm);
      const double ss = 2 * (1 + fac * m2) / m2;
      g += e;
      w[0] += e * (1 - ss * mv[0] * mv[0]);
      w[1] += e * (1 - ss * mv[1] * mv[1]);
      w[2] += e * (1 - ss * mv[2] * mv[2]);
      w[3] -= e * ss * mv[0] * mv[1];
      w[4] -= e * ss * mv[0] * mv[2];
      w[5] -= e * ss * mv[1] * mv[2];
    }
    gt[t] = R(g / ns);
    for (int k = 0; k < 6; ++k) wt[6 * t + k] = R(w[k] / ns);
  }
}

// K-GATHER: F_i -= q_i sum_d K_d (row d of h^-1) dE/du_d (caps_kspace.f90:965-992), L lanes per atom, each taking every
// L-th plane c of its P^3 points (the splines by each lane for itself: cheaper than a stage in shared memory). One lane per
// atom reads fewest instructions, four fill the GPU and shorten the chain of loads where atoms are few.
template <class R, class G, int P, int L>
static __global__ void __launch_bounds__(128) k_gather(PmeArgs A, const G* __restrict__ gr, ForceSink<R> F) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / L, lane = t % L;
  if (i >= A.n) return;
  const double qi = A.q[i];
  if (qi == 0) return;   // the same for an atom's lanes
  R th[3][P], dth[3][P];
  int base[3];
  atom_splines<R, P>(A, i, th, dth, base);
  int ia[P], ib[P];
#pragma unroll
  for (int a = 0; a < P; ++a) ia[a] = wrapk(base[0] + a, A.k1), ib[a] = wrapk(base[1] + a, A.k2);
  R gs0 = 0, gs1 = 0, gs2 = 0;
#pragma unroll
  for (int c0 = 0; c0 < P; c0 += L) {
    const int c = c0 + lane;
    if (P % L != 0 && c >= P) break;
    R tc = th[2][c0], dc = dth[2][c0];   // of plane c, by selects (an index would put the arrays in memory)
#pragma unroll
    for (int m = 1; m < L; ++m)
      if (c0 + m < P && lane == m) tc = th[2][c0 + m], dc = dth[2][c0 + m];
    const int ic = wrapk(base[2] + c, A.k3);
#pragma unroll
    for (int b = 0; b < P; ++b) {
      const R tb = th[1][b], db = dth[1][b];
      const size_t row = size_t(A.k1) * (size_t(ib[b]) + size_t(A.k2) * size_t(ic));
#pragma unroll
      for (int a = 0; a < P; ++a) {
        const R st = R(gr[row + ia[a]]);
        gs0 += dth[0][a] * tb * tc * st;
        gs1 += th[0][a] * db * tc * st;
        gs2 += th[0][a] * tb * dc * st;
      }
    }
  }
  if (L > 1) {
    const unsigned m = (L == 32 ? 0xffffffffu : (1u << L) - 1) << (threadIdx.x & 31 & ~(L - 1));
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
      gs0 += __shfl_xor_sync(m, gs0, o);
      gs1 += __shfl_xor_sync(m, gs1, o);
      gs2 += __shfl_xor_sync(m, gs2, o);
    }
    if (lane) return;
  }
  R f[3];
  for (int r = 0; r < 3; ++r)
    f[r] = -R(qi) * (R(A.k1) * gs0 * R(A.cell.hi[0][r]) + R(A.k2) * gs1 * R(A.cell.hi[1][r]) + R(A.k3) * gs2 * R(A.cell.hi[2][r]));
  F.add(i, f[0], f[1], f[2]);
}

}  // namespace capsb
