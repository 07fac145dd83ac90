// Types of the device PME shared by the host engine and the PME kernels (pme.cuh).
#pragma once
#include "common.cuh"

namespace capsb {

constexpr int kMaxRadices = 8;
constexpr int kMaxOrder = 8;

template <class R> struct Cpx;
template <> struct Cpx<float> { using T = float2; };
template <> struct Cpx<double> { using T = double2; };

template <class T> __device__ __forceinline__ T cmul(T a, T b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
template <class T> __device__ __forceinline__ T cadd(T a, T b) { return {a.x + b.x, a.y + b.y}; }
template <class T> __device__ __forceinline__ T csub(T a, T b) { return {a.x - b.x, a.y - b.y}; }

// A line transform of length n = rad[0] rad[1] ... as Stockham passes. For pass p: nb = n / rad[p] butterflies per line,
// ns = the product of the radices before it; m_nb and m_ns divide by them (div_by).
template <class R>
struct FftPlan {
  int n, nst;
  int rad[kMaxRadices], nb[kMaxRadices], ns[kMaxRadices];
  unsigned m_nb[kMaxRadices], m_ns[kMaxRadices];
  const typename Cpx<R>::T* tw;   // exp(-2 pi i k / n), k < n
};

// t / d by the multiplier m = floor(2^32 / d) + 1 (0 for d = 1), exact for t d < 2^32.
__host__ __device__ inline unsigned div_magic(unsigned d) { return d == 1 ? 0u : unsigned(0xffffffffu / d) + 1u; }
__device__ __forceinline__ int div_by(int t, unsigned m) { return m ? int(__umulhi(unsigned(t), m)) : t; }

}  // namespace capsb
