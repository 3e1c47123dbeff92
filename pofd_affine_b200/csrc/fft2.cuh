// fft2.cuh -- FP64 DFTs of one length by a group of threads in shared memory
// (rows and columns of the two-band grid, small 1D grids).
//
// One DFT, n = 16 M, M = 16 M3 (n a power of two in [512, 4096]), runs on M threads with 16 values each: with
// input j = n1 M + u, u = m M3 + s and output k = k1 + 16 k2 + 256 k3,
//   stage 1: 16-point register DFTs over n1, times W_n^{u k1};
//   stage 2: 16-point register DFTs over m, times W_M^{s k2};
//   stage 3: M3-point register DFTs over s;
// thread u holds (k1, s) = (u / M3, u % M3) in stage 2 and the outputs of
// p = k1 + 16 k2 = u, u + M, ... in stage 3.  The two exchanges go through
// shared memory, pitched so that neither side has bank conflicts.  A column
// goes back through the same stages transposed.  Twiddle powers come from
// four table entries per thread and stage (W^x, W^2x, W^4x, W^8x, made in
// long double), the other eleven by one product each: a table of all of
// them would cost as much shared memory traffic again as the exchanges.
#ifndef POFD_FFT2_CUH
#define POFD_FFT2_CUH

#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "fft1d.cuh"

namespace pofd {
namespace fft {

template <int N>
struct Fft2 {
  static constexpr int M = N / 16, M3 = N / 256;
  static constexpr int PITCH = M + M3;        // of the first exchange, [k1][u]
  static constexpr int SL = 256 * (M3 + 1);   // slots per DFT: [p][s], one pad
  static constexpr int PP = 16 / M3;          // stage-3 DFTs per thread
};

template <int S>
__device__ __forceinline__ void tw16(double2* v, const double2* __restrict__ T, int M) {
  double2 w1 = __ldg(T), w2 = __ldg(T + M), w4 = __ldg(T + 2 * M), w8 = __ldg(T + 3 * M);
  if (S > 0) {
    w1.y = -w1.y;
    w2.y = -w2.y;
    w4.y = -w4.y;
    w8.y = -w8.y;
  }
  const double2 w3 = cmul(w1, w2);
  v[1] = cmul(v[1], w1);
  v[2] = cmul(v[2], w2);
  v[3] = cmul(v[3], w3);
  v[4] = cmul(v[4], w4);
  v[8] = cmul(v[8], w8);
  v[9] = cmul(v[9], cmul(w1, w8));
  v[10] = cmul(v[10], cmul(w2, w8));
  v[11] = cmul(v[11], cmul(w3, w8));
  const double2 w5 = cmul(w1, w4), w6 = cmul(w2, w4), w7 = cmul(w3, w4);
  v[5] = cmul(v[5], w5);
  v[6] = cmul(v[6], w6);
  v[7] = cmul(v[7], w7);
  v[12] = cmul(v[12], cmul(w4, w8));
  v[13] = cmul(v[13], cmul(w5, w8));
  v[14] = cmul(v[14], cmul(w6, w8));
  v[15] = cmul(v[15], cmul(w7, w8));
}

// Stages 1 and 2: v[n1] = input n1 M + u of the thread; leaves the stage-3
// inputs in the slots b[p (M3 + 1) + s].
// Only the DFT's own M threads meet, at named barrier `bar` (one per DFT of
// the block): DFTs of one block run apart, and threads without one idle.
template <int N>
__device__ __forceinline__ void fft2_sync(int bar) {
  constexpr int M = Fft2<N>::M;
  if (M == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" : : "r"(bar), "r"(M) : "memory");
}

template <int N, int S>
__device__ __forceinline__ void fft2_head(double2* v, double2* b, int u,
                                          const double2* __restrict__ TW, int bar) {
  using F = Fft2<N>;
  dft<16, S>(v);
  tw16<S>(v, TW + u, F::M);
#pragma unroll
  for (int k1 = 0; k1 < 16; ++k1) b[k1 * F::PITCH + u] = v[k1];
  fft2_sync<N>(bar);
  const int k1 = u / F::M3, s = u % F::M3;
#pragma unroll
  for (int m = 0; m < 16; ++m) v[m] = b[k1 * F::PITCH + m * F::M3 + s];
  dft<16, S>(v);
  tw16<S>(v, TW + 16 * s, F::M);
  fft2_sync<N>(bar);
#pragma unroll
  for (int k2 = 0; k2 < 16; ++k2) b[(k1 + 16 * k2) * (F::M3 + 1) + s] = v[k2];
  fft2_sync<N>(bar);
}

// The transposed stages 2 and 1 of the inverse, from the slots to v[n1] =
// output n1 M + u.
template <int N>
__device__ __forceinline__ void fft2_tail_inv(double2* v, double2* b, int u,
                                              const double2* __restrict__ TW, int bar) {
  using F = Fft2<N>;
  const int k1 = u / F::M3, s = u % F::M3;
#pragma unroll
  for (int k2 = 0; k2 < 16; ++k2) v[k2] = b[(k1 + 16 * k2) * (F::M3 + 1) + s];
  tw16<1>(v, TW + 16 * s, F::M);
  dft<16, 1>(v);
  fft2_sync<N>(bar);
#pragma unroll
  for (int m = 0; m < 16; ++m) b[k1 * F::PITCH + m * F::M3 + s] = v[m];
  fft2_sync<N>(bar);
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = b[j * F::PITCH + u];
  tw16<1>(v, TW + u, F::M);
  dft<16, 1>(v);
}

// The twiddle table of both stages: W_n^{u 2^i} at [i][u], u < n / 16, i < 4
// (the second stage's W_{n/16}^s at u = 16 s).
inline std::vector<double2> fft2_twiddles(unsigned n) {
  std::vector<double2> tw(n / 4);
  const long double tau = 6.283185307179586476925286766559005768L;
  for (unsigned u = 0; u < n / 16; ++u)
    for (unsigned i = 0; i < 4; ++i) {
      const unsigned e = (u << i) % n;
      const long double a = -tau * static_cast<long double>(e) / static_cast<long double>(n);
      tw[i * (n / 16) + u] = make_double2(static_cast<double>(cosl(a)), static_cast<double>(sinl(a)));
    }
  return tw;
}

}  // namespace fft
}  // namespace pofd
#endif
