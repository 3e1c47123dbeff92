// fftmix.cuh -- FP64 DFT of any length N = 2^a 3^b 5^c 7^d up to 4096 by one
// block in shared memory (1D grids whose size is no power of two).
//
// Stockham stages of radix 7, 5, 3, 8, 4, 2 in place: with Ns the product of
// the radices done, butterfly j < N / R takes inputs j + q N / R, times
// W_{Ns R}^{q (j mod Ns)}, and its outputs go to (j / Ns) Ns R + j mod Ns + q
// Ns.  Every thread has its inputs in registers before the block's barrier and
// writes after it, so that one buffer is enough; input and output are in
// natural order.  The odd radices go first: in the first stage neighbouring
// threads write R values apart, which for odd R are all different banks (a
// first stage of radix 8 would serialise eight ways).  The inverse is the
// forward transform with real and imaginary parts exchanged on the way in and
// out.  Bound by latency, about 2 us a stage: two barriers, a twiddle load and
// a dependent butterfly at 16 warps.  N = 3000 (n = 6000) takes five stages;
// both transforms together are 22 us, cuFFT's two launches 45 and more.
#ifndef POFD_FFTMIX_CUH
#define POFD_FFTMIX_CUH

#include <cuda_runtime.h>

#include "fft1d.cuh"

namespace pofd {
namespace fft {

constexpr int MIX_MAXN = 4096, MIX_STAGES = 8;

// The radices of N in the order of the stages; 0 if another prime divides it
// or the stages would be too many.
inline int mix_factor(int N, int* f) {
  int k = 0;
  for (int r : {7, 5, 3, 8, 4, 2})
    while (N % r == 0 && (r != 8 || N >= 8)) {
      if (k == MIX_STAGES) return 0;
      f[k++] = r;
      N /= r;
    }
  return N == 1 ? k : 0;
}

// In-register DFT of odd R points, forward: pairs j and R - j share cosines
// and sines.
template <int R>
__device__ __forceinline__ void dft_odd(double2* v) {
  static_assert(R == 3 || R == 5 || R == 7, "radix");
  // cos and sin of 2 pi j / R, j = 1 ... (R - 1) / 2
  constexpr double C3[1] = {-0.5}, S3[1] = {0.86602540378443864676};
  constexpr double C5[2] = {0.30901699437494742410, -0.80901699437494742410};
  constexpr double S5[2] = {0.95105651629515357212, 0.58778525229247312917};
  constexpr double C7[3] = {0.62348980185873353053, -0.22252093395631440429,
                            -0.90096886790241912624};
  constexpr double S7[3] = {0.78183148246802980871, 0.97492791218182360702,
                            0.43388373911755812048};
  constexpr int H = (R - 1) / 2;
  double2 a[H], b[H];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    a[j] = cadd(v[1 + j], v[R - 1 - j]);
    b[j] = csub(v[1 + j], v[R - 1 - j]);
  }
  const double2 v0 = v[0];
#pragma unroll
  for (int j = 0; j < H; ++j) v[0] = cadd(v[0], a[j]);
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    double2 p = v0, q = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      const int e = (j * k) % R, i = (e <= H ? e : R - e) - 1;
      const double c = R == 3 ? C3[R == 3 ? i : 0] : R == 5 ? C5[R == 5 ? i : 0] : C7[R == 7 ? i : 0];
      const double s0 = R == 3 ? S3[R == 3 ? i : 0] : R == 5 ? S5[R == 5 ? i : 0] : S7[R == 7 ? i : 0];
      const double s = e <= H ? s0 : -s0;
      p.x = fma(c, a[j - 1].x, p.x);
      p.y = fma(c, a[j - 1].y, p.y);
      q.x = fma(s, b[j - 1].x, q.x);
      q.y = fma(s, b[j - 1].y, q.y);
    }
    v[k] = make_double2(p.x + q.y, p.y - q.x);      // p - i q
    v[R - k] = make_double2(p.x - q.y, p.y + q.x);  // p + i q
  }
}

// Where a transform takes its input from and leaves its output.
struct MixIo {
  const double* grid = nullptr;  // values 2 i, 2 i + 1, one pad per 16, are input i
  int kc = -1;                   // input i past the cut-off (min(i, N - i) > kc) is zero
  bool swap = false;             // real and imaginary part exchanged, in and out
  double2* out = nullptr;
};

// One stage from z to z; first and last by io.  Not inlined: the stages of
// one kernel together spill at 128 registers.
template <int R, int T>
__device__ __noinline__ void mix_stage(int N, int Ns, const double2* __restrict__ W, double2* z,
                                       MixIo io, bool first, bool last) {
  constexpr int C = (MIX_MAXN / R + T - 1) / T;  // most butterflies of a thread
  const int nb = N / R, step = N / (Ns * R);
  double2 v[C][R];
  int k[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = static_cast<int>(threadIdx.x) + c * T;
    k[c] = 0;
    if (j < nb) {
      if (first) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const int i = j + q * nb;
          if (io.grid) {
            const int o = 2 * i + (i >> 3);
            v[c][q] = make_double2(io.grid[o], io.grid[o + 1]);
          } else {
            v[c][q] = (min(i, N - i) <= io.kc) ? z[i] : make_double2(0.0, 0.0);
          }
          if (io.swap) v[c][q] = make_double2(v[c][q].y, v[c][q].x);
        }
      } else {
        k[c] = j % Ns;
        v[c][0] = z[j];
#pragma unroll
        for (int q = 1; q < R; ++q) v[c][q] = cmul(z[j + q * nb], __ldg(W + q * k[c] * step));
      }
    }
  }
  __syncthreads();
  double2* dst = last ? io.out : z;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = static_cast<int>(threadIdx.x) + c * T;
    if (j < nb) {
      if constexpr (R % 2 == 0) dft<R, -1>(v[c]);
      else dft_odd<R>(v[c]);
      const int o = (j - k[c]) * R + k[c];
#pragma unroll
      for (int q = 0; q < R; ++q)
        dst[o + q * Ns] = (last && io.swap) ? make_double2(v[c][q].y, v[c][q].x) : v[c][q];
    }
  }
  __syncthreads();
}

// The transform, all stages: input by io, between the stages through z (N
// values), output to io.out.  W: e^{-2 pi i k / N}, k < N.  The block's T
// threads all call it.
template <int T>
__device__ __forceinline__ void mix_fft(int N, int nf, const unsigned char* f, const double2* W,
                                        double2* z, const MixIo& io) {
  int Ns = 1;
  for (int s = 0; s < nf; ++s) {
    const bool first = s == 0, last = s == nf - 1;
    const int r = f[s];
    switch (r) {
      case 7: mix_stage<7, T>(N, Ns, W, z, io, first, last); break;
      case 5: mix_stage<5, T>(N, Ns, W, z, io, first, last); break;
      case 3: mix_stage<3, T>(N, Ns, W, z, io, first, last); break;
      case 8: mix_stage<8, T>(N, Ns, W, z, io, first, last); break;
      case 4: mix_stage<4, T>(N, Ns, W, z, io, first, last); break;
      default: mix_stage<2, T>(N, Ns, W, z, io, first, last); break;
    }
    Ns *= r;
  }
}

}  // namespace fft
}  // namespace pofd
#endif
