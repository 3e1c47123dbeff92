// surrogate.cu -- BF16 tensor-core MLP surrogate of the log-likelihood:
// forward, backward and Adam on sm_100a (tcgen05 / TMEM GEMMs from
// umma.cuh), trained online on exact (theta, logL) pairs.
//
// Network: x (free parameters, standardised, zero-padded to 16 inputs)
//   -> 3 hidden layers of H SiLU units -> 1 output, the standardised
//   logL - running max.  BF16 weights and activations, FP32 accumulation,
//   FP32 master weights and Adam moments.
#include "surrogate.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <sstream>

#include "setup.hh"
#include "umma.cuh"

namespace pofd {

namespace {

using bf16 = __nv_bfloat16;
constexpr int NT = umma::kThreads;

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    std::ostringstream s;
    s << what << ": " << cudaGetErrorString(e);
    throw Error(e == cudaErrorMemoryAllocation ? POFD_E_NOMEM : POFD_E_CUDA, s.str());
  }
}

template <class T>
T* dal(size_t n) {
  void* p = nullptr;
  ck(cudaMalloc(&p, (n ? n : 1) * sizeof(T)), "cudaMalloc");
  ck(cudaMemset(p, 0, (n ? n : 1) * sizeof(T)), "cudaMemset");
  return static_cast<T*>(p);
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// ------------------------------------------------------------ GEMM kernels
#define UMMA_PROLOGUE                                                         \
  extern __shared__ __align__(1024) uint8_t smem[];                          \
  __shared__ umma::Barriers bs;                                               \
  const int m0 = blockIdx.x * umma::kRows, n0 = blockIdx.y * g.ntile;         \
  const uint32_t tb = umma::mainloop(g, &tmA, &tmB, m0, n0, smem, bs);        \
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;                 \
  const int row = m0 + (warp & 3) * 32 + lane;                                \
  const uint32_t tlane = static_cast<uint32_t>((warp & 3) * 32) << 16;        \
  const int wg = warp >> 2; /* warps w, w + 4, ... share the rows' columns */

__device__ __forceinline__ void st_bf16x4(bf16* dst, const float* v) {
  __align__(8) bf16 h[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __float2bfloat16_rn(v[j]);
  *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
}

// The kernels of a training iteration overlap their launches (each waits for
// the one before it inside, umma::mainloop or pdl_wait).  What an earlier
// kernel of the sequence writes therefore comes through pointers without
// __restrict__: the compiler may move loads that it takes for invariant
// ahead of the wait.
//
// The epilogues are chains of dependent special functions and divisions over
// few elements: with four columns a thread (512 threads a block; 16 columns a
// tile) instead of sixteen they are a quarter as long.
constexpr int NTE = 512;

// Plain product C = A B^T in FP32 (a checkable entry point of the tensor-core
// main loop).
__global__ void __launch_bounds__(NT) k_gemm_f32(const __grid_constant__ CUtensorMap tmA,
                                                 const __grid_constant__ CUtensorMap tmB,
                                                 umma::GemmShape g, float* __restrict__ C,
                                                 int ldc) {
  UMMA_PROLOGUE
  static_cast<void>(wg);
  if (tb != 0xFFFFFFFFu) {
    for (int c0 = 0; c0 < g.ntile; c0 += 16) {
      float v[16];
      umma::tmem_ld16(tb + tlane + c0, v);
      if (row < g.M)
        for (int j = 0; j < 16; ++j) C[static_cast<size_t>(row) * ldc + n0 + c0 + j] = v[j];
    }
  }
  umma::release(bs, g.ntile);
}

// Hidden layer forward: z = A W^T + b, h = silu(z); writes what is given of
// h (bf16, [M][ldh]), z (fp32 [M][N]) and h^T (bf16 [N][ldt]).  The last
// hidden layer also writes this column tile's part of the network output,
// ypart[tile][row] = h . w4 (+ b4 in tile 0), summed in column order.
__global__ void __launch_bounds__(NTE) k_fwd(const __grid_constant__ CUtensorMap tmA,
                                             const __grid_constant__ CUtensorMap tmB,
                                             umma::GemmShape g, const float* bias, bf16* h,
                                             int ldh, float* z, bf16* ht, int ldt,
                                             const float* w4, const float* b4, float* ypart) {
  UMMA_PROLOGUE
  if (tb != 0xFFFFFFFFu) {
    float yacc = 0.0f;
    float* hs = reinterpret_cast<float*>(smem);  // the operands are done with
    for (int c0 = wg * 4; c0 < g.ntile; c0 += 16) {
      float v[4], hv[4];
      umma::tmem_ld4(tb + tlane + c0, v);
      const int cb = n0 + c0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] += bias[cb + j];
        hv[j] = silu(v[j]);
      }
      if (row < g.M) {
        if (h) st_bf16x4(h + static_cast<size_t>(row) * ldh + cb, hv);
        if (z)
          *reinterpret_cast<float4*>(z + static_cast<size_t>(row) * g.N + cb) =
              make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bf16 hb = __float2bfloat16_rn(hv[j]);
          if (ht) ht[static_cast<size_t>(cb + j) * ldt + row] = hb;
          if (w4) hs[(c0 + j) * umma::kRows + (row - m0)] = __bfloat162float(hb);
        }
      }
    }
    if (w4) {
      __syncthreads();
      if (wg == 0 && row < g.M) {
        for (int c = 0; c < g.ntile; ++c) yacc += hs[c * umma::kRows + (row - m0)] * w4[n0 + c];
        ypart[static_cast<size_t>(blockIdx.y) * g.M + row] = yacc + (blockIdx.y == 0 ? b4[0] : 0.0f);
      }
    }
  }
  umma::release(bs, g.ntile);
}

// Backward through a hidden layer: dh = dZ_next W_next (this GEMM, with B =
// W_next^T), dz = dh * silu'(z); writes dz (bf16 [M][N], when given) and dz^T
// (bf16 [N][ldt]).
__global__ void __launch_bounds__(NTE) k_bwd_dx(const __grid_constant__ CUtensorMap tmA,
                                                const __grid_constant__ CUtensorMap tmB,
                                                umma::GemmShape g, const float* z, bf16* dz,
                                                bf16* dzt, int ldt) {
  UMMA_PROLOGUE
  if (tb != 0xFFFFFFFFu) {
    for (int c0 = wg * 4; c0 < g.ntile; c0 += 16) {
      float v[4];
      umma::tmem_ld4(tb + tlane + c0, v);
      const int cb = n0 + c0;
      if (row < g.M) {
        const float4 zz = *reinterpret_cast<const float4*>(z + static_cast<size_t>(row) * g.N + cb);
        v[0] *= dsilu(zz.x);
        v[1] *= dsilu(zz.y);
        v[2] *= dsilu(zz.z);
        v[3] *= dsilu(zz.w);
        if (dz) st_bf16x4(dz + static_cast<size_t>(row) * g.N + cb, v);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          dzt[static_cast<size_t>(cb + j) * ldt + row] = __float2bfloat16_rn(v[j]);
      }
    }
  }
  umma::release(bs, g.ntile);
}

struct AdamArgs {
  float lr, b1, b2, eps, bc1, bc2;  // bc = 1 - beta^t
};

// One Adam step of one weight.  The roundings are spelled out: which product
// of a sum goes into the fused operation is the compiler's choice otherwise,
// and the weights and the biases keep the one that each has had.
template <bool kBias>
__device__ __forceinline__ void adam_step(const AdamArgs& ad, float g, float* p, float* m,
                                          float* v) {
  const float g1 = 1.0f - ad.b1, g2 = (1.0f - ad.b2) * g;
  *m = kBias ? __fmaf_rn(g1, g, __fmul_rn(ad.b1, *m)) : __fmaf_rn(ad.b1, *m, __fmul_rn(g1, g));
  *v = kBias ? __fmaf_rn(g2, g, __fmul_rn(ad.b2, *v)) : __fmaf_rn(ad.b2, *v, __fmul_rn(g2, g));
  *p = __fsub_rn(*p, ad.lr * (*m / ad.bc1) / (sqrtf(*v / ad.bc2) + ad.eps));
}

// Gradients of w4 (sum_r dy h3[r]), b4 (sum dy) and the hidden biases
// (column sums of dz) and their Adam steps.
struct BiasArgs {
  int Mp, H;
  const float* dy;
  const bf16* h3t;      // [H][Mp]
  const bf16* dzt[3];   // [H][Mp]
  float* p[5];   // b1, b2, b3, w4, b4
  float* m[5];
  float* v[5];
  float* grad_out[5];
};

// One warp per entry e: 0 .. 3H - 1 the hidden biases, 3H .. 4H - 1 w4, 4H
// b4.  256 partial sums over rows 256 apart, each 32 of them (a lane's w-th)
// added across the lanes, the eight in order.
__device__ __forceinline__ void bias_adam(const BiasArgs& a, const AdamArgs& ad, int e) {
  const int H = a.H, lane = threadIdx.x & 31;
  if (e > 4 * H) return;
  const int which = e / H, c = e - which * H;
  const bf16* col = which < 3 ? a.dzt[which] + static_cast<size_t>(c) * a.Mp
                   : which == 3 ? a.h3t + static_cast<size_t>(c) * a.Mp : nullptr;
  float s[8];
#pragma unroll
  for (int w = 0; w < 8; ++w) s[w] = 0.0f;
  for (int r0 = lane; r0 < a.Mp; r0 += 256) {
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int r = r0 + 32 * w;
      if (r < a.Mp) {
        if (which < 3) s[w] += __bfloat162float(col[r]);
        else if (which == 3) s[w] = __fadd_rn(s[w], __fmul_rn(a.dy[r], __bfloat162float(col[r])));
        else s[w] += a.dy[r];
      }
    }
  }
#pragma unroll
  for (int w = 0; w < 8; ++w)
    for (int o = 16; o > 0; o >>= 1) s[w] += __shfl_xor_sync(0xffffffffu, s[w], o);
  if (lane == 0) {
    float g = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) g += s[w];
    if (a.grad_out[which]) a.grad_out[which][c] = g;
    else adam_step<true>(ad, g, &a.p[which][c], &a.m[which][c], &a.v[which][c]);
  }
}

// One weight matrix of k_update: G = dZ^T X (A = dZ^T [Nout x M], B = X^T
// [Nin x M]), the Adam step of W [Nout][Nin] and its bf16 copies W
// (row-major) and W^T (may be null).  grad_out, when given, receives G
// instead of the update (gradient checks).
struct UpdateArgs {
  CUtensorMap a, b;
  umma::GemmShape g;
  int blocks, rowtiles;
  float *W, *m, *v, *grad_out;
  bf16 *Wb, *Wt;
};
struct UpdateAll {
  UpdateArgs w[3];
};

// All updates of an iteration in one launch: the tiles of the three weight
// gradients, then the bias entries, 16 to a block.  They are independent once
// the backward pass is through, and a few dozen tiles each: as launches of
// their own, with 16 elements of Adam a thread, the three took 78 us and the
// biases (one block per entry, columns of dz 2 H bytes apart) 6.5 us of the
// iteration's 150 (512 rows, H = 256).
__global__ void __launch_bounds__(NTE) k_update(const __grid_constant__ UpdateAll u, BiasArgs ba,
                                                AdamArgs ad) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ umma::Barriers bs;
  int blk = static_cast<int>(blockIdx.x), l = 0;
  while (l < 3 && blk >= u.w[l].blocks) blk -= u.w[l++].blocks;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (l == 3) {
    dev::pdl_launch();
    dev::pdl_wait();
    bias_adam(ba, ad, blk * (NTE / 32) + warp);
    return;
  }
  const UpdateArgs& q = u.w[l];
  const umma::GemmShape g = q.g;
  const int m0 = (blk % q.rowtiles) * umma::kRows, n0 = (blk / q.rowtiles) * g.ntile;
  const uint32_t tb = umma::mainloop(g, &q.a, &q.b, m0, n0, smem, bs);
  const int row = m0 + (warp & 3) * 32 + lane;
  const uint32_t tlane = static_cast<uint32_t>((warp & 3) * 32) << 16;
  if (tb != 0xFFFFFFFFu) {
    for (int c0 = (warp >> 2) * 4; c0 < g.ntile; c0 += 16) {
      float gv[4];
      umma::tmem_ld4(tb + tlane + c0, gv);
      const int cb = n0 + c0;
      if (row < g.M) {
        const size_t i0 = static_cast<size_t>(row) * g.N + cb;
        if (q.grad_out) {
          *reinterpret_cast<float4*>(q.grad_out + i0) = make_float4(gv[0], gv[1], gv[2], gv[3]);
        } else {
          const float4 m4 = *reinterpret_cast<const float4*>(q.m + i0);
          const float4 v4 = *reinterpret_cast<const float4*>(q.v + i0);
          const float4 w4 = *reinterpret_cast<const float4*>(q.W + i0);
          float m[4] = {m4.x, m4.y, m4.z, m4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w};
          float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) adam_step<false>(ad, gv[j], &w[j], &m[j], &v[j]);
          *reinterpret_cast<float4*>(q.m + i0) = make_float4(m[0], m[1], m[2], m[3]);
          *reinterpret_cast<float4*>(q.v + i0) = make_float4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<float4*>(q.W + i0) = make_float4(w[0], w[1], w[2], w[3]);
          st_bf16x4(q.Wb + i0, w);
          if (q.Wt)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              q.Wt[static_cast<size_t>(cb + j) * g.M + row] = __float2bfloat16_rn(w[j]);
        }
      }
    }
  }
  umma::release(bs, g.ntile);
}

// ------------------------------------------------------ elementwise kernels
__device__ __forceinline__ int pick_row(const Pick& p, int r) {
  if (p.n == 0) return r;
  unsigned long long x = p.seed ^ (p.it * 0x9E3779B97F4A7C15ull) ^
                         (static_cast<unsigned long long>(r) * 0xBF58476D1CE4E5B9ull);
  // splitmix64 finaliser (Steele, Lea & Flood 2014)
  x ^= x >> 30;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return static_cast<int>((x >> 32) * static_cast<unsigned long long>(p.n) >> 32);
}


// Whitened, zero-padded bf16 inputs x [Mp][16] and x^T [16][Mp] (may be
// null) from theta rows (free parameters only): x = W (theta_free - mu), W
// [16][16] row-major (lower triangular); rows >= M are zero.  And the rows'
// targets, and the loss to zero.  A thread per (row, input): with a thread
// per row its 256 loads of W and products were 12 us for 512 rows.
__global__ void __launch_bounds__(256) k_pack_inputs(int M, int Mp, const float* theta, int npar,
                                                     const int* idx, int nin, const float* mu,
                                                     const float* wm, Pick pick, Targets tg,
                                                     bf16* x, bf16* xt) {
  static_assert(Surrogate::kInPad == 16, "half a warp to a row");
  dev::pdl_launch();
  dev::pdl_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = e >> 4, k = e & 15;  // Mp * 16 is a multiple of the block size
  const int src = (r < M) ? pick_row(pick, r) : -1;
  const float dk =
      (src >= 0 && k < nin) ? theta[static_cast<size_t>(src) * npar + idx[k]] - mu[k] : 0.0f;
  float w[16];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 f = reinterpret_cast<const float4*>(wm)[k * 4 + q];
    w[4 * q] = f.x;
    w[4 * q + 1] = f.y;
    w[4 * q + 2] = f.z;
    w[4 * q + 3] = f.w;
  }
  float v = 0.0f;
#pragma unroll
  for (int j = 0; j < 16; ++j) v = fmaf(w[j], __shfl_sync(0xffffffffu, dk, j, 16), v);
  const bf16 b = __float2bfloat16_rn(v);
  x[e] = b;
  if (xt) xt[static_cast<size_t>(k) * Mp + r] = b;
  if (tg.t && k == 0) {
    if (r == 0) *tg.loss = 0.0f;
    if (r < M) {
      const double d = tg.logl[src] - tg.ymax;
      tg.t[r] = static_cast<float>((d < -tg.clip ? -tg.clip : d) * tg.iys);
    }
  }
}

// Network output y = sum of the column-tile parts, the loss, dy = 2 (y - t)
// / M and dz3 = dy w4 * silu'(z3); one thread per (4-column chunk, row), the
// first chunk's writes the row's values.
__global__ void __launch_bounds__(256) k_out_dz(int M, int Mp, int H, int ntiles,
                                                const float* ypart, const float* t, float* y,
                                                float* dy_out, float* loss, const float* w4,
                                                const float* z3, bf16* dz3, bf16* dz3t) {
  dev::pdl_launch();
  dev::pdl_wait();
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= static_cast<long long>(Mp) * (H / 4)) return;
  const int r = static_cast<int>(e % Mp), c0 = static_cast<int>(e / Mp) * 4;
  const float4 zz = *reinterpret_cast<const float4*>(z3 + static_cast<size_t>(r) * H + c0);
  float yy = 0.0f;
  for (int k = 0; k < ntiles; ++k) yy += ypart[static_cast<size_t>(k) * Mp + r];
  const float d = (r < M) ? (yy - t[r]) : 0.0f;
  const float dy = 2.0f * d / static_cast<float>(M);
  if (c0 == 0) {
    y[r] = yy;
    dy_out[r] = dy;
    float q = d * d / static_cast<float>(M);  // 0 past M; a warp is 32 rows
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, q);
  }
  const float v[4] = {dy * w4[c0] * dsilu(zz.x), dy * w4[c0 + 1] * dsilu(zz.y),
                      dy * w4[c0 + 2] * dsilu(zz.z), dy * w4[c0 + 3] * dsilu(zz.w)};
  st_bf16x4(dz3 + static_cast<size_t>(r) * H + c0, v);
#pragma unroll
  for (int j = 0; j < 4; ++j) dz3t[static_cast<size_t>(c0 + j) * Mp + r] = __float2bfloat16_rn(v[j]);
}

// Network output to log-likelihood units: logL = ymax + ys * y.
__global__ void k_unscale(int M, int Mp, int ntiles, const float* ypart, double ymax, double ys,
                          double* out, int* status) {
  dev::pdl_wait();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= M) return;
  float yy = 0.0f;
  for (int k = 0; k < ntiles; ++k) yy += ypart[static_cast<size_t>(k) * Mp + r];
  out[r] = ymax + ys * static_cast<double>(yy);
  if (status) status[r] = POFD_OK;
}

// Appends the valid rows (status OK, finite logL) to the pair ring in row
// order: one block walks the rows in chunks, a ballot prefix gives each
// valid row its slot, so the ring's contents -- and every minibatch drawn
// from it -- depend only on the inputs (ranks that train on the same pairs
// train the same network).
__global__ void k_append_pairs(int n, const float* __restrict__ theta, int npar,
                               const double* __restrict__ logl, const int* __restrict__ status,
                               float* __restrict__ ptheta, double* __restrict__ plogl,
                               unsigned* __restrict__ counters, unsigned cap) {
  // counters[0] = pairs written (ring), counters[1] = pairs held
  __shared__ unsigned wsum[32];
  __shared__ unsigned base;
  if (threadIdx.x == 0) base = counters[0];
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c0 = 0; c0 < n; c0 += blockDim.x) {
    const int r = c0 + static_cast<int>(threadIdx.x);
    const bool ok = r < n && (!status || status[r] == POFD_OK) && isfinite(logl[r]);
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) wsum[wid] = __popc(bal);
    __syncthreads();
    unsigned off = base;
    for (int k = 0; k < wid; ++k) off += wsum[k];
    if (ok) {
      const unsigned slot = (off + __popc(bal & ((1u << lane) - 1u))) % cap;
      for (int p = 0; p < npar; ++p)
        ptheta[static_cast<size_t>(slot) * npar + p] = theta[static_cast<size_t>(r) * npar + p];
      plogl[slot] = logl[r];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned tot = 0;
      for (int k = 0; k < static_cast<int>(blockDim.x >> 5); ++k) tot += wsum[k];
      base += tot;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    counters[0] = base;
    counters[1] = min(max(counters[1], base), cap);
  }
}

// --------------------------------------------- weights and scaling on device
// bf16 copies of the weights, W and W^T.
__global__ void k_pack_weights(int H, const float* __restrict__ W1, const float* __restrict__ W2,
                               const float* __restrict__ W3, bf16* __restrict__ w1b,
                               bf16* __restrict__ w2b, bf16* __restrict__ w2t,
                               bf16* __restrict__ w3b, bf16* __restrict__ w3t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < H * Surrogate::kInPad) w1b[i] = __float2bfloat16_rn(W1[i]);
  if (i >= H * H) return;
  const int r = i / H, k = i - r * H;
  const bf16 b = __float2bfloat16_rn(W2[i]), c = __float2bfloat16_rn(W3[i]);
  w2b[i] = b;
  w2t[k * H + r] = b;
  w3b[i] = c;
  w3t[k * H + r] = c;
}

// Sums for the scaling of inputs and target over the n pairs held, in FP64:
// three passes, since each needs the one before (the largest logL; the means
// over the pairs near it; the covariance about them).  Block b takes rows [b
// R, (b + 1) R); every entry is one thread's, which walks the block's rows;
// the blocks' parts are added by whoever needs them next, in block order.  On
// the host, with the pairs copied there, this was 0.5 ms for 8000 pairs of 14
// inputs and grew with the pairs held; now 0.12 ms with the transfers.
constexpr int kScT = 160;           // threads: covariance entries and more
constexpr int kScCov = Surrogate::kInPad * (Surrogate::kInPad + 1) / 2;
constexpr int kScPart = 160;        // doubles a block writes per pass
// pass 1: sums over the pairs near the maximum and over all, count, target
constexpr int kScAll = 16, kScCount = 32, kScTarget = 33;
static_assert(kScCov < kScT && kScCov < kScPart, "one thread per entry");

struct ScaleArgs {
  int n, R, G, npar, nin;
  double clip;
  const float* theta;
  const double* logl;
  const int* idx;
  double* part[3];  // [G][kScPart] of each pass
  double* out;      // [kScPart] pass 1 sums, [kScPart] pass 2 sums, max
};

__device__ __forceinline__ double scale_max(const ScaleArgs& a, double* sh) {
  const double none = -__longlong_as_double(0x7ff0000000000000ll);
  double mx = none;
  for (int b = threadIdx.x; b < a.G; b += kScT) mx = fmax(mx, a.part[0][static_cast<size_t>(b) * kScPart]);
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = sh[0];
  for (int w = 1; w < kScT / 32; ++w) mx = fmax(mx, sh[w]);
  __syncthreads();
  return mx;
}

__device__ __forceinline__ double scale_total(const ScaleArgs& a, int pass, int e) {
  double s = 0.0;
#pragma unroll 8
  for (int b = 0; b < a.G; ++b) s += a.part[pass][static_cast<size_t>(b) * kScPart + e];
  return s;
}

template <int PASS>
__global__ void __launch_bounds__(kScT) k_scale(ScaleArgs a) {
  __shared__ double sh[kScT], mean[Surrogate::kInPad];
  const int e = threadIdx.x, b = blockIdx.x, K = a.nin;
  const int r0 = min(b * a.R, a.n), r1 = min(r0 + a.R, a.n);
  if (PASS == 0) {
    double mx = -__longlong_as_double(0x7ff0000000000000ll);
    for (int r = r0 + e; r < r1; r += kScT) mx = fmax(mx, a.logl[r]);
    sh[e] = mx;
    __syncthreads();
    if (e == 0) {
      for (int w = 1; w < kScT; ++w) mx = fmax(mx, sh[w]);
      a.part[0][static_cast<size_t>(b) * kScPart] = mx;
    }
    return;
  }
  const double mx = scale_max(a, sh);
  if (PASS == 1) {
    double s = 0.0;
    const bool col = e < K || (e >= kScAll && e < kScAll + K);
    if (col) {
      const int p = a.idx[e & 15];
#pragma unroll 8
      for (int r = r0; r < r1; ++r) {
        const double v = a.theta[static_cast<size_t>(r) * a.npar + p];
        s += (e >= kScAll || a.logl[r] - mx > -a.clip) ? v : 0.0;
      }
    } else if (e == kScCount) {
      for (int r = r0; r < r1; ++r) s += (a.logl[r] - mx > -a.clip) ? 1.0 : 0.0;
    } else if (e == kScTarget) {
#pragma unroll 8
      for (int r = r0; r < r1; ++r) {
        const double d = a.logl[r] - mx;
        s += d < -a.clip ? -a.clip : d;
      }
    }
    a.part[1][static_cast<size_t>(b) * kScPart + e] = s;
    return;
  }
  // means over the pairs within the clip of the maximum if they are enough
  sh[e] = e <= kScTarget ? scale_total(a, 1, e) : 0.0;
  __syncthreads();
  const bool all = sh[kScCount] < (2 * K > 64 ? 2 * K : 64);
  const double nu = all ? a.n : sh[kScCount];
  if (e < K) mean[e] = sh[(all ? kScAll : 0) + e] / nu;
  const double m = sh[kScTarget] / a.n;
  if (b == 0) {
    a.out[e] = sh[e];
    if (e == 0) a.out[2 * kScPart] = mx;
  }
  __syncthreads();
  double s = 0.0;
  if (e < K * (K + 1) / 2) {
    int i = 0;
    while ((i + 1) * (i + 2) / 2 <= e) ++i;
    const int j = e - i * (i + 1) / 2, pi = a.idx[i], pj = a.idx[j];
#pragma unroll 8
    for (int r = r0; r < r1; ++r) {
      const float* t = a.theta + static_cast<size_t>(r) * a.npar;
      const double q = (t[pi] - mean[i]) * (t[pj] - mean[j]);
      s += (all || a.logl[r] - mx > -a.clip) ? q : 0.0;
    }
  } else if (e == kScT - 1) {
#pragma unroll 8
    for (int r = r0; r < r1; ++r) {
      const double d = a.logl[r] - mx;
      const double q = (d < -a.clip ? -a.clip : d) - m;
      s += q * q;
    }
  }
  a.part[2][static_cast<size_t>(b) * kScPart + e] = s;
}

__global__ void __launch_bounds__(kScT) k_scale_out(ScaleArgs a) {
  a.out[kScPart + threadIdx.x] = scale_total(a, 2, threadIdx.x);
}

// ----------------------------------------------------------- tensor maps
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                              const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    ck(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q),
       "cuTensorMapEncodeTiled entry point");
    if (q != cudaDriverEntryPointSuccess || !p) throw Error(POFD_E_CUDA, "cuTensorMapEncodeTiled unavailable");
    fn = reinterpret_cast<EncodeFn>(p);
  }
  return fn;
}

// A row-major bf16 matrix [rows][K] (leading dimension ld elements) in boxes
// of box_rows x 64, 128 bytes of K a row, swizzled as the MMA descriptors of
// umma::mainloop assume; rows and K beyond the matrix read as zero.
CUtensorMap kmajor_map(const bf16* base, int rows, int K, int ld, int box_rows) {
  if (reinterpret_cast<uintptr_t>(base) % 16 || ld % 8 || K % 16)
    throw Error(POFD_E_ARG, "tensor map: base 16-byte aligned, ld multiple of 8, K multiple of 16");
  CUtensorMap m;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  // the box is always whole: rows and K past the matrix are zero-filled, so
  // every stage holds exactly stage_bytes()
  const cuuint32_t box[2] = {umma::kKChunk, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t es[2] = {1, 1};
  const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base),
                                 dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw Error(POFD_E_CUDA, "cuTensorMapEncodeTiled failed");
  return m;
}

struct Gemm {
  umma::GemmShape g;
  CUtensorMap a, b;
  dim3 grid;
  size_t smem;
};

// N tile of a GEMM: the widest of 128, 64, 32 dividing N that still gives at
// least one CTA per SM, else 16.  The surrogate's GEMMs are small (a few
// hundred rows); narrower tiles spread them -- and the fused epilogues, the
// Adam update of the weight gradient above all -- over more SMs.
int ntile_for(int M, int N) {
  static int nsm = 0;
  if (nsm == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0)
      nsm = 148;
  }
  const int rt = (M + umma::kRows - 1) / umma::kRows;
  for (int nt : {128, 64, 32})
    if (N % nt == 0 && rt * (N / nt) >= nsm) return nt;
  return 16;
}

// C[M x N] = A[M x K] B[N x K]^T with A (lda) and B (ldb) row-major bf16.
Gemm plan_gemm(int M, int N, int K, const bf16* A, int lda, const bf16* B, int ldb, int* err) {
  if (M <= 0 || N < 16 || N > umma::kMaxN || N % 16 || K < 16 || K % 16)
    throw Error(POFD_E_ARG, "gemm: need N in [16, 512] and K >= 16, both multiples of 16");
  Gemm q;
  const int nt = ntile_for(M, N);
  q.g = umma::GemmShape{M, N, K, nt, err};
  q.a = kmajor_map(A, M, K, lda, umma::kRows);
  q.b = kmajor_map(B, N, K, ldb, nt);
  q.grid = dim3(static_cast<unsigned>((M + umma::kRows - 1) / umma::kRows),
                static_cast<unsigned>(N / nt));
  q.smem = umma::smem_bytes(nt);
  return q;
}

void set_gemm_attributes() {
  static bool done = false;
  if (done) return;
  const int sm = static_cast<int>(umma::smem_bytes(umma::kMaxNTile));
  ck(cudaFuncSetAttribute(k_gemm_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, sm), "attr");
  ck(cudaFuncSetAttribute(k_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, sm), "attr");
  ck(cudaFuncSetAttribute(k_bwd_dx, cudaFuncAttributeMaxDynamicSharedMemorySize, sm), "attr");
  ck(cudaFuncSetAttribute(k_update, cudaFuncAttributeMaxDynamicSharedMemorySize, sm), "attr");
  done = true;
}

}  // namespace

// ===================================================================== host

Surrogate::Surrogate(int device, cudaStream_t stream, unsigned npar, const int* free_idx,
                     unsigned nin, unsigned hidden, unsigned capacity, uint64_t seed)
    : device_(device), stream_(stream), npar_(npar), nin_(nin), H_(hidden), cap_(capacity),
      seed_(seed) {
  if (device < 0) throw Error(POFD_E_CUDA, "host-only context has no GPU");
  if (nin == 0 || nin > static_cast<unsigned>(kInPad)) throw Error(POFD_E_ARG, "1..16 inputs");
  if (hidden < 16 || hidden > 512 || hidden % 16) throw Error(POFD_E_ARG, "hidden width must be a multiple of 16 in [16, 512]");
  if (capacity < 128) throw Error(POFD_E_ARG, "capacity must be >= 128");
  for (unsigned i = 0; i < nin; ++i)
    if (free_idx[i] < 0 || static_cast<unsigned>(free_idx[i]) >= npar) throw Error(POFD_E_ARG, "input index out of range");
  ck(cudaSetDevice(device_), "cudaSetDevice");
  idx_ = dal<int>(kInPad);
  ck(cudaMemcpy(idx_, free_idx, nin * sizeof(int), cudaMemcpyHostToDevice), "upload");
  wm_ = dal<float>(kInPad * kInPad + kInPad);
  mu_ = wm_ + kInPad * kInPad;
  std::vector<float> eye(kInPad * kInPad, 0.0f);
  for (int k = 0; k < kInPad; ++k) eye[k * kInPad + k] = 1.0f;
  ck(cudaMemcpy(wm_, eye.data(), eye.size() * sizeof(float), cudaMemcpyHostToDevice), "upload");
  const size_t H = H_;
  const size_t sz[kNumTensors] = {H * kInPad, H, H * H, H, H * H, H, H, 1};
  for (int t = 0; t < kNumTensors; ++t) {
    size_[t] = sz[t];
    slab_ += (sz[t] + 63) / 64 * 64;
  }
  p_[0] = dal<float>(slab_);  // all tensors in one allocation, 256-byte aligned
  m_[0] = dal<float>(slab_);
  v_[0] = dal<float>(slab_);
  for (int t = 1; t < kNumTensors; ++t) {
    const size_t step = (sz[t - 1] + 63) / 64 * 64;
    p_[t] = p_[t - 1] + step;
    m_[t] = m_[t - 1] + step;
    v_[t] = v_[t - 1] + step;
  }
  w1b_ = dal<bf16>(H * kInPad);
  w2b_ = dal<bf16>(H * H);
  w3b_ = dal<bf16>(H * H);
  w2t_ = dal<bf16>(H * H);
  w3t_ = dal<bf16>(H * H);
  ptheta_ = dal<float>(static_cast<size_t>(cap_) * npar_);
  plogl_ = dal<double>(cap_);
  counters_ = dal<unsigned>(4);
  err_ = dal<int>(1);
  int sms = 0;
  ck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_), "attr");
  scale_blocks_ = sms > 0 ? sms : 1;
  scale_ = dal<double>(static_cast<size_t>(3 * scale_blocks_ + 3) * kScPart);
  static_assert(3 * kScPart * sizeof(double) >= (kInPad + 1) * kInPad * sizeof(float), "staging");
  ck(cudaMallocHost(reinterpret_cast<void**>(&h_stage_), 3 * kScPart * sizeof(double)), "cudaMallocHost");
  set_gemm_attributes();
  init_weights();
}

Surrogate::~Surrogate() {
  cudaSetDevice(device_);
  if (h_stage_) cudaFreeHost(h_stage_);
  void* q[] = {p_[0], m_[0], v_[0], scale_, idx_, wm_, w1b_, w2b_, w3b_, w2t_, w3t_, ptheta_, plogl_, counters_, err_,
               ws_.x, ws_.xt, ws_.h[0], ws_.h[1], ws_.h[2], ws_.ht[0], ws_.ht[1], ws_.ht[2],
               ws_.z[0], ws_.z[1], ws_.z[2], ws_.dz[0], ws_.dz[1], ws_.dz[2], ws_.dzt[0],
               ws_.dzt[1], ws_.dzt[2], ws_.y, ws_.ypart, ws_.t, ws_.dy, ws_.loss};
  for (void* p : q)
    if (p) cudaFree(p);
}

// He-style uniform initialisation (fan-in) from a seeded host generator.
void Surrogate::init_weights() {
  uint64_t s = seed_ ? seed_ : 0x1234567ull;
  auto next = [&s]() {
    s += 0x9E3779B97F4A7C15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return static_cast<double>(z >> 11) * (1.0 / 9007199254740992.0);
  };
  const int fan[kNumTensors] = {static_cast<int>(nin_), 1, static_cast<int>(H_), 1,
                                static_cast<int>(H_), 1, static_cast<int>(H_), 1};
  std::vector<std::vector<float>> host(kNumTensors);
  for (int t = 0; t < kNumTensors; ++t) {
    host[t].assign(size_[t], 0.0f);
    if (t == 1 || t == 3 || t == 5 || t == 7) continue;  // biases start at 0
    const double a = std::sqrt(6.0 / fan[t]) * (t == 6 ? 0.5 : 1.0);
    for (size_t i = 0; i < size_[t]; ++i) {
      if (t == 0 && (i % kInPad) >= nin_) continue;  // padded inputs
      host[t][i] = static_cast<float>((2.0 * next() - 1.0) * a);
    }
  }
  const float* ptr[kNumTensors];
  for (int t = 0; t < kNumTensors; ++t) ptr[t] = host[t].data();
  set_params_host(ptr);
}

void Surrogate::set_params_host(const float* const* host) {
  ck(cudaSetDevice(device_), "cudaSetDevice");
  for (int t = 0; t < kNumTensors; ++t)
    ck(cudaMemcpyAsync(p_[t], host[t], size_[t] * sizeof(float), cudaMemcpyHostToDevice, stream_), "upload");
  ck(cudaMemsetAsync(m_[0], 0, slab_ * sizeof(float), stream_), "memset");
  ck(cudaMemsetAsync(v_[0], 0, slab_ * sizeof(float), stream_), "memset");
  step_ = 0;
  const int H = static_cast<int>(H_);
  k_pack_weights<<<(H * H + 255) / 256, 256, 0, stream_>>>(H, p_[0], p_[2], p_[4], w1b_, w2b_, w2t_,
                                                         w3b_, w3t_);
  ck(cudaGetLastError(), "k_pack_weights");
  ck(cudaStreamSynchronize(stream_), "synchronize");  // other streams may use the weights
}

void Surrogate::get_param_host(int t, float* out) const {
  ck(cudaSetDevice(device_), "cudaSetDevice");
  ck(cudaMemcpyAsync(out, p_[t], size_[t] * sizeof(float), cudaMemcpyDeviceToHost, stream_), "D2H");
  ck(cudaStreamSynchronize(stream_), "synchronize");
}

void Surrogate::ensure_work(int Mp) {
  if (Mp <= ws_.Mp) return;
  void* q[] = {ws_.x, ws_.xt, ws_.h[0], ws_.h[1], ws_.h[2], ws_.ht[0], ws_.ht[1], ws_.ht[2],
               ws_.z[0], ws_.z[1], ws_.z[2], ws_.dz[0], ws_.dz[1], ws_.dz[2], ws_.dzt[0],
               ws_.dzt[1], ws_.dzt[2], ws_.y, ws_.ypart, ws_.t, ws_.dy, ws_.loss};
  for (void* p : q)
    if (p) cudaFree(p);
  ws_ = Work{};
  const size_t M = static_cast<size_t>(Mp), H = H_;
  ws_.Mp = Mp;
  ws_.x = dal<bf16>(M * kInPad);
  ws_.xt = dal<bf16>(M * kInPad);
  for (int l = 0; l < 3; ++l) {
    ws_.h[l] = dal<bf16>(M * H);
    ws_.ht[l] = dal<bf16>(M * H);
    ws_.z[l] = dal<float>(M * H);
    ws_.dz[l] = dal<bf16>(M * H);
    ws_.dzt[l] = dal<bf16>(M * H);
  }
  ws_.y = dal<float>(M);
  ws_.ypart = dal<float>(M * (umma::kMaxN / 16));
  ws_.t = dal<float>(M);
  ws_.dy = dal<float>(M);
  ws_.loss = dal<float>(1);
}

// Forward of M rows of theta (row r, or the picked one) into ws_.ypart; when
// targets are given (training) keeps z and h^T and writes them too.
void Surrogate::forward(int M, const float* theta, int npar, const Pick& pick, const Targets& tg,
                        cudaStream_t st) {
  const int Mp = (M + umma::kRows - 1) / umma::kRows * umma::kRows;
  ensure_work(Mp);
  const int H = static_cast<int>(H_);
  const bool train = tg.t != nullptr;
  launch_pdl(k_pack_inputs, dim3(Mp * kInPad / 256), dim3(256), 0, st, M, Mp, theta, npar, idx_,
             static_cast<int>(nin_), mu_, wm_, pick, tg, ws_.x, train ? ws_.xt : nullptr);
  const bf16* Ws[3] = {w1b_, w2b_, w3b_};
  const bf16* in = ws_.x;
  int ldin = kInPad;
  for (int l = 0; l < 3; ++l) {
    const int K = (l == 0) ? kInPad : H;
    const Gemm q = plan_gemm(Mp, H, K, in, ldin, Ws[l], K, err_);
    const bool last = (l == 2);
    launch_pdl(k_fwd, q.grid, dim3(NTE), q.smem, st, q.a, q.b, q.g, p_[2 * l + 1],
               last ? nullptr : ws_.h[l], H, train ? ws_.z[l] : nullptr,
               train ? ws_.ht[l] : nullptr, Mp, last ? p_[6] : nullptr, last ? p_[7] : nullptr,
               ws_.ypart);
    in = ws_.h[l];
    ldin = H;
  }
  ck(cudaGetLastError(), "surrogate forward");
}

void Surrogate::predict(unsigned n, const float* theta, unsigned npar, double* out, int* status,
                        cudaStream_t st) {
  if (n == 0) return;
  if (npar < npar_) throw Error(POFD_E_ARG, "Not enough elements in params");
  ck(cudaSetDevice(device_), "cudaSetDevice");
  if (!st) st = stream_;
  forward(static_cast<int>(n), theta, static_cast<int>(npar), Pick{}, Targets{}, st);
  const int Mp = (static_cast<int>(n) + umma::kRows - 1) / umma::kRows * umma::kRows;
  const int ntiles = static_cast<int>(H_) / ntile_for(Mp, static_cast<int>(H_));
  launch_pdl(k_unscale, dim3((n + 127) / 128), dim3(128), 0, st, static_cast<int>(n), Mp, ntiles,
             ws_.ypart, ymax_, ys_, out, status);
  ck(cudaGetLastError(), "k_unscale");
}

void Surrogate::add_pairs(unsigned n, const float* theta, unsigned npar, const double* logl,
                          const int* status, cudaStream_t st) {
  if (n == 0) return;
  if (npar != npar_) throw Error(POFD_E_ARG, "parameter count differs from the surrogate's");
  ck(cudaSetDevice(device_), "cudaSetDevice");
  if (!st) st = stream_;
  k_append_pairs<<<1, 1024, 0, st>>>(static_cast<int>(n), theta, static_cast<int>(npar), logl,
                                     status, ptheta_, plogl_, counters_, cap_);
  ck(cudaGetLastError(), "k_append_pairs");
}

unsigned Surrogate::npairs() const {
  unsigned c[4];
  ck(cudaSetDevice(device_), "cudaSetDevice");
  ck(cudaStreamSynchronize(stream_), "synchronize");
  ck(cudaMemcpy(c, counters_, sizeof(c), cudaMemcpyDeviceToHost), "D2H");
  return c[1];
}

void Surrogate::pairs_host(unsigned n, float* theta, double* logl) const {
  if (n > npairs()) throw Error(POFD_E_ARG, "more pairs asked for than are held");
  if (n == 0) return;
  if (theta)
    ck(cudaMemcpy(theta, ptheta_, static_cast<size_t>(n) * npar_ * sizeof(float),
                  cudaMemcpyDeviceToHost), "D2H pairs");
  if (logl) ck(cudaMemcpy(logl, plogl_, n * sizeof(double), cudaMemcpyDeviceToHost), "D2H pairs");
}

// Standardisation of the inputs (mean, 1/sd of the free parameters) and of
// the target (running max, sd of logL) from the pairs held.
unsigned Surrogate::refresh_scaling() {
  const unsigned n = npairs();
  if (n < 2) throw Error(POFD_E_ARG, "need at least two training pairs");
  // inputs standardised over the pairs whose target is not clipped (the
  // region the sampler explores once burnt in), when there are enough of
  // them; far-off burn-in points then sit at large |x| instead of setting
  // the scale
  const double clip = 25.0 + 2.5 * nin_;
  const unsigned K = nin_;
  ScaleArgs a{};
  a.n = static_cast<int>(n);
  a.R = static_cast<int>((n + scale_blocks_ - 1) / scale_blocks_);
  a.G = (a.n + a.R - 1) / a.R;
  a.npar = static_cast<int>(npar_);
  a.nin = static_cast<int>(K);
  a.clip = clip;
  a.theta = ptheta_;
  a.logl = plogl_;
  a.idx = idx_;
  for (int k = 0; k < 3; ++k) a.part[k] = scale_ + static_cast<size_t>(k) * scale_blocks_ * kScPart;
  a.out = scale_ + static_cast<size_t>(3) * scale_blocks_ * kScPart;
  k_scale<0><<<a.G, kScT, 0, stream_>>>(a);
  k_scale<1><<<a.G, kScT, 0, stream_>>>(a);
  k_scale<2><<<a.G, kScT, 0, stream_>>>(a);
  k_scale_out<<<1, kScT, 0, stream_>>>(a);
  ck(cudaGetLastError(), "k_scale");
  ck(cudaMemcpyAsync(h_stage_, a.out, 3 * kScPart * sizeof(double), cudaMemcpyDeviceToHost, stream_), "D2H");
  ck(cudaStreamSynchronize(stream_), "synchronize");
  // Whitening: mean and covariance of the inputs over those pairs, W = L^-1
  // with L L^T the covariance (Cholesky), so that the network sees
  // decorrelated unit-variance inputs (the knot values of a P(D) posterior
  // are strongly correlated).  A covariance that is not positive definite
  // falls back to the diagonal (1/sd) scaling.
  const bool all = h_stage_[kScCount] < std::max<size_t>(2 * K, 64);
  const double nu = all ? n : h_stage_[kScCount];
  std::vector<double> mean_in(K, 0.0), cov(K * K, 0.0);
  for (unsigned k = 0; k < K; ++k) mean_in[k] = h_stage_[(all ? kScAll : 0) + k] / nu;
  for (unsigned i = 0, e = 0; i < K; ++i)
    for (unsigned j = 0; j <= i; ++j, ++e) cov[i * K + j] = h_stage_[kScPart + e] / nu;
  std::vector<double> L(K * K, 0.0), Winv(K * K, 0.0);
  bool chol = true;
  for (unsigned a = 0; a < K && chol; ++a) {
    for (unsigned b = 0; b <= a; ++b) {
      double v = cov[a * K + b];
      for (unsigned c = 0; c < b; ++c) v -= L[a * K + c] * L[b * K + c];
      if (a == b) {
        if (!(v > 1e-12 * std::fabs(cov[a * K + a])) || !(v > 0)) {
          chol = false;
          break;
        }
        L[a * K + a] = std::sqrt(v);
      } else {
        L[a * K + b] = v / L[b * K + b];
      }
    }
  }
  if (chol) {
    // inverse of the lower-triangular factor, column by column
    for (unsigned c = 0; c < K; ++c)
      for (unsigned a = c; a < K; ++a) {
        double v = (a == c) ? 1.0 : 0.0;
        for (unsigned b = c; b < a; ++b) v -= L[a * K + b] * Winv[b * K + c];
        Winv[a * K + c] = v / L[a * K + a];
      }
  } else {
    for (unsigned k = 0; k < K; ++k) {
      const double sd = std::sqrt(std::max(cov[k * K + k], 0.0));
      Winv[k * K + k] = sd > 0 ? 1.0 / sd : 1.0;
    }
  }
  // target: logL - max, floored at -clip so that far-off burn-in points do
  // not set the scale; the floor grows with the number of inputs (a
  // chi-square of nin degrees of freedom sits near -nin/2)
  const double mx = h_stage_[2 * kScPart], s2 = h_stage_[kScPart + kScT - 1];
  float* wm = reinterpret_cast<float*>(h_stage_);  // the sums are done with
  float* mu = wm + kInPad * kInPad;
  std::fill(wm, mu + kInPad, 0.0f);
  for (unsigned a = 0; a < K; ++a) {
    mu[a] = static_cast<float>(mean_in[a]);
    for (unsigned b = 0; b < K; ++b) wm[a * kInPad + b] = static_cast<float>(Winv[a * K + b]);
  }
  whitened_ = chol;
  const double sd = std::sqrt(s2 / n);
  ymax_ = mx;
  clip_ = clip;
  ys_ = (sd > 0) ? sd : 1.0;
  ck(cudaMemcpyAsync(wm_, wm, (kInPad + 1) * kInPad * sizeof(float), cudaMemcpyHostToDevice, stream_),
     "upload");
  ck(cudaStreamSynchronize(stream_), "synchronize");  // other streams may use them
  scaled_ = true;
  return n;
}

// One training iteration on Mb rows (picked from the pair buffer, or its
// first Mb).  grads (8 tensors), when given, receive the loss gradients and
// the weights are not updated.  Eight launches: inputs and targets, three
// layers forward, output, two layers backward, all updates.
void Surrogate::iteration(int Mb, const Pick& pick, float lr, float** grads, cudaStream_t st) {
  const int Mp = (Mb + umma::kRows - 1) / umma::kRows * umma::kRows;
  const int H = static_cast<int>(H_);
  forward(Mb, ptheta_, static_cast<int>(npar_), pick,
          Targets{plogl_, ymax_, clip_, 1.0 / ys_, ws_.t, ws_.loss}, st);
  const int ntiles = H / ntile_for(Mp, H);
  const long long ne = static_cast<long long>(Mp) * (H / 4);
  launch_pdl(k_out_dz, dim3(static_cast<unsigned>((ne + 255) / 256)), dim3(256), 0, st, Mb, Mp, H,
             ntiles, ws_.ypart, ws_.t, ws_.y, ws_.dy, ws_.loss, p_[6], ws_.z[2], ws_.dz[2],
             ws_.dzt[2]);
  ++step_;
  AdamArgs ad{lr, 0.9f, 0.999f, 1e-8f, 1.0f - std::pow(0.9f, static_cast<float>(step_)),
              1.0f - std::pow(0.999f, static_cast<float>(step_))};
  bf16* Wb[3] = {w1b_, w2b_, w3b_};
  bf16* Wt[3] = {nullptr, w2t_, w3t_};
  for (int l = 2; l > 0; --l) {
    // dh_{l-1} = dz_l W_l: A = dz_l [Mp x H], B = W_l^T [H x H]
    const Gemm q = plan_gemm(Mp, H, H, ws_.dz[l], H, Wt[l], H, err_);
    launch_pdl(k_bwd_dx, q.grid, dim3(NTE), q.smem, st, q.a, q.b, q.g, ws_.z[l - 1],
               l > 1 ? ws_.dz[l - 1] : nullptr, ws_.dzt[l - 1], Mp);
  }
  UpdateAll u;
  size_t smem = 0;
  int blocks = 0;
  for (int l = 0; l < 3; ++l) {
    // G_l = dz_l^T X_l: A = dz_l^T [H x Mp], B = X_l^T [Nin x Mp]
    const int nin = (l == 0) ? kInPad : H;
    const Gemm q = plan_gemm(H, nin, Mp, ws_.dzt[l], Mp, (l == 0) ? ws_.xt : ws_.ht[l - 1], Mp, err_);
    u.w[l] = UpdateArgs{q.a, q.b, q.g, static_cast<int>(q.grid.x * q.grid.y),
                        static_cast<int>(q.grid.x), p_[2 * l], m_[2 * l], v_[2 * l],
                        grads ? grads[2 * l] : nullptr, Wb[l], Wt[l]};
    blocks += u.w[l].blocks;
    smem = std::max(smem, q.smem);
  }
  BiasArgs ba{};
  ba.Mp = Mp;
  ba.H = H;
  ba.dy = ws_.dy;
  ba.h3t = ws_.ht[2];
  for (int l = 0; l < 3; ++l) ba.dzt[l] = ws_.dzt[l];
  const int map[5] = {1, 3, 5, 6, 7};
  for (int q = 0; q < 5; ++q) {
    ba.p[q] = p_[map[q]];
    ba.m[q] = m_[map[q]];
    ba.v[q] = v_[map[q]];
    ba.grad_out[q] = grads ? grads[map[q]] : nullptr;
  }
  blocks += (4 * H + 1 + NTE / 32 - 1) / (NTE / 32);
  launch_pdl(k_update, dim3(blocks), dim3(NTE), smem, st, u, ba, ad);
  ck(cudaGetLastError(), "surrogate training");
}

void Surrogate::train(unsigned iters, unsigned batch, float lr, float* last_loss) {
  if (batch == 0 || batch > 65536) throw Error(POFD_E_ARG, "batch must be in [1, 65536]");
  ck(cudaSetDevice(device_), "cudaSetDevice");
  const unsigned n = refresh_scaling();
  const int Mb = static_cast<int>(batch);
  ensure_work((Mb + umma::kRows - 1) / umma::kRows * umma::kRows);
  ck(cudaMemset(err_, 0, sizeof(int)), "memset");
  for (unsigned it = 0; it < iters; ++it) {
    iteration(Mb, Pick{n, static_cast<unsigned long long>(step_) + 1, seed_}, lr, nullptr, stream_);
  }
  ck(cudaStreamSynchronize(stream_), "synchronize");
  check_err();
  if (last_loss) ck(cudaMemcpy(last_loss, ws_.loss, sizeof(float), cudaMemcpyDeviceToHost), "D2H");
}

void Surrogate::gradients(unsigned n, float** grads_dev, float* loss) {
  ck(cudaSetDevice(device_), "cudaSetDevice");
  if (!scaled_) refresh_scaling();
  if (n == 0 || n > npairs()) throw Error(POFD_E_ARG, "rows beyond the pairs held");
  ensure_work((static_cast<int>(n) + umma::kRows - 1) / umma::kRows * umma::kRows);
  ck(cudaMemset(err_, 0, sizeof(int)), "memset");
  const unsigned s0 = step_;
  iteration(static_cast<int>(n), Pick{}, 0.0f, grads_dev, stream_);
  step_ = s0;
  ck(cudaStreamSynchronize(stream_), "synchronize");
  check_err();
  if (loss) ck(cudaMemcpy(loss, ws_.loss, sizeof(float), cudaMemcpyDeviceToHost), "D2H");
}

void Surrogate::check_err() {
  int e = 0;
  ck(cudaMemcpy(&e, err_, sizeof(int), cudaMemcpyDeviceToHost), "D2H err");
  if (e) {
    ck(cudaMemset(err_, 0, sizeof(int)), "memset");
    throw Error(POFD_E_CUDA, "tensor-core wait timed out");
  }
}

void Surrogate::scaling(double* out) const {
  std::vector<float> mu(kInPad), wm(kInPad * kInPad);
  ck(cudaMemcpy(mu.data(), mu_, kInPad * sizeof(float), cudaMemcpyDeviceToHost), "D2H");
  ck(cudaMemcpy(wm.data(), wm_, wm.size() * sizeof(float), cudaMemcpyDeviceToHost), "D2H");
  for (int k = 0; k < kInPad; ++k) out[k] = mu[k];
  for (int k = 0; k < kInPad * kInPad; ++k) out[kInPad + k] = wm[k];
  const int o = kInPad + kInPad * kInPad;
  out[o] = ymax_;
  out[o + 1] = ys_;
  out[o + 2] = clip_;
  out[o + 3] = whitened_ ? 1.0 : 0.0;
}

// The tensor-core main loop on its own: C = A B^T (fp32).
void bf16_gemm(int M, int N, int K, const void* A, int lda, const void* B, int ldb, float* C,
               int ldc, int* err, cudaStream_t st) {
  set_gemm_attributes();
  const Gemm q = plan_gemm(M, N, K, static_cast<const bf16*>(A), lda, static_cast<const bf16*>(B),
                           ldb, err);
  k_gemm_f32<<<q.grid, NT, q.smem, st>>>(q.a, q.b, q.g, C, ldc);
  ck(cudaGetLastError(), "k_gemm_f32");
}

}  // namespace pofd
