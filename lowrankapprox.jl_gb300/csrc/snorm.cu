// The spectral norm's power iteration (src/snorm.jl:14-45) in one
// cooperative launch: y = D x, x = D' y with D = A, or D = A - B formed entry
// by entry, until the estimate settles or the iterations run out.
//
// Bound: FP64 arithmetic.  An iteration is 4 m n FP64 operations (96 us at 1.25
// TFLOP/s for 6000 x 5003) against two reads of A (71 us of HBM); Float32
// is bound by HBM.  So the kernel spends no FP64 instruction that is not one
// of the products where it can help it: the forward product gives a lane one
// row (no reduction across lanes), the adjoint product sums four columns per
// warp and folds the four totals together in one butterfly, and one
// warp per CTA takes the norm of its slice.  The iteration stays on the device:
// three grid barriers replace five launches, a one-warp norm of the whole
// vector (36 us at 5003 entries) and a host round trip.  6000 x 5003 Float64, 32
// iterations: 6.45 -> 4.93 ms (154 us an iteration, the FP64 unit two thirds
// busy).

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "internal.hpp"
#include "waits.cuh"

namespace lra {

namespace {

constexpr int PNT = 512;
constexpr int PNW = PNT / 32;

template <typename T>
struct PowerArgs {
  int64_t m, n;
  const T* A;
  int64_t lda;
  const T* B;  // null: D = A
  int64_t ldb;
  int herm;  // D = D' (m == n): one product per step
  int64_t niter;
  double atol, rtol;
  T* x;              // n: the start vector, then the iterate (unscaled)
  T* y;              // m
  T* part;           // partial sums of the forward (nch x m) or adjoint (gr x n) product
  int64_t nch, chunk;  // forward: column chunks
  int64_t gr, rchunk;  // adjoint: row chunks (a multiple of 64 rows)
  int* pexp;         // per CTA: its slice's largest binary exponent and the
  double* psum;      // sum of squares at that scale
  double* out;       // the estimate
  GridBar* bar;
};

// this CTA's slice [lo, hi) of x, by warp 0: the binary exponent of its
// largest entry (kZero: none nonzero, kInf: infinite) and the sum of squares
// at that scale.  One warp, and maxima as integers: a block-wide FP64
// reduction in every CTA costs more of the FP64 unit than the slice itself.
constexpr int kZero = -100000, kInf = 100000;

template <typename T>
__device__ void slice_norm(const PowerArgs<T>& P, int64_t lo, int64_t hi) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  unsigned long long mb = 0;
  for (int64_t i = lo + lane; i < hi; i += 32) {
    const double v = fabs((double)__ldcg(P.x + i));
    if (v == v) mb = max(mb, (unsigned long long)__double_as_longlong(v));
  }
  mb = warp_max(mb);
  const double mx = __longlong_as_double((long long)mb);
  const int e = mb == 0 ? kZero : isfinite(mx) ? ilogb(mx) : kInf;
  double s = 0;
  const double sc = e == kZero || e == kInf ? 1.0 : ldexp(1.0, -e);
  for (int64_t i = lo + lane; i < hi; i += 32) {
    const double t = (double)__ldcg(P.x + i) * sc;
    s = fma(t, t, s);
  }
  s = warp_sum(s);
  if (lane == 0) {
    P.pexp[blockIdx.x] = e;
    P.psum[blockIdx.x] = s;
  }
}

// the 2-norm from all slices, the same value in every CTA (rounded to T, as
// the vector's own norm would be)
template <typename T>
__device__ double full_norm(const PowerArgs<T>& P, double* s_nrm) {
  if (threadIdx.x < 32) {
    int e = kZero;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) e = max(e, __ldcg(P.pexp + b));
    e = warp_max(e);
    double r = e == kInf ? INFINITY : 0.0;
    if (e != kZero && e != kInf) {
      double s = 0;
      for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) {
        const int eb = __ldcg(P.pexp + b);
        const double q = __ldcg(P.psum + b);
        s += eb == kZero ? q : ldexp(q, 2 * max(eb - e, -2000));
      }
      s = warp_sum(s);
      r = ldexp(sqrt(s), e);
    }
    if (threadIdx.x == 0) *s_nrm = (double)(T)r;
  }
  __syncthreads();
  const double r = *s_nrm;
  __syncthreads();
  return r;
}

template <typename T, bool DIFF>
__global__ void __launch_bounds__(PNT, 2) snorm_power_kernel(const PowerArgs<T> P) {
  __shared__ double s_nrm;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t m = P.m, n = P.n;
  // warp-major order: a remainder of units spreads over all SMs
  const int64_t gw = (int64_t)wid * gridDim.x + blockIdx.x, W = (int64_t)gridDim.x * PNW;
  const int64_t gt = (int64_t)blockIdx.x * PNT + threadIdx.x, GT = (int64_t)gridDim.x * PNT;
  const int64_t xlo = n * blockIdx.x / gridDim.x, xhi = n * (blockIdx.x + 1) / gridDim.x;

  slice_norm(P, xlo, xhi);
  if (!grid_sync(P.bar)) return;
  double xnrm = full_norm(P, &s_nrm);
  double s = 1, t = 0;
  int64_t it = 0;
  while (s > 0 && fabs(s - t) > fmax(P.atol, t * P.rtol)) {
    if (it == P.niter) break;
    ++it;
    const T inv = (T)(1.0 / xnrm);
    // ---- forward: unit (row block of 32, column chunk) per warp, a lane per
    // row; x is scaled as it is read, 32 entries a load, and broadcast
    {
      const int64_t nrb = (m + 31) / 32, units = nrb * P.nch;
      for (int64_t u = gw; u < units; u += W) {
        const int64_t rb = u % nrb, c = u / nrb;
        const int64_t i = rb * 32 + lane;
        const bool in = i < m;
        const int64_t j0 = c * P.chunk, j1 = min(n, j0 + P.chunk);
        const T* a = P.A + (in ? i : m - 1);
        const T* b = DIFF ? P.B + (in ? i : m - 1) : nullptr;
        T acc = 0;
        for (int64_t j = j0; j < j1; j += 32) {
          const T xv = j + lane < j1 ? __ldcg(P.x + j + lane) * inv : T(0);
          const int cnt = (int)min((int64_t)32, j1 - j);
          for (int q0 = 0; q0 < cnt; q0 += 8) {
            T av[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const bool on = q0 + q < cnt;
              av[q] = on ? a[(j + q0 + q) * P.lda] : T(0);
              if (DIFF && on) av[q] -= b[(j + q0 + q) * P.ldb];
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) acc = fma(av[q], __shfl_sync(0xffffffffu, xv, q0 + q), acc);
          }
        }
        if (in) P.part[c * m + i] = acc;
      }
    }
    if (!grid_sync(P.bar)) return;
    // ---- y = the sum over the chunks
    T* yo = P.herm ? P.x : P.y;
    if (P.herm) {
      // (the slices of x, for the norm)
      for (int64_t i = xlo + threadIdx.x; i < xhi; i += PNT) {
        T v = 0;
        for (int64_t c = 0; c < P.nch; ++c) v += __ldcg(P.part + c * m + i);
        yo[i] = v;
      }
      __syncthreads();
      slice_norm(P, xlo, xhi);
      if (!grid_sync(P.bar)) return;
      xnrm = full_norm(P, &s_nrm);
      t = s;
      s = xnrm;
      continue;
    }
    for (int64_t i = gt; i < m; i += GT) {
      T v = 0;
      for (int64_t c = 0; c < P.nch; ++c) v += __ldcg(P.part + c * m + i);
      yo[i] = v;
    }
    if (!grid_sync(P.bar)) return;
    // ---- adjoint: unit (four columns, row chunk) per warp, so that a load of y
    // serves four columns
    {
      const int64_t nq = (n + 3) / 4, units = nq * P.gr;
      for (int64_t u = gw; u < units; u += W) {
        const int64_t j = u % nq * 4, br = u / nq;
        const int64_t r0 = br * P.rchunk, r1 = min(m, r0 + P.rchunk);
        const T* a[4];
        const T* b[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int64_t jj = min(j + g, n - 1);
          a[g] = P.A + jj * P.lda;
          b[g] = DIFF ? P.B + jj * P.ldb : nullptr;
        }
        T d[4] = {T(0), T(0), T(0), T(0)};
        int64_t i = r0 + lane;
        for (; i + 32 < r1; i += 64) {
          const T y0 = __ldcg(P.y + i), y1 = __ldcg(P.y + i + 32);
          T v0[4], v1[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            v0[g] = a[g][i];
            v1[g] = a[g][i + 32];
            if (DIFF) {
              v0[g] -= b[g][i];
              v1[g] -= b[g][i + 32];
            }
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) d[g] = fma(v1[g], y1, fma(v0[g], y0, d[g]));
        }
        if (i < r1) {
          const T y0 = __ldcg(P.y + i);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            T v = a[g][i];
            if (DIFF) v -= b[g][i];
            d[g] = fma(v, y0, d[g]);
          }
        }
        // transposed butterfly: lanes 8g..8g+7 end with column g's total
        const bool up = lane & 16;
        const T e0 = (up ? d[2] : d[0]) + __shfl_xor_sync(0xffffffffu, up ? d[0] : d[2], 16);
        const T e1 = (up ? d[3] : d[1]) + __shfl_xor_sync(0xffffffffu, up ? d[1] : d[3], 16);
        const bool hi = lane & 8;
        T v = (hi ? e1 : e0) + __shfl_xor_sync(0xffffffffu, hi ? e0 : e1, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const int64_t jl = j + (lane >> 3);
        if ((lane & 7) == 0 && jl < n) P.part[br * n + jl] = v;
      }
    }
    if (!grid_sync(P.bar)) return;
    for (int64_t i = xlo + threadIdx.x; i < xhi; i += PNT) {
      T v = 0;
      for (int64_t r = 0; r < P.gr; ++r) v += __ldcg(P.part + r * n + i);
      P.x[i] = v;
    }
    __syncthreads();
    slice_norm(P, xlo, xhi);
    if (!grid_sync(P.bar)) return;
    xnrm = full_norm(P, &s_nrm);
    t = s;
    s = sqrt(xnrm);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.out = s;
}

}  // namespace

WaitUnit wait_unit_snorm() { return this_wait_unit("snorm"); }

template <typename T>
double snorm_power(lra_ctx* ctx, int64_t m, int64_t n, const T* A, int64_t lda, const T* B, int64_t ldb, bool herm,
                   int64_t niter, double atol, double rtol, T* x) {
  const void* fn = B ? (const void*)snorm_power_kernel<T, true> : (const void*)snorm_power_kernel<T, false>;
  int per = 0;
  LRA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, PNT, 0));
  if (per < 1) fail(LRA_ECUDA, "snorm_power_kernel cannot be resident");
  // a CTA per 16K entries, up to two an SM: fewer CTAs make the grid barriers
  // of a small matrix cheaper than its share of the work saves
  const int64_t most = (int64_t)ctx->num_sms * std::min(per, 2);
  const int64_t G = std::max<int64_t>(1, std::min<int64_t>(most, (m * n + 16383) / 16384));
  PowerArgs<T> P;
  P.m = m;
  P.n = n;
  P.A = A;
  P.lda = lda;
  P.B = B;
  P.ldb = ldb;
  P.herm = herm ? 1 : 0;
  P.niter = niter;
  P.atol = atol;
  P.rtol = rtol;
  P.x = x;
  P.y = ctx->arena.alloc_n<T>(m);
  // forward units: (block of 32 rows) x nch column chunks; adjoint units: (four
  // columns) x gr row chunks, in whole groups of loads: at most one unit a warp
  // (a few second units would run alone, at latency speed), or several times
  // as many units as warps
  const int64_t W = G * PNW, nrb = (m + 31) / 32, nq = (n + 3) / 4;
  auto cut = [&](int64_t len, int64_t others, int64_t step) {
    const int64_t parts = others <= W ? W / others : (4 * W + others - 1) / others;
    return ((len + parts - 1) / parts + step - 1) / step * step;
  };
  P.chunk = cut(n, nrb, 8);
  P.nch = (n + P.chunk - 1) / P.chunk;
  P.rchunk = cut(m, nq, 64);
  P.gr = (m + P.rchunk - 1) / P.rchunk;
  P.part = ctx->arena.alloc_n<T>((size_t)std::max(P.nch * m, P.gr * n));
  P.pexp = ctx->arena.alloc_n<int>(G);
  P.psum = ctx->arena.alloc_n<double>(G);
  P.out = ctx->arena.alloc_n<double>(1);
  P.bar = reinterpret_cast<GridBar*>(ctx->arena.alloc(sizeof(GridBar)));
  LRA_CUDA(cudaMemsetAsync(P.bar, 0, sizeof(GridBar), ctx->stream));
  void* args[] = {&P};
  LRA_CUDA(cudaLaunchCooperativeKernel(fn, dim3((unsigned)G), dim3(PNT), args, 0, ctx->stream));
  post_launch(ctx, "snorm_power_kernel");
  double s = 0;
  GridBar hb;
  LRA_CUDA(cudaMemcpyAsync(&s, P.out, sizeof s, cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaMemcpyAsync(&hb, P.bar, sizeof hb, cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
  if (hb.err != 0) fail(LRA_ETIMEDOUT, "snorm: a grid barrier timed out");
  return s;
}

template double snorm_power<float>(lra_ctx*, int64_t, int64_t, const float*, int64_t, const float*, int64_t, bool,
                                   int64_t, double, double, float*);
template double snorm_power<double>(lra_ctx*, int64_t, int64_t, const double*, int64_t, const double*, int64_t, bool,
                                    int64_t, double, double, double*);

}  // namespace lra
