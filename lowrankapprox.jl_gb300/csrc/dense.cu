// Small dense factorizations of the post-processing stages, FP64 (input
// precision) on CUDA cores:
//   - one-sided (Hestenes) Jacobi SVD of a square k x k matrix, used for the
//     core SVD of psvdfact (src/psvd.jl:245) after a QR of (R V)^T, and --
//     on the shifted positive semidefinite B + s I -- for the k x k Hermitian
//     eigenproblem of pheigfact (src/pheig.jl:284);
//   - a symmetry test (ishermitian on a dense real matrix).
// One cooperative launch runs all sweeps: each round of the round-robin
// ordering rotates n/2 disjoint column pairs in parallel (one warp per
// pair), separated by bounded grid barriers.

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <mutex>
#include <set>
#include <vector>

#include "common.cuh"
#include "df64.cuh"
#include "internal.hpp"
#include "waits.cuh"

namespace lra {

namespace {

template <typename T>
struct JacParams {
  int64_t n;
  T* X;
  int64_t ldx;
  T* V;
  int64_t ldv;
  T* S;
  double tol;
  double stop;  // a sweep whose largest rotated cosine is below this is the last
  int max_sweeps;
  double* part;
  GridBar* bar;
  int* sweeps_out;
  // block Jacobi: V stays in global memory (only X's block pair in shared
  // memory), so that longer columns fit 8-column blocks
  int vglobal = 0;
  // LRA_TRACE: CTA 0's time in each phase of the block kernel, summed over
  // its block pairs (ns): load, local rounds, V, write-back, barrier
  unsigned long long* phase_ns = nullptr;
};

constexpr int JCH = 16;  // rows per lane per register chunk (512 rows)

__device__ __forceinline__ void rr_pair(int64_t r, int64_t s, int64_t nn, int64_t& p, int64_t& q) {
  auto pos = [&](int64_t i) -> int64_t { return i == 0 ? 0 : 1 + (i - 1 + r) % (nn - 1); };
  p = pos(s);
  q = pos(nn - 1 - s);
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT) jacobi_kernel(JacParams<T> P) {
  __shared__ double red[32];
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t gw = (int64_t)blockIdx.x * NW + wid;
  const int64_t W = (int64_t)gridDim.x * NW;
  const int64_t n = P.n;
  const int64_t nn = n + (n & 1);
  int sweep = 0;
  for (; sweep < P.max_sweeps; ++sweep) {
    double off = 0;
    for (int64_t r = 0; r < nn - 1; ++r) {
      for (int64_t s = gw; s < nn / 2; s += W) {
        int64_t p, q;
        rr_pair(r, s, nn, p, q);
        if (p >= n || q >= n) continue;
        if (p > q) {
          const int64_t t = p;
          p = q;
          q = t;
        }
        T* xp = P.X + p * P.ldx;
        T* xq = P.X + q * P.ldx;
        // both columns are pulled into registers with independent loads
        // (one L2 round trip per chunk), reduced, rotated and stored
        T a = 0, b = 0, g = 0;
        T u[JCH], w[JCH];
        const bool one = n <= 32 * JCH;
        for (int64_t b0 = 0; b0 < n; b0 += 32 * JCH) {
#pragma unroll
          for (int t = 0; t < JCH; ++t) {
            const int64_t i = b0 + lane + 32 * t;
            u[t] = i < n ? __ldcg(xp + i) : T(0);
            w[t] = i < n ? __ldcg(xq + i) : T(0);
          }
#pragma unroll
          for (int t = 0; t < JCH; ++t) {
            a = fma(u[t], u[t], a);
            b = fma(w[t], w[t], b);
            g = fma(u[t], w[t], g);
          }
        }
        a = warp_sum(a);
        b = warp_sum(b);
        g = warp_sum(g);
        if (a == 0 || b == 0) continue;
        const T rel = fabs(g) / sqrt(a * b);
        if (!(rel > (T)P.tol)) continue;
        off = fmax(off, (double)rel);
        const T zeta = (b - a) / (T(2) * g);
        const T t = copysign(T(1), zeta) / (fabs(zeta) + sqrt(T(1) + zeta * zeta));
        const T c = T(1) / sqrt(T(1) + t * t);
        const T sn = c * t;
        for (int64_t b0 = 0; b0 < n; b0 += 32 * JCH) {
          if (!one) {
#pragma unroll
            for (int tt = 0; tt < JCH; ++tt) {
              const int64_t i = b0 + lane + 32 * tt;
              u[tt] = i < n ? __ldcg(xp + i) : T(0);
              w[tt] = i < n ? __ldcg(xq + i) : T(0);
            }
          }
#pragma unroll
          for (int tt = 0; tt < JCH; ++tt) {
            const int64_t i = b0 + lane + 32 * tt;
            if (i < n) {
              xp[i] = c * u[tt] - sn * w[tt];
              xq[i] = sn * u[tt] + c * w[tt];
            }
          }
        }
        T* vp = P.V + p * P.ldv;
        T* vq = P.V + q * P.ldv;
        for (int64_t b0 = 0; b0 < n; b0 += 32 * JCH) {
#pragma unroll
          for (int tt = 0; tt < JCH; ++tt) {
            const int64_t i = b0 + lane + 32 * tt;
            u[tt] = i < n ? __ldcg(vp + i) : T(0);
            w[tt] = i < n ? __ldcg(vq + i) : T(0);
          }
#pragma unroll
          for (int tt = 0; tt < JCH; ++tt) {
            const int64_t i = b0 + lane + 32 * tt;
            if (i < n) {
              vp[i] = c * u[tt] - sn * w[tt];
              vq[i] = sn * u[tt] + c * w[tt];
            }
          }
        }
      }
      if (!grid_sync(P.bar)) return;
    }
    off = block_max(off, red);
    if (threadIdx.x == 0) P.part[blockIdx.x] = off;
    if (!grid_sync(P.bar)) return;
    double mx = 0;
    for (int b = threadIdx.x; b < gridDim.x; b += NT) mx = fmax(mx, __ldcg(P.part + b));
    mx = block_max(mx, red);
    if (!grid_sync(P.bar)) return;  // everyone read part before it is rewritten
    if (mx <= P.stop) {
      ++sweep;
      break;
    }
  }
  // singular values = column norms
  for (int64_t j = gw; j < n; j += W) {
    const T* x = P.X + j * P.ldx;
    double a = 0;
    for (int64_t i = lane; i < n; i += 32) {
      const double u = __ldcg(x + i);
      a = fma(u, u, a);
    }
    a = warp_sum(a);
    if (lane == 0) P.S[j] = (T)sqrt(a);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.sweeps_out = sweep;
}

// One CTA per column pair for Float64: the rows of the two columns are
// spread over all threads of the CTA (a warp-wide FP64 instruction costs
// tens of cycles on this part, so fewer rows per thread shorten every
// dependent chain), the three dot products are reduced through shared
// memory, and the rotation test g^2 > tol^2 a b needs no division or
// square root.
constexpr int JP_RCH = 8;  // rows per thread per register chunk

template <typename T, int NT>
__global__ void __launch_bounds__(NT) jacobi_pair_kernel(JacParams<T> P) {
  constexpr int NW = NT / 32;
  __shared__ T red[2][NT][3];
  __shared__ T rot_c[2], rot_s[2];
  __shared__ int rot_on[2];
  __shared__ int s_flag;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t n = P.n;
  const int64_t nn = n + (n & 1);
  const T tol2 = (T)(P.tol * P.tol), stop2 = (T)(P.stop * P.stop);
  int sweep = 0;
  int buf = 0;
  for (; sweep < P.max_sweeps; ++sweep) {
    int above = 0;  // a pair of this CTA had a cosine above the stopping level
    for (int64_t r = 0; r < nn - 1; ++r) {
      for (int64_t s = blockIdx.x; s < nn / 2; s += gridDim.x) {
        int64_t p, q;
        rr_pair(r, s, nn, p, q);
        if (p >= n || q >= n) continue;
        if (p > q) {
          const int64_t t = p;
          p = q;
          q = t;
        }
        T* xp = P.X + p * P.ldx;
        T* xq = P.X + q * P.ldx;
        T a = 0, b = 0, g = 0;
        T u[JP_RCH], w[JP_RCH];
        const bool one = n <= (int64_t)NT * JP_RCH;
        for (int64_t b0 = 0; b0 < n; b0 += (int64_t)NT * JP_RCH) {
#pragma unroll
          for (int c = 0; c < JP_RCH; ++c) {
            if (b0 + (int64_t)NT * c >= n) break;
            const int64_t i = b0 + threadIdx.x + (int64_t)NT * c;
            u[c] = i < n ? __ldcg(xp + i) : T(0);
            w[c] = i < n ? __ldcg(xq + i) : T(0);
          }
#pragma unroll
          for (int c = 0; c < JP_RCH; ++c) {
            if (b0 + (int64_t)NT * c >= n) break;
            a = fma(u[c], u[c], a);
            b = fma(w[c], w[c], b);
            g = fma(u[c], w[c], g);
          }
        }
        // partial dot products to shared memory; warp 0 alone reduces them
        // and computes the rotation (FP64 instructions cost tens of cycles
        // each here, so they are not repeated in every warp)
        red[buf][threadIdx.x][0] = a;
        red[buf][threadIdx.x][1] = b;
        red[buf][threadIdx.x][2] = g;
        __syncthreads();
        if (wid == 0) {
          T ra = 0, rb = 0, rg = 0;
#pragma unroll
          for (int k = 0; k < NW; ++k) {
            ra += red[buf][lane + 32 * k][0];
            rb += red[buf][lane + 32 * k][1];
            rg += red[buf][lane + 32 * k][2];
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            ra += __shfl_xor_sync(0xffffffffu, ra, o);
            rb += __shfl_xor_sync(0xffffffffu, rb, o);
            rg += __shfl_xor_sync(0xffffffffu, rg, o);
          }
          T cs = 1, sn = 0;
          int rot = 0;
          if (ra != 0 && rb != 0) {
            const T g2 = rg * rg, ab = ra * rb;
            if (g2 > tol2 * ab) {
              rot = 1;
              if (g2 > stop2 * ab) above = 1;
              // t = tan of the rotation angle, the smaller root of t^2 + 2 zeta t - 1
              const T d = rb - ra;
              const T t = (T(2) * rg) / (d + copysign(sqrt(fma(d, d, T(4) * g2)), d));
              cs = T(1) / sqrt(fma(t, t, T(1)));
              sn = cs * t;
            }
          }
          if (lane == 0) {
            rot_c[buf] = cs;
            rot_s[buf] = sn;
            rot_on[buf] = rot;
          }
        }
        __syncthreads();
        const int on = rot_on[buf];
        const T c = rot_c[buf], sn = rot_s[buf];
        buf ^= 1;  // the next pair reduces through the other buffer
        if (!on) continue;
        for (int64_t b0 = 0; b0 < n; b0 += (int64_t)NT * JP_RCH) {
          if (!one) {
#pragma unroll
            for (int cc = 0; cc < JP_RCH; ++cc) {
              if (b0 + (int64_t)NT * cc >= n) break;
              const int64_t i = b0 + threadIdx.x + (int64_t)NT * cc;
              u[cc] = i < n ? __ldcg(xp + i) : T(0);
              w[cc] = i < n ? __ldcg(xq + i) : T(0);
            }
          }
#pragma unroll
          for (int cc = 0; cc < JP_RCH; ++cc) {
            if (b0 + (int64_t)NT * cc >= n) break;
            const int64_t i = b0 + threadIdx.x + (int64_t)NT * cc;
            if (i < n) {
              xp[i] = c * u[cc] - sn * w[cc];
              xq[i] = sn * u[cc] + c * w[cc];
            }
          }
        }
        T* vp = P.V + p * P.ldv;
        T* vq = P.V + q * P.ldv;
        for (int64_t b0 = 0; b0 < n; b0 += (int64_t)NT * JP_RCH) {
#pragma unroll
          for (int cc = 0; cc < JP_RCH; ++cc) {
            if (b0 + (int64_t)NT * cc >= n) break;
            const int64_t i = b0 + threadIdx.x + (int64_t)NT * cc;
            u[cc] = i < n ? __ldcg(vp + i) : T(0);
            w[cc] = i < n ? __ldcg(vq + i) : T(0);
          }
#pragma unroll
          for (int cc = 0; cc < JP_RCH; ++cc) {
            if (b0 + (int64_t)NT * cc >= n) break;
            const int64_t i = b0 + threadIdx.x + (int64_t)NT * cc;
            if (i < n) {
              vp[i] = c * u[cc] - sn * w[cc];
              vq[i] = sn * u[cc] + c * w[cc];
            }
          }
        }
      }
      if (!grid_sync(P.bar)) return;
    }
    // any CTA above the stopping level keeps the sweeps going (warp 0 holds
    // the flag of this CTA)
    if (threadIdx.x == 0) P.part[blockIdx.x] = above ? 1.0 : 0.0;
    if (!grid_sync(P.bar)) return;
    if (threadIdx.x == 0) {
      int any = 0;
      for (int k = 0; k < (int)gridDim.x; ++k) any |= __ldcg(P.part + k) != 0.0;
      s_flag = any;
    }
    __syncthreads();
    const int any = s_flag;
    if (!grid_sync(P.bar)) return;  // everyone read part before it is rewritten
    if (!any) {
      ++sweep;
      break;
    }
  }
  // singular values = column norms, a warp per column
  const int64_t gw = (int64_t)blockIdx.x * NW + wid, W = (int64_t)gridDim.x * NW;
  for (int64_t j = gw; j < n; j += W) {
    const T* x = P.X + j * P.ldx;
    double acc = 0;
    for (int64_t i = lane; i < n; i += 32) {
      const double v = __ldcg(x + i);
      acc = fma(v, v, acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) P.S[j] = (T)sqrt(acc);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.sweeps_out = sweep;
}

// two FP32 values in one 64-bit register pair, for the packed FP32 pipe
// (fma/mul .f32x2: one instruction for both halves)
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
  f2_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float f2_lo(f2_t v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float f2_hi(f2_t v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
  f2_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
  f2_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// Block one-sided Jacobi for the FP32 sweeps: the columns are grouped in
// blocks of JBT; each grid-wide round pairs the blocks round-robin, and the
// CTA holding a block pair loads its 2 JBT columns of X and V into shared
// memory and rotates every pair among them there (2 JBT - 1 local rounds of
// JBT pairs, a warp per pair) before writing them back.  A sweep then costs
// about n / JBT grid barriers instead of n, and the local rotations also
// reach the pairs inside each block.  The local rotations are applied to X
// one by one and gathered into a 2 JBT x 2 JBT orthogonal matrix, which is
// applied to the block's columns of V once, a thread per row, after the
// local rounds.
constexpr int JB_RPL = 16;  // rows per lane in registers (columns up to 512 long)
constexpr int JB_QMAX = 16;  // 16-byte chunks a lane holds in the inter-block steps (columns up to 2048 long)

// 16 bytes, of which the first `bytes` come from src and the rest are zero
__device__ __forceinline__ void cp_async16z(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <int JBT>
__global__ void __launch_bounds__(JBT * 32) jacobi_block_kernel(JacParams<float> P) {
  extern __shared__ float jb_smem[];
  __shared__ double red[32];
  __shared__ __align__(16) float Ql[2 * JBT][2 * JBT];  // column k of the block's local rotation at Ql[k][.]
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t n = P.n;
  // column stride in shared memory: n rounded up to 16 bytes, the padding
  // rows zero, so that long columns move in 16-byte vectors
  const int64_t ld = (n + 3) & ~(int64_t)3;
  float* Xs = jb_smem;                        // [2 JBT][ld]
  float* Vs = jb_smem + (size_t)2 * JBT * ld;  // [2 JBT][ld], unless V stays in global memory
  const bool vg = P.vglobal != 0;
  // columns that start on 16 bytes move as 16-byte vectors
  const bool vec16 = (P.ldx & 3) == 0 && ((uintptr_t)P.X & 15) == 0 &&
                     (vg || ((P.ldv & 3) == 0 && ((uintptr_t)P.V & 15) == 0));
  const int64_t nblk = (n + JBT - 1) / JBT;
  const int64_t nbb = nblk + (nblk & 1);
  const float tol = (float)P.tol;
  int sweep = 0;
  for (; sweep < P.max_sweeps; ++sweep) {
    float off = 0;
    for (int64_t r = 0; r < nbb - 1; ++r) {
      for (int64_t s = blockIdx.x; s < nbb / 2; s += gridDim.x) {
        const bool stamp = P.phase_ns && blockIdx.x == 0 && threadIdx.x == 0;
        uint64_t t_ph = stamp ? globaltimer_ns() : 0;
        auto phase = [&](int i) {
          if (!stamp) return;
          const uint64_t t = globaltimer_ns();
          P.phase_ns[i] += t - t_ph;
          t_ph = t;
        };
        int64_t b1, b2;
        rr_pair(r, s, nbb, b1, b2);
        // local column k < JBT is column b1 JBT + k, k >= JBT is b2 JBT + k - JBT
        auto gcol = [&](int k) -> int64_t {
          const int64_t b = k < JBT ? b1 : b2;
          if (b >= nblk) return -1;
          const int64_t j = b * JBT + (k % JBT);
          return j < n ? j : -1;
        };
        // all 4 JBT n elements in flight at once (asynchronous copies), in
        // 16-byte vectors when the columns start on 16 bytes (the rows past n
        // zero-filled)
        for (int k = 0; k < 2 * JBT; ++k) {
          const int64_t j = gcol(k);
          if (vec16) {
            for (int64_t i = 4 * (int64_t)threadIdx.x; i < ld; i += 4 * JBT * 32) {
              const int bytes = j >= 0 ? (int)(4 * min((int64_t)4, n - i)) : 0;
              cp_async16z(Xs + k * ld + i, P.X + (j >= 0 ? i + j * P.ldx : 0), bytes);
              if (!vg) cp_async16z(Vs + k * ld + i, P.V + (j >= 0 ? i + j * P.ldv : 0), bytes);
            }
            continue;
          }
          for (int64_t i = threadIdx.x; i < ld; i += JBT * 32) {
            if (j >= 0 && i < n) {
              cp_async4(Xs + k * ld + i, P.X + i + j * P.ldx);
              if (!vg) cp_async4(Vs + k * ld + i, P.V + i + j * P.ldv);
            } else {
              Xs[k * ld + i] = 0.0f;
              if (!vg) Vs[k * ld + i] = 0.0f;
            }
          }
        }
        for (int e = threadIdx.x; e < 4 * JBT * JBT; e += JBT * 32)
          Ql[e / (2 * JBT)][e % (2 * JBT)] = e / (2 * JBT) == e % (2 * JBT) ? 1.0f : 0.0f;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        phase(0);
        unsigned long long vmask = 0;  // local columns that exist
#pragma unroll
        for (int k = 0; k < 2 * JBT; ++k) vmask |= (gcol(k) >= 0 ? 1ull : 0ull) << k;
        const int ni = (int)n;
        // Past the first round of a sweep (whose full local sweeps also
        // rotate the pairs inside each block, once a sweep), the block pair
        // of long columns takes inter-block steps only: warp w keeps column w
        // of block b1 in registers and meets column (w + step) mod JBT of
        // block b2, which moves from warp to warp through shared memory --
        // every inter-block pair once, in JBT steps that read and write one
        // column a warp instead of 2 JBT - 1 rounds that read and write all.
        // (registers for up to 2048 rows with 8-column blocks and fewer;
        // larger blocks have too few registers a thread)
        constexpr int QM = JBT <= 8 ? JB_QMAX : 1;
        const bool inter = r > 0 && ni > 32 * JB_RPL && ld <= (int64_t)4 * 32 * QM;
        if (inter) {
          const int p = wid;
          const int nq = (int)(ld / 4);
          const ulonglong2 z2 = make_ulonglong2(0ull, 0ull);
          ulonglong2* tp = reinterpret_cast<ulonglong2*>(Xs + p * ld);
          ulonglong2 top[QM];
#pragma unroll
          for (int c = 0; c < QM; ++c) {
            const int v = lane + 32 * c;
            top[c] = v < nq ? tp[v] : z2;
          }
          const bool pe = (vmask >> p) & 1ull;
          for (int st = 0; st < JBT; ++st) {
            const int q = JBT + (wid + st) % JBT;
            if (pe && ((vmask >> q) & 1ull)) {
              ulonglong2* qp = reinterpret_cast<ulonglong2*>(Xs + q * ld);
              ulonglong2 bot[QM];
#pragma unroll
              for (int c = 0; c < QM; ++c) {
                const int v = lane + 32 * c;
                bot[c] = v < nq ? qp[v] : z2;
              }
              f2_t a2 = 0, b2 = 0, g2 = 0;
#pragma unroll
              for (int c = 0; c < QM; ++c) {
                a2 = f2_fma(top[c].x, top[c].x, a2);
                a2 = f2_fma(top[c].y, top[c].y, a2);
                b2 = f2_fma(bot[c].x, bot[c].x, b2);
                b2 = f2_fma(bot[c].y, bot[c].y, b2);
                g2 = f2_fma(top[c].x, bot[c].x, g2);
                g2 = f2_fma(top[c].y, bot[c].y, g2);
              }
              const float a = warp_sum(f2_lo(a2) + f2_hi(a2));
              const float b = warp_sum(f2_lo(b2) + f2_hi(b2));
              const float g = warp_sum(f2_lo(g2) + f2_hi(g2));
              if (a != 0 && b != 0) {
                const float rel = fabsf(g) * rsqrtf(a * b);
                if (rel > tol) {
                  off = fmaxf(off, rel);
                  const float zeta = (b - a) / (2.0f * g);
                  const float t = copysignf(1.0f, zeta) / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
                  const float c = rsqrtf(1.0f + t * t);
                  const float sn = c * t;
                  const f2_t cc = f2_pack(c, c), ss = f2_pack(sn, sn), ns = f2_pack(-sn, -sn);
#pragma unroll
                  for (int k = 0; k < QM; ++k) {
                    const ulonglong2 u = top[k], w = bot[k];
                    top[k].x = f2_fma(ns, w.x, f2_mul(cc, u.x));
                    top[k].y = f2_fma(ns, w.y, f2_mul(cc, u.y));
                    bot[k].x = f2_fma(cc, w.x, f2_mul(ss, u.x));
                    bot[k].y = f2_fma(cc, w.y, f2_mul(ss, u.y));
                    const int v = lane + 32 * k;
                    if (v < nq) qp[v] = bot[k];
                  }
                  for (int l = lane; l < 2 * JBT; l += 32) {
                    const float qu = Ql[p][l], qw = Ql[q][l];
                    Ql[p][l] = c * qu - sn * qw;
                    Ql[q][l] = sn * qu + c * qw;
                  }
                }
              }
            }
            __syncthreads();
          }
#pragma unroll
          for (int c = 0; c < QM; ++c) {
            const int v = lane + 32 * c;
            if (v < nq) tp[v] = top[c];
          }
          __syncthreads();
        } else {
          for (int lr = 0; lr < 2 * JBT - 1; ++lr) {
            // round-robin pair of this warp among the 2 JBT local columns
            auto lpos = [&](int i) { return i == 0 ? 0 : 1 + (i - 1 + lr) % (2 * JBT - 1); };
            int p = lpos(wid), q = lpos(2 * JBT - 1 - wid);
            if (p > q) {
              const int t = p;
              p = q;
              q = t;
            }
            if (((vmask >> p) & 1ull) && ((vmask >> q) & 1ull)) {
              float* xp = Xs + p * ld;
              float* xq = Xs + q * ld;
              float a = 0, b = 0, g = 0;
              if (ni <= 32 * JB_RPL) {
                // both columns in registers for the dots and the update
                float u[JB_RPL], w[JB_RPL];
  #pragma unroll
                for (int t = 0; t < JB_RPL; ++t) {
                  const int i = lane + 32 * t;
                  u[t] = i < ni ? xp[i] : 0.0f;
                  w[t] = i < ni ? xq[i] : 0.0f;
                }
  #pragma unroll
                for (int t = 0; t < JB_RPL; ++t) {
                  a = fmaf(u[t], u[t], a);
                  b = fmaf(w[t], w[t], b);
                  g = fmaf(u[t], w[t], g);
                }
                a = warp_sum(a);
                b = warp_sum(b);
                g = warp_sum(g);
                if (a != 0 && b != 0) {
                  const float rel = fabsf(g) * rsqrtf(a * b);
                  if (rel > tol) {
                    off = fmaxf(off, rel);
                    const float zeta = (b - a) / (2.0f * g);
                    const float t = copysignf(1.0f, zeta) / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
                    const float c = rsqrtf(1.0f + t * t);
                    const float sn = c * t;
  #pragma unroll
                    for (int tt = 0; tt < JB_RPL; ++tt) {
                      const int i = lane + 32 * tt;
                      if (i < ni) {
                        xp[i] = c * u[tt] - sn * w[tt];
                        xq[i] = sn * u[tt] + c * w[tt];
                      }
                    }
                    for (int l = lane; l < 2 * JBT; l += 32) {
                      const float qu = Ql[p][l], qw = Ql[q][l];
                      Ql[p][l] = c * qu - sn * qw;
                      Ql[q][l] = sn * qu + c * qw;
                    }
                  }
                }
              } else {
                // long columns: 16-byte vectors (rows 4v .. 4v + 3 in lane v
                // mod 32) and the packed FP32 pipe, two accumulators a value
                const ulonglong2* vp = reinterpret_cast<const ulonglong2*>(xp);
                const ulonglong2* vq = reinterpret_cast<const ulonglong2*>(xq);
                const int nv = (int)(ld / 4);
                f2_t a2 = 0, b2 = 0, g2 = 0;
  #pragma unroll 4
                for (int v = lane; v < nv; v += 32) {
                  const ulonglong2 u = vp[v], w = vq[v];
                  a2 = f2_fma(u.x, u.x, a2);
                  a2 = f2_fma(u.y, u.y, a2);
                  b2 = f2_fma(w.x, w.x, b2);
                  b2 = f2_fma(w.y, w.y, b2);
                  g2 = f2_fma(u.x, w.x, g2);
                  g2 = f2_fma(u.y, w.y, g2);
                }
                a = warp_sum(f2_lo(a2) + f2_hi(a2));
                b = warp_sum(f2_lo(b2) + f2_hi(b2));
                g = warp_sum(f2_lo(g2) + f2_hi(g2));
                if (a != 0 && b != 0) {
                  const float rel = fabsf(g) * rsqrtf(a * b);
                  if (rel > tol) {
                    off = fmaxf(off, rel);
                    const float zeta = (b - a) / (2.0f * g);
                    const float t = copysignf(1.0f, zeta) / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
                    const float c = rsqrtf(1.0f + t * t);
                    const float sn = c * t;
                    const f2_t cc = f2_pack(c, c), ss = f2_pack(sn, sn), ns = f2_pack(-sn, -sn);
                    ulonglong2* wp = reinterpret_cast<ulonglong2*>(xp);
                    ulonglong2* wq = reinterpret_cast<ulonglong2*>(xq);
  #pragma unroll 4
                    for (int v = lane; v < nv; v += 32) {
                      const ulonglong2 u = wp[v], w = wq[v];
                      ulonglong2 up, uq;
                      up.x = f2_fma(ns, w.x, f2_mul(cc, u.x));
                      up.y = f2_fma(ns, w.y, f2_mul(cc, u.y));
                      uq.x = f2_fma(cc, w.x, f2_mul(ss, u.x));
                      uq.y = f2_fma(cc, w.y, f2_mul(ss, u.y));
                      wp[v] = up;
                      wq[v] = uq;
                    }
                    for (int l = lane; l < 2 * JBT; l += 32) {
                      const float qu = Ql[p][l], qw = Ql[q][l];
                      Ql[p][l] = c * qu - sn * qw;
                      Ql[q][l] = sn * qu + c * qw;
                    }
                  }
                }
              }
            }
            __syncthreads();
          }
        }
        phase(1);
        // the block's columns of V times the gathered rotation, a thread per
        // row (rows of V read and written in place, coalesced, when V stays
        // in global memory)
        if constexpr (JBT <= 8) {
          // two rows a thread at once: their 4 JBT entries are loaded
          // together (the latencies overlap), and each 16-byte read of the
          // rotation (which the compiler may not hoist out of the row loop)
          // serves both
          constexpr int NT = JBT * 32;
          for (int i = threadIdx.x; i < ni; i += 2 * NT) {
            const int i2 = i + NT;
            const bool two = i2 < ni;
            float v0[2 * JBT], v1[2 * JBT];
#pragma unroll
            for (int j = 0; j < 2 * JBT; ++j) {
              if (vg) {
                const int64_t gj = gcol(j);
                v0[j] = gj >= 0 ? P.V[i + gj * P.ldv] : 0.0f;
                v1[j] = gj >= 0 && two ? P.V[i2 + gj * P.ldv] : 0.0f;
              } else {
                v0[j] = Vs[j * ld + i];
                v1[j] = two ? Vs[j * ld + i2] : 0.0f;
              }
            }
#pragma unroll
            for (int k = 0; k < 2 * JBT; ++k) {
              float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
              for (int j = 0; j < 2 * JBT; j += 4) {
                float4 q;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w)
                             : "r"((uint32_t)__cvta_generic_to_shared(&Ql[k][j])));
                s0 = fmaf(v0[j], q.x, s0);
                s0 = fmaf(v0[j + 1], q.y, s0);
                s0 = fmaf(v0[j + 2], q.z, s0);
                s0 = fmaf(v0[j + 3], q.w, s0);
                s1 = fmaf(v1[j], q.x, s1);
                s1 = fmaf(v1[j + 1], q.y, s1);
                s1 = fmaf(v1[j + 2], q.z, s1);
                s1 = fmaf(v1[j + 3], q.w, s1);
              }
              if (vg) {
                const int64_t gk = gcol(k);
                if (gk >= 0) {
                  P.V[i + gk * P.ldv] = s0;
                  if (two) P.V[i2 + gk * P.ldv] = s1;
                }
              } else {
                Vs[k * ld + i] = s0;
                if (two) Vs[k * ld + i2] = s1;
              }
            }
          }
        } else {
          for (int i = threadIdx.x; i < ni; i += JBT * 32) {
            float acc[2 * JBT];
#pragma unroll
            for (int k = 0; k < 2 * JBT; ++k) acc[k] = 0.0f;
#pragma unroll 1
            for (int j = 0; j < 2 * JBT; ++j) {  // (not unrolled: Ql would be hoisted into registers)
              float v;
              if (vg) {
                const int64_t gj = gcol(j);
                v = gj >= 0 ? P.V[i + gj * P.ldv] : 0.0f;
              } else {
                v = Vs[j * ld + i];
              }
#pragma unroll
              for (int k = 0; k < 2 * JBT; ++k) acc[k] = fmaf(v, Ql[k][j], acc[k]);
            }
            if (vg) {
#pragma unroll
              for (int k = 0; k < 2 * JBT; ++k) {
                const int64_t gk = gcol(k);
                if (gk >= 0) P.V[i + gk * P.ldv] = acc[k];
              }
            } else {
#pragma unroll
              for (int k = 0; k < 2 * JBT; ++k) Vs[k * ld + i] = acc[k];
            }
          }
        }
        __syncthreads();
        phase(2);
        for (int k = 0; k < 2 * JBT; ++k) {
          const int64_t j = gcol(k);
          if (j < 0) continue;
          if (vec16) {
            // whole vectors up to the last full one, the rest by element
            const int64_t n4 = n & ~(int64_t)3;
            for (int64_t i = 4 * (int64_t)threadIdx.x; i < n4; i += 4 * JBT * 32) {
              *reinterpret_cast<float4*>(P.X + i + j * P.ldx) = *reinterpret_cast<const float4*>(Xs + k * ld + i);
              if (!vg)
                *reinterpret_cast<float4*>(P.V + i + j * P.ldv) = *reinterpret_cast<const float4*>(Vs + k * ld + i);
            }
            for (int64_t i = n4 + threadIdx.x; i < n; i += JBT * 32) {
              P.X[i + j * P.ldx] = Xs[k * ld + i];
              if (!vg) P.V[i + j * P.ldv] = Vs[k * ld + i];
            }
            continue;
          }
          for (int64_t i = threadIdx.x; i < n; i += JBT * 32) {
            P.X[i + j * P.ldx] = Xs[k * ld + i];
            if (!vg) P.V[i + j * P.ldv] = Vs[k * ld + i];
          }
        }
        __syncthreads();
        phase(3);
      }
      {
        const uint64_t t0 = P.phase_ns && blockIdx.x == 0 && threadIdx.x == 0 ? globaltimer_ns() : 0;
        if (!grid_sync(P.bar)) return;
        if (t0) P.phase_ns[4] += globaltimer_ns() - t0;
      }
    }
    const double offd = block_max((double)off, red);
    if (threadIdx.x == 0) P.part[blockIdx.x] = offd;
    if (!grid_sync(P.bar)) return;
    double mx = 0;
    for (int b = threadIdx.x; b < gridDim.x; b += JBT * 32) mx = fmax(mx, __ldcg(P.part + b));
    mx = block_max(mx, red);
    if (!grid_sync(P.bar)) return;
    if (mx <= P.stop) {
      ++sweep;
      break;
    }
  }
  // singular values = column norms, a warp per column
  const int64_t gw = (int64_t)blockIdx.x * JBT + wid, W = (int64_t)gridDim.x * JBT;
  for (int64_t j = gw; j < n; j += W) {
    const float* x = P.X + j * P.ldx;
    double acc = 0;
    for (int64_t i = lane; i < n; i += 32) {
      const double v = __ldcg(x + i);
      acc = fma(v, v, acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) P.S[j] = (float)sqrt(acc);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.sweeps_out = sweep;
}

// ---- FP32 one-sided Jacobi in one thread-block cluster ---------------------------
// Every column pair sits in the registers of one warp (X and V, RPL rows a
// lane), the whole n x n matrix across the CTAs of one cluster.  Each step
// rotates all nn/2 pairs at once; then the columns move one position along
// the round-robin tournament (slot 0 fixed, slot i <- slot i + 1, slot nn - 1
// <- slot 1), which pairs every two columns once in nn - 1 steps and brings
// every column back to its slot at the end of a sweep.  A column moves by the
// sender's stores into the receiver's shared-memory mailbox, double-buffered
// by step parity: within a CTA plain stores and a release arrival on the
// receiver's mbarrier, across CTAs stores into its distributed shared memory
// that count their bytes on that mbarrier (st.async); the receiver waits for
// the mbarrier's phase, with no barrier across the cluster per step.  Warp w owns slots w (top) and nn - 1 - w
// (bottom): its top moves to warp w - 1's top (warp 1's to warp 0's bottom,
// warp 0's stays), its bottom to warp w + 1's bottom (the last warp's to its
// own top).  The rotation of a pair is that of jacobi_block_kernel.
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory offset in CTA `rank`
__device__ __forceinline__ uint32_t dsmem_addr(const void* local, unsigned rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(r)
               : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
  return r;
}
// 16 / 8 bytes into this CTA's shared memory
__device__ __forceinline__ void mbox_st4(uint32_t a, f2_t x, f2_t y) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ void mbox_st2(uint32_t a, f2_t x) {
  asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(x) : "memory");
}

// A column in a mailbox: rows lane + 32 t of lane `lane` as 16-byte chunks
// (t = 4q .. 4q + 3 at float offset 4 (32 q + lane)), and when RPL is not a
// multiple of 4 the last two at 4 32 (RPL / 4) + 2 lane.  In registers the
// rows come in pairs: pair p holds t = 2p (low half) and 2p + 1 (high).
template <int RPL>
__device__ __forceinline__ void mbox_send(uint32_t base, int lane, const f2_t (&c)[RPL / 2]) {
#pragma unroll
  for (int q = 0; q < RPL / 4; ++q) mbox_st4(base + (uint32_t)((q * 32 + lane) * 16), c[2 * q], c[2 * q + 1]);
  if constexpr (RPL % 4 == 2) mbox_st2(base + (uint32_t)((RPL / 4) * 512 + lane * 8), c[RPL / 2 - 1]);
}
template <int RPL>
__device__ __forceinline__ void mbox_recv(const float* box, int lane, f2_t (&c)[RPL / 2]) {
  const ulonglong2* b4 = reinterpret_cast<const ulonglong2*>(box);
#pragma unroll
  for (int q = 0; q < RPL / 4; ++q) {
    const ulonglong2 v = b4[q * 32 + lane];
    c[2 * q] = v.x;
    c[2 * q + 1] = v.y;
  }
  if constexpr (RPL % 4 == 2) c[RPL / 2 - 1] = reinterpret_cast<const f2_t*>(box + (RPL / 4) * 128)[lane];
}

// Point-to-point exchange: a remote store that counts its bytes on the
// receiver's mbarrier (st.async ... complete_tx), a release arrival for a
// sender in the receiver's own CTA, and the receiver's bounded wait.
__device__ __forceinline__ void st_async16(uint32_t a, f2_t x, f2_t y, uint32_t mbar) {
  asm volatile(
      "{\n\t.reg .b32 x0, x1, y0, y1;\n\tmov.b64 {x0, x1}, %1;\n\tmov.b64 {y0, y1}, %2;\n\t"
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {x0, x1, y0, y1}, [%3];\n}" ::"r"(a),
      "l"(x), "l"(y), "r"(mbar)
      : "memory");
}
__device__ __forceinline__ void st_async8(uint32_t a, f2_t x, uint32_t mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a), "l"(x), "r"(mbar)
               : "memory");
}
template <int RPL>
__device__ __forceinline__ void mbox_send_async(uint32_t base, uint32_t mbar, int lane, const f2_t (&c)[RPL / 2]) {
#pragma unroll
  for (int q = 0; q < RPL / 4; ++q) st_async16(base + (uint32_t)((q * 32 + lane) * 16), c[2 * q], c[2 * q + 1], mbar);
  if constexpr (RPL % 4 == 2) st_async8(base + (uint32_t)((RPL / 4) * 512 + lane * 8), c[RPL / 2 - 1], mbar);
}
__device__ __forceinline__ void jc_mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void jc_arrive_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void jc_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(bar))
               : "memory");
}
__device__ __forceinline__ bool jc_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
      "p;\n}\n"
      : "=r"(ok)
      : "r"((uint32_t)__cvta_generic_to_shared(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait for a phase of `bar`, bounded: a wait that outlasts the limit, or an
// error word already set, sets / keeps the error and gives up.  Returns
// whether the data arrived; the whole warp agrees.
__device__ __forceinline__ bool jc_wait(uint64_t* bar, unsigned parity, int* err) {
  bool ok = true;
  if (*((volatile int*)err) != 0) {
    ok = false;
  } else {
    uint64_t t0 = 0;
    int spins = 0;
    while (!jc_try_wait(bar, parity)) {
      if (++spins < 64) continue;
      spins = 0;
      if (*((volatile int*)err) != 0) {
        ok = false;
        break;
      }
      const uint64_t t = globaltimer_ns();
      if (t0 == 0) {
        t0 = t;
      } else if (t - t0 > wait_limit_ns()) {
        atomicCAS(err, 0, 6);
        ok = false;
        break;
      }
    }
  }
  return __all_sync(0xffffffffu, ok);
}

template <int RPL>
__global__ void __launch_bounds__(512, 1) jacobi_cluster_kernel(JacParams<float> P, int nn) {
  static_assert(RPL % 2 == 0, "rows of a lane go in pairs");
  constexpr int NP = RPL / 2;
  extern __shared__ float4 jc_smem4[];
  float* mbox = reinterpret_cast<float*>(jc_smem4);
  __shared__ unsigned offv[3];  // the sweep's largest cosine (bits of a float >= 0), CTA 0's copy counts
  constexpr int COL = RPL * 32;  // floats of one column in a mailbox
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int NW = blockDim.x >> 5;
  const unsigned rank = cluster_rank();
  const int w = (int)rank * NW + wl;
  const int PW = nn / 2;
  const int n = (int)P.n;
  const float tol = (float)P.tol;
  // mailbox of local warp l, buffer b, slot s (0 top, 1 bottom), X (0) / V (1)
  auto box = [&](int b, int l, int sl, int xv) { return mbox + ((((size_t)b * NW + l) * 2 + sl) * 2 + xv) * COL; };
  f2_t xt[NP], xb[NP], vt[NP], vb[NP];
  {
    const int ct = w, cb = nn - 1 - w;
    auto ld = [&](const float* M, int64_t ldm, int col, int t) -> float {
      const int i = lane + 32 * t;
      return i < n && col < n ? M[i + (int64_t)col * ldm] : 0.0f;
    };
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      xt[p] = f2_pack(ld(P.X, P.ldx, ct, 2 * p), ld(P.X, P.ldx, ct, 2 * p + 1));
      vt[p] = f2_pack(ld(P.V, P.ldv, ct, 2 * p), ld(P.V, P.ldv, ct, 2 * p + 1));
      xb[p] = f2_pack(ld(P.X, P.ldx, cb, 2 * p), ld(P.X, P.ldx, cb, 2 * p + 1));
      vb[p] = f2_pack(ld(P.V, P.ldv, cb, 2 * p), ld(P.V, P.ldv, cb, 2 * p + 1));
    }
  }
  if (threadIdx.x < 3) offv[threadIdx.x] = 0u;
  // destinations of this warp's top and bottom columns
  int dt_w = -1, dt_s = 0;  // warp 0's top stays
  if (w >= 2) {
    dt_w = w - 1;
    dt_s = 0;
  } else if (w == 1) {
    dt_w = 0;
    dt_s = 1;
  }
  const int db_w = w <= PW - 2 ? w + 1 : w, db_s = w <= PW - 2 ? 1 : 0;
  const unsigned dt_r = dt_w >= 0 ? (unsigned)(dt_w / NW) : rank, db_r = (unsigned)(db_w / NW);
  const uint32_t off_remote = dsmem_addr(offv, 0);
  // Point-to-point: full[b][l] completes a phase when the columns of local
  // warp l for a step of parity b have arrived -- its own arrival with the
  // bytes the remote senders store (st.async counts them), plus one release
  // arrival from each sender in this CTA.  A sender never overwrites a
  // buffer before its receiver has read it: every receiver of a warp also
  // sends to it each step, so data of step s + 1 from the receiver means
  // step s was read before step s + 2 reuses the buffer.
  __shared__ __align__(8) uint64_t full[2][16];
  const int ts_w = w == 0 ? -1 : (w == PW - 1 ? w : w + 1);  // sender of this warp's top
  const int bs_w = w >= 1 ? w - 1 : 1;                       // of its bottom
  const bool ts_local = ts_w >= 0 && ts_w / NW == (int)rank, bs_local = bs_w / NW == (int)rank;
  const unsigned remote_bytes = (unsigned)(((ts_w >= 0 && !ts_local) ? 1 : 0) + (bs_local ? 0 : 1)) * 2u * 128u * RPL;
  if (lane == 0) {
    const unsigned cnt = 1u + (ts_local ? 1u : 0u) + (bs_local ? 1u : 0u);
    jc_mbar_init(&full[0][wl], cnt);
    jc_mbar_init(&full[1][wl], cnt);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster_barrier();  // every CTA of the cluster runs (its barriers set up) before any remote store
  int sweep = 0;
  unsigned step_par = 0;
  bool alive = true;  // no wait has given up
  for (; sweep < P.max_sweeps; ++sweep) {
    if (rank == 0 && threadIdx.x == 0) offv[(sweep + 1) % 3] = 0u;
    float off = 0;
    for (int step = 0; step < nn - 1; ++step) {
      if (lane == 0) jc_arrive_tx(&full[step_par & 1u][wl], remote_bytes);
      f2_t a2 = 0, b2 = 0, g2 = 0;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        a2 = f2_fma(xt[p], xt[p], a2);
        b2 = f2_fma(xb[p], xb[p], b2);
        g2 = f2_fma(xt[p], xb[p], g2);
      }
      float a = warp_sum(f2_lo(a2) + f2_hi(a2));
      float b = warp_sum(f2_lo(b2) + f2_hi(b2));
      float g = warp_sum(f2_lo(g2) + f2_hi(g2));
      if (a != 0 && b != 0) {
        const float rel = fabsf(g) * rsqrtf(a * b);
        if (rel > tol) {
          off = fmaxf(off, rel);
          // the angle need not be correctly rounded: (c, s) is a rotation
          // to rounding whatever t is
          const float zeta = __fdividef(b - a, 2.0f * g);
          const float tn = copysignf(__fdividef(1.0f, fabsf(zeta) + sqrtf(fmaf(zeta, zeta, 1.0f))), zeta);
          const float c = rsqrtf(fmaf(tn, tn, 1.0f));
          const float sn = c * tn;
          const f2_t cc = f2_pack(c, c), ss = f2_pack(sn, sn), ns = f2_pack(-sn, -sn);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const f2_t u = xt[p], v = xb[p];
            xt[p] = f2_fma(ns, v, f2_mul(cc, u));
            xb[p] = f2_fma(cc, v, f2_mul(ss, u));
            const f2_t pu = vt[p], pv = vb[p];
            vt[p] = f2_fma(ns, pv, f2_mul(cc, pu));
            vb[p] = f2_fma(cc, pv, f2_mul(ss, pu));
          }
        }
      }
      if (step == nn - 2 && lane == 0) {
        const uint32_t oa = off_remote + (uint32_t)((sweep % 3) * sizeof(unsigned));
        asm volatile("red.shared::cluster.max.u32 [%0], %1;" ::"r"(oa), "r"(__float_as_uint(off)) : "memory");
      }
      const int buf = (int)(step_par & 1u);
      // a local receiver's arrival releases the whole warp's stores
      if (alive && dt_w >= 0) {
        if (dt_r == rank) {
          mbox_send<RPL>((uint32_t)__cvta_generic_to_shared(box(buf, dt_w % NW, dt_s, 0)), lane, xt);
          mbox_send<RPL>((uint32_t)__cvta_generic_to_shared(box(buf, dt_w % NW, dt_s, 1)), lane, vt);
          __syncwarp();
          if (lane == 0) jc_arrive(&full[buf][dt_w % NW]);
        } else {
          const uint32_t mb = dsmem_addr(&full[buf][dt_w % NW], dt_r);
          mbox_send_async<RPL>(dsmem_addr(box(buf, dt_w % NW, dt_s, 0), dt_r), mb, lane, xt);
          mbox_send_async<RPL>(dsmem_addr(box(buf, dt_w % NW, dt_s, 1), dt_r), mb, lane, vt);
        }
      }
      if (alive) {
        if (db_r == rank) {
          mbox_send<RPL>((uint32_t)__cvta_generic_to_shared(box(buf, db_w % NW, db_s, 0)), lane, xb);
          mbox_send<RPL>((uint32_t)__cvta_generic_to_shared(box(buf, db_w % NW, db_s, 1)), lane, vb);
          __syncwarp();
          if (lane == 0) jc_arrive(&full[buf][db_w % NW]);
        } else {
          const uint32_t mb = dsmem_addr(&full[buf][db_w % NW], db_r);
          mbox_send_async<RPL>(dsmem_addr(box(buf, db_w % NW, db_s, 0), db_r), mb, lane, xb);
          mbox_send_async<RPL>(dsmem_addr(box(buf, db_w % NW, db_s, 1), db_r), mb, lane, vb);
        }
      }
      if (alive) alive = jc_wait(&full[buf][wl], (step_par >> 1) & 1u, &P.bar->err);
      if (w != 0) {
        mbox_recv<RPL>(box(buf, wl, 0, 0), lane, xt);
        mbox_recv<RPL>(box(buf, wl, 0, 1), lane, vt);
      }
      mbox_recv<RPL>(box(buf, wl, 1, 0), lane, xb);
      mbox_recv<RPL>(box(buf, wl, 1, 1), lane, vb);
      ++step_par;
    }
    // a cluster barrier a sweep orders every warp's maximum; a wait that
    // gave up anywhere ends the sweeps everywhere at the same point
    cluster_barrier();
    unsigned mb;
    asm volatile("ld.shared::cluster.u32 %0, [%1];"
                 : "=r"(mb)
                 : "r"(off_remote + (uint32_t)((sweep % 3) * sizeof(unsigned)))
                 : "memory");
    const bool failed = *((volatile int*)&P.bar->err) != 0;
    if ((double)__uint_as_float(mb) <= P.stop || failed) {
      ++sweep;
      break;
    }
  }
  // every column is back in its slot: slot c holds column c
  {
    const int ct = w, cb = nn - 1 - w;
    double st = 0, sb = 0;
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
      const int i = lane + 32 * t;
      const float x0 = t & 1 ? f2_hi(xt[t / 2]) : f2_lo(xt[t / 2]);
      const float x1 = t & 1 ? f2_hi(xb[t / 2]) : f2_lo(xb[t / 2]);
      if (i < n) {
        if (ct < n) {
          P.X[i + (int64_t)ct * P.ldx] = x0;
          P.V[i + (int64_t)ct * P.ldv] = t & 1 ? f2_hi(vt[t / 2]) : f2_lo(vt[t / 2]);
        }
        if (cb < n) {
          P.X[i + (int64_t)cb * P.ldx] = x1;
          P.V[i + (int64_t)cb * P.ldv] = t & 1 ? f2_hi(vb[t / 2]) : f2_lo(vb[t / 2]);
        }
      }
      st = fma((double)x0, (double)x0, st);
      sb = fma((double)x1, (double)x1, sb);
    }
    st = warp_sum(st);
    sb = warp_sum(sb);
    if (lane == 0) {
      if (ct < n) P.S[ct] = (float)sqrt(st);
      if (cb < n) P.S[cb] = (float)sqrt(sb);
    }
  }
  if (rank == 0 && threadIdx.x == 0) *P.sweeps_out = sweep;
  cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

// Double-float block Jacobi: the polish sweeps of the mixed-precision path,
// the same block-pair schedule as jacobi_block_kernel with X and V held as
// float pairs (df64.cuh) and every dot, rotation and update done in
// double-float arithmetic on the FP32 pipes.  Columns are kept orthogonal
// to about 1e-13, ample for the tolerances the mixed path accepts.
//
// Bound: the chain of a step (dot, warp reduction, angle, update), 2 JBT - 1
// steps a block pair and one pair a round.  Half the warps rotate X, the others
// apply the same rotations to V one step later, beside the next dots; a lane
// holds no more rows than the order needs; and a round waits for the two blocks
// that it takes, not for the grid.  Order 213, 10 sweeps: 16.2 -> 8.1 ms.
struct JacDf {
  int64_t n, ld;  // ld: a multiple of 4, rows n..ld - 1 zero
  float* Xh;
  float* Xl;
  float* Vh;
  float* Vl;
  double* S;
  double tol, stop;
  int max_sweeps;
  double* part;
  unsigned* done;  // rounds that each block of columns has been through
  GridBar* bar;
  int* sweeps_out;
};

// a pair's rotation, for V: 0 none, 1 a small angle (eps, sn), 2 any (c, s)
struct JdRot {
  int mode;
  float eps, sn;
  Df c, s;
};

__device__ __forceinline__ Df df_rot_a(Df c, Df s, Df u, Df w) { return df_add(df_mul(c, u), df_neg(df_mul(s, w))); }
__device__ __forceinline__ Df df_rot_b(Df c, Df s, Df u, Df w) { return df_add(df_mul(s, u), df_mul(c, w)); }

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// columns p and q (u and w: their values) rotated in place
template <int RPL>
__device__ __forceinline__ void jd_apply(const JdRot& R, int ni, int lane, const Df (&u)[RPL], const Df (&w)[RPL], float* ph,
                                         float* pl, float* qh, float* ql) {
  if (R.mode == 1) {
    // small angle: x' = x + delta, delta = -eps x -/+ s y in FP32
    // (c = 1 - eps, eps = t^2 / (r (1 + r)), r = sqrt(1 + t^2))
    const float eps = R.eps, sn = R.sn;
    auto bump = [&](Df x, float d) {
      float hs, e;
      two_sum(x.h, d, hs, e);
      return quick_two_sum(hs, x.l + e);
    };
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
      const int i = lane + 32 * t;
      if (i < ni) {
        const Df x1 = bump(u[t], fmaf(-sn, w[t].l, fmaf(-sn, w[t].h, -eps * u[t].h)));
        const Df x2 = bump(w[t], fmaf(sn, u[t].l, fmaf(sn, u[t].h, -eps * w[t].h)));
        ph[i] = x1.h;
        pl[i] = x1.l;
        qh[i] = x2.h;
        ql[i] = x2.l;
      }
    }
  } else {
#pragma unroll
    for (int t = 0; t < RPL; ++t) {
      const int i = lane + 32 * t;
      if (i < ni) {
        const Df x1 = df_rot_a(R.c, R.s, u[t], w[t]), x2 = df_rot_b(R.c, R.s, u[t], w[t]);
        ph[i] = x1.h;
        pl[i] = x1.l;
        qh[i] = x2.h;
        ql[i] = x2.l;
      }
    }
  }
}

template <int JBT, int RPL>
__global__ void __launch_bounds__(JBT * 64) jacobi_block_df_kernel(JacDf P) {
  extern __shared__ __align__(16) float jd_smem[];
  __shared__ JdRot s_rot[2][JBT];
  __shared__ int s_any;
  constexpr int NS = JBT * 32;  // threads of a side
  const int lane = threadIdx.x & 31, wid = (threadIdx.x >> 5) % JBT;
  const bool vside = threadIdx.x >= NS;
  const int st = threadIdx.x % NS;
  const int ni = (int)P.n, ld = (int)P.ld;
  const size_t plane = (size_t)2 * JBT * ld;
  float* const Sh = jd_smem + (vside ? 2 * plane : 0);  // this side's columns
  float* const Sl = Sh + plane;
  float* const Gh = vside ? P.Vh : P.Xh;
  float* const Gl = vside ? P.Vl : P.Xl;
  const int nblk = (ni + JBT - 1) / JBT;
  const int nbb = nblk + (nblk & 1);
  const float ftol = (float)P.tol, fstop = (float)P.stop;
  auto side_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(vside ? 2 : 1), "n"(NS) : "memory"); };
  int sweep = 0;
  for (; sweep < P.max_sweeps; ++sweep) {
    int above = 0;
    for (int r = 0; r < nbb - 1; ++r) {
      const unsigned gen = (unsigned)(sweep * (nbb - 1) + r);
      for (int s = blockIdx.x; s < nbb / 2; s += gridDim.x) {
        auto bpos = [&](int i) { return i == 0 ? 0 : 1 + (i - 1 + r) % (nbb - 1); };
        const int b1 = bpos(s), b2 = bpos(nbb - 1 - s);
        auto gcol = [&](int k) -> int {
          const int b = k < JBT ? b1 : b2;
          if (b >= nblk) return -1;
          const int j = b * JBT + (k % JBT);
          return j < ni ? j : -1;
        };
        // both blocks are through the round before (a wait that gives up sets
        // err, ends all waits, and the next grid barrier ends the kernel)
        if (st < 2) {
          const int b = st == 0 ? b1 : b2;
          if (b < nblk) {
            wait_reached(P.done + b, gen, &P.bar->err);
          }
        }
        side_sync();
        for (int t = st; t < 2 * JBT * (ld / 4); t += NS) {
          const int k = t / (ld / 4), i = (t - k * (ld / 4)) * 4, j = gcol(k);
          if (j < 0) continue;
          cp_async16(Sh + (size_t)k * ld + i, Gh + (size_t)j * ld + i);
          cp_async16(Sl + (size_t)k * ld + i, Gl + (size_t)j * ld + i);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        side_sync();
        unsigned vmask = 0;
#pragma unroll
        for (int k = 0; k < 2 * JBT; ++k) vmask |= (gcol(k) >= 0 ? 1u : 0u) << k;
        for (int step = 0; step < 2 * JBT; ++step) {
          const int lr = vside ? step - 1 : step;  // V a step behind
          if (lr >= 0 && lr < 2 * JBT - 1) {
            auto lpos = [&](int i) { return i == 0 ? 0 : 1 + (i - 1 + lr) % (2 * JBT - 1); };
            int p = lpos(wid), q = lpos(2 * JBT - 1 - wid);
            if (p > q) {
              const int t = p;
              p = q;
              q = t;
            }
            float* ph = Sh + p * ld;
            float* pl = Sl + p * ld;
            float* qh = Sh + q * ld;
            float* ql = Sl + q * ld;
            if (((vmask >> p) & 1u) && ((vmask >> q) & 1u) && (!vside || s_rot[lr & 1][wid].mode != 0)) {
              Df u[RPL], w[RPL];
#pragma unroll
              for (int t = 0; t < RPL; ++t) {
                const int i = lane + 32 * t;
                u[t] = i < ni ? Df{ph[i], pl[i]} : Df{0.f, 0.f};
                w[t] = i < ni ? Df{qh[i], ql[i]} : Df{0.f, 0.f};
              }
              if (vside) {
                const JdRot R = s_rot[lr & 1][wid];
                jd_apply<RPL>(R, ni, lane, u, w, ph, pl, qh, ql);
              } else {
                Df a{0.f, 0.f}, b{0.f, 0.f}, g{0.f, 0.f};
#pragma unroll
                for (int t = 0; t < RPL; ++t) {
                  df_fma_acc(a, u[t].h, u[t].l, u[t].h, u[t].l);
                  df_fma_acc(b, w[t].h, w[t].l, w[t].h, w[t].l);
                  df_fma_acc(g, u[t].h, u[t].l, w[t].h, w[t].l);
                }
                a = quick_two_sum(a.h, a.l);
                b = quick_two_sum(b.h, b.l);
                g = quick_two_sum(g.h, g.l);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                  a = df_add(a, df_shfl_xor(a, o));
                  b = df_add(b, df_shfl_xor(b, o));
                  g = df_add(g, df_shfl_xor(g, o));
                }
                JdRot R;
                R.mode = 0;
                R.eps = R.sn = 0.f;
                R.c = R.s = Df{0.f, 0.f};
                if (a.h > 0.f && b.h > 0.f) {
                  const float rel = fabsf(g.h) * rsqrtf(a.h) * rsqrtf(b.h);
                  if (rel > ftol) {
                    if (rel > fstop) above = 1;
                    // tan of the rotation angle from zeta = (b - a) / (2 g) in
                    // double-float; t itself in FP32: a rotation by an angle off
                    // by 1e-7 relative still shrinks g by 1e-7, and the rotation
                    // matrix below is orthogonal to double-float precision
                    const Df zeta = df_div(df_add(b, df_neg(a)), df_mul(Df{2.f, 0.f}, g));
                    const float z = zeta.h;
                    const float t = copysignf(1.0f, z) / (fabsf(z) + sqrtf(fmaf(z, z, 1.0f)));
                    if (fabsf(t) < 9.5367431640625e-07f) {
                      const float rt = sqrtf(fmaf(t, t, 1.0f));
                      R.mode = 1;
                      R.eps = t * t / (rt * (1.0f + rt));
                      R.sn = t / rt;
                    } else {
                      const Df td{t, 0.f};
                      R.mode = 2;
                      R.c = df_div(Df{1.f, 0.f}, df_sqrt(df_add(Df{1.f, 0.f}, df_mul(td, td))));
                      R.s = df_mul(R.c, td);
                    }
                  }
                }
                if (lane == 0) s_rot[lr & 1][wid] = R;
                if (R.mode != 0) jd_apply<RPL>(R, ni, lane, u, w, ph, pl, qh, ql);
              }
            } else if (!vside && lane == 0) {
              s_rot[lr & 1][wid].mode = 0;
            }
          }
          if (step + 1 < 2 * JBT) __syncthreads();
        }
        // X is done a step earlier and is written while V takes its last one
        if (vside) side_sync();
        for (int t = st; t < 2 * JBT * (ld / 4); t += NS) {
          const int k = t / (ld / 4), i = (t - k * (ld / 4)) * 4, j = gcol(k);
          if (j < 0) continue;
          __stcg(reinterpret_cast<float4*>(Gh + (size_t)j * ld + i), *reinterpret_cast<const float4*>(Sh + (size_t)k * ld + i));
          __stcg(reinterpret_cast<float4*>(Gl + (size_t)j * ld + i), *reinterpret_cast<const float4*>(Sl + (size_t)k * ld + i));
        }
        __syncthreads();
        if (threadIdx.x < 2) {
          const int b = threadIdx.x == 0 ? b1 : b2;
          if (b < nblk) {
            __threadfence();
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(P.done + b), "r"(gen + 1u) : "memory");
          }
        }
      }
    }
    // any rotation above the stopping level, over the grid
    above = __syncthreads_or(above);
    if (threadIdx.x == 0) P.part[blockIdx.x] = above ? 1.0 : 0.0;
    if (!grid_sync(P.bar)) return;
    if (threadIdx.x == 0) {
      int any = 0;
      for (int k = 0; k < (int)gridDim.x; ++k) any |= __ldcg(P.part + k) != 0.0;
      s_any = any;
    }
    __syncthreads();
    const int any = s_any;
    if (!grid_sync(P.bar)) return;
    if (!any) {
      ++sweep;
      break;
    }
  }
  // singular values = column norms, a warp per column
  const int gw = blockIdx.x * (2 * JBT) + (threadIdx.x >> 5), W = gridDim.x * (2 * JBT);
  for (int j = gw; j < ni; j += W) {
    Df acc{0.f, 0.f};
    for (int i = lane; i < ni; i += 32) {
      const float h = __ldcg(P.Xh + (size_t)j * ld + i), l = __ldcg(P.Xl + (size_t)j * ld + i);
      df_fma_acc(acc, h, l, h, l);
    }
    acc = quick_two_sum(acc.h, acc.l);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = df_add(acc, df_shfl_xor(acc, o));
    if (lane == 0) P.S[j] = sqrt(df_val(acc.h, acc.l));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.sweeps_out = sweep;
}

__global__ void df_from_double_kernel(int64_t n, const double* __restrict__ A, int64_t lda, float* __restrict__ H,
                                      float* __restrict__ L, int64_t ld, int identity) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ld * n; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % ld, j = t / ld;
    const double x = i >= n ? 0.0 : identity ? (i == j ? 1.0 : 0.0) : A[i + j * lda];
    const Df d = df_split(x);
    H[t] = d.h;
    L[t] = d.l;
  }
}

__global__ void df_to_double_kernel(int64_t n, const float* __restrict__ H, const float* __restrict__ L, int64_t ld,
                                    double* __restrict__ A, int64_t lda) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * n; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % n, j = t / n;
    A[i + j * lda] = df_val(H[i + j * ld], L[i + j * ld]);
  }
}

template <typename T>
__global__ void symcheck_kernel(int64_t n, const T* __restrict__ A, int64_t lda, int* bad) {
  const int64_t total = n * n;
  int local = 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % n, j = t / n;
    if (i < j && A[i + j * lda] != A[j + i * lda]) local = 1;
  }
  if (__syncthreads_or(local) && threadIdx.x == 0) atomicExch(bad, 1);
}

}  // namespace

// LRA_JACOBI_CLUSTER=0 keeps the FP32 sweeps on the block-pair kernel even
// where the matrix fits one cluster (both variants stay testable)
static bool jacobi_cluster_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("LRA_JACOBI_CLUSTER");
    return !(e && *e == '0');
  }();
  return on;
}

// The FP32 sweeps in one cluster (jacobi_cluster_kernel) when the columns fit
// the registers of its warps: false when they do not (or no cluster of the
// size needed can be scheduled), the caller then takes the block-pair kernel.
static bool jacobi_cluster(lra_ctx* ctx, JacParams<float>& P) {
  const int64_t n = P.n;
  if (!jacobi_cluster_enabled() || n < 64 || n > 32 * 14) return false;
  const int rpl = n <= 128 ? 4 : n <= 256 ? 8 : 14;
  const void* kern = rpl == 4   ? (const void*)jacobi_cluster_kernel<4>
                     : rpl == 8 ? (const void*)jacobi_cluster_kernel<8>
                                : (const void*)jacobi_cluster_kernel<14>;
  int optin = 0;
  LRA_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  const size_t per_warp = (size_t)1024 * rpl;  // two buffers x two slots x (X, V) x 32 rpl floats
  const int nw_max = (int)std::min<size_t>(16, ((size_t)optin - 1024) / per_warp);  // static smem below 1 KB
  const int64_t need = (n + 1) / 2;  // column pairs
  raise_smem_limit(ctx, kern);
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> portable_set;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!portable_set.count({kern, ctx->device})) {
      LRA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
      portable_set.insert({kern, ctx->device});
    }
  }
  if (ctx->tuning.jacobi_cluster == 1) return false;
  const int c_max = ctx->tuning.jacobi_cluster > 1 ? ctx->tuning.jacobi_cluster : 16;
  for (int c = c_max; c >= 2; --c) {
    const int64_t nw = (need + c - 1) / c;
    if (nw > nw_max || nw < 1) break;  // fewer CTAs only need more warps each
    const int pw = (int)(c * nw);
    if (pw < 2) continue;
    const size_t smem = per_warp * (size_t)nw;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3((unsigned)(nw * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (clusters < 1) continue;
    int nn = 2 * pw;
    void* args[] = {&P, &nn};
    LRA_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
    post_launch(ctx, "jacobi_cluster_kernel");
    if (trace_on()) std::fprintf(stderr, "[lra] jacobi f32 cluster n=%lld ctas=%d warps=%lld slots=%d\n", (long long)n,
                                 c, (long long)nw, nn);
    return true;
  }
  return false;
}

template <typename T>
void jacobi_svd(lra_ctx* ctx, int64_t n, T* X, int64_t ldx, T* V, int64_t ldv, T* S, bool quadratic_stop,
                double stop) {
  // Float64: a CTA of 128 threads per pair; Float32: block Jacobi with the
  // block pair in shared memory when it fits, else a warp per pair
  constexpr bool pair_cta = sizeof(T) == 8;
  constexpr int NT = 128;
  if (n <= 0) return;
  set_identity(ctx, n, n, V, ldv);
  const ArenaMark mk = ctx->arena.mark();
  // FP32: 8-column blocks (16-column blocks halve the grid barriers but
  // measured slower: the local sweeps become issue-bound on half the SMs);
  // 4-column blocks for the longer columns whose 8-column block pair does
  // not fit shared memory (up to about 3500 rows); a warp per pair beyond
  const size_t blk_cap = 210 * 1024;
  // 8-column blocks with the block pair of X and V in shared memory; for
  // longer columns V stays in global memory (read and written once per block
  // pair), up to about 3400 rows; beyond, a warp per pair
  int jbt = 8;
  const int64_t nld = (n + 3) & ~(int64_t)3;  // the kernel's padded column stride
  bool vglobal = (size_t)4 * jbt * nld * sizeof(float) > blk_cap;
  // the tuning table may ask for another block size (when it fits)
  const int want = ctx->tuning.jacobi_jb;
  if ((want == 4 || want == 8 || want == 16 || want == 32) && (size_t)2 * want * nld * sizeof(float) <= blk_cap) {
    jbt = want;
    vglobal = (size_t)4 * jbt * nld * sizeof(float) > blk_cap;
  }
  const size_t blk_smem = (size_t)(vglobal ? 2 : 4) * jbt * nld * sizeof(float);
  const bool block = !pair_cta && n >= 4 * jbt && blk_smem <= blk_cap;
  const void* kern = pair_cta ? (const void*)jacobi_pair_kernel<T, NT>
                     : !block ? (const void*)jacobi_kernel<T, NT>
                     : jbt == 32 ? (const void*)jacobi_block_kernel<32>
                     : jbt == 16 ? (const void*)jacobi_block_kernel<16>
                     : jbt == 8 ? (const void*)jacobi_block_kernel<8>
                                : (const void*)jacobi_block_kernel<4>;
  const int nt = block ? jbt * 32 : NT;
  const size_t smem = block ? blk_smem : 0;
  if (block) raise_smem_limit(ctx, (const void*)kern);
  int per_sm = 0;
  LRA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nt, smem));
  const int64_t pairs = (n + 1) / 2;
  int64_t units = pair_cta ? pairs : (pairs + NT / 32 - 1) / (NT / 32);
  if (block) {
    const int64_t nblk = (n + jbt - 1) / jbt;
    units = (nblk + 1) / 2;
  }
  // the FP64 pairs all at once (up to two CTAs per SM), the rest one CTA per SM
  int grid = (int)std::min<int64_t>(units, (int64_t)ctx->num_sms * (pair_cta ? 2 : 1));
  grid = std::max(1, std::min(grid, ctx->num_sms * std::max(per_sm, 1)));
  JacParams<T> P;
  P.n = n;
  P.X = X;
  P.ldx = ldx;
  P.V = V;
  P.ldv = ldv;
  P.S = S;
  P.vglobal = block && vglobal ? 1 : 0;
  P.tol = (double)Real<T>::eps * 2.0 * std::sqrt((double)n);
  // A sweep whose cosines were all below sqrt(tol)/10 leaves them near
  // tol^2/100 times a modest gap factor (quadratic convergence), so the
  // sweep that would only confirm it is skipped.
  P.stop = stop > 0 ? stop : (quadratic_stop ? std::sqrt(P.tol) * 0.1 : P.tol);
  P.max_sweeps = 40;
  P.part = ctx->arena.alloc_n<double>(grid);
  P.bar = reinterpret_cast<GridBar*>(ctx->arena.alloc(sizeof(GridBar)));
  P.sweeps_out = ctx->arena.alloc_n<int>(1);
  if (trace_on() && block) {
    P.phase_ns = ctx->arena.alloc_n<unsigned long long>(5);
    LRA_CUDA(cudaMemsetAsync(P.phase_ns, 0, 5 * sizeof(unsigned long long), ctx->stream));
  }
  LRA_CUDA(cudaMemsetAsync(P.bar, 0, sizeof(GridBar), ctx->stream));
  if constexpr (sizeof(T) == 4) {
    if (jacobi_cluster(ctx, P)) {
      int sweeps = 0;
      GridBar hb;
      LRA_CUDA(cudaMemcpyAsync(&hb, P.bar, sizeof(GridBar), cudaMemcpyDeviceToHost, ctx->stream));
      if (trace_on())
        LRA_CUDA(cudaMemcpyAsync(&sweeps, P.sweeps_out, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      LRA_CUDA(cudaStreamSynchronize(ctx->stream));
      ctx->arena.release(mk);
      if (hb.err != 0) fail(LRA_ETIMEDOUT, "jacobi: a column exchange between the cluster's CTAs timed out");
      if (trace_on()) std::fprintf(stderr, "[lra] jacobi f32 cluster n=%lld sweeps=%d\n", (long long)n, sweeps);
      return;
    }
  }
  void* args[] = {&P};
  LRA_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(nt), args, smem, ctx->stream));
  post_launch(ctx, pair_cta ? "jacobi_pair_kernel" : (block ? "jacobi_block_kernel" : "jacobi_kernel"));
  GridBar hb;
  int sweeps = 0;
  unsigned long long ph[5] = {0, 0, 0, 0, 0};
  LRA_CUDA(cudaMemcpyAsync(&hb, P.bar, sizeof(GridBar), cudaMemcpyDeviceToHost, ctx->stream));
  if (trace_on())
    LRA_CUDA(cudaMemcpyAsync(&sweeps, P.sweeps_out, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  if (P.phase_ns) LRA_CUDA(cudaMemcpyAsync(ph, P.phase_ns, sizeof(ph), cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
  ctx->arena.release(mk);
  if (hb.err != 0) fail(LRA_ETIMEDOUT, "jacobi: a grid barrier timed out");
  if (P.phase_ns)
    std::fprintf(stderr, "[lra] jacobi block CTA 0 ms: load %.2f local %.2f V %.2f write %.2f barrier %.2f\n",
                 ph[0] * 1e-6, ph[1] * 1e-6, ph[2] * 1e-6, ph[3] * 1e-6, ph[4] * 1e-6);
  if (trace_on())
    std::fprintf(stderr, "[lra] jacobi %s%s n=%lld sweeps=%d grid=%d\n", sizeof(T) == 8 ? "f64" : "f32",
                 block ? " block" : "", (long long)n, sweeps, grid);
}

bool jacobi_svd_df(lra_ctx* ctx, int64_t n, double* X, int64_t ldx, double* V, int64_t ldv, double* S, bool clusters) {
  // 4-column blocks: the double-float rotations are issue-bound, so the work
  // is spread over as many SMs as the block pairs allow
  constexpr int JDF = 4;
  if (n < 2 || n > 32 * JB_RPL) return false;
  const int64_t ld = (n + 3) / 4 * 4;
  const size_t smem = (size_t)8 * JDF * ld * sizeof(float);
  if (smem > 200 * 1024) return false;
  // rows a lane, the next power of two
  const void* kern = n <= 128 ? (const void*)jacobi_block_df_kernel<JDF, 4>
                     : n <= 256 ? (const void*)jacobi_block_df_kernel<JDF, 8>
                                : (const void*)jacobi_block_df_kernel<JDF, 16>;
  raise_smem_limit(ctx, kern);
  int per_sm = 0;
  LRA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, JDF * 64, smem));
  if (per_sm < 1) return false;
  const ArenaMark mk = ctx->arena.mark();
  const int64_t nblk = (n + JDF - 1) / JDF;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((nblk + 1) / 2, (int64_t)ctx->num_sms * per_sm));
  JacDf P;
  P.n = n;
  P.ld = ld;
  for (float** q : {&P.Xh, &P.Xl, &P.Vh, &P.Vl}) *q = ctx->arena.alloc_n<float>((size_t)ld * n);
  P.done = ctx->arena.alloc_n<unsigned>((size_t)nblk);
  LRA_CUDA(cudaMemsetAsync(P.done, 0, (size_t)nblk * sizeof(unsigned), ctx->stream));
  P.S = S;
  // double-float resolves cosines down to a few units of 2^-46 sqrt(n)
  P.tol = std::max((double)Real<double>::eps * 2.0 * std::sqrt((double)n), 8.0 * std::ldexp(1.0, -46) * std::sqrt((double)n));
  // quadratic convergence from the FP32 sweeps; but not among columns of equal
  // norms, whose rounding-level cosines no single sweep removes
  P.stop = clusters ? 4.0 * P.tol : std::sqrt(P.tol) * 0.1;
  P.max_sweeps = 40;
  P.part = ctx->arena.alloc_n<double>(grid);
  P.bar = reinterpret_cast<GridBar*>(ctx->arena.alloc(sizeof(GridBar)));
  P.sweeps_out = ctx->arena.alloc_n<int>(1);
  LRA_CUDA(cudaMemsetAsync(P.bar, 0, sizeof(GridBar), ctx->stream));
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n * n + 255) / 256, ctx->num_sms * 8));
  df_from_double_kernel<<<g, 256, 0, ctx->stream>>>(n, X, ldx, P.Xh, P.Xl, ld, 0);
  post_launch(ctx, "df_from_double_kernel");
  df_from_double_kernel<<<g, 256, 0, ctx->stream>>>(n, nullptr, n, P.Vh, P.Vl, ld, 1);
  post_launch(ctx, "df_from_double_kernel");
  void* args[] = {&P};
  LRA_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(JDF * 64), args, smem, ctx->stream));
  post_launch(ctx, "jacobi_block_df_kernel<JDF>");
  df_to_double_kernel<<<g, 256, 0, ctx->stream>>>(n, P.Xh, P.Xl, ld, X, ldx);
  post_launch(ctx, "df_to_double_kernel");
  df_to_double_kernel<<<g, 256, 0, ctx->stream>>>(n, P.Vh, P.Vl, ld, V, ldv);
  post_launch(ctx, "df_to_double_kernel");
  GridBar hb;
  int sweeps = 0;
  LRA_CUDA(cudaMemcpyAsync(&hb, P.bar, sizeof(GridBar), cudaMemcpyDeviceToHost, ctx->stream));
  if (trace_on())
    LRA_CUDA(cudaMemcpyAsync(&sweeps, P.sweeps_out, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
  ctx->arena.release(mk);
  if (hb.err != 0) fail(LRA_ETIMEDOUT, "jacobi: a grid barrier timed out");
  if (trace_on())
    std::fprintf(stderr, "[lra] jacobi df block n=%lld sweeps=%d grid=%d\n", (long long)n, sweeps, grid);
  return true;
}

template <typename T>
bool is_symmetric(lra_ctx* ctx, int64_t n, const T* A, int64_t lda) {
  if (ctx->linop) return ctx->linop->hermitian != 0;  // a HermitianLinearOperator is, by its type
  const ArenaMark mk = ctx->arena.mark();
  int* bad = ctx->arena.alloc_n<int>(1);
  LRA_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n * n + 255) / 256, (int64_t)ctx->num_sms * 16));
  symcheck_kernel<T><<<g, 256, 0, ctx->stream>>>(n, A, lda, bad);
  post_launch(ctx, "symcheck_kernel");
  int h = 0;
  LRA_CUDA(cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
  ctx->arena.release(mk);
  return h == 0;
}

template void jacobi_svd<float>(lra_ctx*, int64_t, float*, int64_t, float*, int64_t, float*, bool, double);
template void jacobi_svd<double>(lra_ctx*, int64_t, double*, int64_t, double*, int64_t, double*, bool, double);
template bool is_symmetric<float>(lra_ctx*, int64_t, const float*, int64_t);
template bool is_symmetric<double>(lra_ctx*, int64_t, const double*, int64_t);

}  // namespace lra

// ---- blocked Cholesky and right triangular solve ----------------------------------
// Used by the sketch-preconditioned Cholesky QR of the post-processing: the
// skeleton columns A[:, sk] times R11^{-1} (R11 from the pivoted QR of the
// sketch) are well conditioned, so their Gram matrix factors stably.

namespace lra {

namespace {

constexpr int CB = 32;  // diagonal block size

// Upper Cholesky of a jb x jb diagonal block in shared memory (256 threads), its
// upper triangle in place; *bad set when the block is not positive definite.
// LAPACK xPOTF2's order: R(c, c) = sqrt(.), row c times 1 / R(c, c), then the
// trailing block.  Lane j of warp i mod 8 keeps entry (i, j); the warp of row c
// updates it first, takes the root, the reciprocal and the scaling itself and
// leaves the row in xs (two buffers): one barrier a column.  Bound: that chain, a
// root and a divide.  With one thread for the scalars, three barriers and an
// index division an entry, order 370 took 329 us in FP32 and 365 us of order 213
// in FP64 (the whole factorization); 227 and 311 us with this block.
template <typename T>
__device__ void potrf_block(T (*a)[CB + 1], int jb, T (*xs)[CB], int* bad) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  T v[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) v[t] = wid + 8 * t < jb && lane < jb ? a[wid + 8 * t][lane] : T(0);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    for (int w = 0; w < 8; ++w) {
      const int c = 8 * t + w;
      if (c >= jb) break;
      if (wid == w) {
        T d = __shfl_sync(0xffffffffu, v[t], c);
        if (!(d > T(0))) {
          if (lane == 0) atomicExch(bad, 1);
          d = T(1);
        }
        const T r = sqrt(d), inv = T(1) / r;
        v[t] = lane == c ? r : v[t] * inv;
        xs[c & 1][lane] = v[t];
      }
      __syncthreads();
      const T xj = xs[c & 1][lane];
      // rows of this group of eight first: the next pivot row is among them
#pragma unroll
      for (int u = t; u < 4; ++u) {
        const int i = wid + 8 * u;
        if (i > c && lane >= i) v[u] = fma(-xs[c & 1][i], xj, v[u]);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int i = wid + 8 * t;
    if (i <= lane && lane < jb) a[i][lane] = v[t];
  }
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(256) potrf_diag_kernel(int jb, T* G, int64_t ldg, int* bad) {
  __shared__ T a[CB][CB + 1];
  __shared__ T xs[2][CB];
  for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
    const int i = t % jb, j = t / jb;
    a[i][j] = G[i + j * ldg];
  }
  __syncthreads();
  potrf_block<T>(a, jb, xs, bad);
  for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
    const int i = t % jb, j = t / jb;
    G[i + j * ldg] = i <= j ? a[i][j] : T(0);
  }
}

// The whole blocked right-looking Cholesky in one cooperative launch, of
// one matrix or two independent ones at once, each on CTAs of its own: every
// CTA factors each 32-wide diagonal block itself (the same operations, so the
// same bits; no barrier and no trip through memory between the block and its
// row), the CTAs solve the block row with a warp per column (lane i holds x_i)
// and update the upper trailing triangle in tiles of 32 x 32, with a bounded
// barrier of the matrix's CTAs after either.  Order 370 in FP32: 227 us with one CTA at
// the block and an element a thread, 142 us now; 213 in FP64: 311 and 281 us.
template <typename T>
struct PotrfJobs {
  int n;           // 1 or 2
  int64_t k[2];
  T* G[2];
  int64_t ldg[2];
  int* bad;        // one flag per matrix
};

template <typename T>
__global__ void __launch_bounds__(256) potrf_coop_kernel(PotrfJobs<T> J, GridBar* bars) {
  __shared__ T a[CB][CB + 1], pj[CB][CB + 1];
  __shared__ T rinv[CB];
  __shared__ T xs[2][CB];
  const int m = (int)blockIdx.x % J.n, g = (int)blockIdx.x / J.n;
  const int Gm = ((int)gridDim.x - m + J.n - 1) / J.n;  // CTAs of this matrix
  GridBar* bar = bars + m;
  const int64_t k = J.k[m], ldg = J.ldg[m];
  T* const G = J.G[m];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int64_t j0 = 0; j0 < k; j0 += CB) {
    // ---- 1. the diagonal block ----
    // (every read of G goes around L1: other CTAs wrote it in earlier phases)
    const int jb = (int)min((int64_t)CB, k - j0);
    const int64_t rest = k - j0 - jb, o = j0 + jb;
    if (rest <= 0 && g != 0) break;
    T* Gjj = G + j0 + j0 * ldg;
    for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) a[t % jb][t / jb] = __ldcg(Gjj + t % jb + (t / jb) * ldg);
    __syncthreads();
    potrf_block<T>(a, jb, xs, J.bad + m);
    // back to memory by one CTA, once every CTA has read the block as it was
    auto store_block = [&]() {
      for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
        const int i = t % jb, j = t / jb;
        if (i <= j) Gjj[i + j * ldg] = a[i][j];
      }
    };
    if (rest <= 0) {
      store_block();
      break;
    }
    // ---- 2. the block row: R_{b,>b} = R_bb^{-T} G_{b,>b}, a warp per column ----
    if (threadIdx.x < jb) rinv[threadIdx.x] = T(1) / a[threadIdx.x][threadIdx.x];
    __syncthreads();
    for (int64_t col = (int64_t)wid * Gm + g; col < rest; col += (int64_t)Gm * 8) {
      T* p = G + j0 + (o + col) * ldg;
      T x = lane < jb ? __ldcg(p + lane) : T(0);
      // x_i = (g_i - sum_{q<i} R_qi x_q) / R_ii, the sums accumulated lane-wise
      for (int i = 0; i < jb; ++i) {
        const T xi = __shfl_sync(0xffffffffu, x, i) * rinv[i];
        if (lane == i) x = xi;
        if (lane > i && lane < jb) x -= a[i][lane] * xi;
      }
      if (lane < jb) p[lane] = x;
    }
    if (!group_sync(bar, Gm)) return;
    if (g == 0) {
      store_block();
      __syncthreads();
    }
    // ---- 3. trailing upper triangle: G(i, j) -= sum_q R(q, i) R(q, j), o <= i <= j ----
    // (jb = 32 here)
    const int64_t nt = (rest + CB - 1) / CB;
    for (int64_t t = g; t < nt * nt; t += Gm) {
      const int64_t ti = t % nt * CB, tj = t / nt * CB;
      if (ti > tj) continue;
      T gij[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int64_t ci = ti + wid + 8 * r, cj = tj + wid + 8 * r;
        a[wid + 8 * r][lane] = ci < rest ? __ldcg(G + j0 + lane + (o + ci) * ldg) : T(0);
        pj[wid + 8 * r][lane] = cj < rest ? __ldcg(G + j0 + lane + (o + cj) * ldg) : T(0);
        gij[r] = ti + lane < rest && cj < rest && ti + lane <= cj ? __ldcg(G + o + ti + lane + (o + cj) * ldg) : T(0);
      }
      __syncthreads();
      T s[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 8
      for (int q = 0; q < CB; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r] = fma(a[lane][q], pj[wid + 8 * r][q], s[r]);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int64_t i = ti + lane, j = tj + wid + 8 * r;
        if (i <= j && j < rest) G[o + i + (o + j) * ldg] = gij[r] - s[r];
      }
      __syncthreads();
    }
    if (!group_sync(bar, Gm)) return;
  }
}

// panel: R_{b, >b} = R_bb^{-T} G_{b, >b} (jb x nc), one thread per column
template <typename T>
__global__ void potrf_panel_kernel(int jb, int64_t nc, const T* Rbb, int64_t ldr, T* P, int64_t ldp) {
  __shared__ T r[CB][CB + 1];
  __shared__ T rinv[CB];
  for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
    const int i = t % jb, j = t / jb;
    r[i][j] = Rbb[i + j * ldr];
  }
  if (threadIdx.x < jb) rinv[threadIdx.x] = T(1) / Rbb[threadIdx.x + threadIdx.x * ldr];
  __syncthreads();
  for (int64_t col = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; col < nc; col += (int64_t)gridDim.x * blockDim.x) {
    T* p = P + col * ldp;
    T x[CB];
#pragma unroll
    for (int i = 0; i < CB; ++i)
      if (i < jb) x[i] = p[i];
#pragma unroll
    for (int i = 0; i < CB; ++i) {
      if (i < jb) {
        T s = x[i];
#pragma unroll
        for (int q = 0; q < CB; ++q)
          if (q < i) s -= r[q][i] * x[q];
        x[i] = s * rinv[i];
      }
    }
#pragma unroll
    for (int i = 0; i < CB; ++i)
      if (i < jb) p[i] = x[i];
  }
}

// X_b <- X_b R_bb^{-1} (m x jb), one thread per row
template <typename T>
__global__ void trsm_right_diag_kernel(int64_t m, int jb, const T* Rbb, int64_t ldr, T* X, int64_t ldx) {
  __shared__ T r[CB][CB + 1];
  __shared__ T rinv[CB];
  for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
    const int i = t % jb, j = t / jb;
    r[i][j] = Rbb[i + j * ldr];
  }
  if (threadIdx.x < jb) rinv[threadIdx.x] = T(1) / Rbb[threadIdx.x + threadIdx.x * ldr];
  __syncthreads();
  for (int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; row < m; row += (int64_t)gridDim.x * blockDim.x) {
    T x[CB];
#pragma unroll
    for (int j = 0; j < CB; ++j)
      if (j < jb) x[j] = X[row + j * ldx];
    // x R = b: x_j = (b_j - sum_{i<j} x_i R_ij) / R_jj
#pragma unroll
    for (int j = 0; j < CB; ++j) {
      if (j < jb) {
        T s = x[j];
#pragma unroll
        for (int i = 0; i < CB; ++i)
          if (i < j) s -= x[i] * r[i][j];
        x[j] = s * rinv[j];
      }
    }
#pragma unroll
    for (int j = 0; j < CB; ++j)
      if (j < jb) X[row + j * ldx] = x[j];
  }
}

// X[0:jb, :] <- Rbb^{-1} X[0:jb, :] for an upper-triangular jb x jb block
template <typename T>
__global__ void trsm_left_diag_kernel(int jb, int64_t nrhs, const T* Rbb, int64_t ldr, T* X, int64_t ldx) {
  __shared__ T r[CB][CB + 1];
  __shared__ T rinv[CB];
  for (int t = threadIdx.x; t < jb * jb; t += blockDim.x) {
    const int i = t % jb, j = t / jb;
    r[i][j] = Rbb[i + j * ldr];
  }
  if (threadIdx.x < jb) rinv[threadIdx.x] = T(1) / Rbb[threadIdx.x + threadIdx.x * ldr];
  __syncthreads();
  for (int64_t col = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; col < nrhs;
       col += (int64_t)gridDim.x * blockDim.x) {
    T* xc = X + col * ldx;
    T x[CB];
#pragma unroll
    for (int i = 0; i < CB; ++i)
      if (i < jb) x[i] = xc[i];
    // R x = b: x_i = (b_i - sum_{q>i} R_iq x_q) / R_ii, bottom up
#pragma unroll
    for (int i = CB - 1; i >= 0; --i) {
      if (i < jb) {
        T s = x[i];
#pragma unroll
        for (int q = CB - 1; q > i; --q)
          if (q < jb) s -= r[i][q] * x[q];
        x[i] = s * rinv[i];
      }
    }
#pragma unroll
    for (int i = 0; i < CB; ++i)
      if (i < jb) xc[i] = x[i];
  }
}

// ---- the whole Float32 solve in one launch ------------------------------------
// trsm_upper's and trsm_right_upper's recursion (halves of multiples of 32, a
// product between them, blocks of at most 32) on a few right-hand sides a CTA,
// which wait in shared memory: kTfN columns of R^{-1} X, or rows of X R^{-1}.
// Every entry sees the recursion's operations in its order: a product's sum
// from 0 over its inner index, subtracted once; within a block its own chain.
// Same bits as the recursion in launches, which cost one per block and product
// (rank 363: 23 launches of 9 to 14 us).  Bound: the chain of the blocks and R's
// way through L2, read once by every CTA; hence the limit on the right-hand sides.
// Rank 757, 3339 columns: 0.61 ms in launches, 0.385 so; the five solves of a psvd of
// rank 302: 1.0 and 0.39 ms.
constexpr int kTfN = 8;      // right-hand sides a CTA, a warp each in a block
constexpr int kTfMax = 1024;

template <int NCT>
__device__ __forceinline__ void tf_load(const float* x, float (&v)[NCT]) {
  if constexpr (NCT >= 4) {
#pragma unroll
    for (int c = 0; c < NCT; c += 4) {
      const float4 t = *reinterpret_cast<const float4*>(x + c);
      v[c] = t.x, v[c + 1] = t.y, v[c + 2] = t.z, v[c + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int c = 0; c < NCT; ++c) v[c] = x[c];
  }
}

template <bool RIGHT, int NCT>
__device__ __forceinline__ void tf_update(const float* __restrict__ R, int64_t ldr, float* xs, int r0, int nr, int q0, int nq,
                                          int tid, int nthreads) {
  // rows r0..r0+nr (RIGHT: columns) of each right-hand side take those q0..q0+nq away
  const int groups = kTfN / NCT, per = nthreads / groups;
  const int g = tid / per;
  for (int i = tid % per; i < nr; i += per) {
    float acc[NCT];
#pragma unroll
    for (int c = 0; c < NCT; ++c) acc[c] = 0.f;
    const float* r = RIGHT ? R + q0 + (int64_t)(r0 + i) * ldr : R + r0 + i + (int64_t)q0 * ldr;
    const int64_t step = RIGHT ? 1 : ldr;
    const float* x = xs + q0 * kTfN + g * NCT;
    float rn[8];  // the next eight entries of R are on their way
#pragma unroll
    for (int u = 0; u < 8; ++u) rn[u] = u < nq ? __ldg(r + u * step) : 0.f;
    for (int q = 0; q < nq; q += 8) {
      float rv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        rv[u] = rn[u];
        rn[u] = q + 8 + u < nq ? __ldg(r + (q + 8 + u) * step) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (q + u < nq) {
          float xv[NCT];
          tf_load<NCT>(x + (q + u) * kTfN, xv);
#pragma unroll
          for (int c = 0; c < NCT; ++c) acc[c] = fmaf(rv[u], xv[c], acc[c]);
        }
    }
    float* y = xs + (r0 + i) * kTfN + g * NCT;
#pragma unroll
    for (int c = 0; c < NCT; ++c) y[c] -= acc[c];
  }
}

template <bool RIGHT>
__global__ void __launch_bounds__(kTfN * 32) trsm_fused_kernel(int k, int64_t nrhs, const float* __restrict__ R, int64_t ldr,
                                                               float* X, int64_t ldx) {
  extern __shared__ __align__(16) float tf_x[];  // [k][kTfN]: a product reads all right-hand sides of an entry
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int64_t c0 = (int64_t)blockIdx.x * kTfN;
  const int nc = (int)min((int64_t)kTfN, nrhs - c0);
  for (int t = tid; t < k * kTfN; t += kTfN * 32) {
    const int c = RIGHT ? t % kTfN : t / k, i = RIGHT ? t / kTfN : t % k;
    tf_x[i * kTfN + c] = c < nc ? (RIGHT ? X[c0 + c + i * ldx] : X[i + (c0 + c) * ldx]) : 0.f;
  }
  __syncthreads();
  // the recursion: (begin, length) still to be solved, or (begin, length) whose
  // product is due (length negative)
  int sb[24], sl[24], top = 0;
  sb[0] = 0;
  sl[0] = k;
  top = 1;
  while (top > 0) {
    --top;
    const int b = sb[top];
    int len = sl[top];
    if (len > 32) {
      const int k1 = (len / 2 + 31) / 32 * 32;
      // done last, pushed first
      sb[top] = RIGHT ? b + k1 : b;
      sl[top++] = RIGHT ? len - k1 : k1;
      sb[top] = b;
      sl[top++] = -len;
      sb[top] = RIGHT ? b : b + k1;
      sl[top++] = RIGHT ? k1 : len - k1;
      continue;
    }
    if (len < 0) {
      len = -len;
      const int k1 = (len / 2 + 31) / 32 * 32, k2 = len - k1;
      const int r0 = RIGHT ? b + k1 : b, nr = RIGHT ? k2 : k1, q0 = RIGHT ? b : b + k1, nq = RIGHT ? k1 : k2;
      if (nr > 128)
        tf_update<RIGHT, 8>(R, ldr, tf_x, r0, nr, q0, nq, tid, kTfN * 32);
      else if (nr > 64)
        tf_update<RIGHT, 4>(R, ldr, tf_x, r0, nr, q0, nq, tid, kTfN * 32);
      else if (nr > 32)
        tf_update<RIGHT, 2>(R, ldr, tf_x, r0, nr, q0, nq, tid, kTfN * 32);
      else
        tf_update<RIGHT, 1>(R, ldr, tf_x, r0, nr, q0, nq, tid, kTfN * 32);
      __syncthreads();
      continue;
    }
    // a block: warp = right-hand side, lane = entry
    const float* Rb = R + b + (int64_t)b * ldr;
    const float rinv = lane < len ? 1.0f / __ldg(Rb + lane + (int64_t)lane * ldr) : 0.f;
    float s = lane < len ? tf_x[(b + lane) * kTfN + wid] : 0.f, y = 0.f;
    float rr[32];
#pragma unroll
    for (int q = 0; q < 32; ++q)
      rr[q] = q < len && lane < len && (RIGHT ? q < lane : lane < q)
                  ? __ldg(RIGHT ? Rb + q + (int64_t)lane * ldr : Rb + lane + (int64_t)q * ldr)
                  : 0.f;
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const int q = RIGHT ? t : 31 - t;
      if (q < len) {
        const float xq = __shfl_sync(0xffffffffu, s * rinv, q);
        if (lane == q) y = xq;
        if (RIGHT ? lane > q : lane < q) s = fmaf(-rr[q], xq, s);
      }
    }
    if (lane < len) tf_x[(b + lane) * kTfN + wid] = y;
    __syncthreads();
  }
  for (int t = tid; t < k * kTfN; t += kTfN * 32) {
    const int c = RIGHT ? t % kTfN : t / k, i = RIGHT ? t / kTfN : t % k;
    if (c < nc) (RIGHT ? X[c0 + c + i * ldx] : X[i + (c0 + c) * ldx]) = tf_x[i * kTfN + c];
  }
}

}  // namespace

bool trsm_fused(lra_ctx* ctx, bool right, int64_t k, int64_t nrhs, const float* R, int64_t ldr, float* X, int64_t ldx) {
  if (k > kTfMax || nrhs > (int64_t)ctx->num_sms * 4 * kTfN) return false;
  const size_t smem = (size_t)kTfN * (size_t)k * sizeof(float);
  const unsigned g = (unsigned)((nrhs + kTfN - 1) / kTfN);
  if (right)
    trsm_fused_kernel<true><<<g, kTfN * 32, smem, ctx->stream>>>((int)k, nrhs, R, ldr, X, ldx);
  else
    trsm_fused_kernel<false><<<g, kTfN * 32, smem, ctx->stream>>>((int)k, nrhs, R, ldr, X, ldx);
  post_launch(ctx, "trsm_fused_kernel");
  return true;
}

// one or two Cholesky factorizations G_m = R_m^T R_m in place (upper R,
// lower part zeroed) in one cooperative launch; ok[m] false when G_m is not
// numerically positive definite
template <typename T>
void potrf_upper_batch(lra_ctx* ctx, int n, const int64_t* k, T* const* G, const int64_t* ldg, bool* ok);

// Blocked right-looking Cholesky on the tensor-core path for orders past
// kPotrfPanel * 2: per panel of kPotrfPanel columns the diagonal blocks of
// all matrices factored in one cooperative launch, the block rows R12 =
// R11^-T G12 = Dr^-1 (Y^T G12) with Y = R11^-1 Dr (tri_inv_upper), and the
// trailing G22 -= R12^T R12 as a tensor-core GEMM; the cooperative kernel's
// FP64 trailing updates (k^3 / 3 FMAs on the FP64 pipe) are the cost this
// removes.
constexpr int64_t kPotrfPanel = 256;

template <typename T>
void potrf_upper_blocked(lra_ctx* ctx, int n, const int64_t* k, T* const* G, const int64_t* ldg, bool* ok) {
  int64_t kmax = 0;
  for (int m = 0; m < n; ++m) {
    ok[m] = true;
    kmax = std::max(kmax, k[m]);
  }
  for (int64_t j0 = 0; j0 < kmax; j0 += kPotrfPanel) {
    int64_t kb[2] = {0, 0}, lb[2] = {1, 1};
    T* Gb[2] = {nullptr, nullptr};
    bool okb[2] = {true, true};
    int idx[2] = {-1, -1}, nb = 0;
    for (int m = 0; m < n; ++m) {
      if (!ok[m] || j0 >= k[m]) continue;
      idx[nb] = m;
      kb[nb] = std::min(kPotrfPanel, k[m] - j0);
      Gb[nb] = G[m] + j0 + j0 * ldg[m];
      lb[nb] = ldg[m];
      ++nb;
    }
    if (nb == 0) break;
    potrf_upper_batch<T>(ctx, nb, kb, Gb, lb, okb);
    for (int b = 0; b < nb; ++b) {
      const int m = idx[b];
      if (!okb[b]) {
        ok[m] = false;
        continue;
      }
      const int64_t jb = kb[b], rest = k[m] - j0 - jb, ld = ldg[m];
      if (rest <= 0) continue;
      const ArenaMark mk = ctx->arena.mark();
      T* Y = ctx->arena.alloc_n<T>((size_t)jb * jb);
      T* W = ctx->arena.alloc_n<T>((size_t)jb * rest);
      tri_inv_upper<T>(ctx, jb, Gb[b], ld, Y, jb);
      T* G12 = G[m] + j0 + (j0 + jb) * ld;
      gemm<T>(ctx, 't', 'n', jb, rest, jb, T(1), Y, jb, G12, ld, T(0), W, jb);
      div_by_diag<T>(ctx, jb, rest, Gb[b], ld, 'l', W, jb, G12, ld);
      T* G22 = G[m] + (j0 + jb) + (j0 + jb) * ld;
      gemm<T>(ctx, 't', 'n', rest, rest, jb, T(-1), G12, ld, G12, ld, T(1), G22, ld);
      ctx->arena.release(mk);  // stream-ordered reuse
    }
  }
  for (int m = 0; m < n; ++m)
    if (k[m] > 0) zero_lower(ctx, k[m], k[m], G[m], ldg[m]);
}

template <typename T>
void potrf_upper_batch(lra_ctx* ctx, int n, const int64_t* k, T* const* G, const int64_t* ldg, bool* ok) {
  if (sizeof(T) == 8 && ctx->gemm_tc) {
    int64_t kmax = 0;
    for (int m = 0; m < n; ++m) kmax = std::max(kmax, k[m]);
    if (kmax > 2 * kPotrfPanel) {
      potrf_upper_blocked<T>(ctx, n, k, G, ldg, ok);
      return;
    }
  }
  const ArenaMark mk = ctx->arena.mark();
  int* bad = ctx->arena.alloc_n<int>(2);
  LRA_CUDA(cudaMemsetAsync(bad, 0, 2 * sizeof(int), ctx->stream));
  PotrfJobs<T> J{};
  J.n = 0;
  J.bad = bad;
  int slot[2] = {-1, -1};
  for (int m = 0; m < n; ++m) {
    ok[m] = true;
    if (k[m] <= 0) continue;
    slot[m] = J.n;
    J.k[J.n] = k[m];
    J.G[J.n] = G[m];
    J.ldg[J.n] = ldg[m];
    ++J.n;
  }
  if (J.n > 0) {
    int per_sm = 0;
    LRA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, potrf_coop_kernel<T>, 256, 0));
    const int grid = std::max(J.n, std::min(ctx->num_sms, ctx->num_sms * per_sm));
    GridBar* bar = reinterpret_cast<GridBar*>(ctx->arena.alloc(2 * sizeof(GridBar)));
    LRA_CUDA(cudaMemsetAsync(bar, 0, 2 * sizeof(GridBar), ctx->stream));
    void* args[] = {&J, &bar};
    LRA_CUDA(cudaLaunchCooperativeKernel((const void*)potrf_coop_kernel<T>, dim3(grid), dim3(256), args, 0,
                                         ctx->stream));
    post_launch(ctx, "potrf_coop_kernel");
    for (int m = 0; m < J.n; ++m) zero_lower(ctx, J.k[m], J.k[m], J.G[m], J.ldg[m]);
    int h[2] = {0, 0};
    GridBar hb[2];
    LRA_CUDA(cudaMemcpyAsync(h, bad, 2 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    LRA_CUDA(cudaMemcpyAsync(hb, bar, 2 * sizeof(GridBar), cudaMemcpyDeviceToHost, ctx->stream));
    LRA_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->arena.release(mk);
    if (hb[0].err != 0 || hb[1].err != 0) fail(LRA_ETIMEDOUT, "potrf: a grid barrier timed out");
    for (int m = 0; m < n; ++m)
      if (slot[m] >= 0) ok[m] = h[slot[m]] == 0;
    return;
  }
  ctx->arena.release(mk);
}

template <typename T>
bool potrf_upper(lra_ctx* ctx, int64_t k, T* G, int64_t ldg) {
  if (k <= 0) return true;
  if (k > CB) {
    bool ok = true;
    potrf_upper_batch<T>(ctx, 1, &k, &G, &ldg, &ok);
    return ok;
  }
  const ArenaMark mk = ctx->arena.mark();
  int* bad = ctx->arena.alloc_n<int>(1);
  LRA_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
  for (int64_t j0 = 0; j0 < k; j0 += CB) {
    const int jb = (int)std::min<int64_t>(CB, k - j0);
    T* Gjj = G + j0 + j0 * ldg;
    potrf_diag_kernel<T><<<1, 256, 0, ctx->stream>>>(jb, Gjj, ldg, bad);
    post_launch(ctx, "potrf_diag_kernel");
    const int64_t rest = k - j0 - jb;
    if (rest > 0) {
      T* P = G + j0 + (j0 + jb) * ldg;
      const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((rest + 127) / 128, ctx->num_sms * 4));
      potrf_panel_kernel<T><<<g, 128, 0, ctx->stream>>>(jb, rest, Gjj, ldg, P, ldg);
      post_launch(ctx, "potrf_panel_kernel");
      // trailing: G_{>b,>b} -= P^T P
      T* Gt = G + (j0 + jb) + (j0 + jb) * ldg;
      gemm<T>(ctx, 't', 'n', rest, rest, jb, T(-1), P, ldg, P, ldg, T(1), Gt, ldg);
    }
  }
  zero_lower(ctx, k, k, G, ldg);  // the factor is used as a dense matrix later
  int h = 0;
  LRA_CUDA(cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
  ctx->arena.release(mk);
  return h == 0;
}

template <typename T>
void trsm_left_diag(lra_ctx* ctx, int jb, int64_t nrhs, const T* R, int64_t ldr, T* X, int64_t ldx) {
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((nrhs + 127) / 128, ctx->num_sms * 8));
  trsm_left_diag_kernel<T><<<g, 128, 0, ctx->stream>>>(jb, nrhs, R, ldr, X, ldx);
  post_launch(ctx, "trsm_left_diag_kernel");
}

namespace {

// Y = R^-1 D with D = diag(R), the inverse of the unit upper triangular
// D^-1 R (k x k, strictly lower part zero), a CTA per column: column j
// solves R y = R_jj e_j by column-oriented back substitution -- y_j = 1,
// then a_i -= R_iq y_q for i < q and y_q = a_q / R_qq from q = j down.  A graded R
// (|R_iq| <= |R_ii|, as a
// pivoted QR leaves it) has an inverse whose rows span its whole diagonal
// range, which a GEMM that scales each row by its largest entry would
// truncate; R^-1 D has entries of order one.
//
// Bound: the chain of FP64 operations.  Blocks of 32 rows from the bottom: warp 0
// solves the block on its diagonal, a row a lane, its entries of R loaded while
// the block before was applied; then all threads subtract the 32 columns from
// the rows above, each entry in the order of q, with no barrier among them (a
// barrier a column before: 200 us for order 460, 92 us now).  1 / R_qq is
// computed for every q first, so that no FP64 division sits on the chain (a
// product with the reciprocal instead, within an ulp of the quotient).
constexpr int kTiNT = 128;
constexpr int kTiMax = 2048;
constexpr int kTiLeaf = 512;  // larger orders split in two on the tensor-core path

template <typename T>
__global__ void __launch_bounds__(kTiNT) tri_inv_upper_kernel(int64_t k, const T* __restrict__ R, int64_t ldr,
                                                              T* __restrict__ Y, int64_t ldy) {
  extern __shared__ __align__(16) unsigned char ti_smem[];
  T* ys = reinterpret_cast<T*>(ti_smem);  // k: the partial sums a_i, then y
  T* rdi = ys + k;                        // 1 / R_qq
  const int tid = threadIdx.x, lane = tid & 31;
  for (int64_t q = tid; q < k; q += kTiNT) rdi[q] = T(1) / R[q + q * ldr];
  for (int64_t j = blockIdx.x; j < k; j += gridDim.x) {
    for (int64_t i = tid; i <= j; i += kTiNT) ys[i] = T(0);
    T rr[32];  // warp 0: R(qb + lane, qb + t) of the next diagonal block
    auto fetch = [&](int64_t qb) {
#pragma unroll
      for (int t = 0; t < 32; ++t) rr[t] = lane < t && qb + t <= j ? __ldg(R + qb + lane + (qb + t) * ldr) : T(0);
    };
    int64_t qb = j / 32 * 32;
    if (tid < 32) fetch(qb);
    __syncthreads();
    for (; qb >= 0; qb -= 32) {
      if (tid < 32) {
        T a = qb + lane <= j ? ys[qb + lane] : T(0), y = T(0);
#pragma unroll
        for (int t = 31; t >= 0; --t) {
          const int64_t q = qb + t;
          if (q <= j) {
            const T yq = q == j ? T(1) : __shfl_sync(0xffffffffu, a, t) * rdi[q];
            if (lane == t) y = yq;
            if (lane < t) a = fma(-rr[t], yq, a);
          }
        }
        if (qb + lane <= j) ys[qb + lane] = y;
        if (qb > 0) fetch(qb - 32);
      }
      __syncthreads();
      const int nq = (int)min((int64_t)32, j - qb + 1);
      for (int64_t i = tid; i < qb; i += kTiNT) {
        T a = ys[i];
        const T* r = R + i + qb * ldr;
        int t = nq - 1;
        for (; t >= 7; t -= 8) {
          T rv[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) rv[u] = __ldg(r + (t - u) * ldr);
#pragma unroll
          for (int u = 0; u < 8; ++u) a = fma(-rv[u], ys[qb + t - u], a);
        }
        for (; t >= 0; --t) a = fma(-__ldg(r + t * ldr), ys[qb + t], a);
        ys[i] = a;
      }
      __syncthreads();
    }
    for (int64_t i = tid; i < k; i += kTiNT) Y[i + j * ldy] = i <= j ? ys[i] : T(0);
    __syncthreads();  // ys is rewritten for the next column
  }
}

// dst = src with row i (side 'l') or column j (side 'r') divided by R's
// diagonal entry, as the substitution divides
template <typename T>
__global__ void div_by_diag_kernel(int64_t m, int64_t n, const T* __restrict__ R, int64_t ldr, bool rows,
                                   const T* __restrict__ src, int64_t lds, T* __restrict__ dst, int64_t ldd) {
  const int64_t total = m * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % m, j = t / m;
    const int64_t d = rows ? i : j;
    dst[i + j * ldd] = src[i + j * lds] / R[d + d * ldr];
  }
}

}  // namespace

template <typename T>
void div_by_diag(lra_ctx* ctx, int64_t m, int64_t n, const T* R, int64_t ldr, char side, const T* src, int64_t lds,
                 T* dst, int64_t ldd) {
  if (m <= 0 || n <= 0) return;
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((m * n + 255) / 256, ctx->num_sms * 8));
  div_by_diag_kernel<T><<<g, 256, 0, ctx->stream>>>(m, n, R, ldr, side == 'l', src, lds, dst, ldd);
  post_launch(ctx, "div_by_diag_kernel");
}
template void div_by_diag<float>(lra_ctx*, int64_t, int64_t, const float*, int64_t, char, const float*, int64_t,
                                 float*, int64_t);
template void div_by_diag<double>(lra_ctx*, int64_t, int64_t, const double*, int64_t, char, const double*, int64_t,
                                  double*, int64_t);

template <typename T>
bool tri_inv_upper(lra_ctx* ctx, int64_t k, const T* R, int64_t ldr, T* Y, int64_t ldy) {
  if (k <= 0) return true;
  if (k > kTiMax) return false;
  if (sizeof(T) == 8 && ctx->gemm_tc && k > kTiLeaf) {
    // Recursive on the tensor-core path: with R = [A B; 0 C] and D = diag(R),
    // R^-1 D = [Ya, -Ya (Da^-1 B) Yc; 0, Yc] for Ya = A^-1 Da, Yc = C^-1 Dc.
    // Every factor has entries of order one (Da^-1 B because |R_iq| <=
    // |R_ii| in a pivoted QR's R), so the two products are accurate on the
    // tensor cores; the leaves' column substitutions are shorter.
    const int64_t k1 = (k / 2 + 31) / 32 * 32, k2 = k - k1;
    tri_inv_upper<T>(ctx, k1, R, ldr, Y, ldy);
    tri_inv_upper<T>(ctx, k2, R + k1 + k1 * ldr, ldr, Y + k1 + k1 * ldy, ldy);
    const ArenaMark mk = ctx->arena.mark();
    T* W = ctx->arena.alloc_n<T>((size_t)k1 * k2);
    T* W2 = ctx->arena.alloc_n<T>((size_t)k1 * k2);
    div_by_diag<T>(ctx, k1, k2, R, ldr, 'l', R + k1 * ldr, ldr, W, k1);
    gemm<T>(ctx, 'n', 'n', k1, k2, k2, T(1), W, k1, Y + k1 + k1 * ldy, ldy, T(0), W2, k1);
    gemm<T>(ctx, 'n', 'n', k1, k2, k1, T(-1), Y, ldy, W2, k1, T(0), Y + k1 * ldy, ldy);
    zero_lower(ctx, k, k, Y, ldy);  // the block below the diagonal
    ctx->arena.release(mk);  // stream-ordered reuse
    return true;
  }
  const size_t smem = (size_t)2 * k * sizeof(T);
  if (smem > 48 * 1024) raise_smem_limit(ctx, (const void*)tri_inv_upper_kernel<T>);
  tri_inv_upper_kernel<T><<<(unsigned)k, kTiNT, smem, ctx->stream>>>(k, R, ldr, Y, ldy);
  post_launch(ctx, "tri_inv_upper_kernel");
  return true;
}

template bool tri_inv_upper<float>(lra_ctx*, int64_t, const float*, int64_t, float*, int64_t);
template bool tri_inv_upper<double>(lra_ctx*, int64_t, const double*, int64_t, double*, int64_t);

// Whether a triangular solve with a k x k factor and `other` right-hand
// sides should multiply by the explicit inverse instead: on the tensor-core
// path for FP64, where the substitution's diagonal blocks run on the FP64
// pipe (a few FMAs a clock per SM) and the inverse costs one GEMM
template <typename T>
bool trsm_by_inverse(const lra_ctx* ctx, int64_t k, int64_t other) {
  if (sizeof(T) != 8 || !ctx->gemm_tc || ctx->tuning.trsm_inv == 1) return false;
  return k > 2 * CB && k <= kTiMax && tc_gemm_worthwhile(other, k, k);
}
template bool trsm_by_inverse<float>(const lra_ctx*, int64_t, int64_t);
template bool trsm_by_inverse<double>(const lra_ctx*, int64_t, int64_t);

// X <- X triu(R)^{-1}, recursive like trsm_upper: the leading half, a GEMM
// update of the trailing columns, the trailing half; on the tensor-core
// path X times the explicit inverse
template <typename T>
void trsm_right_upper(lra_ctx* ctx, int64_t m, int64_t k, const T* R, int64_t ldr, T* X, int64_t ldx, const T* Yd) {
  if (m <= 0 || k <= 0) return;
  if (trsm_by_inverse<T>(ctx, k, m)) {
    const ArenaMark mk = ctx->arena.mark();
    T* Y = Yd ? nullptr : ctx->arena.alloc_n<T>((size_t)k * k);
    T* W = ctx->arena.alloc_n<T>((size_t)m * k);
    // X R^-1 = (X Y) D^-1 with Y = R^-1 D (Yd when the caller has it)
    if (Y) tri_inv_upper<T>(ctx, k, R, ldr, Y, k);
    gemm<T>(ctx, 'n', 'n', m, k, k, T(1), X, ldx, Yd ? Yd : Y, k, T(0), W, m);
    div_by_diag<T>(ctx, m, k, R, ldr, 'r', W, m, X, ldx);
    ctx->arena.release(mk);  // stream-ordered reuse
    return;
  }
  if constexpr (sizeof(T) == 4)
    if (trsm_fused(ctx, true, k, m, R, ldr, X, ldx)) return;
  if (k <= CB) {
    const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((m + 127) / 128, ctx->num_sms * 8));
    trsm_right_diag_kernel<T><<<g, 128, 0, ctx->stream>>>(m, (int)k, R, ldr, X, ldx);
    post_launch(ctx, "trsm_right_diag_kernel");
    return;
  }
  const int64_t k1 = (k / 2 + CB - 1) / CB * CB, k2 = k - k1;
  trsm_right_upper(ctx, m, k1, R, ldr, X, ldx);
  gemm<T>(ctx, 'n', 'n', m, k2, k1, T(-1), X, ldx, R + k1 * ldr, ldr, T(1), X + k1 * ldx, ldx);
  trsm_right_upper(ctx, m, k2, R + k1 + k1 * ldr, ldr, X + k1 * ldx, ldx);
}

template bool potrf_upper<float>(lra_ctx*, int64_t, float*, int64_t);
template bool potrf_upper<double>(lra_ctx*, int64_t, double*, int64_t);
template void potrf_upper_batch<float>(lra_ctx*, int, const int64_t*, float* const*, const int64_t*, bool*);
template void potrf_upper_batch<double>(lra_ctx*, int, const int64_t*, double* const*, const int64_t*, bool*);
template void trsm_right_upper<float>(lra_ctx*, int64_t, int64_t, const float*, int64_t, float*, int64_t,
                                      const float*);
template void trsm_right_upper<double>(lra_ctx*, int64_t, int64_t, const double*, int64_t, double*, int64_t,
                                       const double*);
// ---- T = R11^{-1} R12 by back substitution --------------------------------------
// The ID's solve (src/id.jl:447, R11 \ R12) for ranks up to kBsMax.  From the
// bottom row: x_j = s_j / R_jj, and s_i -= R_ij x_j with j falling, which lets
// all rows take x_j at once.  Every path runs these operations in this order: a
// batch gives the bits of its single calls.
// Bound: the FP64 unit, 64 cycles a warp instruction on each quarter of an SM.
constexpr int kBsLd = 33;  // row stride of the tile
template <typename T>
constexpr size_t bs_smem_bytes(int64_t k) {
  return (size_t)k * (kBsLd + 1) * sizeof(T);
}

// s / r from inv = 1 / r: one Newton step on the quotient, 3 instructions for
// the divide's 10; what over- or underflows there is divided.
template <typename T>
__device__ __forceinline__ T bs_inv(T r) {
  const T big = sizeof(T) == 8 ? (T)1e300 : (T)1e36;
  return fabs(r) < big ? (T)1 / r : (T)INFINITY;
}
__device__ __forceinline__ bool bs_finite(double q) { return (__double2hiint(q) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool bs_finite(float q) { return (__float_as_int(q) & 0x7f800000) != 0x7f800000; }
template <typename T>
__device__ __forceinline__ T bs_div(T s, T r, T inv) {
  T q = s * inv;
  q = fma(fma(-q, r, s), inv, q);
  return bs_finite(q) ? q : s / r;
}

// 32 right-hand sides of a warp in shared memory, a lane each (with the columns
// in global memory a load takes 32 sectors: 160 solves of rank 41 and 2000
// columns 1.19 ms so, 0.52 now; their FP64 instructions take 0.5 on all SMs).
// A block is one warp.
template <typename T>
__device__ __forceinline__ void bs_tile(int k, int nc, const T* __restrict__ R, int64_t ldr, const T* __restrict__ src,
                                        int64_t lds, T* __restrict__ dst, int64_t ldd, T* xs) {
  const int lane = threadIdx.x;
  T* inv = xs + k * kBsLd;
  for (int i = lane; i < k; i += 32) inv[i] = bs_inv(R[i + i * ldr]);
  for (int c = 0; c < nc; ++c)
    for (int i = lane; i < k; i += 32) xs[i * kBsLd + c] = src[i + c * lds];
  __syncwarp();
  if (lane < nc) {
    T* x = xs + lane;
    for (int i = k - 1; i >= 0; --i) {
      T t = x[i * kBsLd];
      const T* r = R + i;
      int j = k - 1;
      for (; j - 4 >= i; j -= 4) {
        T rv[4], xv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          rv[q] = __ldg(r + (j - q) * ldr);
          xv[q] = x[(j - q) * kBsLd];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) t = fma(-rv[q], xv[q], t);
      }
      for (; j > i; --j) t = fma(-__ldg(r + j * ldr), x[j * kBsLd], t);
      x[i * kBsLd] = bs_div(t, __ldg(r + i * ldr), inv[i]);
    }
  }
  __syncwarp();
  for (int c = 0; c < nc; ++c)
    for (int i = lane; i < k; i += 32) dst[i + c * ldd] = xs[i * kBsLd + c];
}

template <typename T>
__global__ void __launch_bounds__(32) trsm_bs_kernel(int k, int64_t nrhs, const T* __restrict__ R, int64_t ldr, T* X,
                                                     int64_t ldx) {
  extern __shared__ __align__(16) unsigned char bs_smem[];
  const int64_t c0 = (int64_t)blockIdx.x * 32;
  T* x = X + c0 * ldx;
  bs_tile(k, (int)min((int64_t)32, nrhs - c0), R, ldr, x, ldx, x, ldx, reinterpret_cast<T*>(bs_smem));
}

// Few right-hand sides: four a warp, eight lanes a column, lane l with the
// rows l, l + 8, ... in registers, so that an instruction updates eight rows and
// eight times the warps share the work.
template <typename T>
__global__ void __launch_bounds__(32) trsm_bs_lanes_kernel(int k, int64_t nrhs, const T* __restrict__ R, int64_t ldr, T* X,
                                                           int64_t ldx) {
  constexpr int NB = kBsMax / 8;
  __shared__ T inv[kBsMax];
  const int lane = threadIdx.x, l = lane & 7;
  const int64_t c = (int64_t)blockIdx.x * 4 + (lane >> 3);
  for (int i = lane; i < k; i += 32) inv[i] = bs_inv(R[i + i * ldr]);
  T x[NB], rn[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int i = b * 8 + l;
    x[b] = c < nrhs && i < k ? X[i + c * ldx] : (T)0;
    rn[b] = i < k ? __ldg(R + i + (int64_t)(k - 1) * ldr) : (T)0;
  }
  __syncwarp();
#pragma unroll
  for (int b = NB - 1; b >= 0; --b) {
    for (int jj = min(7, k - 1 - b * 8); jj >= 0; --jj) {
      const int j = b * 8 + jj;
      T r[NB];
#pragma unroll
      for (int a = 0; a <= b; ++a) {  // this column of R, and the next on its way
        r[a] = rn[a];
        if (j > 0 && a * 8 + l < j) rn[a] = __ldg(R + a * 8 + l + (int64_t)(j - 1) * ldr);
      }
      const T rjj = __shfl_sync(0xffffffffu, r[b], jj, 8);
      const T xj = bs_div(__shfl_sync(0xffffffffu, x[b], jj, 8), rjj, inv[j]);
      if (l == jj)
        x[b] = xj;
      else if (l < jj)
        x[b] = fma(-r[b], xj, x[b]);
#pragma unroll
      for (int a = 0; a < b; ++a) x[a] = fma(-r[a], xj, x[a]);
    }
  }
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int i = b * 8 + l;
    if (c < nrhs && i < k) X[i + c * ldx] = x[b];
  }
}

template <typename T>
void trsm_bs(lra_ctx* ctx, int64_t k, int64_t nrhs, const T* R, int64_t ldr, T* X, int64_t ldx) {
  if (k <= 0 || nrhs <= 0) return;
  if (k > kBsMax) fail(LRA_EINVAL, "trsm_bs: k > %d", kBsMax);
  // A warp takes k^2 / 2 updates and 3 k of quotients for 32 columns, or k^2 / 16
  // and 3 k for 4: the second is less until each quarter of the chip has about
  // four of its warps.  2000 columns, the whole stage: rank 41 0.087 and 0.054 ms,
  // rank 125 0.35 and 0.135.
  if (nrhs <= (int64_t)ctx->num_sms * 64) {
    trsm_bs_lanes_kernel<T><<<(unsigned)((nrhs + 3) / 4), 32, 0, ctx->stream>>>((int)k, nrhs, R, ldr, X, ldx);
    post_launch(ctx, "trsm_bs_lanes_kernel");
    return;
  }
  trsm_bs_kernel<T><<<(unsigned)((nrhs + 31) / 32), 32, bs_smem_bytes<T>(k), ctx->stream>>>((int)k, nrhs, R, ldr, X, ldx);
  post_launch(ctx, "trsm_bs_kernel");
}

// one matrix of the batch: T (k x nr, ld k) = R11^{-1} R12, both read from B
struct BsJob {
  int64_t k, nr, ldb;
  const double* B;
  double* T;
};

// blocks (matrix, 32 right-hand sides)
__global__ void __launch_bounds__(32) trsm_bs_group_kernel(const BsJob* __restrict__ jobs) {
  extern __shared__ __align__(16) unsigned char bs_smem[];
  const BsJob J = jobs[blockIdx.x];
  const int64_t c0 = (int64_t)blockIdx.y * 32;
  if (c0 >= J.nr) return;
  bs_tile((int)J.k, (int)min((int64_t)32, J.nr - c0), J.B, J.ldb, J.B + (J.k + c0) * J.ldb, J.ldb, J.T + c0 * J.k, J.k,
          reinterpret_cast<double*>(bs_smem));
}

void trsm_bs_batch(lra_ctx* ctx, int64_t count, const BsItem* items) {
  if (count <= 0) return;
  std::vector<BsJob> jobs;
  jobs.reserve((size_t)count);
  int64_t nrmax = 1, kmax = 1;
  for (int64_t i = 0; i < count; ++i) {
    const BsItem& it = items[i];
    if (it.k > kBsMax) fail(LRA_EINVAL, "trsm_bs_batch: k > %d", kBsMax);
    if (it.k > 0 && it.nr > 0) jobs.push_back(BsJob{it.k, it.nr, it.ldb, it.B, it.T});
    nrmax = std::max(nrmax, it.nr);
    kmax = std::max(kmax, it.k);
  }
  if (jobs.empty()) return;
  BsJob* d = ctx->arena.alloc_n<BsJob>(jobs.size());
  LRA_CUDA(cudaMemcpyAsync(d, jobs.data(), jobs.size() * sizeof(BsJob), cudaMemcpyHostToDevice, ctx->stream));
  trsm_bs_group_kernel<<<dim3((unsigned)jobs.size(), (unsigned)((nrmax + 31) / 32)), 32,
                         bs_smem_bytes<double>(kmax), ctx->stream>>>(d);
  post_launch(ctx, "trsm_bs_group_kernel");
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
}

__global__ void pack_results_kernel(const PackItem* __restrict__ items, char* __restrict__ out) {
  const PackItem it = items[blockIdx.x];
  int64_t* p = reinterpret_cast<int64_t*>(out + it.off);
  for (int64_t i = threadIdx.x; i < it.n; i += blockDim.x) p[i] = it.jpvt[i];
  double* t = reinterpret_cast<double*>(out + it.off + 8 * (size_t)it.n);
  for (int64_t i = threadIdx.x; i < it.nt; i += blockDim.x) t[i] = it.T[i];
}

void pack_results(lra_ctx* ctx, int64_t count, const PackItem* items, char* out) {
  if (count <= 0) return;
  PackItem* d = ctx->arena.alloc_n<PackItem>((size_t)count);
  LRA_CUDA(cudaMemcpyAsync(d, items, (size_t)count * sizeof(PackItem), cudaMemcpyHostToDevice, ctx->stream));
  pack_results_kernel<<<(unsigned)count, 256, 0, ctx->stream>>>(d, out);
  post_launch(ctx, "pack_results_kernel");
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
}

template void trsm_bs<float>(lra_ctx*, int64_t, int64_t, const float*, int64_t, float*, int64_t);
template void trsm_bs<double>(lra_ctx*, int64_t, int64_t, const double*, int64_t, double*, int64_t);
template void trsm_left_diag<float>(lra_ctx*, int, int64_t, const float*, int64_t, float*, int64_t);
template void trsm_left_diag<double>(lra_ctx*, int, int64_t, const double*, int64_t, double*, int64_t);

WaitUnit wait_unit_dense() { return this_wait_unit("dense"); }

}  // namespace lra
