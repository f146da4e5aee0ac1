// FP32 one-sided block Jacobi through Gram products: the sweeps that bring
// the columns of a core matrix X close to orthogonal (largest cosine near
// 1e-2) before the Gram-matrix polish of the mixed path finishes in double
// precision, with the rotations accumulated in V.
//
// Columns are grouped in blocks of 32.  A round pairs the blocks
// (round-robin); for each pair of blocks the 64 x 64 Gram matrix of its
// columns is formed, the rotations of the 32 x 32 inter-block column pairs
// (all 64 x 63 / 2 pairs in a sweep's first round) are taken on the Gram
// matrix alone, two-sided, and gathered in a 64 x 64 orthogonal Q, and X and V
// are multiplied by Q.  A pair of blocks belongs to a group of c CTAs, each
// with a chunk of the rows: the group's CTAs exchange their partial Gram
// matrices, run the same rotations on the sum (the same bits in each, so Q
// need not be sent), and apply Q to their rows, which stayed in shared memory
// since the Gram product.  One barrier inside a group and one across the grid
// a round.
//
// Why: rotating the columns themselves pair by pair is bound by the traffic
// and the reductions of 2 n-long dots per rotation (a round of 8-column
// blocks: 31 us at n = 1803, 2260 rounds).  Here the n-long work is two dense
// products a round (4 n^3 multiply-adds a sweep on packed FP32), a rotation
// step is a few hundred cycles on 64 x 64, and a round covers 32 columns.
// The cosines the rotations are taken from are FP32 sums like the dots they
// replace; the two-sided updates keep each entry's error relative to the norms
// of its own two columns, so graded columns stay as accurate as their own
// scale.  The diagonal blocks of the Gram matrix are carried from round to
// round (32 x 32 inter-block entries are fresh each round) and formed anew in
// a sweep's first round: a group's CTAs have them in shared memory before they
// meet, after which its first CTA writes them back rotated.

#include <algorithm>
#include <cmath>
#include <cstdio>

#include "common.cuh"
#include "internal.hpp"
#include "waits.cuh"

namespace lra {

namespace {

constexpr int JB = 32;         // columns per block
constexpr int JC = 2 * JB;     // columns per pair of blocks
constexpr int JNT = 512;
constexpr int JNW = JNT / 32;
constexpr int JGS = JC + 1;    // row stride of the Gram matrix (conflict-free columns)
constexpr int JQS = JC + 4;    // row stride of Q (16-byte rows)
static_assert(JNW == 16 && JC * JGS >= 4 * (JNW + 1) * JB, "16 warps hold G; the exchange buffers fit over it");
constexpr int JMAXC = 8;       // CTAs per pair of blocks, at most

typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float lo2(f2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// the rotation of a column pair from its Gram entries (a, b the squared norms,
// g the product): c, s with [x_p x_q] <- [c x_p - s x_q, s x_p + c x_q].
// t = tan = 2 g / ((b - a) + sign(b - a) sqrt((b - a)^2 + 4 g^2)), the smaller
// root, at the power-of-two scale of the larger norm (squares of graded
// columns' entries would underflow).  The angle needs few digits (the next
// sweep corrects it), the pair (c, s) its unit length: an approximate root and
// reciprocal, s = c t; three special-function operations in a chain, as every
// warp computes all 32 angles of a step.
__device__ __forceinline__ void jg_angle(float a, float b, float g, float tol2, float& cs, float& sn) {
  const float inv = __uint_as_float(0x7f000000u - (__float_as_uint(fmaxf(a, b)) & 0x7f800000u));
  const float u = (b - a) * inv, v = 2.0f * g * inv;
  float root, q, c;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(root) : "f"(fmaf(u, u, v * v)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(fmaxf(fabsf(u) + root, 1e-30f)));
  const float t = copysignf(1.0f, u) * v * q;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(fmaf(t, t, 1.0f)));
  // no rotation where the cosine is rounding (tol2 = 4 tol^2; columns of equal
  // norms would turn by a large angle for it), a column is zero, or a sum
  // overflowed
  const bool ok = v * v > tol2 * (a * inv) * (b * inv) && fabsf(t) <= 1.000001f;
  cs = ok ? c : 1.f;
  sn = ok ? c * t : 0.f;
}

// its cosine
__device__ __forceinline__ float jg_cosine(float a, float b, float g) {
  const float rel = fabsf(g) * rsqrtf(a) * rsqrtf(b);
  return a > 0.f && b > 0.f ? rel : 0.f;
}

// two-sided rotation of a 2 x 2 block: its rows by (cs, sn), its columns by
// (c2, s2)
__device__ __forceinline__ void jg_two_sided(float cs, float sn, float c2, float s2, float& x00, float& x01,
                                             float& x10, float& x11) {
  const float y00 = cs * x00 - sn * x10, y01 = cs * x01 - sn * x11;
  const float y10 = sn * x00 + cs * x10, y11 = sn * x01 + cs * x11;
  x00 = c2 * y00 - s2 * y01;
  x01 = s2 * y00 + c2 * y01;
  x10 = c2 * y10 - s2 * y11;
  x11 = s2 * y10 + c2 * y11;
}

struct JgParams {
  int n;
  float* X;
  float* V;
  int64_t ld;  // of both, a multiple of 4
  float tol2;  // 4 tol^2: column pairs with a cosine below tol are left alone
  double stop;
  int max_sweeps;
  int c;        // CTAs (row chunks) per pair of blocks
  int chunk;    // rows per chunk, a multiple of 4
  int rt, lds;  // rows per tile in shared memory, column stride of a tile
  float* part;  // [pairs][c][3][JB * JB] partial Gram blocks AB, AA, BB
  float* diag;  // [blocks][JB * JB] the diagonal Gram blocks
  unsigned* arrive;  // one counter per group, a 128-byte line apart
  double* off;  // per CTA
  GridBar* bar;
  int* sweeps_out;
  // LRA_TRACE: CTA 0's time in each phase (ns): Gram product, the group's
  // meeting, rotations, X and V, barrier
  unsigned long long* phase_ns = nullptr;
};

__device__ __forceinline__ void cp16z(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}

__global__ void __launch_bounds__(JNT, 1) jacobi_gram_kernel(const JgParams P) {
  extern __shared__ __align__(16) float jg_smem[];
  __shared__ int s_ok;
  __shared__ double red[32];
  __shared__ float s_abg[2][3][JB];  // a step's (a, b, g) of each pair, by parity
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n = P.n, lds = P.lds;
  float* tile0 = jg_smem;                       // JC columns x rt rows
  float* tile1 = tile0 + (size_t)JC * lds;      // the same; the Gram product's per-warp sums before that
  const size_t t1 = max((size_t)JC * lds, (size_t)JNW * JB * JB);
  float* G = tile1 + t1;                        // JC x JGS
  float* Q = G + JC * JGS + (4 - (JC * JGS) % 4) % 4;  // JC x JQS, Q[i][k]
  const int nblk = (n + JB - 1) / JB, nbb = nblk + (nblk & 1);
  const int group = blockIdx.x / P.c, rank = blockIdx.x % P.c;
  const int row0 = rank * P.chunk, row1 = min(n, row0 + P.chunk);
  const int nsub = max(1, (row1 - row0 + P.rt - 1) / P.rt);
  unsigned meets = 0;
  int b1 = 0, b2 = 0;

  // the tile's columns (JB of block b1, JB of b2) of M, rows r0 .. r0 + rt,
  // zero past the ends
  auto load = [&](float* dst, const float* M, int sub) {
    const int r0 = row0 + sub * P.rt;
    const int rows = max(0, min(P.rt, row1 - r0));
    const int nv = (P.rt + 3) / 4;
    for (int e = threadIdx.x; e < JC * nv; e += JNT) {
      const int k = e / nv, v = e % nv;
      const int b = k < JB ? b1 : b2;
      const int j = b * JB + (k & (JB - 1));
      const int left = rows - 4 * v;
      const bool on = b < nblk && j < n && left > 0;
      cp16z(dst + k * lds + 4 * v, on ? M + (int64_t)j * P.ld + r0 + 4 * v : M, on ? 4 * min(4, left) : 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // acc += (columns A0..A0+31)' (columns B0..B0+31) over the rows of a tile:
  // warp w takes row pairs w, w + 16, ...; a lane 8 x 4 of the 32 x 32 sums
  const int la = lane >> 3, lb = lane & 7;
  auto gram = [&](f2 (&acc)[8][4], const float* t, int A0, int B0) {
    for (int r = 2 * wid; r < P.rt; r += 2 * JNW) {
      f2 a[8], b[4];
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = *reinterpret_cast<const f2*>(t + (A0 + la + 4 * q) * lds + r);
#pragma unroll
      for (int q = 0; q < 4; ++q) b[q] = *reinterpret_cast<const f2*>(t + (B0 + lb + 8 * q) * lds + r);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i], b[j], acc[i][j]);
    }
  };

  uint64_t t_ph = 0;
  auto phase = [&](int i) {
    if (!P.phase_ns || blockIdx.x != 0 || threadIdx.x != 0) return;
    const uint64_t t = globaltimer_ns();
    if (i >= 0) P.phase_ns[i] += t - t_ph;
    t_ph = t;
  };
  int sweep = 0;
  for (; sweep < P.max_sweeps; ++sweep) {
    float off = 0;
    for (int r = 0; r < nbb - 1; ++r) {
      {
        auto pos = [&](int i) { return i == 0 ? 0 : 1 + (i - 1 + r) % (nbb - 1); };
        b1 = pos(group);
        b2 = pos(nbb - 1 - group);
        if (b1 > b2) {
          const int t = b1;
          b1 = b2;
          b2 = t;
        }
      }
      const bool first = r == 0;
      phase(-1);
      // a block paired with none has only its own column pairs to rotate
      if (b2 < nblk || first) {
        // ---- partial Gram blocks of this CTA's rows; the diagonal blocks, settled
        // by the grid's barrier, are on their way meanwhile
        const int nprod = first ? 3 : 1;
        float aa[JB * JB / JNT], bb[JB * JB / JNT];
        if (!first) {
#pragma unroll
          for (int h = 0; h < JB * JB / JNT; ++h) {
            aa[h] = __ldcg(P.diag + (size_t)b1 * JB * JB + threadIdx.x + h * JNT);
            bb[h] = __ldcg(P.diag + (size_t)b2 * JB * JB + threadIdx.x + h * JNT);
          }
        }
        for (int pr = 0; pr < nprod; ++pr) {
          f2 acc[8][4];
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0;
          for (int sub = 0; sub < nsub; ++sub) {
            if (pr == 0 || nsub > 1) {
              __syncthreads();
              load(tile0, P.X, sub);
              asm volatile("cp.async.wait_all;" ::: "memory");
              __syncthreads();
            }
            gram(acc, tile0, pr == 2 ? JB : 0, pr == 1 ? 0 : JB);
          }
          // the warps' sums through shared memory
          float* ws = tile1 + wid * JB * JB;
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) ws[(la + 4 * i) * JB + lb + 8 * j] = lo2(acc[i][j]) + hi2(acc[i][j]);
          __syncthreads();
          float* dst = P.part + (((size_t)group * P.c + rank) * 3 + pr) * JB * JB;
          for (int e = threadIdx.x; e < JB * JB; e += JNT) {
            float s = 0;
#pragma unroll
            for (int w = 0; w < JNW; ++w) s += tile1[w * JB * JB + e];
            __stcg(dst + e, s);
          }
          // the diagonal blocks are in G before this CTA arrives at the meeting:
          // after it rank 0 overwrites them
          if (!first) {
#pragma unroll
            for (int h = 0; h < JB * JB / JNT; ++h) {
              const int e = threadIdx.x + h * JNT, i = e / JB, j = e % JB;
              G[i * JGS + j] = aa[h];
              G[(JB + i) * JGS + JB + j] = bb[h];
            }
          }
          __syncthreads();
        }
        phase(0);
        // ---- the group's CTAs meet (bounded)
        ++meets;
        if (threadIdx.x == 0) {
          unsigned* cnt = P.arrive + group * 32;
          const unsigned target = meets * (unsigned)P.c;
          __threadfence();
          atomicAdd(cnt, 1u);
          s_ok = wait_reached(cnt, target, &P.bar->err);
          __threadfence();
        }
        __syncthreads();
        if (!s_ok) return;
        phase(1);
        // (V's rows arrive while the rotations are found)
        if (nsub == 1) {
          load(tile1, P.V, 0);
        } else {
          load(tile0, P.X, 0);
          load(tile1, P.X, 1);
        }
        // ---- G = [AA AB; AB' BB]
        {
          // every load in flight at once
          float ab[JB * JB / JNT][JMAXC];
#pragma unroll
          for (int h = 0; h < JB * JB / JNT; ++h) {
            const int e = threadIdx.x + h * JNT;
            const float* src = P.part + (size_t)group * P.c * 3 * JB * JB + e;
#pragma unroll
            for (int q = 0; q < JMAXC; ++q) ab[h][q] = q < P.c ? __ldcg(src + (size_t)q * 3 * JB * JB) : 0.f;
            if (first) {
              aa[h] = bb[h] = 0.f;
              for (int q = 0; q < P.c; ++q) {
                aa[h] += __ldcg(src + ((size_t)q * 3 + 1) * JB * JB);
                bb[h] += __ldcg(src + ((size_t)q * 3 + 2) * JB * JB);
              }
            }
          }
#pragma unroll
          for (int h = 0; h < JB * JB / JNT; ++h) {
            const int e = threadIdx.x + h * JNT, i = e / JB, j = e % JB;
            float s = 0;
#pragma unroll
            for (int q = 0; q < JMAXC; ++q) s += ab[h][q];
            if (first) {
              G[i * JGS + j] = aa[h];
              G[(JB + i) * JGS + JB + j] = bb[h];
            }
            G[i * JGS + JB + j] = s;
            G[(JB + j) * JGS + i] = s;
          }
        }
        __syncthreads();
        phase(5);
        if (first) {
          // ---- all 64 x 63 / 2 pairs, G and Q in shared memory: a step rotates
          // 32 disjoint pairs; lane = pair (its angle in every warp), a thread
          // two of the 32 x 32 blocks of 2 x 2 entries and four rows of Q
          for (int e = threadIdx.x; e < JC * JC; e += JNT) Q[(e / JC) * JQS + e % JC] = e / JC == e % JC ? 1.f : 0.f;
          __syncthreads();
          for (int st = 0; st < JC - 1; ++st) {
            const int p = lane == 0 ? 0 : 1 + (lane - 1 + st) % (JC - 1);
            const int q = 1 + (JC - 2 - lane + st) % (JC - 1);
            float cs, sn;
            const float a = G[p * JGS + p], b = G[q * JGS + q], g = G[p * JGS + q];
            jg_angle(a, b, g, P.tol2, cs, sn);
            if (wid == 8) off = fmaxf(off, jg_cosine(a, b, g));
            float x[2][4];
            int cp[2], cq[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int o = wid + h * JNW;  // the column pair of this block
              cp[h] = __shfl_sync(0xffffffffu, p, o);
              cq[h] = __shfl_sync(0xffffffffu, q, o);
              const float c2 = __shfl_sync(0xffffffffu, cs, o), s2 = __shfl_sync(0xffffffffu, sn, o);
              x[h][0] = G[p * JGS + cp[h]];
              x[h][1] = G[p * JGS + cq[h]];
              x[h][2] = G[q * JGS + cp[h]];
              x[h][3] = G[q * JGS + cq[h]];
              jg_two_sided(cs, sn, c2, s2, x[h][0], x[h][1], x[h][2], x[h][3]);
            }
            float qp[4], qq[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int i = wid + h * JNW;
              const float u = Q[i * JQS + p], w = Q[i * JQS + q];
              qp[h] = cs * u - sn * w;
              qq[h] = sn * u + cs * w;
            }
            __syncthreads();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              G[p * JGS + cp[h]] = x[h][0];
              G[p * JGS + cq[h]] = x[h][1];
              G[q * JGS + cp[h]] = x[h][2];
              G[q * JGS + cq[h]] = x[h][3];
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int i = wid + h * JNW;
              Q[i * JQS + p] = qp[h];
              Q[i * JQS + q] = qq[h];
            }
            __syncthreads();
          }
          if (rank == 0)
            for (int e = threadIdx.x; e < JB * JB; e += JNT) {
              const int i = e / JB, j = e % JB;
              __stcg(P.diag + (size_t)b1 * JB * JB + e, G[i * JGS + j]);
              if (b2 < nblk) __stcg(P.diag + (size_t)b2 * JB * JB + e, G[(JB + i) * JGS + JB + j]);
            }
        } else {
          // ---- the inter-block pairs, step st pairing column i of b1 (p_i) with
          // column q_i = (i + st) mod 32 of b2, with G and Q in registers.  G
          // is symmetric: the 2 x 2 blocks of pairs (i, i - d) for d = 0 .. 16
          // hold it all; warp d has block (lane, lane - d), the last warp d = 15
          // and 16.  After a step every q moves on by one: entries (q_i, q_j) along
          // the lanes by a shuffle, entries (p_i, q_j) and (q_i, p_j) to the warps of d - 1
          // and d + 1 through shared memory (double-buffered, one barrier a step);
          // past the ends of the range of d their mirror images step in.
          const bool two = wid == JNW - 1;
          const int nx = (lane + 1) & 31, pv = (lane + 31) & 31;
          float x[2][4], qa[4], qb[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int o = (lane - wid - h) & 31;
            x[h][0] = G[lane * JGS + o];
            x[h][1] = G[lane * JGS + JB + o];
            x[h][2] = G[(JB + lane) * JGS + o];
            x[h][3] = G[(JB + lane) * JGS + JB + o];
          }
          if (wid == 0) {
            s_abg[0][0][lane] = x[0][0];
            s_abg[0][1][lane] = x[0][3];
            s_abg[0][2][lane] = x[0][1];
          }
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int i = wid + h * JNW;
            qa[h] = i == lane ? 1.f : 0.f;
            qb[h] = i == JB + lane ? 1.f : 0.f;
          }
          __syncthreads();
          for (int st = 0; st < JB; ++st) {
            const int par = st & 1;
            float cs, sn;
            const float a = s_abg[par][0][lane], b = s_abg[par][1][lane], g = s_abg[par][2][lane];
            jg_angle(a, b, g, P.tol2, cs, sn);
            if (wid == 8) off = fmaxf(off, jg_cosine(a, b, g));
            // (over G) [entry (p, q) or (q, p)][d][lane] of the next step's parity
            float* e01 = G + (par ^ 1) * 2 * (JNW + 1) * JB;
            float* e10 = e01 + (JNW + 1) * JB;
            auto turn = [&](int h) {
              const int d = wid + h, o = (lane - d) & 31;
              const float c2 = __shfl_sync(0xffffffffu, cs, o), s2 = __shfl_sync(0xffffffffu, sn, o);
              jg_two_sided(cs, sn, c2, s2, x[h][0], x[h][1], x[h][2], x[h][3]);
              if (st == JB - 1) return;
              e01[d * JB + lane] = x[h][1];
              e10[d * JB + lane] = x[h][2];
              if (d == 0) {
                s_abg[par ^ 1][0][lane] = x[h][0];
                s_abg[par ^ 1][1][pv] = x[h][3];
              }
              if (d == 1) s_abg[par ^ 1][2][pv] = x[h][2];
              x[h][3] = __shfl_sync(0xffffffffu, x[h][3], nx);
            };
            turn(0);
            if (two) turn(1);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const float u = qa[h], w = qb[h];
              qa[h] = cs * u - sn * w;
              qb[h] = sn * u + cs * w;
              if (st < JB - 1) qb[h] = __shfl_sync(0xffffffffu, qb[h], nx);
            }
            __syncthreads();
            if (st < JB - 1) {
              x[0][1] = wid > 0 ? e01[(wid - 1) * JB + lane] : e10[JB + nx];
              x[0][2] = e10[(wid + 1) * JB + nx];
              if (two) {
                x[1][1] = e01[wid * JB + lane];
                x[1][2] = e01[(JNW - 1) * JB + ((lane + 16) & 31)];
              }
            }
          }
          const int lq = (lane + JB - 1) & 31;  // the b2 column of pair `lane` in the last step
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int i = wid + h * JNW;
            Q[i * JQS + lane] = qa[h];
            Q[i * JQS + JB + lq] = qb[h];
          }
          if (rank == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (h == 1 && !two) continue;
              // block (lane, o) and its mirror image
              const int o = (lane - wid - h) & 31, oq = (o + JB - 1) & 31;
              float* d1 = P.diag + (size_t)b1 * JB * JB;
              float* d2 = P.diag + (size_t)b2 * JB * JB;
              __stcg(d1 + lane * JB + o, x[h][0]);
              __stcg(d1 + o * JB + lane, x[h][0]);
              __stcg(d2 + lq * JB + oq, x[h][3]);
              __stcg(d2 + oq * JB + lq, x[h][3]);
            }
          }
          __syncthreads();
        }
        phase(2);
        // ---- X <- X Q, V <- V Q on this CTA's rows: a warp 64 rows by 32 columns at
        // a time, a lane 8 x 8 of it (four 16-byte shared loads for 64
        // multiply-adds a step of the sum, as the loads are the bound of smaller
        // lane tiles: 27.7 against 13 us a round at n = 1803 with 4 x 4)
        for (int it = 0; it < 2 * nsub; ++it) {
          float* M = it < nsub ? P.X : P.V;
          const int sub = it < nsub ? it : it - nsub;
          float* t = (it & 1) ? tile1 : tile0;
          if (nsub == 1) {
            if (it == 1) asm volatile("cp.async.wait_group 0;" ::: "memory");
          } else {
            if (it + 1 < 2 * nsub)
              asm volatile("cp.async.wait_group 1;" ::: "memory");
            else
              asm volatile("cp.async.wait_group 0;" ::: "memory");
          }
          __syncthreads();
          const int r0 = row0 + sub * P.rt;
          const int rows = max(0, min(P.rt, row1 - r0));
          const int k0 = 32 * (wid & 1) + 4 * (lane >> 3);  // columns k0 .. k0 + 3 and k0 + 16 ..
          for (int rb = 64 * (wid >> 1); rb < rows; rb += 64 * (JNW / 2)) {
            const int rr = rb + 4 * (lane & 7);  // rows rr .. rr + 3 and rr + 32 ..
            const float* ta = t + (rr < rows ? rr : 0);
            const float* tb = t + (rr + 32 < rows ? rr + 32 : 0);
            f2 acc[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[i][j] = 0;
#pragma unroll 4
            for (int i = 0; i < JC; ++i) {
              const ulonglong2 xa = *reinterpret_cast<const ulonglong2*>(ta + i * lds);
              const ulonglong2 xb = *reinterpret_cast<const ulonglong2*>(tb + i * lds);
              const float4 wa = *reinterpret_cast<const float4*>(Q + i * JQS + k0);
              const float4 wb = *reinterpret_cast<const float4*>(Q + i * JQS + k0 + 16);
              const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const f2 ww = pack2(w[j], w[j]);
                acc[0][j] = fma2(xa.x, ww, acc[0][j]);
                acc[1][j] = fma2(xa.y, ww, acc[1][j]);
                acc[2][j] = fma2(xb.x, ww, acc[2][j]);
                acc[3][j] = fma2(xb.y, ww, acc[3][j]);
              }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int k = k0 + (j & 3) + 16 * (j >> 2);
              const int b = k < JB ? b1 : b2;
              const int col = b * JB + (k & (JB - 1));
              if (b >= nblk || col >= n) continue;
              // (the padding rows up to ld hold zeros and get zeros)
              float* o = M + (int64_t)col * P.ld + r0 + rr;
              if (rr < rows) *reinterpret_cast<ulonglong2*>(o) = make_ulonglong2(acc[0][j], acc[1][j]);
              if (rr + 32 < rows) *reinterpret_cast<ulonglong2*>(o + 32) = make_ulonglong2(acc[2][j], acc[3][j]);
            }
          }
          if (nsub > 1 && it + 2 < 2 * nsub) {
            __syncthreads();
            const int nx = it + 2;
            load(t, nx < nsub ? P.X : P.V, nx < nsub ? nx : nx - nsub);
          }
        }
      }
      phase(3);
      if (!grid_sync(P.bar)) return;
      phase(4);
    }
    const double offd = block_max((double)off, red);
    if (threadIdx.x == 0) P.off[blockIdx.x] = offd;
    if (!grid_sync(P.bar)) return;
    double mx = 0;
    for (int b = threadIdx.x; b < gridDim.x; b += JNT) mx = fmax(mx, __ldcg(P.off + b));
    mx = block_max(mx, red);
    if (!grid_sync(P.bar)) return;
    if (mx <= P.stop) {
      ++sweep;
      break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.sweeps_out = sweep;
}

}  // namespace

WaitUnit wait_unit_jg() { return this_wait_unit("jacobi_gram"); }

// X (n x n) and V (n x n, the identity on entry) with one leading dimension,
// a multiple of 4, rows n .. ld zero; false when the shape does not fit
bool jacobi_gram_sweeps(lra_ctx* ctx, int64_t n, float* X, float* V, int64_t ld, double stop) {
  if (n < 2 * JB || n > 1 << 20 || (ld & 3)) return false;
  raise_smem_limit(ctx, (const void*)jacobi_gram_kernel);
  cudaFuncAttributes fa;
  LRA_CUDA(cudaFuncGetAttributes(&fa, jacobi_gram_kernel));
  const int64_t cap = fa.maxDynamicSharedSizeBytes / 4 - (JC * JGS + 4 + JC * JQS);  // floats
  const int64_t nblk = (n + JB - 1) / JB, pairs = (nblk + 1) / 2;
  if (pairs > ctx->num_sms) return false;
  JgParams P;
  // row chunks: as many CTAs per pair as there are SMs, at least 32 rows each
  P.c = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(ctx->num_sms / pairs, JMAXC), n / 32));
  P.chunk = (int)(((n + P.c - 1) / P.c + 3) / 4 * 4);
  P.c = (int)((n + P.chunk - 1) / P.chunk);
  // a tile's column stride: 4 mod 8 words keeps the Gram product's columns off
  // one another's banks
  auto stride = [](int64_t rows) { return (rows + 3) / 8 * 8 + 4; };
  auto words = [&](int64_t rows) {
    return JC * stride(rows) + std::max<int64_t>(JC * stride(rows), (int64_t)JNW * JB * JB);
  };
  int64_t rt = P.chunk;
  while (rt > 4 && words(rt) > cap) rt = rt > 512 ? 512 : rt - 4;
  if (words(rt) > cap) return false;
  P.rt = (int)rt;
  P.lds = (int)stride(rt);
  const size_t smem = (size_t)(words(rt) + JC * JGS + 4 + JC * JQS) * 4;
  P.n = (int)n;
  P.X = X;
  P.V = V;
  P.ld = ld;
  const double tol = (double)Real<float>::eps * 2.0 * std::sqrt((double)n);
  P.tol2 = (float)(4.0 * tol * tol);
  P.stop = stop;
  P.max_sweeps = 40;
  const int grid = (int)(pairs * P.c);
  const ArenaMark mk = ctx->arena.mark();
  P.part = ctx->arena.alloc_n<float>((size_t)grid * 3 * JB * JB);
  P.diag = ctx->arena.alloc_n<float>((size_t)nblk * JB * JB);
  P.arrive = ctx->arena.alloc_n<unsigned>((size_t)pairs * 32);
  P.off = ctx->arena.alloc_n<double>(grid);
  P.bar = reinterpret_cast<GridBar*>(ctx->arena.alloc(sizeof(GridBar)));
  P.sweeps_out = ctx->arena.alloc_n<int>(1);
  LRA_CUDA(cudaMemsetAsync(P.arrive, 0, (size_t)pairs * 32 * sizeof(unsigned), ctx->stream));
  LRA_CUDA(cudaMemsetAsync(P.bar, 0, sizeof(GridBar), ctx->stream));
  if (trace_on()) {
    P.phase_ns = ctx->arena.alloc_n<unsigned long long>(6);
    LRA_CUDA(cudaMemsetAsync(P.phase_ns, 0, 6 * sizeof(unsigned long long), ctx->stream));
  }
  void* args[] = {&P};
  LRA_CUDA(cudaLaunchCooperativeKernel((const void*)jacobi_gram_kernel, dim3((unsigned)grid), dim3(JNT), args, smem,
                                       ctx->stream));
  post_launch(ctx, "jacobi_gram_kernel");
  GridBar hb;
  int sweeps = 0;
  unsigned long long ph[6] = {0, 0, 0, 0, 0, 0};
  if (P.phase_ns) LRA_CUDA(cudaMemcpyAsync(ph, P.phase_ns, sizeof ph, cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaMemcpyAsync(&hb, P.bar, sizeof(GridBar), cudaMemcpyDeviceToHost, ctx->stream));
  if (trace_on())
    LRA_CUDA(cudaMemcpyAsync(&sweeps, P.sweeps_out, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LRA_CUDA(cudaStreamSynchronize(ctx->stream));
  ctx->arena.release(mk);
  if (hb.err != 0) fail(LRA_ETIMEDOUT, "jacobi: a wait between CTAs timed out");
  if (trace_on())
    std::fprintf(stderr, "[lra] jacobi f32 gram n=%lld ctas=%d x %d rows/tile=%d sweeps=%d; CTA 0 ms: gram %.2f meet %.2f "
                 "collect %.2f rotations %.2f X, V %.2f barrier %.2f\n", (long long)n, (int)pairs, P.c, P.rt, sweeps, ph[0] * 1e-6,
                 ph[1] * 1e-6, ph[5] * 1e-6, ph[2] * 1e-6, ph[3] * 1e-6, ph[4] * 1e-6);
  return true;
}

}  // namespace lra
