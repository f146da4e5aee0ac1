// Pivoted QRs that hold their columns in shared memory at input precision
// (ComplexF32, ComplexF64, Float64 native): norms on their bits and the pivot
// exchange between the blocks.
#pragma once

#include "common.cuh"

namespace lra {

template <typename R>
struct NormBits;
template <>
struct NormBits<double> {
  // a norm as an integer of the same order, -1 for a NaN
  static __device__ long long key(double v) {
    const long long k = __double_as_longlong(v) & 0x7fffffffffffffffll;
    return k > 0x7ff0000000000000ll ? -1 : k;
  }
  static __device__ double value(long long k) { return __longlong_as_double(k); }
  // the leading bits of |v|, their exponent, whether its square and root are safe
  static __device__ unsigned lead(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
  static __device__ int expo(unsigned h) { return (int)(h >> 20) - 1023; }
  static __device__ bool safe(unsigned h) { return h >= (123u << 20) && h < (1923u << 20); }
  static __device__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }
};
template <>
struct NormBits<float> {
  static __device__ long long key(float v) {
    const unsigned k = __float_as_uint(v) & 0x7fffffffu;
    return k > 0x7f800000u ? -1 : (long long)k;
  }
  static __device__ float value(long long k) { return __uint_as_float((unsigned)k); }
  static __device__ unsigned lead(float v) { return __float_as_uint(v) & 0x7fffffffu; }
  static __device__ int expo(unsigned h) { return (int)(h >> 23) - 127; }
  static __device__ bool safe(unsigned h) { return h >= (27u << 23) && h < (227u << 23); }
  static __device__ float pow2(int e) { return __int_as_float((e + 127) << 23); }
};

// The blocks' candidates: word and staged column by the parity of the exchange.
template <typename E>
struct ColXch {
  ulonglong2* word;  // [2][G], zeroed before the launch
  E* stage;          // [2][G][m]
};
struct ColXchShared {
  long long key;
  int64_t id;
  int q, owner, any, bad, pay;
};

// Exchange e.  find(lane, v, i), by warp 0: the best of the block's candidates
// as (key, id << 24 | slot); pay(slot) goes with it.  Ids and payloads are below
// 2^24, equal keys go to the smaller id.  The winner's rows from..m-1 are staged, then
// offered in one 16-byte word (release), and warp 0 reads all G <= 256 words until
// they are this exchange's: one trip through L2 a pivot.  Two parities are
// enough: whoever offers exchange e + 2 has read all of e + 1, whose offers
// come after the reads of e.  On return s holds the best key, its id (none: n),
// payload and block, and the OR of the flags; false if a wait ran out.
template <int NT, typename E, typename F, typename Y>
__device__ __forceinline__ bool col_exchange(ColXchShared& s, const ColXch<E>& x, GridBar* bar, int e, int from, int m, int64_t n,
                                             const E* cols, int flag, F find, Y pay) {
  constexpr int PW = 256 / 32;  // words a lane
  const int G = gridDim.x, b = blockIdx.x, lane = threadIdx.x & 31;
  __syncthreads();
  if (threadIdx.x < 32) {
    long long v = -1;
    int64_t i = n << 24;
    find(lane, v, i);
    warp_argmax(v, i);
    if (lane == 0) {
      s.q = v >= 0 ? (int)(i & 0xffffff) : -1;
      s.key = v;
      s.id = v >= 0 ? i >> 24 : n;
      s.pay = v >= 0 ? pay(s.q) : 0;
    }
  }
  __syncthreads();
  E* st = x.stage + ((size_t)(e & 1) * G + b) * m;
  if (s.q >= 0) {
    const E* a = cols + (size_t)s.q * m;
    for (int i = from + threadIdx.x; i < m; i += NT) st[i] = a[i];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    ulonglong2* const wd = x.word + (size_t)(e & 1) * G;
    const unsigned long long seq = (unsigned long long)((e + 1) & 0x3fff) << 50;
    if (lane == 0)
      st_word(wd + b, (unsigned long long)s.key,
              seq | (unsigned long long)s.id << 25 | (unsigned long long)s.pay << 1 | (unsigned long long)flag);
    ulonglong2 w[PW];
    uint64_t t0 = 0;
    bool bad = false;
    for (int it = 1;; ++it) {
      bool all = true;
#pragma unroll
      for (int k = 0; k < PW; ++k)
        if (k * 32 + lane < G) w[k] = ld_word(wd + k * 32 + lane);
#pragma unroll
      for (int k = 0; k < PW; ++k)
        if (k * 32 + lane < G) all &= (w[k].y >> 50) == seq >> 50;
      if (__all_sync(0xffffffffu, all)) break;
      if ((it & 63) == 0) {
        const uint64_t t = globaltimer_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > wait_limit_ns()) atomicCAS(&bar->err, 0, 4);
        bad = __any_sync(0xffffffffu, *((volatile int*)&bar->err) != 0);
        if (bad) break;
      }
    }
    __threadfence();
    long long v = -1;
    int64_t i = n << 16;
    bool fl = false;
#pragma unroll
    for (int k = 0; k < PW; ++k)
      if (k * 32 + lane < G) {
        fl |= (w[k].y & 1) != 0;
        argmax_merge<long long>(v, i, (long long)w[k].x, (int64_t)((w[k].y >> 25) & 0x1ffffff) << 16 | (k * 32 + lane));
      }
    warp_argmax(v, i);
    fl = __any_sync(0xffffffffu, fl);
    const int owner = (int)(i & 0xffff);
    int py = 0;
#pragma unroll
    for (int k = 0; k < PW; ++k)
      if (k * 32 + lane == owner && owner < G) py = (int)((w[k].y >> 1) & 0xffffff);
    py = __shfl_sync(0xffffffffu, py, owner & 31);
    if (lane == 0) {
      s.key = v;
      s.pay = py;
      s.id = v >= 0 ? i >> 16 : n;
      s.owner = owner;
      s.any = fl;
      s.bad = bad;
    }
  }
  __syncthreads();
  return s.bad == 0;
}

// Of two blocks one offers and the other never does: the wait runs out.  (gb, zeros,
// returned: as probe_wait_kernel's)
template <typename E>
__global__ void __launch_bounds__(32) probe_col_exchange_kernel(GridBar* gb, unsigned long long* zeros, int* returned) {
  __shared__ ColXchShared s;
  if (blockIdx.x == 0) {
    const ColXch<E> x{reinterpret_cast<ulonglong2*>(zeros), reinterpret_cast<E*>(zeros + 64)};
    const bool ok = col_exchange<32>(s, x, gb, 0, 0, 1, 1, static_cast<const E*>(nullptr), 0,
                                     [](int, long long&, int64_t&) {}, [](int) { return 0; });
    if (threadIdx.x == 0 && ok) atomicAdd(returned, 1000);
  }
  if (threadIdx.x == 0) atomicAdd(returned, 1);
}

}  // namespace lra
