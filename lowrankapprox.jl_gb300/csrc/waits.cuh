// The bounded waits of a translation unit: its limit, and kernels whose waits
// nothing ends, for the self-test.
#pragma once

#include "common.cuh"
#include "internal.hpp"

namespace lra {

namespace {

// Two CTAs meet at a grid barrier whose arrival count starts at the grid
// size, so that no arrival completes it, and wait for a word that nobody
// raises: every wait ends by its limit, records the time-out, and both CTAs
// return.
__global__ void probe_wait_kernel(GridBar* gb, unsigned long long* zeros, int* returned) {
  const bool met = grid_sync(gb);
  if (threadIdx.x != 0) return;
  int* err = reinterpret_cast<int*>(zeros + 1 + blockIdx.x);  // (gb->err would end this wait at once)
  const bool reached = wait_reached(reinterpret_cast<const unsigned*>(zeros), 1u, err);
  atomicAdd(returned, met || reached || *((volatile int*)err) != 4 ? 1000 : 1);
}

inline WaitUnit this_wait_unit(const char* name, const void* probe2 = nullptr) {
  return WaitUnit{name, [](uint64_t ns) { return set_unit_wait_limit(ns); }, {(const void*)probe_wait_kernel, probe2}};
}

}  // namespace

}  // namespace lra
