// Bounded device-side waits shared by the persistent kernels: the limits, the
// acquire loads and the grid barrier of a cooperative launch.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>

namespace e2e {

// A wait gives up after `spins` polls or `timeout_ns`, sets an error bit the
// host reads (E2E_ERR_DEVICE) and lets the launch drain.  `extra` raises every
// wait's target so that no wait can complete: the test hook that makes the
// bounded waits run out on purpose, without any fault.
struct WaitBound {
  unsigned long long timeout_ns;
  long long spins;
  unsigned int extra;
};

// Host: E2E_WAIT_LIMIT_MS (default 2000) bounds each wait; with
// E2E_TEST_UNREACHABLE_WAIT=1 the targets are raised by one (tests only).
inline WaitBound wait_bound_from_env() {
  WaitBound w{2000000000ull, 1ll << 22, 0u};
  if (const char* ms = std::getenv("E2E_WAIT_LIMIT_MS")) {
    const double v = std::atof(ms);
    if (v > 0 && v <= 60000) w.timeout_ns = (unsigned long long)(v * 1e6);
  }
  if (const char* u = std::getenv("E2E_TEST_UNREACHABLE_WAIT")) w.extra = (u[0] == '1') ? 1u : 0u;
  return w;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// orders the CTA's earlier writes (behind a __syncthreads) before the count;
// against a fence and an addition 0.3 us less a barrier
__device__ __forceinline__ void add_release(unsigned int* p, unsigned int n) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(n) : "memory");
}

// The limits of one wait.  The clock is read on every 32nd poll only: the read
// takes longer than a wait that is about to end.
struct WaitClock {
  static constexpr int kEvery = 32;
  long long polls = 0;
  unsigned long long t0 = 0;
  __device__ __forceinline__ bool over(const WaitBound& wb) {
    if (++polls % kEvery) return false;
    const unsigned long long now = global_ns();
    if (t0 == 0) t0 = now;
    return polls > wb.spins || now - t0 > wb.timeout_ns;
  }
};

// Grid-wide barrier of a cooperative launch, in two halves so that work which needs
// no other CTA can stand between them.  sync[0] counts arrivals (never reset inside
// a launch); a wait that outlives its limit sets bit 1 of sync[1] and every later
// wait returns false at once.
__device__ __forceinline__ void grid_arrive(unsigned int* sync) {
  __syncthreads();
  if (threadIdx.x == 0) add_release(sync, 1u);
}

__device__ __forceinline__ bool grid_wait(unsigned int* sync, unsigned int target, const WaitBound& wb) {
  __shared__ int ok;
  if (threadIdx.x == 0) {
    int good = 1;
    WaitClock clock;
    while (ld_acquire(sync) < target + wb.extra) {
      if (clock.over(wb) || (clock.polls % WaitClock::kEvery == 0 && ld_acquire(sync + 1) != 0u)) {
        atomicOr(sync + 1, 2u);
        good = 0;
        break;
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

__device__ __forceinline__ bool grid_barrier(unsigned int* sync, unsigned int target, const WaitBound& wb) {
  grid_arrive(sync);
  return grid_wait(sync, target, wb);
}

}  // namespace e2e
