// Grid-wide barrier of the persistent cooperative kernels (recur.cu, nonorth.cu).
//
// All CTAs of a cooperative launch are co-resident, so they can wait for each other.  One
// counter only grows: a CTA arrives with a release addition, and barrier k is passed when the
// counter has reached k times the number of CTAs, which each CTA polls with acquire loads.  So
// a barrier costs the stores' acknowledgement, the addition's way to L2 and one poll, about
// 1 us; a last arrival that resets a count and bumps a generation adds two dependent round
// trips, and sleeping between polls half of a poll (a recursion step of 961 rows on 4 CTAs took
// 4.4 us with these and takes 2.3 us; of 65536 rows on 256 CTAs, 4.5 and 2.4 us).
// Arrival and wait are separate, so that work whose results no other CTA reads in the next step
// (the dot products) runs between them.
//
// The wait is bounded: after kSpinLimit polls a CTA sets the error flag and every waiting CTA
// gives up, so a bad launch ends instead of hanging the GPU; the host turns the flag into
// LINQT_ERR_TIMEOUT (check_device_errors).  For tests, a session can make its barriers wait
// for CTAs that were never launched, with a short poll limit
// (linqt_session_inject_barrier_timeout): the kernel then returns through the same path.
// Release: bar.sync, then the addition at gpu scope, which orders the whole CTA's stores;
// acquire: the poll, then bar.sync.  The acquire drops stale L1 lines, so data written by other
// CTAs before the barrier may be read through L1 after it.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace linqt {

struct GridBarrier {
  unsigned count;  // arrivals since the launch
  int err;
  int extra;              // fault injection (tests): arrivals awaited beyond the launched CTAs
  long long spin_limit;   // fault injection (tests): polls before giving up (0: kSpinLimit)
};
// bytes of GridBarrier that restart at zero for every launch
constexpr size_t kBarrierResetBytes = offsetof(GridBarrier, err);

constexpr unsigned kFewCtas = 2 * 148;  // two CTAs on each of a B200's SMs

constexpr long long kSpinLimit = 1LL << 24;  // polls of a few 0.1 us: well above any step, far below a hang

// One CTA's state of the barrier, used by its thread 0.  In shared memory: the kernels around it
// are short of registers.
struct GridSyncState {
  unsigned need, target;
  long long limit;
};
__device__ __forceinline__ GridSyncState &grid_sync_state() {
  __shared__ GridSyncState st;
  return st;
}

// Once, by every thread, before the first barrier of a launch.
__device__ __forceinline__ void grid_init(GridBarrier *bar, unsigned nblocks) {
  if (threadIdx.x == 0) {
    GridSyncState &st = grid_sync_state();
    st.need = nblocks + (unsigned)bar->extra;
    st.target = 0;
    st.limit = bar->spin_limit > 0 ? bar->spin_limit : kSpinLimit;
  }
}

// This CTA's stores so far are what the next step of every CTA may read.
__device__ __forceinline__ void grid_arrive(GridBarrier *bar) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(&bar->count) : "memory");
    GridSyncState &st = grid_sync_state();
    st.target += st.need;
  }
}

__device__ __forceinline__ unsigned load_acquire(const unsigned *p) {
  unsigned c;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(c) : "l"(p) : "memory");
  return c;
}
__device__ __forceinline__ unsigned load_relaxed(const unsigned *p) {
  unsigned c;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(c) : "l"(p) : "memory");
  return c;
}

// False if the wait gave up (the error flag is then set).
__device__ __forceinline__ bool grid_wait(GridBarrier *bar) {
  int bad = 0;
  if (threadIdx.x == 0) {
    const GridSyncState &st = grid_sync_state();
    const unsigned target = st.target;
    // An acquire drops the SM's L1 lines.  Up to two CTAs an SM (256 CTAs: 0.4 us less a
    // barrier than a fence after the poll) every poll is one; with more, whose other CTAs
    // would read on through a cold L1 meanwhile, only the last load is.
    const bool few = st.need <= kFewCtas;
    for (long long spins = 1;; ++spins) {
      const unsigned c = few ? load_acquire(&bar->count) : load_relaxed(&bar->count);
      if ((int)(c - target) >= 0) break;
      if ((spins & 1023) == 0 || spins >= st.limit) {
        if (*(volatile int *)&bar->err) {
          bad = 1;
          break;
        }
        if (spins >= st.limit) {
          atomicExch(&bar->err, 1);
          bad = 1;
          break;
        }
      }
    }
    if (!few) (void)load_acquire(&bar->count);
  }
  return __syncthreads_or(bad) == 0;
}

__device__ __forceinline__ bool grid_barrier(GridBarrier *bar) {
  grid_arrive(bar);
  return grid_wait(bar);
}

}  // namespace linqt
