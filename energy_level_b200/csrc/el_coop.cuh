// Grid barrier of the cooperative kernels.
#pragma once

#include "el_internal.cuh"

namespace el {

// All CTAs of the launch meet: an arrival counter (zero at launch) polled by
// one thread per CTA.  Writes before the barrier are released with the
// arrival and acquired with the poll that sees the count complete.  The wait
// is bounded: after poll_limit polls the error flag is set, and every later
// barrier returns at once.
__device__ __forceinline__ void coop_sync(unsigned *bar, int *err, int nctas, int poll_limit, unsigned &gen) {
  __syncthreads();
  gen += (unsigned)nctas;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    if (!*(volatile int *)err) {
      int polls = 0;
      unsigned v;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        if (v >= gen) break;
        if (++polls > poll_limit) { atomicExch(err, 1); break; }
        if ((polls & 255) == 0 && *(volatile int *)err) break;
      }
    }
  }
  __syncthreads();
}

}  // namespace el
