// solve.cuh - what solver.cu (preparation, colouring) and solve.cu (the solve
// kernels) share: the block shape, the bounded grid barrier, and the solve's
// instances.
#pragma once

#include "avbd_device.cuh"

namespace avbd {
namespace {

constexpr int kSolveBlock = 128;   // threads of a solve block (3 blocks per SM)
static_assert(kSolveBlock == kLaneMaxGroup, "a lane chunk is one solve block");
constexpr int kStageSlots = 4;     // contacts a lane stages in shared memory at a time
constexpr int kStageVecs = 9;      // float4 per staged contact
constexpr size_t kSolveSmem = (size_t)kSolveBlock * kStageSlots * kStageVecs * sizeof(float4);  // 73,728 B

// ---------------------------------------------------------------------------
// Bounded grid barrier (all blocks are co-resident: cooperative launch), in
// two halves. Arrivals are counted in one word (zeroed with the step's
// counters), and barrier k of `blocks` blocks is over when it reaches
// k * blocks. Waiters poll the word the arrivals go to, and the timeout flag
// in the same round trip: with a generation word that the last arrival
// writes, a second fence and a closing flag read, a barrier of one busy block
// took 3,800 cycles, with this 2,200. grid_wait returns false when the wait
// gave up or another block reported a timeout; the caller must then return.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void grid_arrive(unsigned *arrivals) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrivals) : "memory");
}
__device__ __forceinline__ bool grid_wait(Control *ctl, const unsigned *arrivals, unsigned target, long long limit) {
  __shared__ int ok;
  if (threadIdx.x == 0) {
    int good = 1;
    long long spins = 0;
    for (;;) {
      const unsigned f = *((volatile unsigned *)&ctl->flags);  // in flight together with the count
      unsigned v;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrivals) : "memory");
      if (f & kOvfTimeout) good = 0;
      if ((int)(v - target) >= 0 || !good) break;
      // give up after `limit` polls, or at once when another block gave up
      if (++spins > limit) {
        atomicOr(&ctl->flags, kOvfTimeout);
        good = 0;
        break;
      }
      __nanosleep(20);
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// A step skipped for a candidate overflow (Control::skip): its kernels after
// the broad phase return at once and leave every state array untouched.
__device__ __forceinline__ bool step_skipped(const World &w) { return *((volatile int *)&w.ctl->skip) != 0; }

}  // namespace

// The solve's instantiations: the contact extensions
// (AVBD_CONTACT_MATERIALS), joints and springs, and the FP64 bodies each in
// kernels of their own, so that the others carry none of their registers. The
// joints' calls cost some 180 bytes of spills, the FP64 path's a 1.5 KB stack
// frame and 800, which every grid barrier's acquire throws out of L1; without
// them there are none (168 registers; solve of piles of 200 / 8,192 bodies 0.30
// -> 0.27 / 0.60 -> 0.55 ms, the crushed 36-layer pyramid 4.96 -> 4.58).
// Each is a unit of its own (solve.cu compiled once per instance): a unit's
// code is loaded whole when a process first needs any of it, and with all
// instances in one the first pack of a process took 15 ms.
using SolveInstance = const void *(bool wave);  // the colour-phase or the wavefront kernel
SolveInstance solve_plain, solve_forces, solve_forces_fp64;
SolveInstance solve_materials, solve_materials_forces, solve_materials_forces_fp64;

}  // namespace avbd
