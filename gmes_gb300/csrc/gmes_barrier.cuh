// Grid-wide barrier of the cooperative kernels.
#pragma once

#include "gmes_internal.cuh"

namespace gmes {
namespace {

// Polls of the barrier's word before a block gives up (each poll is a
// round trip to L2, about a microsecond: some seconds), sets the error word
// and returns; every other block then gives up too.
constexpr int kBarrierPolls = 1 << 22;

// A barrier slot: the blocks' arrivals (zero low bits after every barrier) and
// the blocks that have left the launch's last one.
struct alignas(32) Slot {
  unsigned word, left;
};
__device__ Slot slots[kStreamSlots + kGraphSlots];

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned add_acq_rel(unsigned* p, unsigned v) {
  unsigned old;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;"
               : "=r"(old)
               : "l"(p), "r"(v)
               : "memory");
  return old;
}

// All blocks of the (cooperative) launch arrive before any leaves.  Each adds
// one, block 0 the rest of 2^31, so the word's top bit flips when the last
// block has arrived and the low bits are zero again (the arrival scheme of the
// grid barrier in CUDA's cooperative groups header).  False: gave up.
__device__ __forceinline__ bool grid_barrier(const Meeting& m, int* error) {
  __shared__ int good;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned* const word = &slots[m.slot].word;
    const unsigned old =
        add_acq_rel(word, blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u);
    int n = 0;
    while (((old ^ load_acquire(word)) & 0x80000000u) == 0 && n < kBarrierPolls) ++n;
    good = n < kBarrierPolls;
    if (!good) *error = 1;
  }
  __syncthreads();
  return good != 0;
}

// After a launch's last barrier: once all its blocks are here, the slot may go
// to another stream.
__device__ __forceinline__ void leave_barrier(const Meeting& m) {
  if (m.done == nullptr || threadIdx.x != 0) return;
  Slot& s = slots[m.slot];
  if (add_acq_rel(&s.left, 1u) != gridDim.x - 1) return;
  s.left = 0;
  __threadfence_system();
  *static_cast<volatile uint32_t*>(m.done) = m.number;
}

}  // namespace
}  // namespace gmes
