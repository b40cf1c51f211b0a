// Grid-wide barrier of the cooperative kernels.
#pragma once

#include "gmes_internal.cuh"

namespace gmes {
namespace {

// Arrivals (low half) and the failed word (high half) of a slot.
__device__ __forceinline__ unsigned long long load_slot(const Slot* s) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(s) : "memory");
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
// grid barrier in CUDA's cooperative groups header).  False: gave up, after
// m.polls polls (each a round trip to L2, about a microsecond) or because a
// block before has; what meets at the slot after that gives up too, until
// clear_slots.
__device__ __forceinline__ bool grid_barrier(const Meeting& m, int* error) {
  __shared__ int good;
  __syncthreads();
  if (threadIdx.x == 0) {
    Slot* const s = m.at;
    const unsigned old =
        add_acq_rel(&s->word, blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u);
    unsigned long long v;
    int n = 0;
    do
      v = load_slot(s);
    while (((old ^ (unsigned)v) & 0x80000000u) == 0 && v >> 32 == 0 && ++n < m.polls);
    good = ((old ^ (unsigned)v) & 0x80000000u) != 0 && v >> 32 == 0;
    if (!good) {
      *static_cast<volatile unsigned*>(&s->failed) = 1;
      *static_cast<volatile int*>(error) = 1;
    }
  }
  __syncthreads();
  return good != 0;
}

// The results of a launch that gave up read as NaN: each block that gives up
// fills its share of them with ones.
__device__ __noinline__ void spoil(void* p, int64_t bytes) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < bytes / 4;
       k += (int64_t)gridDim.x * blockDim.x)
    static_cast<uint32_t*>(p)[k] = 0xffffffffu;
}

// After a launch's last barrier: once all its blocks are here, the slot may go
// to another stream.
__device__ __forceinline__ void leave_barrier(const Meeting& m) {
  if (m.done == nullptr || threadIdx.x != 0) return;
  Slot& s = *m.at;
  if (add_acq_rel(&s.left, 1u) != gridDim.x - 1) return;
  s.left = 0;
  __threadfence_system();
  *static_cast<volatile uint32_t*>(m.done) = m.number;
}

}  // namespace
}  // namespace gmes
