// last_block.cuh -- which of a launch's blocks finishes last, for reductions
// whose last block adds what the others stored.
#pragma once

namespace dyn {

// Called by every thread of each of 'nb' blocks after its stores: true in the
// block that takes the last ticket, which may then read what every thread of
// every block stored.  The barrier stands between the block's stores and its
// ticket: a thread's fence orders its own stores only, so without it the ticket
// could be taken before the other threads' stores.
__device__ inline bool last_block(unsigned* counter, unsigned nb) {
  __shared__ unsigned ticket;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) ticket = atomicAdd(counter, 1u);
  __syncthreads();
  if (ticket != nb - 1) return false;
  __threadfence();
  return true;
}

}  // namespace dyn
