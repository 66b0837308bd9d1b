// The last-block ticket of the ICP's reductions (dynamap_b200/csrc/last_block.cuh)
// under the thread-block emulation, whose threads run one after another up to
// the next barrier: when a block takes its ticket, all its stores must be there.
#include "cuda_emu.h"

#include <vector>

static std::vector<int>* g_row;  // what the running block has stored
static int g_early = 0;          // tickets taken before the whole row was there
inline void __threadfence() {}
inline unsigned atomicAdd(unsigned* p, unsigned v) {
  for (const int x : *g_row) g_early += x == 0;
  const unsigned old = *p;
  *p += v;
  return old;
}

#include "../../dynamap_b200/csrc/last_block.cuh"

// Blocks of 'threads' threads each store 'values' of theirs and take the ticket;
// returns the stores that a ticket did not wait for, and in *last the number of
// blocks that were told to be the last one.
extern "C" int last_block_check(int blocks, int threads, int values, int* last) {
  unsigned counter = 0;
  std::vector<int> row(values, 0), told(blocks, 0);
  g_row = &row;
  g_early = 0;
  emu::launch(blocks, threads, [&] {
    const int t = (int)threadIdx.x;
    if (t == 0) std::fill(row.begin(), row.end(), 0);
    __syncthreads();
    if (t < values) row[t] = 1 + t;
    if (dyn::last_block(&counter, (unsigned)blocks)) told[blockIdx.x] = 1;
    __syncthreads();
  });
  *last = 0;
  for (const int x : told) *last += x;
  return g_early;
}
