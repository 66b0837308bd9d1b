// The persistent ICP's host arithmetic (dynamap_b200/csrc/icp.cuh).  Its rows, in the order that
// lets a block fall behind: one that has left after its last level's rows were
// complete, but has not read them yet, while the others run every later level.
#include "cuda_emu.h"

#include <cstdint>
#include <set>
#include <vector>

#include "../../dynamap_b200/csrc/icp.cuh"

extern "C" int icp_tiles_of(int npx, int kahan) { return dyn::icp_tiles(npx, kahan); }

// Level slots of npx[0..2] pixels, iters[0..2] executed iterations each, a block
// per tile.  Returns the rows of some block's last level that a later level
// overwrites (of *leavers levels that some block leaves after).
extern "C" int icp_rows_overwritten(const int* npx, const int* iters, int kahan, int* leavers) {
  using namespace dyn;
  int nt[3], bad = 0;
  *leavers = 0;
  for (int pl = 0; pl < 3; ++pl) nt[pl] = iters[pl] > 0 ? icp_tiles(npx[pl], kahan) : 0;
  for (int pl = 0; pl < 3; ++pl) {
    int later = 0;
    for (int q = pl + 1; q < 3; ++q) later = nt[q] > later ? nt[q] : later;
    if (nt[pl] <= later || nt[pl] == 0) continue;  // every block goes on
    ++*leavers;
    std::set<int> rows;  // what a block that leaves reads last
    for (int t = 0; t < nt[pl]; ++t) rows.insert(icp_row(pl, iters[pl], t));
    for (int q = pl + 1; q < 3; ++q) {
      for (int it = 1; it <= iters[q]; ++it)
        for (int t = 0; t < nt[q]; ++t) bad += rows.count(icp_row(q, it, t)) != 0;
      bad += rows.count(icp_state_row(q)) != 0;
    }
  }
  return bad;
}

// Every row and state word lies in the scratch; rows of one level and parity
// are distinct.
extern "C" int icp_rows_in_scratch() {
  using namespace dyn;
  std::set<int> seen;
  for (int pl = 0; pl < 3; ++pl) {
    for (int par = 0; par < 2; ++par)
      for (int t = 0; t < kIcpMaxTiles; ++t) seen.insert(icp_row(pl, 2 + par, t));
    seen.insert(icp_state_row(pl));
  }
  const size_t end = icp_rows_offset() + ((size_t)*seen.rbegin() + 1) * kIcpRowWords * 8;
  return *seen.begin() == 0 && (int)seen.size() == 6 * kIcpMaxTiles + 3 &&
         end <= icp_frame_scratch_bytes();
}

// The epoch after the one given, over a scratch filled with 'fill': returns the
// new epoch; *rows the bytes of the rows that still hold the fill, *before those
// of what lies before the rows.
extern "C" unsigned icp_next_epoch(unsigned epoch, int fill, int64_t* rows, int64_t* before) {
  using namespace dyn;
  std::vector<unsigned char> scratch(icp_frame_scratch_bytes() + 16, (unsigned char)fill);
  unsigned bar[kIcpBarWords] = {epoch};
  unsigned char* base = scratch.data();
  while (reinterpret_cast<uintptr_t>(base) & 15) ++base;
  advance_epoch(bar, base);
  *rows = *before = 0;
  for (size_t i = 0; i < icp_frame_scratch_bytes(); ++i)
    (i < icp_rows_offset() ? *before : *rows) += base[i] == (unsigned char)fill;
  return bar[0];
}

extern "C" void icp_budgets(const long long* weight, const int* count, int k, int cap, int* out) {
  dyn::icp_group_budgets(weight, count, k, cap, out);
}
extern "C" long long icp_weight_of(int npx, int kahan) { return dyn::icp_weight(npx, kahan); }

// The parts of a table (0: chained): their grids per kind and first sessions.
extern "C" int icp_table(const int* npx, const int* kahan, int n, int budget, int* grid,
                         int* first) {
  const dyn::IcpLaunches L = dyn::icp_launches(npx, kahan, n, budget);
  for (int p = 0; p < L.parts; ++p)
    for (int k = 0; k < 2; ++k) grid[2 * p + k] = L.grid[p][k];
  for (int p = 0; p <= L.parts && L.parts > 0; ++p) first[p] = dyn::icp_part_first(n, L.parts, p);
  return L.parts;
}
