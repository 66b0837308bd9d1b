// icp.cuh -- projective point-to-plane (+photometric) ICP normal equations
// and the on-device Gauss-Newton step.
#pragma once
#include "common.cuh"

namespace dyn {

// Per-session solver state, device resident.
struct IcpState {
  double inc[6];      // xi accumulated over the frame's levels (gnSolver.cu:345)
  double prev[6];     // prev_increment (gnSolver.cu:347,415)
  float T[16];        // float exp(v2t(inc)) used by the next reduction
  int converged;      // current level stopped (|delta| <= minIncrement)
  int have_target;    // 0 until a target exists (first frame: no tracking)
  unsigned int ticket;  // last-block-done counter
  int iters[3];
  int inliers[3];
  float rms[3];
};

// Pose of the session, device resident.
struct PoseState {
  double pose[16];    // camera-to-world (row-major, double)
  float posef[16];    // float copy used by the kernels
  float invf[16];     // float4x4::getInverse of posef (utils_matrix.h:970-1086)
  double last_inc[6];
  int reset;          // NaN / maxIncrement guard fired this frame
  int frame;
};

struct IcpLevel {
  const float* sd;     // source depth
  const float4* sn;    // source normals
  const float* si;     // source intensity (may be null if cw == 0)
  const float* td;     // target depth
  const float4* tn;    // target normals
  const float* ti;     // target intensity (may be null if cw == 0)
  DSensor s;
};

struct IcpParams {
  float dmin, dmax;    // icp depth window
  float cos_thr;
  float cw;            // color weight
  float min_inc, max_inc, reg;
  int compose_left;
  int kahan;           // compensated FP32 per-thread sums (mixed precision)
};

constexpr int kIcpVals = 29;
// The stage entry points' reduction (icp_reduce_kernel).
constexpr int kIcpThreads = 256;
constexpr int kIcpMaxBlocks = 148 * 8;
// The per-frame ICP: one 512-thread block per SM, and its normal equations
// summed per tile of a level; a tile's partial sums are the same whichever
// block computes them, and the level's total adds the tiles in a fixed order.
// So the result does not depend on how many blocks work on a level, nor on the
// sessions that share the launch.  A tile is a run of icp_tile_slots(n, kahan)
// slots: 256 (half of a block's warps, so that a level of 19,200 pixels still
// spreads over 75 SMs) or a whole number per thread, the least that gives at
// most 160 tiles -- about one per SM; every block reads every tile's row.  A
// slot of the plain form is a pixel; of the compensated form a group of
// icp_group(n) pixels 256 apart (of runs of 256 times as many pixels), which
// one thread sums in plain FP32.
constexpr int kIcpFrameThreads = 512;
constexpr int kIcpMaxTiles = 160;
inline __host__ __device__ int icp_group(int npx) { return npx <= 8192 ? 1 : (npx <= 65536 ? 2 : 4); }
inline __host__ __device__ int icp_slots(int npx, int kahan) {
  if (!kahan) return npx;
  const int run = icp_group(npx) * 256;
  return (npx + run - 1) / run * 256;
}
inline __host__ __device__ int icp_tile_slots(int npx, int kahan) {
  const int n = icp_slots(npx, kahan);
  if (n <= 148 * 256) return 256;
  return (n + kIcpMaxTiles * kIcpFrameThreads - 1) / (kIcpMaxTiles * kIcpFrameThreads) *
         kIcpFrameThreads;
}
inline __host__ __device__ int icp_tiles(int npx, int kahan) {
  const int t = icp_tile_slots(npx, kahan);
  return (icp_slots(npx, kahan) + t - 1) / t;
}

// Weight of a session in the shares of a table's blocks: its level-0 pixels and
// two pixels' worth per slot for the warps' sums.
inline __host__ __device__ long long icp_weight(int npx, int kahan) {
  return npx + (kahan ? 2ll * icp_slots(npx, kahan) : 0ll);
}

// Scratch of a stage reduction: per-block partial sums (kIcpMaxBlocks*29 doubles).
size_t icp_scratch_bytes();
// Scratch of a session's per-frame ICP: the chained kernels' row of partial
// sums per tile, then the persistent kernel's rows (kIcpRowWords tagged words
// each): per level slot two per tile, by the iteration's parity, and the level's
// state.  A level has rows of its own: a block that leaves after its last level
// still reads that level's last rows, and says nothing to the others, who may be
// two iterations into the next level by then (as with two rows per tile for all
// levels; 161 KB per session, now 481).
constexpr int kIcpRowWords = 64;
inline __host__ __device__ size_t icp_rows_offset() {  // bytes
  return ((size_t)kIcpMaxTiles * kIcpVals * sizeof(double) + 255) / 256 * 256;
}
// The row of tile 'tile' in iteration 'it' of level slot pl.
inline __host__ __device__ int icp_row(int pl, int it, int tile) {
  return (2 * pl + (it & 1)) * kIcpMaxTiles + tile;
}
// The row that level slot pl's state is left in.
inline __host__ __device__ int icp_state_row(int pl) { return 6 * kIcpMaxTiles + pl; }
constexpr int kIcpRows = 6 * kIcpMaxTiles + 3;
inline size_t icp_frame_scratch_bytes() {
  return icp_rows_offset() + (size_t)kIcpRows * kIcpRowWords * 8;
}

// The persistent ICP (one cooperative launch per frame and summation kind, or
// one per part of a large table): the blocks that can be resident at once on
// 'device' (0: cooperative launches unavailable).
int icp_persistent_capacity(int device);
// Blocks of a session of npx pixels in a persistent launch over sessions that
// weigh 'sum' in all: its part of 'pool' blocks beside 'base', at least one.
__host__ __device__ inline int icp_share(int npx, int kahan, long long sum, int pool, int base) {
  const int tiles = icp_tiles(npx, kahan);
  long long b = base + (long long)pool * icp_weight(npx, kahan) / (sum > 0 ? sum : 1);
  if (b > tiles) b = tiles;
  if (b < 1) b = 1;
  return (int)b;
}

// The launches of a table of n sessions within 'budget' blocks: the table in
// 'parts' runs one after another (0: the chained kernels run it, with the same
// results), each with a launch per summation kind of grid[part][kind] blocks (0:
// no session of that kind).  Every session needs a block: a table of more
// sessions than blocks takes the fewest parts that give them one.  (160 sessions
// of 64x48 in two parts: 266 us of ICP, in the chained kernels 459; 580 in four:
// 550 and 1349; 200 of 320x240 in two: 2281 and 4671.)  Blocks follow the
// sessions' weights; where that leaves small sessions less than one each, all get
// one first and the weights share out the rest.
constexpr int kIcpMaxParts = 4;
struct IcpLaunches {
  int parts;
  int grid[kIcpMaxParts][2], pool[kIcpMaxParts][2], base[kIcpMaxParts][2];
};
inline __host__ __device__ int icp_part_first(int n, int parts, int part) {
  return (int)((long long)n * part / parts);
}
inline IcpLaunches icp_launches(const int* npx, const int* kahan, int n, int budget) {
  IcpLaunches L = {};
  if (budget <= 0 || n <= 0 || n > (long long)kIcpMaxParts * budget) return L;
  L.parts = (n + budget - 1) / budget;
  for (int part = 0; part < L.parts; ++part) {
    const int first = icp_part_first(n, L.parts, part), end = icp_part_first(n, L.parts, part + 1);
    for (int kind = 0; kind < 2; ++kind) {
      long long sum = 0;
      int members = 0;
      for (int j = first; j < end; ++j)
        if ((kahan[j] != 0) == (kind == 1)) {
          sum += icp_weight(npx[j], kind);
          ++members;
        }
      for (int base = 0; base < 2; ++base) {
        const int pool = budget - base * members;
        long long g = 0;
        for (int j = first; j < end; ++j)
          if ((kahan[j] != 0) == (kind == 1)) g += icp_share(npx[j], kind, sum, pool, base);
        L.grid[part][kind] = (int)g;
        L.pool[part][kind] = pool;
        L.base[part][kind] = base;
        if (g <= budget) break;
      }
    }
  }
  return L;
}
// Resident blocks that each of k groups of sessions may take for its persistent
// ICP, out[g], when the groups run at once: 'weight' a group's icp_weight in all,
// 'count' its sessions.  The shares never add up to more than 'cap', so that all
// launches can be resident together (their blocks wait for one another: a launch
// that is resident in part beside another such would wait out its bound); a
// group without a block runs the chained kernels.  Shares follow the weights,
// except that a group whose share would be less than a block per session is given
// just that while there are blocks for every session.
inline void icp_group_budgets(const long long* weight, const int* count, int k, int cap,
                              int* out) {
  long long sessions = 0;
  for (int g = 0; g < k; ++g) {
    sessions += count[g];
    out[g] = 0;
  }
  if (cap <= 0) return;
  const bool all_fit = sessions <= cap;
  long long left = cap, rest = 0;  // blocks and weight of the groups not yet settled
  for (int g = 0; g < k; ++g) rest += weight[g];
  for (bool again = all_fit; again;) {
    again = false;
    for (int g = 0; g < k; ++g)
      if (out[g] == 0 && count[g] > 0 && left * weight[g] < rest * count[g]) {
        out[g] = count[g];
        left -= count[g];
        rest -= weight[g];
        again = true;
      }
  }
  for (int g = 0; g < k; ++g)
    if (out[g] == 0 && rest > 0) out[g] = (int)(left * weight[g] / rest);
}

// The persistent ICP's words of a session: the epoch of the next launch's tags
// (advance_epoch) and, on a line of its own, the abort word (zero before a launch).
constexpr int kIcpAbort = 32;
constexpr int kIcpBarWords = 64;
constexpr unsigned kIcpEpochStep = 4096;
// Called by one thread after a launch: the next launch's epoch.  Tags are 32
// bits, so an epoch comes again after 2^20 launches; a row that none of them
// wrote would then pass for this launch's, so the rows are emptied where the
// epochs start again (481 KB by one thread, once in 9.7 hours at 30 Hz).  0 is no
// epoch: an empty row carries no tag of any launch.
inline __host__ __device__ void advance_epoch(unsigned* bar, void* scratch) {
  unsigned e = bar[0] + kIcpEpochStep;
  if (e < kIcpEpochStep) {
    uint4* const rows = reinterpret_cast<uint4*>(static_cast<char*>(scratch) + icp_rows_offset());
    const int n = kIcpRows * kIcpRowWords / 2;
    for (int i = 0; i < n; ++i) rows[i] = make_uint4(0u, 0u, 0u, 0u);
    e = kIcpEpochStep;
  }
  bar[0] = e;
}
// The bounded wait of the persistent ICP's blocks, as a barrier run alone:
// 'blocks' blocks wait for blocks + missing arrivals (bar_dev: kIcpBarWords
// words).  DYN_OK when it completes, DYN_ERR_TIMEOUT when the wait ran out,
// DYN_ERR_INVALID_ARG when the blocks cannot all be resident.
dyn_status icp_barrier_selftest(int blocks, int missing, unsigned* bar_dev, cudaStream_t st);
// After the last level: guards, pose composition, float pose + inverse, reset
// of the solver state.  Runs with one thread.
void launch_pose_finalize(const IcpParams& P, IcpState* st, PoseState* ps,
                          cudaStream_t stream);
// Tracking of the next frame starts from the motion from the current pose
// to 'hint' (double[16], camera-to-world): the solver's increment becomes
// its SE(3) logarithm (before the first target, the hint becomes the pose).
void launch_pose_hint(PoseState* ps, IcpState* st, const double* hint_dev, int compose_left,
                      cudaStream_t stream);
// Set the pose from the host (double[16]); recomputes posef/invf.
void launch_pose_set(PoseState* ps, const double* pose_dev, cudaStream_t stream);
// Normal equations only (no solve): out[29] doubles on the device or in pinned
// host memory.
void launch_icp_reduce_only(const IcpLevel& L, const IcpParams& P, const M4f& T,
                            double* partials, unsigned int* ticket, double* out,
                            cudaStream_t stream);
// The same reduction on an explicit grid, T on the device ('partials' holds grid * 29
// doubles; pixels beyond grid * kIcpThreads are covered by the grid-stride
// loop).
void launch_icp_reduce_grid(const IcpLevel& L, const IcpParams& P, const float* T_dev,
                            double* partials, unsigned int* ticket, double* out_dev, int grid,
                            cudaStream_t stream);

}  // namespace dyn
