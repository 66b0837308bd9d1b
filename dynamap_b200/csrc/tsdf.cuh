// tsdf.cuh -- voxel-hashed TSDF: allocation, visibility, integration, raycast.
// The per-frame stages run as fused launches over a table of sessions
// (sessdev.cuh); the raycast also has a one-session form for
// tsdfVolume::GenerateDepth / GenerateRgb.
#pragma once
#include "common.cuh"
#include "icp.cuh"

namespace dyn {

// The box of the raycast's block grid: block coordinates (x0, y0, z0) and
// extents, z fastest; ok 0 where the pose is not finite or the box exceeds
// the grid's capacity (the raycast then looks blocks up in the hash).
struct GridBox {
  int x0, y0, z0;
  int nx, ny, nz;
  int ok;
};

struct VolumeDev {
  Entry* entries;                 // num_buckets * bucket_size
  unsigned long long* block_keys; // key of each heap index
  dyn_voxel* voxels;              // FP32 form: num_blocks * 512, x-major per block
  unsigned* vox16;                // mixed form: {f16 sdf | u16 weight << 16} per voxel
  uchar4* colors;                 // mixed form: r,g,b per voxel (null: no colour kept)
  int fp16;                       // 1: mixed-precision voxels (vox16 [+ colors])
  Counters* cnt;
  DTsdf t;
  // Free-space summaries per heap index, kept for the mixed form (null in
  // the FP32 form, whose raycast evaluates every sample, and with band
  // allocation, which allocates no free space to step through): nonsat = voxels
  // that are observed and not saturated, kept exact by the integration;
  // freecell = 1 when every voxel a trilinear cell keyed in the block can
  // read (the block and its seven upper neighbours, missing neighbours
  // included) is unobserved or saturated, so the raycast's interpolated sdf
  // there is the truncation distance.  freecell may be 0 where it could be
  // 1, never the reverse.  A mixed voxel is saturated when its f16 value is
  // exactly 1 (free space); an FP32 voxel (the upload's count, for a volume
  // that keeps summaries) when sdf >= sat_lo, the truncation distance to
  // within 1e-6 relative.  free_ok: sat_lo >= vs, so a saturated sample
  // never ends a march (flags are set only then).
  int* nonsat;
  unsigned char* freecell;
  float sat_lo;
  int free_ok;
  // The raycast's block grid, rebuilt for every raycast (null: the session's
  // rays reach a box too large for one): per block of the box its first
  // voxel, 512 x heap index, with the free-cell flag in bit 0, or that of the
  // empty block num_blocks, whose voxels are zero.
  unsigned* grid;
  GridBox* gbox;
  int grid_cap;  // entries
};

// Entries of a grid that covers whatever box the rays of sensor s reach up to
// dmax (any rotation), 0 where that exceeds kGridMax.  The widest box's side
// is the largest distance between two points of the viewing pyramid.  The line
// at 2^24 entries (64 MB, rewritten every frame, half of L2) keeps the grid in
// cache beside the voxels: 4 mm voxels at 3 m of range need 3.1 M entries,
// 4 mm at 8 m 67 M.
constexpr long long kGridMax = 1ll << 24;
inline long long grid_entries(const DSensor& s, const DTsdf& t) {
  const double u0 = (0.0 - s.cx) / s.fx, u1 = (s.cols - 1.0 - s.cx) / s.fx;
  const double v0 = (0.0 - s.cy) / s.fy, v1 = (s.rows - 1.0 - s.cy) / s.fy;
  double d2 = (u1 - u0) * (u1 - u0) + (v1 - v0) * (v1 - v0);
  for (int k = 0; k < 4; ++k) {
    const double u = (k & 1) ? u1 : u0, v = (k & 2) ? v1 : v0;
    const double e = u * u + v * v + 1.0;
    d2 = d2 > e ? d2 : e;
  }
  const double side = __builtin_sqrt(d2) * t.dmax / t.bsm + 6.0;
  if (!(side < 256.0) || t.num_blocks >= (1 << 23) - 1) return 0;
  const long long n = (long long)(side * side * side);
  return n <= kGridMax ? n : 0;
}

// Allocation's form of a session (walk_rays).  The tile-local keys' 10 bits an axis
// hold a ray of the step cap from the camera; a band ray's start as well, up to
// twice the sensor range away.
inline __host__ __device__ bool narrow_keys(const DTsdf& t) {
  return t.dda_cap <= (t.band ? 300 : 509);
}
// Whether neighbouring rays run through the same blocks: a block spans at least
// four of them at the sensor range.  Allocation in us with CLOSE / without:
// 640x480, 5 mm, 3 m and 5 m of range (7 and 4.2 rays) 63 / 108 and 78 / 141;
// 1280x720, 4 mm, 5 m (6.7) 424 / 688; 320x240, 5 mm, 3 m (3.5) 72 / 66, 4 m (2.6)
// 123 / 89; 160x120, 5 mm, 3 m (1.8) 274 / 151; 640x480, 4 mm, 8 m (2.1) 1505 / 819.
// Rays of more steps than the narrow keys hold fill the set either way: 1280x720,
// 2 mm, 3 m (5.6) 491 / 406, 3 mm, 6 m (4.2) 1376 / 1081, 4 mm, 8 m (4.2) 813 / 824.
// A band ray's few blocks do not: 160x120, 5 mm, 3 m 14 / 20, and the sessions of
// a batch stay in one launch.
inline __host__ __device__ bool close_rays(const DTsdf& t, const DSensor& s) {
  return narrow_keys(t) && (t.band || t.bsm * (s.fx < s.fy ? s.fx : s.fy) >= 4.0f * t.dmax);
}

void launch_volume_clear(const VolumeDev& v, cudaStream_t st);
// GenerateDepthKernel / GenerateRgbKernel (tsdf.cu:471-526).  pose_override
// (device float[16]) replaces the session pose when non-null.  use_grid:
// through the volume's block grid, rebuilt here.
void launch_raycast(const VolumeDev& v, const DSensor& s, const PoseState* ps,
                    const float* pose_override, float* depth_out, uint8_t* rgb_out,
                    bool use_grid, cudaStream_t st);
// Download helpers: block coordinates of heap indices [0, n).
void launch_block_coords(const VolumeDev& v, int n, int* coords, cudaStream_t st);
// Heap index (or -1) of each of n block coordinates (x, y, z triples).
void launch_find_blocks(const VolumeDev& v, const int* coords, int n, int* ptr_out,
                        cudaStream_t st);

}  // namespace dyn
