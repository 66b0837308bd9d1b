// ray_grid.cuh -- the raycast's block grid (its box, clearing and entries) and
// the ranges within which a march may use it.  On their own, because every
// index of the grid march is unchecked: what lets a ray take it is decided
// here (and by tests on the CPU).
#pragma once
#include "common.cuh"
#include "tsdf.cuh"

namespace dyn {

namespace {

// ------------------------------------------------------------ the block grid
// The raycast looks blocks up by their coordinates far more often than
// anything else (every sample, up to eight blocks), so each frame's blocks are
// also laid out in a dense grid over the box the frame's rays can reach
// (GridBox; z fastest): entry = first voxel of the block (512 x heap index),
// or of the empty block after the heap.  A lookup is one multiply-add chain
// and one load without branches, where the hash takes a bucket scan in a
// divergent branch for every lane that changes block.  A 640x480 FP32 target with
// colours: 327 M warp instructions at 25 of 32 lanes and 485 us before, and no
// faster with the exact march alone; with the grid 181 M at 28 lanes and 264 us
// (320x240 225 -> 99).  The mixed march, whose arithmetic did not change: 640x480
// 136 -> 62 us, 1280x720 band 200 -> 100 us, and a 32-session band batch 667 ->
// 358 us.
__device__ inline GridBox grid_box(const float* __restrict__ T, const DSensor& s, const DTsdf& t,
                                   int cap) {
  GridBox b;
  float lo[3], hi[3];
  // (each corner takes in every entry of its row: a NaN or an infinity shows in
  // its value, while the minimum and maximum would skip a NaN)
  bool fin = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) lo[a] = hi[a] = T[4 * a + 3];
  const float u0 = (0.0f - s.cx) / s.fx, u1 = ((float)(s.cols - 1) - s.cx) / s.fx;
  const float v0 = (0.0f - s.cy) / s.fy, v1 = ((float)(s.rows - 1) - s.cy) / s.fy;
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float e = (T[4 * a] * ((k & 1) ? u1 : u0) + T[4 * a + 1] * ((k & 2) ? v1 : v0) +
                       T[4 * a + 2]) * t.dmax + T[4 * a + 3];
      fin = fin && fabsf(e) <= 3.4e38f;
      lo[a] = fminf(lo[a], e);
      hi[a] = fmaxf(hi[a], e);
    }
  int n[3], o[3];
  bool ok = cap > 0 && fin;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    // a block of margin below, two above (a cell's high corners); 2^20 blocks
    // is the key's range
    const float l = floorf(lo[a] / t.bsm) - 1.0f, h = floorf(hi[a] / t.bsm) + 2.0f;
    ok = ok && l > -1048576.0f && h < 1048576.0f;
    o[a] = ok ? (int)l : 0;
    n[a] = ok ? (int)h - (int)l + 1 : 0;
  }
  ok = ok && (double)n[0] * (double)n[1] * (double)n[2] <= (double)cap;
  b.x0 = o[0];
  b.y0 = o[1];
  b.z0 = o[2];
  b.nx = n[0];
  b.ny = n[1];
  b.nz = n[2];
  b.ok = ok ? 1 : 0;
  return b;
}
// The grid emptied at pose T by 'threads' threads, this one number 'thread'.
__device__ inline void grid_clear(const VolumeDev& v, const float* __restrict__ T,
                                  const DSensor& s, int thread, int threads) {
  const GridBox b = grid_box(T, s, v.t, v.grid_cap);
  if (thread == 0) *v.gbox = b;
  if (!b.ok) return;
  const int n4 = (b.nx * b.ny * b.nz + 3) / 4;  // (the buffer holds whole vectors)
  const unsigned e = (unsigned)v.t.num_blocks * (unsigned)kBlockVox;
  for (int i = thread; i < n4; i += threads)
    reinterpret_cast<uint4*>(v.grid)[i] = make_uint4(e, e, e, e);
}
__device__ inline void grid_put(const VolumeDev& v, const GridBox& b, unsigned long long key,
                                int ptr, unsigned flag) {
  const int x = key_x(key) - b.x0, y = key_y(key) - b.y0, z = key_z(key) - b.z0;
  if ((unsigned)x < (unsigned)b.nx && (unsigned)y < (unsigned)b.ny && (unsigned)z < (unsigned)b.nz)
    v.grid[(x * b.ny + y) * b.nz + z] = ((unsigned)ptr * (unsigned)kBlockVox) | flag;
}

// ------------------------------------------------------------ a ray's range
struct MarchRay {
  float yhx, ylx, yhy, yly;  // reciprocals of fx and fy
};

__device__ inline bool recip_ok(float x) { return moderate(fabsf(x)); }

// Whether the samples of pixel offset (px, py) (per unit depth) from pose T, up
// to dmax, stay within 131072 voxels of the origin on every axis: the range of
// the rounded indices, and with it of the grid's.  False for a pose that is not
// finite (each axis is compared by itself: a NaN fails its own comparison).
__device__ inline bool march_within(const DTsdf& t, const M4f& T, float px, float py,
                                    float inv_vs) {
  bool in = true;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float e = (fabsf(T.m[4 * i]) * fabsf(px) + fabsf(T.m[4 * i + 1]) * fabsf(py) +
                     fabsf(T.m[4 * i + 2])) * t.dmax + fabsf(T.m[4 * i + 3]);
    in = in && e * inv_vs * 1.001f + 2.0f < 131072.0f;
  }
  return in;
}

// Every step of a march is at least min(voxel, truncation): below 4096 of them
// up to dmax the roundings of cur add up to less than a step, so the march
// ends within the step cap (rc_cap, four steps more) and needs no count.
__device__ inline bool march_bounded(const DTsdf& t) {
  return t.dmax <= 4096.0f * fminf(t.vs, t.trunc);
}

// Whether the fast indices and divisions hold along the whole ray of pixel
// offset (ax, ay) from pose T, with their constants.
__device__ inline bool march_setup(const DTsdf& t, const DSensor& s, const M4f& T, float ax,
                                   float ay, float inv_vs, MarchRay& m) {
  const bool ok = recip_ok(s.fx) && recip_ok(s.fy) && (ax == 0.0f || recip_ok(ax)) &&
                  (ay == 0.0f || recip_ok(ay)) && recip_ok(t.vs) && recip_ok(t.trunc) &&
                  recip_ok(t.dmax) && march_bounded(t);
  m.yhx = 1.0f / s.fx;
  m.yhy = 1.0f / s.fy;
  m.ylx = __fmaf_rn(-s.fx, m.yhx, 1.0f) * m.yhx;
  m.yly = __fmaf_rn(-s.fy, m.yhy, 1.0f) * m.yhy;
  return ok && march_within(t, T, ax * m.yhx, ay * m.yhy, inv_vs);
}

}  // namespace

}  // namespace dyn
