// tsdf.cu -- voxel-hashed TSDF kernels.
//
// Reference: include/geometry/tsdf/tsdf.cu (integration :268-344, allocation
// :346-453, raycast :471-526, voxel addressing :47-239),
// include/dataStructure/hashTable/hashTable.cu (:80-163),
// include/geometry/geom_Types.h (Voxel merge :79-103).
//
// Layout in HBM (per session): a bucketed hash of 16-byte entries
// {u64 packed block key, i32 heap index, i32 frame stamp}; a heap-index ->
// key array; voxels as 8-byte {r,g,b,w,f32 sdf} (the reference's Voxel),
// 512 per block in x-major order, so one block is 4 KB contiguous.  The
// mixed form keeps {f16 sdf / truncation, u16 weight} per voxel (2 KB per
// block) and an optional uchar4 colour array.
//
// Each stage is a __device__ body used by a by-value kernel (one session)
// and by a fused kernel over every session of a frame (blockIdx.z).
#include "tsdf.cuh"

#include <cuda_fp16.h>

#include <algorithm>

#include "near_key.cuh"
#include "ray_grid.cuh"
#include "sessdev.cuh"

namespace dyn {

namespace {

// ------------------------------------------------------------ exact shortcuts
// Rounding by adding and subtracting 1.5 * 2^23: two additions and no
// conversion (the conversions run at an eighth of the FP32 rate); the sum's
// low bits are the integer.
constexpr float kRint = 12582912.0f;   // 1.5 * 2^23
constexpr int kRintBits = 0x4B400000;  // its bits: a multiple of 8

// ------------------------------------------------------------ allocation
constexpr int kAllocX = 16, kAllocY = 16, kAllocN = kAllocX * kAllocY;  // pixel tile per CTA
constexpr int kSetProbes = 32;

struct alignas(16) AllocSmem {
  unsigned long long set[kSetSlots];  // keys; all bits set: none; later the claimed entries
  unsigned short list[kSetSlots];     // the keys' slots in order of arrival
  unsigned short claim[kSetSlots];    // the claimed ones'
  M4f T;       // the frame's pose
  int cam[3];  // the camera's block
  int stamp;
  int nkeys, nclaims;
  int base;
  int new_blocks, bucket_full, heap_exhausted, unique, overruns;
};

// bucket_insert (the lock-free unique insert) is in common.cuh.

// AllocateFromDepthKernel (tsdf.cu:346-453) for one pixel: the reference's
// DDA over blocks, exact FP32 (this file is built with -fmad=false), with
// the 'diff' pre-step for negative directions and the step cap.
struct RayWalk {
  int bx, by, bz;  // first block
  int nx, ny, nz;  // pre-step (0 or -1)
  int ex, ey, ez;  // last block
  int sx, sy, sz;
  float mx, my, mz, dtx, dty, dtz;
};
__device__ inline RayWalk ray_walk(F3 start_pt, F3 point, float trunc, float block_size) {
  RayWalk w;
  F3 dir = normalize3(point - start_pt);
  float surface_distance = norm3(start_pt - point);
  F3 ray_start = start_pt;
  F3 ray_end = start_pt + dir * (surface_distance + trunc);
  w.bx = (int)floorf(ray_start.x / block_size);
  w.by = (int)floorf(ray_start.y / block_size);
  w.bz = (int)floorf(ray_start.z / block_size);
  w.ex = (int)floorf(ray_end.x / block_size);
  w.ey = (int)floorf(ray_end.y / block_size);
  w.ez = (int)floorf(ray_end.z / block_size);
  w.sx = (dir.x > 0) - (dir.x < 0);
  w.sy = (dir.y > 0) - (dir.y < 0);
  w.sz = (dir.z > 0) - (dir.z < 0);
  const float FMAX = 3.402823466e+38f;
  w.dtx = dir.x != 0 ? fabsf(block_size / dir.x) : FMAX;
  w.dty = dir.y != 0 ? fabsf(block_size / dir.y) : FMAX;
  w.dtz = dir.z != 0 ? fabsf(block_size / dir.z) : FMAX;
  float bdx = ((float)w.bx + (float)w.sx) * block_size;
  float bdy = ((float)w.by + (float)w.sy) * block_size;
  float bdz = ((float)w.bz + (float)w.sz) * block_size;
  w.mx = dir.x != 0 ? (bdx - ray_start.x) / dir.x : FMAX;
  w.my = dir.y != 0 ? (bdy - ray_start.y) / dir.y : FMAX;
  w.mz = dir.z != 0 ? (bdz - ray_start.z) / dir.z : FMAX;
  w.nx = w.bx != w.ex && dir.x < 0 ? -1 : 0;
  w.ny = w.by != w.ey && dir.y < 0 ? -1 : 0;
  w.nz = w.bz != w.ez && dir.z < 0 ? -1 : 0;
  return w;
}

// The ray of a pixel; false: none (tsdf.cu:442-444)
__device__ inline bool pixel_ray(const float* __restrict__ depth, const DSensor& s, const DTsdf& t,
                                 const M4f& T, int x, int y, RayWalk& w) {
  if (x >= s.cols || y >= s.rows) return false;
  const float d = depth[y * s.cols + x];
  if (d < t.dmin || d > t.dmax) return false;
  const F3 point = xform(T, point3d_uv(x, y, d, s));
  if (point.x == 0 && point.y == 0 && point.z == 0) return false;
  F3 start_pt = f3(T.m[3], T.m[7], T.m[11]);
  // band allocation: the ray starts a truncation distance before the
  // surface point instead of at the camera
  if (t.band) start_pt = point - normalize3(point - start_pt) * t.trunc;
  w = ray_walk(start_pt, point, t.trunc, t.bsm);
  return true;
}

// One block into the global table, its heap index from the volume's counter.
__device__ __forceinline__ void insert_block_inline(const VolumeDev& v, unsigned long long key,
                                                    AllocSmem& sm) {
  const int r = bucket_insert(v.entries, v.t, key, sm.stamp, &sm.unique);
  if (r >= 0) {
    const int ptr = atomicAdd(&v.cnt->nalloc, 1);
    if (ptr < v.t.num_blocks) {
      v.entries[r].ptr = ptr;
      v.block_keys[ptr] = key;
      atomicAdd(&sm.new_blocks, 1);
    } else {
      atomicAdd(&sm.heap_exhausted, 1);
    }
  } else if (r == -2) {
    atomicAdd(&sm.bucket_full, 1);
  }
}

__device__ __noinline__ void insert_block(const VolumeDev& v, unsigned long long key,
                                          AllocSmem& sm) {
  insert_block_inline(v, key, sm);
}

// A pixel's whole ray without the set (anywhere; blocks that other rays enter
// as well are found or claimed once).
__device__ __noinline__ void walk_far(const SessDev& S, int x, int y, AllocSmem& sm) {
  const VolumeDev& v = S.vol;
  RayWalk w;
  if (!pixel_ray(S.raw, S.ls[0], v.t, sm.T, x, y, w)) return;
  int bx = w.bx, by = w.by, bz = w.bz;
  insert_block(v, pack_key(bx, by, bz), sm);
  if (w.nx | w.ny | w.nz) {
    bx += w.nx;
    by += w.ny;
    bz += w.nz;
    insert_block(v, pack_key(bx, by, bz), sm);
  }
  int left = v.t.dda_cap;
  while (bx != w.ex || by != w.ey || bz != w.ez) {
    if (left-- <= 0) {
      atomicAdd(&sm.overruns, 1);
      return;
    }
    const bool xy = w.mx < w.my, xz = w.mx < w.mz, yz = w.my < w.mz;
    const bool gx = xy && xz, gy = !xy && yz;
    if (gx) { bx += w.sx; w.mx += w.dtx; }
    else if (gy) { by += w.sy; w.my += w.dty; }
    else { bz += w.sz; w.mz += w.dtz; }
    insert_block(v, pack_key(bx, by, bz), sm);
  }
}

// One block of a ray into the CTA's set.  Most visits find their key with a plain
// read.  CLOSE (close_rays): of a run of lanes that miss the same key together the first
// enters it (their compare-and-swaps would queue at the slot: half of the shared
// memory cycles there), and the entered slots are listed.  Else nearly every lane
// misses another key, the set fills up, and holding the lanes together for each
// other is what costs; the set is then scanned as a whole.
template <class K, bool CLOSE>
__device__ inline void visit_block(K key, const VolumeDev& v, AllocSmem& sm) {
  K* const set = reinterpret_cast<K*>(sm.set);
  constexpr K none = ~(K)0;
  unsigned slot = NearKey<K>::slot(key);
  for (int p = 0; p < kSetProbes; ++p) {
    K old = *(volatile K*)&set[slot];
    if (old == none) {
      if (CLOSE) {
        const unsigned here = __activemask(), lane = threadIdx.x & 31;
        const K left = __shfl_up_sync(here, key, 1);
        const bool follows = lane > 0 && (here >> (lane - 1) & 1u) && left == key;
        if (!follows) {
          old = atomicCAS(&set[slot], none, key);
          if (old == none) {
            sm.list[atomicAdd(&sm.nkeys, 1)] = (unsigned short)slot;
            old = key;
          }
        }
        __syncwarp(here);
        if (follows) old = *(volatile K*)&set[slot];
      } else {
        old = atomicCAS(&set[slot], none, key);
        if (old == none) old = key;
      }
    }
    if (old == key) return;
    slot = (slot + 1) & (kSetSlots - 1);
  }
  // set saturated
  if (CLOSE)
    insert_block(v, volume_key(key, sm.cam), sm);
  else
    insert_block_inline(v, volume_key(key, sm.cam), sm);
}

// The rays of one pixel tile (tx, ty) of AllocateFromDepthKernel.
template <class K, bool CLOSE>
__device__ inline void walk_rays(const SessDev& S, int tx, int ty, AllocSmem& sm) {
  constexpr int B = NearKey<K>::kBits;
  const VolumeDev& v = S.vol;
  const int tid = threadIdx.x;
  // (a warp's rays are 8x4 pixels)
  const int x = tx * kAllocX + (tid & 7) + (tid >> 2 & (kAllocX - 8)),
            y = ty * kAllocY + (tid >> 3 & 3) + tid / (kAllocX * 4) * 4;
  RayWalk w;
  if (!pixel_ray(S.raw, S.ls[0], v.t, sm.T, x, y, w)) return;
  const int ox = apart_of(w.bx, sm.cam[0]), oy = apart_of(w.by, sm.cam[1]),
            oz = apart_of(w.bz, sm.cam[2]);
  // (a last block beyond the fields is beyond the cap as well)
  const int lx = apart_of(w.ex, sm.cam[0]), ly = apart_of(w.ey, sm.cam[1]),
            lz = apart_of(w.ez, sm.cam[2]);
  constexpr unsigned half = 1u << (B - 1);
  const bool ends = (unsigned)lx + half < 2 * half && (unsigned)ly + half < 2 * half &&
                    (unsigned)lz + half < 2 * half;
  const K last = ends ? near_key<K>(lx, ly, lz) : ~(K)0;
  int left = v.t.dda_cap;
  // (none that could leave the fields is walked with them: band rays of poses
  // that are not rigid start anywhere)
  if (!near_walk<K>(ox, oy, oz, left)) {
    walk_far(S, x, y, sm);
    return;
  }
  const K ix = (K)(long long)w.sx << (2 * B), iy = (K)(long long)w.sy << B, iz = (K)(long long)w.sz;
  K key = near_key<K>(ox, oy, oz);
  visit_block<K, CLOSE>(key, v, sm);
  if (w.nx | w.ny | w.nz) {
    key = near_key<K>(ox + w.nx, oy + w.ny, oz + w.nz);
    visit_block<K, CLOSE>(key, v, sm);
  }
  while (key != last) {
    if (left-- <= 0) {
      atomicAdd(&sm.overruns, 1);
      break;
    }
    const bool xy = w.mx < w.my, xz = w.mx < w.mz, yz = w.my < w.mz;
    const bool gx = xy && xz, gy = !xy && yz;
    key += gx ? ix : (gy ? iy : iz);
    if (gx) w.mx += w.dtx;
    else if (gy) w.my += w.dty;
    else w.mz += w.dtz;
    visit_block<K, CLOSE>(key, v, sm);
  }
}

template <class K, bool CLOSE>
__device__ inline void allocate_tile(const SessDev& S, int tx, int ty, AllocSmem& sm) {
  K* const set = reinterpret_cast<K*>(sm.set);
  const VolumeDev& v = S.vol;
  const DTsdf& t = v.t;
  const int tid = threadIdx.x;
  for (int k = tid; k < kSetSlots * (int)sizeof(K) / 16; k += kAllocN)
    reinterpret_cast<uint4*>(sm.set)[k] = make_uint4(~0u, ~0u, ~0u, ~0u);
  if (tid < 16) {
    const float m = S.pose->posef[tid];
    sm.T.m[tid] = m;
    if ((tid & 3) == 3 && tid < 12) sm.cam[tid >> 2] = (int)floorf(m / t.bsm);
  }
  if (tid == 0) {
    sm.nkeys = sm.nclaims = 0;
    sm.new_blocks = sm.bucket_full = sm.heap_exhausted = sm.unique = sm.overruns = 0;
    sm.stamp = S.pose->frame;
  }
  __syncthreads();
  walk_rays<K, CLOSE>(S, tx, ty, sm);
  __syncthreads();
  // drain the set into the global table
  const int listed = CLOSE ? sm.nkeys : kSetSlots;
  for (int k = tid; k < listed; k += kAllocN) {
    const int slot = CLOSE ? sm.list[k] : k;
    if (!CLOSE && set[slot] == ~(K)0) continue;
    const int r = bucket_insert(v.entries, t, volume_key(set[slot], sm.cam), sm.stamp, &sm.unique);
    if (r >= 0) {
      set[slot] = (K)(unsigned)r;
      sm.claim[atomicAdd(&sm.nclaims, 1)] = (unsigned short)slot;
    } else if (r == -2) {
      atomicAdd(&sm.bucket_full, 1);
    }
  }
  __syncthreads();
  if (tid == 0 && sm.nclaims > 0) sm.base = atomicAdd(&v.cnt->nalloc, sm.nclaims);
  __syncthreads();
  for (int c = tid; c < sm.nclaims; c += kAllocN) {
    int ptr = sm.base + c;
    const int e = (int)set[sm.claim[c]];
    if (ptr < t.num_blocks) {
      v.entries[e].ptr = ptr;
      v.block_keys[ptr] = v.entries[e].key;
      atomicAdd(&sm.new_blocks, 1);
    } else {
      atomicAdd(&sm.heap_exhausted, 1);
    }
  }
  __syncthreads();
  if (tid == 0) {
    if (sm.new_blocks) atomicAdd(&v.cnt->new_blocks, sm.new_blocks);
    if (sm.bucket_full) atomicAdd(&v.cnt->bucket_full, sm.bucket_full);
    if (sm.heap_exhausted) atomicAdd(&v.cnt->heap_exhausted, sm.heap_exhausted);
    if (sm.unique) atomicAdd(&v.cnt->unique_probed, sm.unique);
    if (sm.overruns) atomicAdd(&v.cnt->dda_overruns, sm.overruns);
  }
}

// One kernel per form (sessions of the other form return).  Bound by the walks: a
// 640x480 frame at 5 mm without the drain takes 63 of 69 us, about 30 instructions
// a step and a wait at each block that the tile meets for the first time.  Smaller
// tiles meet more of them (16x8 98 us, 8x8 134), sets twice as large, two to four
// steps looked up together or warps held together at each step are no faster (70
// to 118).  CLOSE: 5 CTAs per SM, 48 registers and nothing spilled in the walk: 63
// us, with 8 CTAs and 32 registers 73, with 64-bit keys packed at each step and a
// compare-and-swap by every lane 85.  Otherwise 8 CTAs (32 registers): rays that
// share no blocks wait on more of them, 640x480 at 4 mm and 8 m 819 us, with 6
// CTAs 942.
// The tiles' rows of CTAs are followed by rows that empty the raycast's grid at
// the frame's pose (memory-bound work beside the rays' latency-bound one).
template <bool CLOSE>
__global__ void __launch_bounds__(kAllocN, CLOSE ? 5 : 8)
    fused_allocate_kernel(const SessDev* __restrict__ tab, int tile_rows) {
  __shared__ SessDev S;
  stage_session(tab + blockIdx.z, &S);
  __syncthreads();
  const DSensor& s = S.ls[0];
  if (close_rays(S.vol.t, s) != CLOSE) return;
  if ((int)blockIdx.y >= tile_rows) {
    if (S.vol.grid && S.mode == 1)
      grid_clear(S.vol, S.pose->posef, s,
                 (((int)blockIdx.y - tile_rows) * (int)gridDim.x + (int)blockIdx.x) * kAllocN +
                     (int)threadIdx.x,
                 ((int)gridDim.y - tile_rows) * (int)gridDim.x * kAllocN);
    return;
  }
  if ((int)blockIdx.x * kAllocX >= s.cols || (int)blockIdx.y * kAllocY >= s.rows) return;
  __shared__ AllocSmem sm;
  if (CLOSE || narrow_keys(S.vol.t))
    allocate_tile<unsigned, CLOSE>(S, blockIdx.x, blockIdx.y, sm);
  else
    allocate_tile<unsigned long long, CLOSE>(S, blockIdx.x, blockIdx.y, sm);
}

// ------------------------------------------------------------ visibility
// IntegrateScanKernel's block test (tsdf.cu:283-300): block origin to the
// camera, z < 0 rejected, the origin plus half a block (in camera axes,
// computed in double) projected into the image.
__device__ inline bool block_visible(unsigned long long key, const DTsdf& t, const DSensor& s,
                                     const M4f& invT) {
  const float vs = t.vs;
  const int bs = kBlockSize;
  F3 position = f3((float)key_x(key) * vs * (float)bs, (float)key_y(key) * vs * (float)bs,
                   (float)key_z(key) * vs * (float)bs);
  F3 pc = xform(invT, position);
  if (pc.z < 0) return false;
  double half = 0.5 * (double)vs * (double)bs;
  F3 bc = f3((float)((double)pc.x + half), (float)((double)pc.y + half),
             (float)((double)pc.z + half));
  int ix, iy;
  if (!project(bc, s, &ix, &iy)) return false;
  return ix >= 0 && iy >= 0 && ix < s.cols && iy < s.rows;
}

// ------------------------------------------------------------ ray depth bounds
// A ray sample whose voxel lies in no allocated block reads weight 0 and
// steps one truncation distance (tsdf.cu:505-507), so for every 8x8 pixel
// tile the frame's raycast gets a lower bound on the camera depth at which
// any of its rays can first enter an allocated block and an upper bound on
// the depth at which the last one leaves one: below the first and above the
// second (and beyond the near distance, where rays are marched normally) a
// sample needs no lookup, the march adds the truncation distance just as
// the lookup would have made it -- the same steps, so the same depths.
// Band sessions (blocks only near surfaces) skip most of every ray; the
// reference's carving allocation fills the space in front of surfaces, so
// there the far bound is what skips (rays past the scene).  Each allocated
// block contributes its box widened by one voxel beyond the rounding cells
// of its outer voxels, clipped to camera depth >= the near distance,
// projected and widened by one pixel: the tiles its bounding rectangle
// touches get min(near, nearest depth of the box) and max(far, farthest
// depth of the box).
// The bounds buffer of a session with tiles_x x tiles_y fine tiles
// (ray_bounds_words): near and far per fine tile, then near and far per
// coarse tile; a pixel's bounds are min(near) / max(far) over both levels.
struct RayBounds {
  unsigned *near8, *far8, *near64, *far64;
  int cx, cy;
};
__device__ inline RayBounds ray_bounds(unsigned* rb, int tiles_x, int tiles_y) {
  RayBounds B;
  B.cx = (tiles_x + kRbCoarse - 1) / kRbCoarse;
  B.cy = (tiles_y + kRbCoarse - 1) / kRbCoarse;
  B.near8 = rb;
  B.far8 = rb + tiles_x * tiles_y;
  B.near64 = B.far8 + tiles_x * tiles_y;
  B.far64 = B.near64 + B.cx * B.cy;
  return B;
}

__device__ inline float ray_near(const DTsdf& t) { return t.bsm; }

__device__ inline void bound_block(unsigned long long key, const DTsdf& t, const DSensor& s,
                                   const M4f& invT, unsigned* __restrict__ rb, int tiles_x,
                                   int tiles_y, bool near, bool far) {
  const float vs = t.vs;
  const float znear = ray_near(t);
  const float lo[3] = {((float)key_x(key) * 8.0f - 1.5f) * vs,
                       ((float)key_y(key) * 8.0f - 1.5f) * vs,
                       ((float)key_z(key) * 8.0f - 1.5f) * vs};
  const float ext = 11.0f * vs;
  F3 c[8];
  float zmin = 3.0e38f, zmax = -3.0e38f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    c[k] = xform(invT, f3(lo[0] + ((k & 1) ? ext : 0.0f), lo[1] + ((k & 2) ? ext : 0.0f),
                          lo[2] + ((k & 4) ? ext : 0.0f)));
    zmin = fminf(zmin, c[k].z);
    zmax = fmaxf(zmax, c[k].z);
  }
  if (!(zmax >= znear)) return;  // wholly nearer than the near distance
  float umin = 3.0e38f, umax = -3.0e38f, vmin = 3.0e38f, vmax = -3.0e38f;
  // (approximate reciprocals: their error is far below the rectangle's margin
  // of a pixel wherever it lies in the image)
  const float rnear = 1.0f / znear;
  auto add = [&](float X, float Y, float rz) {
    const float u = s.fx * X * rz + s.cx, w = s.fy * Y * rz + s.cy;
    umin = fminf(umin, u);
    umax = fmaxf(umax, u);
    vmin = fminf(vmin, w);
    vmax = fmaxf(vmax, w);
  };
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (c[k].z >= znear) add(c[k].x, c[k].y, __fdividef(1.0f, c[k].z));
  // the 12 box edges (corner pairs differing in one bit) cut by z = znear
  if (zmin < znear)
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int bit = 1; bit < 8; bit <<= 1) {
        if (k & bit) continue;
        const F3 a = c[k], b = c[k | bit];
        if ((a.z < znear) != (b.z < znear)) {
          const float f = (znear - a.z) / (b.z - a.z);
          add(a.x + f * (b.x - a.x), a.y + f * (b.y - a.y), rnear);
        }
      }
  umin -= 1.0f;
  vmin -= 1.0f;
  umax += 1.0f;
  vmax += 1.0f;
  if (!(umax >= 0.0f && vmax >= 0.0f && umin <= (float)(s.cols - 1) &&
        vmin <= (float)(s.rows - 1)))
    return;
  const int tx0 = umin <= 0.0f ? 0 : min((int)umin / kRbTile, tiles_x - 1);
  const int ty0 = vmin <= 0.0f ? 0 : min((int)vmin / kRbTile, tiles_y - 1);
  const int tx1 = umax >= (float)(s.cols - 1) ? tiles_x - 1 : (int)umax / kRbTile;
  const int ty1 = vmax >= (float)(s.rows - 1) ? tiles_y - 1 : (int)vmax / kRbTile;
  // Non-negative floats order as their bit patterns.  A block whose
  // rectangle spans more than 16 tiles (one close to the camera) goes to
  // the coarse level instead, so that no thread walks hundreds of tiles;
  // the coarse bounds of such blocks are loose only near the camera.
  // Carving sessions' blocks start at the camera: their near bound comes
  // from the blocks that hold observed non-saturated voxels (mixed form,
  // fused_surface_bound_kernel) or stays 0 (FP32 form).
  const unsigned zb = __float_as_uint(fmaxf(zmin, 0.0f)), ze = __float_as_uint(zmax);
  RayBounds B = ray_bounds(rb, tiles_x, tiles_y);
  unsigned *nb = B.near8, *fb = B.far8;
  int tw = tiles_x, x0 = tx0, x1 = tx1, y0 = ty0, y1 = ty1;
  if ((tx1 - tx0 + 1) * (ty1 - ty0 + 1) > 16) {
    nb = B.near64;
    fb = B.far64;
    tw = B.cx;
    x0 = tx0 / kRbCoarse;
    x1 = tx1 / kRbCoarse;
    y0 = ty0 / kRbCoarse;
    y1 = ty1 / kRbCoarse;
  }
  for (int ty = y0; ty <= y1; ++ty)
    for (int tx = x0; tx <= x1; ++tx) {
      if (near) atomicMin(nb + ty * tw + tx, zb);
      if (far) atomicMax(fb + ty * tw + tx, ze);
    }
}

// Free-space blocks of a depth-only frame.  A voxel whose point is nearer
// than (sdist - truncation) of its pixel takes IntegrateScanKernel's
// free-space branch (sdf = truncation).  A visible block is a free-space
// block when that holds for every voxel: the block's voxel points (the box
// of corners origin .. origin + 7 voxels) lie in front of the camera and
// project inside the image (a pixel of margin around the corners'
// projections), and the farthest corner (with 1e-5 relative + 1e-5 m of
// margin) is nearer than the free-space tile map's least (sdist -
// truncation) over the tiles that rectangle touches -- which is 0 wherever
// a pixel's depth is outside the sensor range.  The per-voxel arithmetic
// rounds far below these margins, so its test takes the free-space branch
// for every voxel of such a block, and integration skips the per-voxel
// projection (colours are zero: no RGB).  Blocks whose rectangle covers
// more than 16 coarse tiles (close to the camera) take the per-voxel test.
__device__ inline bool free_space_block(unsigned long long key, const DTsdf& t, const DSensor& s,
                                        const M4f& invT, const unsigned* __restrict__ ftile,
                                        int tiles_x, int tiles_y, int parity) {
  const float vs = t.vs, e = 7.0f * vs;
  const float ox = (float)key_x(key) * vs * (float)kBlockSize,
              oy = (float)key_y(key) * vs * (float)kBlockSize,
              oz = (float)key_z(key) * vs * (float)kBlockSize;
  float u0 = 3.0e38f, u1 = -3.0e38f, v0 = 3.0e38f, v1 = -3.0e38f, dm = 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const F3 c = xform(invT, f3(ox + ((k & 1) ? e : 0.0f), oy + ((k & 2) ? e : 0.0f),
                                oz + ((k & 4) ? e : 0.0f)));
    if (!(c.z > 0.01f)) return false;
    const float rz = __fdividef(1.0f, c.z);  // far more exact than the pixel of margin
    const float u = s.fx * c.x * rz + s.cx, w = s.fy * c.y * rz + s.cy;
    u0 = fminf(u0, u);
    u1 = fmaxf(u1, u);
    v0 = fminf(v0, w);
    v1 = fmaxf(v1, w);
    dm = fmaxf(dm, dot3(c, c));
  }
  dm = sqrtf(dm);
  // (u0 <= u1 fails where every corner's projection is NaN)
  if (!(u0 >= 1.0f && v0 >= 1.0f && u1 <= (float)(s.cols - 2) && v1 <= (float)(s.rows - 2) &&
        u0 <= u1 && v0 <= v1))
    return false;
  const int x0 = (int)floorf(u0) - 1, x1 = (int)ceilf(u1) + 1;
  const int y0 = (int)floorf(v0) - 1, y1 = (int)ceilf(v1) + 1;
  if (x0 < 0 || y0 < 0 || x1 >= s.cols || y1 >= s.rows) return false;
  int tx0 = x0 / kRbTile, tx1 = x1 / kRbTile, ty0 = y0 / kRbTile, ty1 = y1 / kRbTile;
  const unsigned* m = ftile;
  int tw = tiles_x;
  if ((tx1 - tx0 + 1) * (ty1 - ty0 + 1) > 16) {
    m = ftile + tiles_x * tiles_y + parity * coarse_tiles(tiles_x, tiles_y);
    tw = (tiles_x + kRbCoarse - 1) / kRbCoarse;
    tx0 /= kRbCoarse;
    tx1 /= kRbCoarse;
    ty0 /= kRbCoarse;
    ty1 /= kRbCoarse;
    if ((tx1 - tx0 + 1) * (ty1 - ty0 + 1) > 16) return false;
  }
  // at most 16 tiles, four loads in flight (the last one repeated)
  const int w = tx1 - tx0 + 1, n = w * (ty1 - ty0 + 1);
  unsigned mn = 0xffffffffu;
  for (int k = 0; k < n; k += 4) {
    unsigned q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = min(k + j, n - 1), r = i / w;
      q[j] = __ldg(m + (ty0 + r) * tw + tx0 + (i - r * w));
    }
    mn = min(min(mn, min(q[0], q[1])), min(q[2], q[3]));
  }
  return dm * (1.0f + 1e-5f) + 1e-5f < __uint_as_float(mn);
}

// one volume's grid at a caller's pose: emptied, then its blocks entered
__global__ void grid_clear_kernel(const __grid_constant__ VolumeDev v,
                                  const __grid_constant__ DSensor s,
                                  const float* __restrict__ pose16) {
  grid_clear(v, pose16, s, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void grid_fill_kernel(const __grid_constant__ VolumeDev v) {
  const GridBox b = *v.gbox;
  if (!b.ok) return;
  const int n = min(v.cnt->nalloc, v.t.num_blocks);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    grid_put(v, b, v.block_keys[i], i, v.freecell && v.freecell[i] ? 1u : 0u);
}

// Every session's visible blocks appended to one batch-wide list of
// (session, heap index), so integration balances across sessions; the
// session index carries kVisFree for free-space blocks.
// Bound by latency: a thread's chain (three sets of corners and the tile
// minima), and the list's one counter, which takes an atomic per CTA and step
// (per warp, 1100 of them at 640x480, and with IEEE quotients, 27 us of a
// frame, now 24.6; 27 -> 18.4 at 320x240; more with a CTA's look at the
// bounds before their atomics).  CTAs this small, so that a few thousand blocks reach every
// SM.
constexpr int kVisThreads = 128;
__global__ void __launch_bounds__(kVisThreads) fused_visible_kernel(const SessDev* __restrict__ tab, int2* __restrict__ gvis,
                                     int* __restrict__ gcount) {
  __shared__ SessDev S;
  stage_session(tab + blockIdx.z, &S);
  __syncthreads();
  const VolumeDev& v = S.vol;
  __shared__ M4f invT;
  __shared__ int seen[2][kVisThreads / 32], base_s[2];
  if (threadIdx.x < 16) invT.m[threadIdx.x] = S.pose->invf[threadIdx.x];
  int n = v.cnt->nalloc;
  if (n > v.t.num_blocks) n = v.t.num_blocks;
  if ((int)(blockIdx.x * blockDim.x) >= n) return;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int total = 0, step = 0;
  // (mixed carving sessions' entries get their free-cell flags afterwards)
  GridBox box;
  box.ok = 0;
  if (v.grid && S.mode == 1) box = *v.gbox;
  const bool carve = S.ftile && !v.t.band && !*S.rgb_flag;
  // (the frame counter has advanced since the ingest made the map)
  const int parity = (S.pose->frame - 1) & 1;
  for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    int i = base + threadIdx.x;
    bool vis = false;
    unsigned long long key = 0;
    if (i < n) {
      key = v.block_keys[i];
      if (box.ok) grid_put(v, box, key, i, 0u);
      vis = block_visible(key, v.t, S.ls[0], invT);
      // every allocated block (visible or not) enters the ray-start bound
      if (S.rbound) bound_block(key, v.t, S.ls[0], invT, S.rbound, S.rb_tx, S.rb_ty, v.t.band, true);
    }
    bool fr = false;
    if (vis && carve)
      fr = free_space_block(key, v.t, S.ls[0], invT, S.ftile, S.rb_tx, S.rb_ty, parity);
    const unsigned m = __ballot_sync(0xffffffffu, vis);
    if (lane == 0) seen[step][warp] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kVisThreads / 32; ++w) {
      if (w < warp) before += seen[step][w];
      all += seen[step][w];
    }
    if (threadIdx.x == 0 && all) base_s[step] = atomicAdd(gcount, all);
    total += all;
    __syncthreads();
    if (vis)
      gvis[base_s[step] + before + __popc(m & ((1u << lane) - 1))] =
          make_int2((int)blockIdx.z | (fr ? kVisFree : 0), i);
    step ^= 1;  // (the other buffer: no barrier before its next use)
  }
  if (threadIdx.x == 0 && total) atomicAdd(&v.cnt->visible, total);
}

// The near ray bound of mixed carving sessions, after integration.  A
// sample whose cell and centre voxel lie only in blocks without observed
// non-saturated voxels (unallocated, unobserved or saturated: f16 value 1)
// steps the truncation distance, or the interpolation of saturated values
// -- the truncation up to the rounding of the weights, never ending the
// march (free_ok) -- as the free-cell shortcut does; so the near bound of a
// tile is the nearest depth of the boxes of the blocks that hold such
// voxels (VolumeDev::nonsat > 0), widened as bound_block widens every box.
// Every block also enters the raycast's grid here, with its free-cell flag.
__global__ void __launch_bounds__(kVisThreads) fused_surface_bound_kernel(const SessDev* __restrict__ tab) {
  const SessDev& S = tab[blockIdx.z];
  const VolumeDev& v = S.vol;
  if (!v.nonsat) return;
  const bool bound = S.rbound && v.free_ok && !v.t.band;
  const bool put = v.grid && S.mode == 1 && v.gbox->ok;
  __shared__ M4f invT;
  if (threadIdx.x < 16) invT.m[threadIdx.x] = S.pose->invf[threadIdx.x];
  __syncthreads();
  int n = v.cnt->nalloc;
  if (n > v.t.num_blocks) n = v.t.num_blocks;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
      const unsigned long long key = v.block_keys[i];
      if (put) grid_put(v, *v.gbox, key, i, v.freecell[i] ? 1u : 0u);
      if (bound && v.nonsat[i] > 0)
        bound_block(key, v.t, S.ls[0], invT, S.rbound, S.rb_tx, S.rb_ty, true, false);
    }
}

// ------------------------------------------------------------ integration
// IntegrateScanKernel voxel loop (tsdf.cu:301-341) + Voxel::mergeVoxel
// (geom_Types.h:79-103).  The voxel updated is the thread's own: the
// reference's camera->world round trip through UpdateVoxel lands on the same
// voxel (the oracle checks this).
//
// One warp per block: lane (y, z pair) walks x, so that a step is 64 voxels in
// 512 contiguous bytes (256 in the mixed form), two per lane in one vector,
// and the products of the camera transform that depend on y and z alone are
// taken once per block -- the reference's sums, with their terms computed
// once.  A voxel gathers one word of its pixel (sdist, which carries the
// depth's validity, image.cu) and, when it is updated, the pixel's packed
// colour.  Three of the reference's IEEE operations only decide something for
// few voxels, which alone compute them:
//  * the pixel: an approximate quotient within a margin of its rounding;
//  * the distance from the camera: its approximation tells free space and
//    behind the surface apart, the band takes the square root;
//  * the merge's division by weight + 1: by the tabulated reciprocal with an
//    exact correction (div_by), the colours' by a tabulated multiplier.
// A 640x480 RGB frame (32,000 blocks): the CTA-per-block kernel before it took
// 123 M warp instructions and waited on its barriers and on gathers of five words
// per voxel; this one takes 88 M and issues in 67 % of the cycles (with 80
// registers and 24 warps per SM it was slower).  Live stage before -> now:
// 640x480 RGB FP32 156 -> 112 us, mixed with its free-cell passes 195 -> 141,
// 320x240 FP32 41 -> 36, 32-session band batch 357 -> 194; reading and writing
// the blocks once would take 45 us of the first.
//
// FAST (band sessions, whose allocation already departs from the
// reference's): fused multiply-adds and hardware-approximate division and
// square root throughout.

// The tabulated divisors of the merge, for weights 0 .. 255 (divisor w + 1).
struct MergeTable {
  float2 rcp[256];    // 1 / (w + 1) as yh, yl of div_by
  unsigned mul[256];  // ceil(2^24 / (w + 1))
};
__device__ inline void make_merge_table(MergeTable& t, int k) {
  const float b = (float)(k + 1);
  const float yh = 1.0f / b;
  t.rcp[k] = make_float2(yh, __fmaf_rn(-b, yh, 1.0f) * yh);
  t.mul[k] = (0x1000000u + (unsigned)k) / (unsigned)(k + 1);
}

// Voxel::mergeVoxelColor (geom_Types.h:87-91) of an observation of weight 1
// into a channel of weight w: the byte of (old * w + obs) / (w + 1) in
// FP32.  The numerator is an integer below 2^24 (exact in FP32), and the
// rounded quotient truncates to the floor of the exact one: below an
// integer k <= 255 the quotient is at least 1 / (w + 1) >= 2^-16 away,
// more than the half ulp (at most 2^-17) it would take to round up to k.
// So the integer quotient gives the same byte; for w <= 255 (n <= 65280) it is
// the high part of n * ceil(2^24 / (w + 1)): the multiplier is less than 1 too
// large by (w + 1) parts in 2^24, and n (w + 1) < 2^24.
__device__ inline unsigned colour_merge(unsigned old, unsigned obs, unsigned w, unsigned mul) {
  const unsigned n = old * w + obs;
  return (unsigned)(((unsigned long long)n * mul) >> 24);
}
// the three channels of packed colours (byte 3 zero)
__device__ inline unsigned colours_merge(unsigned old, unsigned obs, unsigned w,
                                         const MergeTable& tb) {
  unsigned r = 0;
  if (w <= 255u) {
    const unsigned m = tb.mul[w];
#pragma unroll
    for (int k = 0; k < 24; k += 8)
      r |= colour_merge((old >> k) & 255u, (obs >> k) & 255u, w, m) << k;
  } else {  // mixed form
#pragma unroll
    for (int k = 0; k < 24; k += 8)
      r |= ((((old >> k) & 255u) * w + ((obs >> k) & 255u)) / (w + 1u)) << k;
  }
  return r;
}

struct FrameView {
  const float* __restrict__ sdist;
  int cols, rows;
  float fx, fy, cx, cy, trunc;
  float mx, my;  // a half less the margin of the approximate pixel coordinate
};

__device__ inline float norm3_fast(F3 v) {
  const float q = __fmaf_rn(v.x, v.x, __fmaf_rn(v.y, v.y, v.z * v.z));
  return q > 0.0f ? q * rsqrtf(q) : 0.0f;
}

// roundf(x) as an integer biased by kRintBits, for |x| < 2^22 (other values
// give integers outside 0 .. 8191, as do NaNs: the addition is monotone).
__device__ inline int round_biased(float x) {
  const float t = x + kRint;
  const float d = x - (t - kRint);  // ties went to even: away from zero instead
  return __float_as_int(t) + (d == 0.5f && x > 0.0f ? 1 : 0) - (d == -0.5f && x < 0.0f ? 1 : 0);
}

// The pixel that camera-frame point p projects to, or -1.
template <bool FAST>
__device__ inline int observed_pixel(const FrameView& f, F3 p) {
  int px, py;
  bool ok = true;
  if (FAST) {
    ok = p.z > 0.0f;
    const float rz = __fdividef(1.0f, p.z);
    px = round_biased(__fmaf_rn(f.fx * p.x, rz, f.cx)) - kRintBits;
    py = round_biased(__fmaf_rn(f.fy * p.y, rz, f.cy)) - kRintBits;
  } else {
    const float ax = f.fx * p.x, ay = f.fy * p.y;
    float rz;
    asm("rcp.approx.f32 %0, %1;" : "=f"(rz) : "f"(p.z));
    const float x = __fmaf_rn(ax, rz, f.cx), y = __fmaf_rn(ay, rz, f.cy);
    const float tx = x + kRint, ty = y + kRint;
    px = __float_as_int(tx) - kRintBits;
    py = __float_as_int(ty) - kRintBits;
    if (!(fabsf(x - (tx - kRint)) < f.mx && fabsf(y - (ty - kRint)) < f.my)) {
      // Project, utils.h:114-119
      const float rx = roundf(ax / p.z + f.cx), ry = roundf(ay / p.z + f.cy);
      ok = fabsf(rx) < 2e9f && fabsf(ry) < 2e9f;
      px = ok ? (int)rx : 0;
      py = ok ? (int)ry : 0;
    }
  }
  ok = ok && (unsigned)px < (unsigned)f.cols && (unsigned)py < (unsigned)f.rows;
  return ok ? py * f.cols + px : -1;
}

// Whether the voxel at camera-frame point p is updated by its pixel's sdist
// word, and with which sdf.
template <bool FAST>
__device__ inline bool observed_sdf(const FrameView& f, F3 p, float sd, float& sdf) {
  const float s = fabsf(sd), lo = s - f.trunc, hi = s + f.trunc;  // (NaN: no depth in range)
  float vd;
  sdf = f.trunc;
  if (FAST) {
    vd = norm3_fast(p);
  } else {
    const float q = p.x * p.x + p.y * p.y + p.z * p.z;
    const float va = q * rsqrtf(q);  // |p| to within 4e-7
    if (va * 1.000002f < lo) return true;
    if (va > hi * 1.000002f) return false;
    vd = sqrtf(q);
  }
  if (vd > lo && vd < hi && __float_as_int(sd) >= 0) {  // sign: depth at the range's end
    sdf = s - vd;
    return true;
  }
  return vd < lo;
}

// Voxel::mergeVoxel (geom_Types.h:79-103) of one observation into an FP32-form
// voxel {r, g, b, w | sdf}.
__device__ inline uint2 merge_fp32(uint2 raw, float sdf, bool has_rgb, unsigned rgb, int max_w,
                                   const MergeTable& tb) {
  const unsigned w = raw.x >> 24;
  const float fw = (float)w, d = fw + 1.0f;
  const float a = __uint_as_float(raw.y) * fw + sdf * 1.0f;
  const float2 r = tb.rcp[w];
  float nsdf = div_by(a, d, r.x, r.y);
  if (!(fabsf(a) > 1e-18f && fabsf(a) < 1e18f)) nsdf = a / d;  // div_by's range
  // a zero colour merged with a zero colour stays exactly zero
  unsigned c = raw.x & 0x00ffffffu;
  if (has_rgb || c) c = colours_merge(c, rgb, w, tb);
  int nw = (uint8_t)(w + 1);
  if (nw > max_w) nw = max_w;
  return make_uint2(c | ((unsigned)nw << 24), __float_as_uint(nsdf));
}

// The same into a mixed-form voxel {f16 sdf / truncation | u16 weight}: the
// FP32 merge, stored as f16 (|value| <= 1, free space exactly 1).  'delta':
// the change of the block's count of observed, non-saturated voxels.
__device__ inline unsigned merge_mixed(unsigned raw, float sdf, float trunc, int max_w, int& delta) {
  const float osdf = __half2float(__ushort_as_half((unsigned short)(raw & 0xffffu))) * trunc;
  const int w = (int)(raw >> 16);
  const float fw = (float)w;
  const float nsdf = __fdividef(osdf * fw + sdf, fw + 1.0f);
  int nw = w + 1;
  if (nw > max_w) nw = max_w;
  const unsigned short nh = __half_as_ushort(__float2half_rn(__fdividef(nsdf, trunc)));
  // saturated: f16 value exactly 1 (free space); unobserved before
  const bool was = w == 0 || (raw & 0xffffu) == 0x3C00u, now = nh == 0x3C00u;
  delta += (int)was - (int)now;
  return (unsigned)nh | ((unsigned)nw << 16);
}

// The frame's update of block 'ptr' by one warp; free: a free-space block
// (every voxel's sdf is the truncation, no colours).
template <bool FP16, bool FAST>
__device__ inline void integrate_block(const SessDev& S, int ptr, bool free,
                                       const MergeTable& tb) {
  const VolumeDev& v = S.vol;
  const DTsdf& t = v.t;
  const int lane = threadIdx.x & 31, y = lane >> 2, z0 = (lane & 3) * 2;
  const unsigned* __restrict__ rgb = (!free && *S.rgb_flag) ? S.rgb4 : nullptr;
  const int max_w = t.max_w;
  const float vs = t.vs, trunc = t.trunc;
  FrameView f;
  f.sdist = S.sdist;
  f.cols = S.ls[0].cols;
  f.rows = S.ls[0].rows;
  f.fx = S.ls[0].fx;
  f.fy = S.ls[0].fy;
  f.cx = S.ls[0].cx;
  f.cy = S.ls[0].cy;
  f.trunc = trunc;
  // the coordinate's error: two roundings of x - cx (2^-22 of it), one of x
  f.mx = 0.5f - 6e-7f * ((float)f.cols + fabsf(f.cx) + 1.0f);
  f.my = 0.5f - 6e-7f * ((float)f.rows + fabsf(f.cy) + 1.0f);
  M4f T;
  const float4* inv = reinterpret_cast<const float4*>(S.pose->invf);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float4 r = __ldg(inv + k);
    T.m[4 * k] = r.x;
    T.m[4 * k + 1] = r.y;
    T.m[4 * k + 2] = r.z;
    T.m[4 * k + 3] = r.w;
  }
  // the block's first voxel and the lane's two, as the reference computes
  // them: key * extent + index * voxel
  const unsigned long long key = v.block_keys[ptr];
  const float ox = (float)key_x(key) * vs * (float)kBlockSize;
  const float vy = (float)key_y(key) * vs * (float)kBlockSize + (float)y * vs;
  const float oz = (float)key_z(key) * vs * (float)kBlockSize;
  const float vz[2] = {oz + (float)z0 * vs, oz + (float)(z0 + 1) * vs};
  float py[3], pz[2][3];  // the transform's terms in y and z
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    py[a] = T.m[4 * a + 1] * vy;
#pragma unroll
    for (int k = 0; k < 2; ++k)
      pz[k][a] = FAST ? __fmaf_rn(T.m[4 * a + 1], vy, __fmaf_rn(T.m[4 * a + 2], vz[k], T.m[4 * a + 3]))
                      : T.m[4 * a + 2] * vz[k];
  }
  const size_t base = (size_t)ptr * kBlockVox + y * 8 + z0;
  int delta = 0;
#pragma unroll 1
  for (int x = 0; x < 8; ++x) {
    const size_t i = base + (size_t)x * 64;
    bool up[2] = {true, true};
    float sdf[2] = {trunc, trunc};
    unsigned col[2] = {0u, 0u};
    if (!free) {
      const float vx = ox + (float)x * vs;
      F3 c[2];
      {
        float e[2][3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (FAST) {
#pragma unroll
            for (int k = 0; k < 2; ++k) e[k][a] = __fmaf_rn(T.m[4 * a], vx, pz[k][a]);
          } else {
            const float xy = T.m[4 * a] * vx + py[a];
#pragma unroll
            for (int k = 0; k < 2; ++k) e[k][a] = xy + pz[k][a] + T.m[4 * a + 3] * 1.0f;
          }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) c[k] = f3(e[k][0], e[k][1], e[k][2]);
      }
      int px[2];
      float sd[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) px[k] = observed_pixel<FAST>(f, c[k]);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        sd[k] = px[k] >= 0 ? __ldg(f.sdist + px[k]) : __int_as_float(0x7fffffff);
      if (rgb) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
          if (px[k] >= 0) col[k] = __ldg(rgb + px[k]);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) up[k] = observed_sdf<FAST>(f, c[k], sd[k], sdf[k]);
      if (!up[0] && !up[1]) continue;
    }
    if (FP16) {
      uint2* vp = reinterpret_cast<uint2*>(v.vox16 + i);
      uint2 r = *vp;
      if (v.colors) {
        uint2* cp = reinterpret_cast<uint2*>(v.colors + i);
        uint2 c = *cp;
        // colour exactly as the FP32 form (truncated to bytes)
        if (up[0]) c.x = (c.x & 0xff000000u) | colours_merge(c.x & 0x00ffffffu, col[0], r.x >> 16, tb);
        if (up[1]) c.y = (c.y & 0xff000000u) | colours_merge(c.y & 0x00ffffffu, col[1], r.y >> 16, tb);
        *cp = c;
      }
      if (up[0]) r.x = merge_mixed(r.x, sdf[0], trunc, max_w, delta);
      if (up[1]) r.y = merge_mixed(r.y, sdf[1], trunc, max_w, delta);
      *vp = r;
    } else {
      uint4* vp = reinterpret_cast<uint4*>(v.voxels + i);
      uint4 r = *vp;
      if (up[0]) {
        const uint2 n = merge_fp32(make_uint2(r.x, r.y), sdf[0], rgb != nullptr, col[0], max_w, tb);
        r.x = n.x;
        r.y = n.y;
      }
      if (up[1]) {
        const uint2 n = merge_fp32(make_uint2(r.z, r.w), sdf[1], rgb != nullptr, col[1], max_w, tb);
        r.z = n.x;
        r.w = n.y;
      }
      *vp = r;
    }
  }
  // the block's non-saturated count follows its voxels exactly (the block is
  // this warp's alone)
  if (FP16 && v.nonsat) {
    const int net = __reduce_add_sync(0xffffffffu, delta);
    if (lane == 0 && net != 0) v.nonsat[ptr] += net;
  }
}

// the batch-wide visible list: each item (session, block) by one warp
constexpr int kIntThreads = 256;
__global__ void __launch_bounds__(kIntThreads, 4)
    fused_integrate_kernel(const SessDev* __restrict__ tab, const int2* __restrict__ gvis,
                           const int* __restrict__ gcount) {
  __shared__ MergeTable tb;
  static_assert(kIntThreads == 256, "a table entry per thread");
  make_merge_table(tb, threadIdx.x);
  __syncthreads();
  const int n = *gcount;
  const int warps = gridDim.x * (kIntThreads / 32);
  for (int b = blockIdx.x * (kIntThreads / 32) + (threadIdx.x >> 5); b < n; b += warps) {
    const int2 entry = gvis[b];
    const SessDev& S = tab[entry.x & ~kVisFree];
    const bool free = (entry.x & kVisFree) != 0;
    if (!S.vol.fp16) integrate_block<false, false>(S, entry.y, free, tb);
    else if (S.vol.t.band) integrate_block<true, true>(S, entry.y, free, tb);
    else integrate_block<true, false>(S, entry.y, free, tb);
    __syncwarp();
  }
}

// Heap indices (or -1) of the seven neighbours of a block to one side: from the
// frame's block grid where it covers them, else from the hash.
__device__ inline void neighbours(const VolumeDev& v, bool grid, int x, int y, int z, int sg,
                                  int (&p)[8]) {
  if (grid) {
    const GridBox b = *v.gbox;
    const int gx = x - b.x0, gy = y - b.y0, gz = z - b.z0;
    const int ux = gx + sg, uy = gy + sg, uz = gz + sg;
    if (min(min(gx, ux), min(min(gy, uy), min(gz, uz))) >= 0 && max(gx, ux) < b.nx &&
        max(gy, uy) < b.ny && max(gz, uz) < b.nz) {
#pragma unroll
      for (int k = 1; k < 8; ++k) {
        const unsigned e = v.grid[((k & 1 ? ux : gx) * b.ny + (k & 2 ? uy : gy)) * b.nz +
                                  (k & 4 ? uz : gz)];
        p[k] = (int)(e / kBlockVox) < v.t.num_blocks ? (int)(e / kBlockVox) : -1;
      }
      return;
    }
  }
#pragma unroll
  for (int k = 1; k < 8; ++k)
    p[k] = find_block(v.entries, v.t, x + (k & 1 ? sg : 0), y + (k & 2 ? sg : 0),
                      z + (k & 4 ? sg : 0));
}

// Free-cell flags of the visible blocks (after their integration): a block's
// flag is set when it and its seven upper neighbours (+x, +y, +z and their
// combinations; missing ones count as free) hold no observed non-saturated
// voxel.  A visible block that holds one clears the flags of its seven lower
// neighbours, whose cells read it; those may be blocks that are not visible
// this frame.  Both writers of a flag agree: a block whose flag a neighbour
// clears computes 0 for itself.  Flags are only ever set here, for visible
// blocks, so a flag is never 1 where a cell of its block reads a
// non-saturated voxel.
__global__ void fused_free_cells_kernel(const SessDev* __restrict__ tab,
                                        const int2* __restrict__ gvis,
                                        const int* __restrict__ gcount) {
  const int n = *gcount;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int2 entry = gvis[i];
    const int2 item = make_int2(entry.x & ~kVisFree, entry.y);
    const VolumeDev& v = tab[item.x].vol;
    if (!v.freecell) continue;
    const unsigned long long key = v.block_keys[item.y];
    const int x = key_x(key), y = key_y(key), z = key_z(key);
    const bool own = v.nonsat[item.y] == 0;
    bool free = own && v.free_ok;
    if (own && !free) {
      v.freecell[item.y] = 0;
      continue;
    }
    // the upper neighbours of a block without such a voxel, the lower ones of
    // one with
    const int sg = own ? 1 : -1;
    int p[8];
    neighbours(v, tab[item.x].mode == 1 && v.grid && v.gbox->ok, x, y, z, sg, p);
#pragma unroll
    for (int k = 1; k < 8; ++k) {
      if (p[k] < 0) continue;
      if (own)
        free = free && v.nonsat[p[k]] == 0;
      else
        v.freecell[p[k]] = 0;
    }
    v.freecell[item.y] = free ? 1 : 0;
  }
}

// ------------------------------------------------------------ raycast
struct VoxelSample {
  float sdf;
  float r, g, b;
  int w;
};

struct BlockCache {
  int x, y, z;
  int ptr;
};
// the cache of the mixed march's cell blocks, with the block's free-cell flag
struct FreeCache : BlockCache {
  int free;
};

// voxel_index, blk_of and loc_of (WorldToGlobalVoxelHashing / WorldToBlock /
// WorldToLocalVoxel) are in common.cuh.

// tsdfVolume::GetVoxel, tsdf.cu:227-239, for a voxel already resolved to
// (block, local index); a one-block lookup cache skips repeated bucket
// scans of the same block.
__device__ inline int block_ptr(const VolumeDev& v, int bx, int by, int bz, BlockCache& bc) {
  if (bx != bc.x || by != bc.y || bz != bc.z) {
    bc.x = bx;
    bc.y = by;
    bc.z = bz;
    bc.ptr = find_block(v.entries, v.t, bx, by, bz);
  }
  return bc.ptr;
}
__device__ inline uint2 load_voxel(const VolumeDev& v, int ptr, int lin) {
  if (ptr < 0) return make_uint2(0u, 0u);
  return __ldg(reinterpret_cast<const uint2*>(v.voxels + (size_t)ptr * kBlockVox + lin));
}
__device__ inline int lin_of(int gx, int gy, int gz) {
  return (loc_of(gx) << 6) | (loc_of(gy) << 3) | loc_of(gz);
}

__device__ inline uint2 get_voxel(const VolumeDev& v, F3 pos, float inv_vs, BlockCache& bc) {
  const float vs = v.t.vs;
  int gx = voxel_index(pos.x, vs, inv_vs), gy = voxel_index(pos.y, vs, inv_vs),
      gz = voxel_index(pos.z, vs, inv_vs);
  return load_voxel(v, block_ptr(v, blk_of(gx), blk_of(gy), blk_of(gz), bc), lin_of(gx, gy, gz));
}

__device__ inline int vw(uint2 r) { return (int)(r.x >> 24); }
__device__ inline float vsdf(uint2 r) { return __uint_as_float(r.y); }

// The heap indices of the (up to eight) blocks a 2x2x2 cell touches: the
// cell's low corner is in block b, its high corner steps into b + 1 along
// the axes where the low corner is the block's last voxel (cx, cy, cz).
// Each distinct block is resolved once (the low one through the ray's
// cache); named fields, so that corner selection folds to a few selects.
struct CellBlocks {
  int p0, px, py, pz, pxy, pxz, pyz, pxyz;
};
__device__ inline void cell_blocks(const VolumeDev& v, int bx, int by, int bz, bool cx, bool cy,
                                   bool cz, BlockCache& bc, CellBlocks& cb) {
  const DTsdf& t = v.t;
  cb.p0 = block_ptr(v, bx, by, bz, bc);
  cb.px = cx ? find_block(v.entries, t, bx + 1, by, bz) : -1;
  cb.py = cy ? find_block(v.entries, t, bx, by + 1, bz) : -1;
  cb.pz = cz ? find_block(v.entries, t, bx, by, bz + 1) : -1;
  cb.pxy = (cx && cy) ? find_block(v.entries, t, bx + 1, by + 1, bz) : -1;
  cb.pxz = (cx && cz) ? find_block(v.entries, t, bx + 1, by, bz + 1) : -1;
  cb.pyz = (cy && cz) ? find_block(v.entries, t, bx, by + 1, bz + 1) : -1;
  cb.pxyz = (cx && cy && cz) ? find_block(v.entries, t, bx + 1, by + 1, bz + 1) : -1;
}
// the block of corner (ox, oy, oz) (compile-time offsets after unrolling)
__device__ inline int corner_block(const CellBlocks& cb, bool cx, bool cy, bool cz, int ox,
                                   int oy, int oz) {
  const bool kx = ox && cx, ky = oy && cy, kz = oz && cz;
  return kx ? (ky ? (kz ? cb.pxyz : cb.pxy) : (kz ? cb.pxz : cb.px))
            : (ky ? (kz ? cb.pyz : cb.py) : (kz ? cb.pz : cb.p0));
}

// tsdfVolume::GetInterpolatedVoxel, tsdf.cu:47-175.  The eight corners are
// pos_dual + {0, vs} per axis, so each axis has two coordinate values: they
// are resolved once (six index computations instead of twenty-four) and
// combined per corner; every corner still gets exactly the reference's
// float coordinate.  When the 2x2x2 corners lie in one block (the common
// case) the block is resolved once.  Corners are summed in the reference's
// order.  COLOR false skips the colour sums (the marching loop only reads
// sdf and weight).
template <bool COLOR>
__device__ inline VoxelSample get_interpolated(const VolumeDev& v, F3 position, float inv_vs,
                                               BlockCache& bc) {
  VoxelSample out;
  uint2 v0 = get_voxel(v, position, inv_vs, bc);
  out.w = vw(v0);
  if (out.w == 0) {
    out.sdf = vsdf(v0);
    out.r = (float)(v0.x & 0xff);
    out.g = (float)((v0.x >> 8) & 0xff);
    out.b = (float)((v0.x >> 16) & 0xff);
    return out;
  }
  const float vs = v.t.vs;
  F3 pos_dual = position - f3(vs / 2.0f, vs / 2.0f, vs / 2.0f);
  const float inv = 1.0f / vs;
  F3 vp = position * inv;
  F3 wt = f3(vp.x - floorf(vp.x), vp.y - floorf(vp.y), vp.z - floorf(vp.z));
  int gx[2], gy[2], gz[2];
  voxel_index_pair(pos_dual.x + 0.0f, pos_dual.x + vs, vs, inv_vs, gx[0], gx[1]);
  voxel_index_pair(pos_dual.y + 0.0f, pos_dual.y + vs, vs, inv_vs, gy[0], gy[1]);
  voxel_index_pair(pos_dual.z + 0.0f, pos_dual.z + vs, vs, inv_vs, gz[0], gz[1]);
  // the high corners lie in the next block along an axis where they cross
  const bool cx = blk_of(gx[1]) != blk_of(gx[0]), cy = blk_of(gy[1]) != blk_of(gy[0]),
             cz = blk_of(gz[1]) != blk_of(gz[0]);
  const int off[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1},
                         {1, 1, 0}, {0, 1, 1}, {1, 0, 1}, {1, 1, 1}};
  // the eight corner voxels: one block and constant strides from the low
  // corner in the common case (no axis crosses a block boundary and each
  // high index is the low one + 1), else each corner's block and index
  uint2 cv[8];
  if (!(cx || cy || cz) && gx[1] - gx[0] == 1 && gy[1] - gy[0] == 1 && gz[1] - gz[0] == 1) {
    const int p0 = block_ptr(v, blk_of(gx[0]), blk_of(gy[0]), blk_of(gz[0]), bc);
    const uint2* base = reinterpret_cast<const uint2*>(v.voxels + (size_t)(p0 < 0 ? 0 : p0) *
                                                                      kBlockVox +
                                                       lin_of(gx[0], gy[0], gz[0]));
#pragma unroll
    for (int k = 0; k < 8; ++k)
      cv[k] = p0 < 0 ? make_uint2(0u, 0u)
                     : __ldg(base + (off[k][0] << 6) + (off[k][1] << 3) + off[k][2]);
  } else {
    CellBlocks cells;
    cell_blocks(v, blk_of(gx[0]), blk_of(gy[0]), blk_of(gz[0]), cx, cy, cz, bc, cells);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int ox = off[k][0], oy = off[k][1], oz = off[k][2];
      cv[k] = load_voxel(v, corner_block(cells, cx, cy, cz, ox, oy, oz),
                         lin_of(gx[ox], gy[oy], gz[oz]));
    }
  }
  float dist = 0.0f;
  float cr = 0.0f, cg = 0.0f, cb = 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ox = off[k][0], oy = off[k][1], oz = off[k][2];
    const uint2 vv = cv[k];
    uint2 src = (vw(vv) == 0) ? v0 : vv;
    float a = ox ? wt.x : 1.0f - wt.x;
    float b = oy ? wt.y : 1.0f - wt.y;
    float c = oz ? wt.z : 1.0f - wt.z;
    float coef = a * b * c;
    dist += coef * vsdf(src);
    if (COLOR) {
      cr = cr + (float)(src.x & 0xff) * coef;
      cg = cg + (float)((src.x >> 8) & 0xff) * coef;
      cb = cb + (float)((src.x >> 16) & 0xff) * coef;
    }
  }
  out.sdf = dist;
  out.r = cr;
  out.g = cg;
  out.b = cb;
  return out;
}

// tsdfVolume raycast (tsdf.cu:471-526) of pixel (x, y) from camera pose T:
// march from 0 by the interpolated sdf (a truncation where unobserved) until
// the sdf drops under a voxel or the depth passes max_sensor_depth; then the
// interpolated colour at the hit.  Beyond the near distance, samples before
// skip_to or after skip_far (the tile's ray depth bounds: no allocated block
// there) step by the truncation without a lookup -- what the lookup would
// have returned.  Returns true when the march hit the step cap.
__device__ inline bool exact_hash_march(const VolumeDev& v, const DSensor& s, const M4f& T, int x,
                                        int y, float skip_to, float skip_far,
                                        float* __restrict__ depth_out,
                                        uint8_t* __restrict__ rgb_out) {
  const int i = y * s.cols + x;
  const DTsdf& t = v.t;
  const float inv_vs = 1.0f / t.vs;
  // getPoint3d (utils.h:104-112) with the pixel's (u - cx), (v - cy) hoisted
  const float ax = (float)x - s.cx, ay = (float)y - s.cy;
  BlockCache bc;
  bc.x = bc.y = bc.z = 0x7fffffff;
  bc.ptr = -1;
  float cur = 0.0f;
  int steps = 0;
  bool over = false;
  const float znear = ray_near(t);
  while (cur < t.dmax) {
    if (steps++ >= t.rc_cap) {
      over = true;
      break;
    }
    if (cur >= znear && (cur < skip_to || cur > skip_far)) {  // no allocated block here
      cur += t.trunc;
      continue;
    }
    F3 pc = f3(ax * cur / s.fx, ay * cur / s.fy, cur);
    F3 point = xform(T, pc);
    VoxelSample vx = get_interpolated<false>(v, point, inv_vs, bc);
    if (vx.w == 0) cur += t.trunc;
    else cur += vx.sdf;
    if (vx.w != 0 && vx.sdf < t.vs) break;
  }
  depth_out[i] = cur;
  if (rgb_out) {
    uint8_t r = 0, g = 0, b = 0;
    if (cur < t.dmax) {
      F3 point = xform(T, point3d_uv(x, y, cur, s));
      VoxelSample vx = get_interpolated<true>(v, point, inv_vs, bc);
      r = (uint8_t)vx.r;
      g = (uint8_t)vx.g;
      b = (uint8_t)vx.b;
    }
    rgb_out[3 * (size_t)i] = r;
    rgb_out[3 * (size_t)i + 1] = g;
    rgb_out[3 * (size_t)i + 2] = b;
  }
  return over;
}

// The same out of line, for the rays of a grid session that its grid does not
// take.
__device__ __noinline__ bool raycast_exact_hash_px(const VolumeDev& v, const DSensor& s,
                                                   const M4f& T, int x, int y, float skip_to,
                                                   float skip_far, float* __restrict__ depth_out,
                                                   uint8_t* __restrict__ rgb_out) {
  return exact_hash_march(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out);
}

// ---- the exact march over the block grid
// A sample of the reference's march needs the voxel its point lies in and the
// low corner of its trilinear cell, each the truncation of an IEEE quotient
// plus or minus a half (voxel_index), and the weights p * (1/vs) - floor.  All
// of them follow from e = p / vs: the voxel is e rounded to nearest, the low
// corner floor(e), the high corner floor(e) + 1.  The march takes both from
// vp = fl(p * fl(1/vs)), which the weights need anyway, rounded by adding and
// subtracting 1.5 * 2^23 (two additions and no conversion: the sum's low bits
// are the integer).  With u = 2^-24 the roundings of vp (2u|e|) and of the
// reference's corner, quotient and half additions (4u|e| + 3u at most, the
// high corner's) move a value across a rounding boundary only within
// 6u|e| + 3u of it, so where every axis is farther than 8u(max|vp| + 2) from
// every multiple of one half the indices are the reference's; else
// (exact_axis) they are computed with its own expressions.
//
// (x - cx) * z / fx by the hoisted reciprocal (div_by), whose range march_setup
// checks; a zero's sign reaches only sums with the pose's translation, where it
// changes no index, weight or depth.
// v rounded to the nearest integer (|v| < 2^22): its integer biased by
// kRintBits, the integer of floor(v) likewise, and v - round(v).
struct Rounded {
  int near, low;
  float diff;
};
__device__ inline Rounded round_near(float v) {
  Rounded r;
  const float t = v + kRint;
  r.near = __float_as_int(t);
  r.diff = v - (t - kRint);
  r.low = r.near - (r.diff < 0.0f ? 1 : 0);  // (not for -0)
  return r;
}
__device__ inline float biased_float(int i) { return __int_as_float(i) - kRint; }

// The block grid of the march (GridBox): entry of the block that holds voxel
// (x, y, z), biased as round_near gives them.
struct GridView {
  const unsigned* __restrict__ e;
  unsigned sx, sy, off;
};
__device__ inline GridView grid_view(const VolumeDev& v) {
  const GridBox& b = *v.gbox;
  GridView g;
  g.e = v.grid;
  g.sy = (unsigned)b.nz;
  g.sx = (unsigned)b.ny * g.sy;
  constexpr unsigned bias = (unsigned)kRintBits >> 3;
  g.off = ((unsigned)b.x0 + bias) * g.sx + ((unsigned)b.y0 + bias) * g.sy + (unsigned)b.z0 + bias;
  return g;
}
__device__ inline unsigned grid_index(const GridView& g, int x, int y, int z) {
  return (unsigned)(x >> 3) * g.sx + (unsigned)(y >> 3) * g.sy + (unsigned)(z >> 3) - g.off;
}

// Voxel indices of the eight corners of the cell whose low corner is (x, y, z)
// (biased), in the reference's order: g the grid index of the low corner's
// block, e0 that block's first voxel; the other blocks are read only where the
// cell crosses a block boundary.  FLAG: entries carry the free-cell flag in
// bit 0.
template <bool FLAG>
__device__ inline void cell_corners(const GridView& G, unsigned g, unsigned e0, int x, int y,
                                    int z, unsigned (&i)[8]) {
  const bool kx = (x & 7) == 7, ky = (y & 7) == 7, kz = (z & 7) == 7;
  unsigned b[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) b[k] = e0;
  if (kx | ky | kz) {
    const unsigned mx = kx ? G.sx : 0u, my = ky ? G.sy : 0u, mz = kz ? 1u : 0u;
    const unsigned gx = g + mx, gy = g + my, gxy = gx + my;
    b[1] = __ldg(G.e + gx);
    b[2] = __ldg(G.e + gy);
    b[3] = __ldg(G.e + (g + mz));
    b[4] = __ldg(G.e + gxy);
    b[5] = __ldg(G.e + (gy + mz));
    b[6] = __ldg(G.e + (gx + mz));
    b[7] = __ldg(G.e + (gxy + mz));
  }
  const unsigned xl = (unsigned)(x & 7) << 6, yl = (unsigned)(y & 7) << 3, zl = (unsigned)(z & 7);
  const unsigned xh = kx ? 0u : xl + 64u, yh = ky ? 0u : yl + 8u, zh = kz ? 0u : zl + 1u;
  if (FLAG) {
#pragma unroll
    for (int k = 0; k < 8; ++k) b[k] &= ~1u;
  }
  i[0] = b[0] + (xl + yl) + zl;
  i[1] = b[1] + (xh + yl) + zl;
  i[2] = b[2] + (xl + yh) + zl;
  i[3] = b[3] + (xl + yl) + zh;
  i[4] = b[4] + (xh + yh) + zl;
  i[5] = b[5] + (xl + yh) + zh;
  i[6] = b[6] + (xh + yl) + zh;
  i[7] = b[7] + (xh + yh) + zh;
}

// The depths of a march: samples below the near distance, then steps without a
// lookup up to the tile's near bound (no allocated block there, so each sample
// would step by the truncation), samples up to the far bound, and steps
// without a lookup to the end.  Depths only grow, so one comparison per sample
// tells whether its range is left.  The sum is taken step by step, as the
// samples would take it.
struct MarchRange {
  float skip_to, last;  // last: the first depth past the far bound or the end
  float lim;
  bool near;
  __device__ MarchRange(float znear, float skip_to_, float skip_far, float dmax)
      : skip_to(fminf(skip_to_, dmax)), near(true) {
    // the least float above skip_far (>= 0)
    last = skip_far < dmax ? fminf(__int_as_float(__float_as_int(skip_far) + 1), dmax) : dmax;
    lim = fminf(znear, dmax);
  }
  // whether a sample is taken at 'cur'; moves it past depths without one
  __device__ bool sample(float& cur, float trunc, float dmax) {
    if (cur < lim) return true;
    if (near) {
      near = false;
      while (cur < skip_to) cur += trunc;
      lim = last;
      if (cur < lim) return true;
    }
    while (cur < dmax) cur += trunc;
    return false;
  }
};

// One axis by the reference's expressions: (low corner, voxel - low corner),
// or a second value of 2 where the high corner is not low + 1 or the voxel is
// neither.  (Quotients too small for div_by's exactness are lost in the half.)
__device__ __noinline__ int2 exact_axis(float p, float vs, float inv_vs) {
  const float yl = __fmaf_rn(-vs, inv_vs, 1.0f) * inv_vs;
  auto index = [&](float q) {
    const float sg = (float)((q > 0.0f) - (q < 0.0f));
    return (int)(div_by(q, vs, inv_vs, yl) + sg * 0.5f);
  };
  const float pd = p - vs / 2.0f;
  const int g = index(p), g0 = index(pd + 0.0f), g1 = index(pd + vs);
  return make_int2(g0, (g1 - g0 == 1 && (g == g0 || g == g1)) ? g - g0 : 2);
}

// get_interpolated without colour, out of line (rare in the march).
__device__ __noinline__ float2 interpolated_generic(const VolumeDev& v, float x, float y, float z,
                                                    float inv_vs) {
  BlockCache bc;
  bc.x = bc.y = bc.z = 0x7fffffff;
  bc.ptr = -1;
  const VoxelSample s = get_interpolated<false>(v, f3(x, y, z), inv_vs, bc);
  return make_float2(s.sdf, s.w ? 1.0f : 0.0f);
}

// exact_hash_march over the block grid (which the volume has): every sample
// reads the entry of its voxel's block, an observed one those of its cell's
// blocks.  Rays outside march_setup's ranges take raycast_exact_hash_px.
__device__ inline bool raycast_exact_px(const VolumeDev& v, const DSensor& s, const M4f& T, int x,
                                        int y, float skip_to, float skip_far,
                                        float* __restrict__ depth_out,
                                        uint8_t* __restrict__ rgb_out) {
  const DTsdf& t = v.t;
  const float inv_vs = 1.0f / t.vs;
  // getPoint3d (utils.h:104-112) with the pixel's (u - cx), (v - cy) hoisted
  const float ax = (float)x - s.cx, ay = (float)y - s.cy;
  MarchRay R;
  if (!v.gbox->ok || !march_setup(t, s, T, ax, ay, inv_vs, R))
    return raycast_exact_hash_px(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out);
  const GridView G = grid_view(v);
  const uint2* __restrict__ vox = reinterpret_cast<const uint2*>(v.voxels);
  const float fx = s.fx, fy = s.fy, dmax = t.dmax, trunc = t.trunc, vs = t.vs;
  const unsigned empty = (unsigned)t.num_blocks * (unsigned)kBlockVox;
  float cur = 0.0f;
  MarchRange range(ray_near(t), skip_to, skip_far, dmax);
  while (range.sample(cur, trunc, dmax)) {
    const F3 p = xform(T, f3(div_by(ax * cur, fx, R.yhx, R.ylx), div_by(ay * cur, fy, R.yhy, R.yly),
                             cur));
    const F3 vp = p * inv_vs;
    const Rounded rx = round_near(vp.x), ry = round_near(vp.y), rz = round_near(vp.z);
    // the weights, from the floors of vp whatever the indices
    const float wx = vp.x - biased_float(rx.low), wy = vp.y - biased_float(ry.low),
                wz = vp.z - biased_float(rz.low);
    int lx = rx.low, ly = ry.low, lz = rz.low, ix = rx.near, iy = ry.near, iz = rz.near;
    int odd = 0;
    // margin: 1/4 - 8u(max|vp| + 2)
    const float thr = __fmaf_rn(fmaxf(fmaxf(fabsf(vp.x), fabsf(vp.y)), fabsf(vp.z)),
                                -4.76837158203125e-7f, 0.25f - 9.5367431640625e-7f);
    if (!(fmaxf(fmaxf(fabsf(fabsf(rx.diff) - 0.25f), fabsf(fabsf(ry.diff) - 0.25f)),
                fabsf(fabsf(rz.diff) - 0.25f)) < thr)) {
      auto check = [&](float diff, float pos, int& l, int& i) {
        if (!(fabsf(fabsf(diff) - 0.25f) < thr)) {
          const int2 e = exact_axis(pos, vs, inv_vs);
          l = e.x + kRintBits;
          i = l + e.y;
          odd |= e.y & 2;
        }
      };
      check(rx.diff, p.x, lx, ix);
      check(ry.diff, p.y, ly, iy);
      check(rz.diff, p.z, lz, iz);
    }
    if (odd) {
      const float2 g = interpolated_generic(v, p.x, p.y, p.z, inv_vs);
      cur += g.y == 0.0f ? trunc : g.x;
      if (g.y != 0.0f && g.x < vs) break;
      continue;
    }
    // (both entries at once: one load's latency instead of two)
    const unsigned g = grid_index(G, lx, ly, lz);
    const unsigned own = __ldg(G.e + grid_index(G, ix, iy, iz)), e0 = __ldg(G.e + g);
    if (own == empty) {  // no block: weight 0
      cur += trunc;
      continue;
    }
    // the voxel and the cell's corners together
    unsigned c[8];
    cell_corners<false>(G, g, e0, lx, ly, lz, c);
    const uint2 v0 = __ldg(vox + (own + (unsigned)(((ix & 7) << 6) | ((iy & 7) << 3) | (iz & 7))));
    uint2 r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = __ldg(vox + c[k]);
    if (v0.x < 0x01000000u) {  // weight 0
      cur += trunc;
      continue;
    }
    const float x0 = 1.0f - wx, y0 = 1.0f - wy, z0 = 1.0f - wz;
    const float a00 = x0 * y0, a10 = wx * y0, a01 = x0 * wy, a11 = wx * wy;
    const float coef[8] = {a00 * z0, a10 * z0, a01 * z0, a00 * wz,
                           a11 * z0, a01 * wz, a10 * wz, a11 * wz};
    // an unobserved corner takes the voxel's value
    const unsigned least = min(min(min(r[0].x, r[1].x), min(r[2].x, r[3].x)),
                               min(min(r[4].x, r[5].x), min(r[6].x, r[7].x)));
    if (least < 0x01000000u) {
#pragma unroll
      for (int k = 0; k < 8; ++k) r[k].y = r[k].x < 0x01000000u ? v0.y : r[k].y;
    }
    float sdf = coef[0] * vsdf(r[0]);
#pragma unroll
    for (int k = 1; k < 8; ++k) sdf += coef[k] * vsdf(r[k]);
    cur += sdf;
    if (sdf < vs) break;
  }
  const int i = y * s.cols + x;
  depth_out[i] = cur;
  if (rgb_out) {
    uint8_t r = 0, g = 0, b = 0;
    if (cur < dmax) {
      BlockCache bc;
      bc.x = bc.y = bc.z = 0x7fffffff;
      bc.ptr = -1;
      F3 point = xform(T, point3d_uv(x, y, cur, s));
      VoxelSample vx = get_interpolated<true>(v, point, inv_vs, bc);
      r = (uint8_t)vx.r;
      g = (uint8_t)vx.g;
      b = (uint8_t)vx.b;
    }
    rgb_out[3 * (size_t)i] = r;
    rgb_out[3 * (size_t)i + 1] = g;
    rgb_out[3 * (size_t)i + 2] = b;
  }
  return false;
}

// ------------------------------------------------------------ mixed-precision raycast
// The mixed forms' march: tsdfVolume::GenerateDepthKernel /
// GenerateRgbKernel (tsdf.cu:471-526) with GetInterpolatedVoxel
// (tsdf.cu:47-175) in voxel units: the sample at depth z is q = o + z * d
// (o the camera centre, d the pixel's ray direction per unit depth, both
// divided by the voxel size) by fused multiply-adds.  The reference's step
// rule is kept: from 0, step by the interpolated sdf where the sample's
// voxel (floor(q + 0.5), the reference's rounding of p / vs up to ties) is
// observed, by the truncation distance where it is not, until the sdf drops
// under a voxel or the depth passes max_sensor_depth.  The trilinear cell
// is floor(q) .. floor(q) + 1 with weights q - floor(q) (the reference's
// rounded p - vs/2 and p + vs/2 and its weights from p / vs); unobserved
// corners take the centre voxel's value.  Two shortcuts give what the full
// sample would give:
//  * beyond the near distance, a sample before the tile's near bound or
//    after its far bound (no allocated block there) steps by the truncation
//    without a lookup;
//  * a sample whose cell lies in a free-cell block (every voxel the cell can
//    read is unobserved or saturated, VolumeDev::freecell) steps by the
//    truncation distance without reading voxels: the reference's step there
//    is the truncation (unobserved centre) or the interpolation of
//    saturated values (f16 value exactly 1), which is the truncation up to
//    the rounding of the weights, and never ends the march (free_ok).
// The FP32 drop-in keeps raycast_exact_px: its targets decide the tracked
// poses, whose bar against the reference (1e-4 m / 1e-4 rad per frame)
// holds only with the reference's own rounding in the march -- with this
// march in the FP32 form, tracked poses left that bar after six to nine
// frames on the parity sequences, through the solver's discrete
// convergence test (an extra or a missing iteration moves a pose by up to
// the 1e-3 increment threshold).
struct MixedVox {
  static __device__ unsigned load(const VolumeDev& v, int ptr, int lin) {
    return ptr < 0 ? 0u : __ldg(v.vox16 + (size_t)ptr * kBlockVox + lin);
  }
  static __device__ int w(unsigned r) { return (int)(r >> 16); }
  static __device__ float val(unsigned r) {
    return __half2float(__ushort_as_half((unsigned short)(r & 0xffffu)));
  }
  static __device__ uchar4 color(const VolumeDev& v, int ptr, int lin) {
    return (v.colors && ptr >= 0) ? v.colors[(size_t)ptr * kBlockVox + lin]
                                  : make_uchar4(0, 0, 0, 0);
  }
};

// The interpolated sample at q (voxel units) whose centre voxel raw0 (heap
// index ptr0, local index lin0) is observed.  Sums by fused multiply-adds
// in the reference's corner order.
template <bool COLOR>
__device__ inline VoxelSample interp(const VolumeDev& v, F3 q, unsigned raw0, int ptr0, int lin0,
                                     BlockCache& bc) {
  using V = MixedVox;
  VoxelSample out;
  const float fx = floorf(q.x), fy = floorf(q.y), fz = floorf(q.z);
  const float wx = q.x - fx, wy = q.y - fy, wz = q.z - fz;
  const int gx = (int)fx, gy = (int)fy, gz = (int)fz;
  const int lx = gx & 7, ly = gy & 7, lz = gz & 7;
  const bool cx = lx == 7, cy = ly == 7, cz = lz == 7;
  CellBlocks cb;
  cell_blocks(v, gx >> 3, gy >> 3, gz >> 3, cx, cy, cz, bc, cb);
  // local index of the low corner and the steps to the high ones (wrapping
  // into the next block where the cell crosses)
  const int base = (lx << 6) | (ly << 3) | lz;
  const int dx = cx ? -448 : 64, dy = cy ? -56 : 8, dz = cz ? -7 : 1;
  const uchar4 c0 = COLOR ? V::color(v, ptr0, lin0) : make_uchar4(0, 0, 0, 0);
  const float n0 = V::val(raw0);
  const float ax[2] = {1.0f - wx, wx}, ay[2] = {1.0f - wy, wy}, az[2] = {1.0f - wz, wz};
  float dist = 0.0f, cr = 0.0f, cg = 0.0f, cbl = 0.0f;
  const int off[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1},
                         {1, 1, 0}, {0, 1, 1}, {1, 0, 1}, {1, 1, 1}};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ox = off[k][0], oy = off[k][1], oz = off[k][2];
    const int ptr = corner_block(cb, cx, cy, cz, ox, oy, oz);
    const int lin = base + (ox ? dx : 0) + (oy ? dy : 0) + (oz ? dz : 0);
    const unsigned r = V::load(v, ptr, lin);
    const bool use0 = V::w(r) == 0;
    const float coef = (ax[ox] * ay[oy]) * az[oz];
    dist = __fmaf_rn(coef, use0 ? n0 : V::val(r), dist);
    if (COLOR) {
      const uchar4 cc = use0 ? c0 : V::color(v, ptr, lin);
      cr = __fmaf_rn((float)cc.x, coef, cr);
      cg = __fmaf_rn((float)cc.y, coef, cg);
      cbl = __fmaf_rn((float)cc.z, coef, cbl);
    }
  }
  out.sdf = dist * v.t.trunc;
  out.w = V::w(raw0);
  out.r = cr;
  out.g = cg;
  out.b = cbl;
  return out;
}

// The interpolated colour at depth 'cur' of the ray q = o + cur * d (voxel
// units); of an unobserved voxel its own.
__device__ __noinline__ uchar4 mixed_colour(const VolumeDev& v, F3 o, F3 d, float cur) {
  using V = MixedVox;
  const F3 q = f3(__fmaf_rn(cur, d.x, o.x), __fmaf_rn(cur, d.y, o.y), __fmaf_rn(cur, d.z, o.z));
  const int gx = (int)floorf(q.x + 0.5f), gy = (int)floorf(q.y + 0.5f),
            gz = (int)floorf(q.z + 0.5f);
  BlockCache bc;
  bc.x = bc.y = bc.z = 0x7fffffff;
  bc.ptr = -1;
  const int ptr = block_ptr(v, blk_of(gx), blk_of(gy), blk_of(gz), bc);
  const int lin = lin_of(gx, gy, gz);
  const unsigned raw = V::load(v, ptr, lin);
  if (V::w(raw) == 0) return V::color(v, ptr, lin);
  const VoxelSample vx = interp<true>(v, q, raw, ptr, lin, bc);
  return make_uchar4((uint8_t)vx.r, (uint8_t)vx.g, (uint8_t)vx.b, 0);
}

// The block of a cell's low corner through the ray's cache, with its
// free-cell flag (0 where no flags are kept).
__device__ inline int cell_block_free(const VolumeDev& v, int bx, int by, int bz, FreeCache& bc,
                                      int* free) {
  if (bx != bc.x || by != bc.y || bz != bc.z) {
    bc.x = bx;
    bc.y = by;
    bc.z = bz;
    bc.ptr = find_block(v.entries, v.t, bx, by, bz);
    bc.free = (v.freecell && bc.ptr >= 0) ? (int)__ldg(v.freecell + bc.ptr) : 0;
  }
  *free = bc.free;
  return bc.ptr;
}

// The march of pixel (x, y) from camera pose T; the colour at the hit when
// rgb_out is given.  skip_to / skip_far: the tile's ray depth bounds.
// Returns true when the march hit the step cap.  FREE: the session keeps
// free-cell flags (mixed form with carving); without them (band sessions)
// the cell's and the centre voxel's blocks share one lookup cache.
template <bool FREE>
__device__ inline bool mixed_hash_march(const VolumeDev& v, const DSensor& s, const M4f& T, int x,
                                        int y, float skip_to, float skip_far,
                                        float* __restrict__ depth_out,
                                        uint8_t* __restrict__ rgb_out) {
  using V = MixedVox;
  const int i = y * s.cols + x;
  const DTsdf& t = v.t;
  const float inv_vs = 1.0f / t.vs;
  const float axf = ((float)x - s.cx) / s.fx, ayf = ((float)y - s.cy) / s.fy;
  const F3 o = f3(T.m[3] * inv_vs, T.m[7] * inv_vs, T.m[11] * inv_vs);
  const F3 d = f3((T.m[0] * axf + T.m[1] * ayf + T.m[2]) * inv_vs,
                  (T.m[4] * axf + T.m[5] * ayf + T.m[6]) * inv_vs,
                  (T.m[8] * axf + T.m[9] * ayf + T.m[10]) * inv_vs);
  FreeCache bc;   // the cell's low-corner block, with its flag
  BlockCache bc0;  // the centre voxel's block where it is another
  bc.x = bc.y = bc.z = bc0.x = bc0.y = bc0.z = 0x7fffffff;
  bc.ptr = bc0.ptr = -1;
  bc.free = 0;
  float cur = 0.0f;
  int steps = 0;
  bool over = false;
  const float znear = ray_near(t);
  while (cur < t.dmax) {
    if (steps++ >= t.rc_cap) {
      over = true;
      break;
    }
    if (cur >= znear && (cur < skip_to || cur > skip_far)) {  // no allocated block: weight 0
      cur += t.trunc;
      continue;
    }
    const F3 q = f3(__fmaf_rn(cur, d.x, o.x), __fmaf_rn(cur, d.y, o.y), __fmaf_rn(cur, d.z, o.z));
    const float flx = floorf(q.x), fly = floorf(q.y), flz = floorf(q.z);
    if (FREE) {
      int free;
      cell_block_free(v, (int)flx >> 3, (int)fly >> 3, (int)flz >> 3, bc, &free);
      if (free) {  // the interpolated sdf is the truncation distance
        cur += t.trunc;
        continue;
      }
    }
    const int gx = (int)flx + (q.x - flx >= 0.5f), gy = (int)fly + (q.y - fly >= 0.5f),
              gz = (int)flz + (q.z - flz >= 0.5f);
    // the centre voxel's block: mostly the cell's own, already resolved
    const int ptr = !FREE ? block_ptr(v, blk_of(gx), blk_of(gy), blk_of(gz), bc)
                    : (blk_of(gx) == bc.x && blk_of(gy) == bc.y && blk_of(gz) == bc.z)
                        ? bc.ptr
                        : block_ptr(v, blk_of(gx), blk_of(gy), blk_of(gz), bc0);
    const int lin = lin_of(gx, gy, gz);
    const unsigned raw = V::load(v, ptr, lin);
    if (V::w(raw) == 0) {
      cur += t.trunc;
      continue;
    }
    const VoxelSample vx = interp<false>(v, q, raw, ptr, lin, bc);
    cur += vx.sdf;
    if (vx.sdf < t.vs) break;
  }
  depth_out[i] = cur;
  if (rgb_out) {
    uchar4 c = make_uchar4(0, 0, 0, 0);
    if (cur < t.dmax) c = mixed_colour(v, o, d, cur);
    rgb_out[3 * (size_t)i] = c.x;
    rgb_out[3 * (size_t)i + 1] = c.y;
    rgb_out[3 * (size_t)i + 2] = c.z;
  }
  return over;
}

// The same out of line (raycast_exact_hash_px).
template <bool FREE>
__device__ __noinline__ bool raycast_hash_px(const VolumeDev& v, const DSensor& s, const M4f& T,
                                             int x, int y, float skip_to, float skip_far,
                                             float* __restrict__ depth_out,
                                             uint8_t* __restrict__ rgb_out) {
  return mixed_hash_march<FREE>(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out);
}

// mixed_hash_march over the block grid: the same samples, each with the entries
// of its cell's blocks read from the grid.  FREE: bit 0 of a block's entry is
// its free-cell flag.
template <bool FREE>
__device__ inline bool raycast_px(const VolumeDev& v, const DSensor& s, const M4f& T, int x,
                                  int y, float skip_to, float skip_far,
                                  float* __restrict__ depth_out, uint8_t* __restrict__ rgb_out) {
  const DTsdf& t = v.t;
  const float inv_vs = 1.0f / t.vs;
  const float axf = ((float)x - s.cx) / s.fx, ayf = ((float)y - s.cy) / s.fy;
  if (!v.gbox->ok || !march_bounded(t) || !march_within(t, T, axf, ayf, inv_vs))
    return raycast_hash_px<FREE>(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out);
  const F3 o = f3(T.m[3] * inv_vs, T.m[7] * inv_vs, T.m[11] * inv_vs);
  const F3 d = f3((T.m[0] * axf + T.m[1] * ayf + T.m[2]) * inv_vs,
                  (T.m[4] * axf + T.m[5] * ayf + T.m[6]) * inv_vs,
                  (T.m[8] * axf + T.m[9] * ayf + T.m[10]) * inv_vs);
  const GridView G = grid_view(v);
  const unsigned* __restrict__ vox = v.vox16;
  const float dmax = t.dmax, trunc = t.trunc, vs = t.vs;
  float cur = 0.0f;
  MarchRange range(ray_near(t), skip_to, skip_far, dmax);
  auto half_of = [](unsigned r) {
    return __half2float(__ushort_as_half((unsigned short)(r & 0xffffu)));
  };
  while (range.sample(cur, trunc, dmax)) {
    const F3 q = f3(__fmaf_rn(cur, d.x, o.x), __fmaf_rn(cur, d.y, o.y), __fmaf_rn(cur, d.z, o.z));
    const int lx = round_near(q.x).low, ly = round_near(q.y).low, lz = round_near(q.z).low;
    const float wx = q.x - biased_float(lx), wy = q.y - biased_float(ly),
                wz = q.z - biased_float(lz);
    const unsigned g = grid_index(G, lx, ly, lz);
    const unsigned e0 = __ldg(G.e + g);
    if (FREE && (e0 & 1u)) {  // the interpolated sdf is the truncation distance
      cur += trunc;
      continue;
    }
    const int ix = lx + (wx >= 0.5f), iy = ly + (wy >= 0.5f), iz = lz + (wz >= 0.5f);
    // the voxel's block: mostly the cell's own
    unsigned own = e0;
    if ((unsigned)((ix ^ lx) | (iy ^ ly) | (iz ^ lz)) >= 8u)
      own = __ldg(G.e + grid_index(G, ix, iy, iz));
    const unsigned raw =
        __ldg(vox + ((FREE ? own & ~1u : own) + (unsigned)(((ix & 7) << 6) | ((iy & 7) << 3) | (iz & 7))));
    if (raw < 0x10000u) {  // weight 0
      cur += trunc;
      continue;
    }
    unsigned c[8], r[8];
    cell_corners<FREE>(G, g, e0, lx, ly, lz, c);
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = __ldg(vox + c[k]);
    const float n0 = half_of(raw);
    const float x0 = 1.0f - wx, y0 = 1.0f - wy, z0 = 1.0f - wz;
    const float a00 = x0 * y0, a10 = wx * y0, a01 = x0 * wy, a11 = wx * wy;
    const float coef[8] = {a00 * z0, a10 * z0, a01 * z0, a00 * wz,
                           a11 * z0, a01 * wz, a10 * wz, a11 * wz};
    float dist = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) dist = __fmaf_rn(coef[k], r[k] < 0x10000u ? n0 : half_of(r[k]), dist);
    const float sdf = dist * trunc;
    cur += sdf;
    if (sdf < vs) break;
  }
  const int i = y * s.cols + x;
  depth_out[i] = cur;
  if (rgb_out) {
    uchar4 c = make_uchar4(0, 0, 0, 0);
    if (cur < dmax) c = mixed_colour(v, o, d, cur);
    rgb_out[3 * (size_t)i] = c.x;
    rgb_out[3 * (size_t)i + 1] = c.y;
    rgb_out[3 * (size_t)i + 2] = c.z;
  }
  return false;
}

// One pixel's ray of a TX x TY pixel tile (bx, by) from pose16 (a float 4x4);
// warps cover 8x4 pixel sub-tiles for coherent rays.  Step-cap overruns are
// counted.  GRID: the volume has a block grid.
template <bool MIXED, bool GRID, int TX, int TY>
__device__ inline void raycast_tile(const VolumeDev& v, const DSensor& s,
                                    const float* __restrict__ pose16, float* __restrict__ depth_out,
                                    uint8_t* __restrict__ rgb_out, int bx, int by,
                                    const unsigned* __restrict__ rbound, int tiles_x) {
  static_assert(TX % 8 == 0 && TY % 4 == 0, "tile of 8x4 warps");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x = bx * TX + (warp % (TX / 8)) * 8 + (lane & 7);
  const int y = by * TY + (warp / (TX / 8)) * 4 + (lane >> 3);
  if (x >= s.cols || y >= s.rows) return;
  M4f T;  // the pose in registers for the whole march
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float4 r = __ldg(reinterpret_cast<const float4*>(pose16) + k);
    T.m[4 * k] = r.x;
    T.m[4 * k + 1] = r.y;
    T.m[4 * k + 2] = r.z;
    T.m[4 * k + 3] = r.w;
  }
  float skip_to = 0.0f, skip_far = 3.402823466e+38f;
  if (rbound) {
    const int tx = x / kRbTile, ty = y / kRbTile;
    const RayBounds B =
        ray_bounds(const_cast<unsigned*>(rbound), tiles_x, (s.rows + kRbTile - 1) / kRbTile);
    const int f = ty * tiles_x + tx, c = (ty / kRbCoarse) * B.cx + tx / kRbCoarse;
    skip_to = fminf(__uint_as_float(B.near8[f]), __uint_as_float(B.near64[c]));
    skip_far = fmaxf(__uint_as_float(B.far8[f]), __uint_as_float(B.far64[c]));
  }
  bool over;
  if (MIXED) {
    const bool free = v.freecell != nullptr;
    if (GRID)
      over = free ? raycast_px<true>(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out)
                  : raycast_px<false>(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out);
    else
      over = free ? mixed_hash_march<true>(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out)
                  : mixed_hash_march<false>(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out);
  } else {
    over = GRID ? raycast_exact_px(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out)
                : exact_hash_march(v, s, T, x, y, skip_to, skip_far, depth_out, rgb_out);
  }
  if (over) atomicAdd(&v.cnt->raycast_overruns, 1);
}

template <bool MIXED, bool GRID>
__global__ void __launch_bounds__(256)
    raycast_kernel(const __grid_constant__ VolumeDev v, const __grid_constant__ DSensor s,
                   const PoseState* __restrict__ ps, const float* __restrict__ pose_override,
                   float* __restrict__ depth_out, uint8_t* __restrict__ rgb_out) {
  raycast_tile<MIXED, GRID, 16, 16>(v, s, pose_override ? pose_override : ps->posef, depth_out, rgb_out,
                                    blockIdx.x, blockIdx.y, nullptr, 0);
}

// next frame's target of every mode-1 session (blockIdx.z) at its new pose;
// one instantiation per voxel form and march, through the block grid or the
// hash (other sessions return), and per tile shape (every pixel's march is
// independent of the tiling)
// (at least 1024 threads resident per SM: the march waits on its own loads --
// grid entry, voxel, corners -- and issues in 67 % of the cycles, and 4 CTAs of
// 256 hide more of it than the 3 that 76 registers allow.  A persistent launch
// whose warps fetch 8x4 tiles from an even sample of the image balanced the
// SMs but spilled in the loop: 272 against 253 us.  All nine loads of a sample
// issued together: 275 against 265 us, the weight test saves more.)
template <bool MIXED, bool GRID, int TX, int TY>
__global__ void __launch_bounds__(TX* TY, 1024 / (TX * TY))
    fused_raycast_kernel(const SessDev* __restrict__ tab) {
  const SessDev& S = tab[blockIdx.z];
  if (S.mode != 1 || (S.vol.fp16 != 0) != MIXED || (S.vol.grid != nullptr) != GRID) return;
  const DSensor& s = S.ls[0];
  if ((int)blockIdx.x * TX >= s.cols || (int)blockIdx.y * TY >= s.rows) return;
  uint8_t* rgb_out = S.use_color ? S.trgb : nullptr;
  raycast_tile<MIXED, GRID, TX, TY>(S.vol, s, S.pose->posef, S.ray, rgb_out, blockIdx.x,
                                    blockIdx.y, S.rbound, S.rb_tx);
}

template <int TX, int TY>
void launch_fused_raycast(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  dim3 grid((b.max_cols + TX - 1) / TX, (b.max_rows + TY - 1) / TY, b.n);
  if (b.ray_mask & 1) fused_raycast_kernel<false, false, TX, TY><<<grid, TX * TY, 0, st>>>(tab);
  if (b.ray_mask & 2) fused_raycast_kernel<true, false, TX, TY><<<grid, TX * TY, 0, st>>>(tab);
  if (b.ray_mask & 4) fused_raycast_kernel<false, true, TX, TY><<<grid, TX * TY, 0, st>>>(tab);
  if (b.ray_mask & 8) fused_raycast_kernel<true, true, TX, TY><<<grid, TX * TY, 0, st>>>(tab);
}

__global__ void clear_entries_kernel(Entry* e, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Entry z;
  z.key = kEmptyKey;
  z.ptr = -1;
  z.stamp = -1;
  e[i] = z;
}

__global__ void block_coords_kernel(VolumeDev v, int n, int* coords) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long k = v.block_keys[i];
  coords[3 * i] = key_x(k);
  coords[3 * i + 1] = key_y(k);
  coords[3 * i + 2] = key_z(k);
}

__global__ void find_blocks_kernel(VolumeDev v, const int* __restrict__ coords, int n,
                                   int* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = find_block(v.entries, v.t, coords[3 * i], coords[3 * i + 1], coords[3 * i + 2]);
  out[i] = (p >= 0 && p < v.t.num_blocks) ? p : -1;
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

void launch_volume_clear(const VolumeDev& v, cudaStream_t st) {
  size_t ne = (size_t)v.t.num_buckets * v.t.bucket_size;
  clear_entries_kernel<<<nblk((long long)ne, 256), 256, 0, st>>>(v.entries, ne);
  const size_t nv = ((size_t)v.t.num_blocks + 1) * kBlockVox;  // and the empty block
  if (v.voxels) cudaMemsetAsync(v.voxels, 0, sizeof(dyn_voxel) * nv, st);
  if (v.vox16) cudaMemsetAsync(v.vox16, 0, sizeof(unsigned) * nv, st);
  if (v.colors) cudaMemsetAsync(v.colors, 0, sizeof(uchar4) * nv, st);
  if (v.nonsat) cudaMemsetAsync(v.nonsat, 0, sizeof(int) * (size_t)v.t.num_blocks, st);
  if (v.freecell) cudaMemsetAsync(v.freecell, 0, (size_t)v.t.num_blocks, st);
  cudaMemsetAsync(v.cnt, 0, sizeof(Counters), st);
}

void launch_raycast(const VolumeDev& v, const DSensor& s, const PoseState* ps,
                    const float* pose_override, float* depth_out, uint8_t* rgb_out,
                    bool use_grid, cudaStream_t st) {
  if (use_grid) {
    grid_clear_kernel<<<148 * 4, 256, 0, st>>>(v, s, pose_override ? pose_override : ps->posef);
    grid_fill_kernel<<<148 * 4, 256, 0, st>>>(v);
  }
  const dim3 grid(nblk(s.cols, 16), nblk(s.rows, 16));
  const auto kernel = v.fp16 ? (use_grid ? raycast_kernel<true, true> : raycast_kernel<true, false>)
                             : (use_grid ? raycast_kernel<false, true> : raycast_kernel<false, false>);
  kernel<<<grid, 256, 0, st>>>(v, s, ps, pose_override, depth_out, rgb_out);
}

void launch_block_coords(const VolumeDev& v, int n, int* coords, cudaStream_t st) {
  if (n > 0) block_coords_kernel<<<nblk(n, 256), 256, 0, st>>>(v, n, coords);
}

void launch_find_blocks(const VolumeDev& v, const int* coords, int n, int* ptr_out,
                        cudaStream_t st) {
  if (n > 0) find_blocks_kernel<<<nblk(n, 256), 256, 0, st>>>(v, coords, n, ptr_out);
}

// ---- fused stages
void fused_allocate(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  const int tx = nblk(b.max_cols, kAllocX), ty = nblk(b.max_rows, kAllocY);
  // about two CTAs per SM for the grids (enough for their writes)
  const int extra = b.max_grid > 0 ? nblk(std::max(8, 148 * 2 / b.n), tx) : 0;
  const dim3 grid(tx, ty + extra, b.n);
  if (b.close_mask & 1) fused_allocate_kernel<false><<<grid, kAllocN, 0, st>>>(tab, ty);
  if (b.close_mask & 2) fused_allocate_kernel<true><<<grid, kAllocN, 0, st>>>(tab, ty);
}

// grid-stride over each session's heap; a wave of CTAs in all
static dim3 visible_grid(const BatchShape& b) {
  return dim3(std::min(nblk(b.max_blocks, kVisThreads), std::max(148 * 12 / b.n, 32)), 1, b.n);
}
void fused_visible(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  fused_visible_kernel<<<visible_grid(b), kVisThreads, 0, st>>>(tab, b.gvis, b.gcount);
}

void fused_integrate(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  fused_integrate_kernel<<<b.integrate_ctas > 0 ? b.integrate_ctas : 148 * 8, kIntThreads, 0,
                           st>>>(tab, b.gvis, b.gcount);
}

void fused_free_cells(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  fused_free_cells_kernel<<<148 * 8, 64, 0, st>>>(tab, b.gvis, b.gcount);
  if (b.fp16_mask & 2) {  // mixed sessions: the near ray bound from their summaries
    fused_surface_bound_kernel<<<visible_grid(b), kVisThreads, 0, st>>>(tab);
  }
}

void fused_raycast(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  switch (b.ray_tile) {
    case 1: launch_fused_raycast<32, 8>(tab, b, st); break;
    case 2: launch_fused_raycast<8, 8>(tab, b, st); break;
    default: launch_fused_raycast<16, 16>(tab, b, st); break;
  }
}

}  // namespace dyn
