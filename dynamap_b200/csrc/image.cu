// image.cu -- depth ingest, bilateral filter, 2x pyramid and normal maps.
//
// Reference: include/image/pyramid/pyramid.cu (bilateral :208-252, pyramid
// :49-143), include/image/sensor/rgbdImage.cu (vertex map :23-38, normals
// :126-157), include/solver/gnSolver/gnSolver.cu:457-465 (intensity).
//
// Each stage's arithmetic is one __device__ function, used by a by-value
// kernel (stage entry points) and by a fused kernel that runs the stage for
// every session of a frame in one launch (blockIdx.z = session).
#include "image.cuh"

#include <cmath>
#include <cstdlib>

#include "dyn_exp.h"
#include "sessdev.cuh"

namespace dyn {

namespace {

// gnSolver::Intensity(ColorToFloat(c)), gnSolver.cu:457-459 + utils.h:98-102:
// channel/255 in float, weighted sum in double, result rounded to float.
__device__ inline float intensity_u8(const uint8_t* c) {
  float r = (float)c[0] / 255.0f, g = (float)c[1] / 255.0f, b = (float)c[2] / 255.0f;
  return (float)(0.2126 * (double)r + 0.7152 * (double)g + 0.0722 * (double)b);
}

// pyramid::applyBilateralFilter, pyramid.cu:213-233, window rows x-r..x+r-1,
// cols y-r..y+r-1, summed row-major.  The depth tile plus halo is staged in
// shared memory (0 where outside the image or not > 0: such taps are skipped,
// such centres stay 0); the spatial weights, a pure function of the tap
// offset, come precomputed on the host in double and rounded to float exactly
// as the reference rounds them per tap (read as warp-uniform values).  The
// range weight uses dyn_expf, the same operation sequence the oracle runs, so
// the filtered depth is bit-identical to the oracle's.
// FAST (mixed-precision sessions): each tap's weight in one hardware
// base-2 exponential, gs * exp(-dn^2 / (2 s^2)) = 2^(log2 gs - dn^2 c) with
// c = log2(e) / (2 s^2), the spatial weights staged as their logarithms;
// the range normalisation 1/(2 pi s^2), common to every weight, cancels in
// acc / wp and is left out.
//
// Bound by the FP32 pipe: 15 operations per tap (dyn_expf's polynomial is 7 of
// them), 256 taps per pixel at the reference's diameter.  So everything else
// is kept off the tap:
//  * SMALL: where the depths of the CTA's tile span so little that every tap's
//    exponent rounds to k = 0 (sigma_i 10 m: always), dyn_expf's reduction is
//    the identity and is left out -- the conversions it needs run at an eighth
//    of the FP32 rate;
//  * MASK false: where no staged pixel is invalid, no test per tap;
//  * the taps of a window row unroll (DT the window size, 0: any), so that
//    their weights overlap; only the two sums are serial.
// A call at diameter 8, before -> now: 160x120 43.1 -> 10.3 us, 320x240 45.1 ->
// 15.3, 640x480 78.3 -> 32.9, 1280x720 145 -> 70.7.  Other diameters keep a loop of
// unknown length with the test per tap: 640x480 at 4, 6, 7 and 16 24.8, 47.6, 61.4
// and 278 us before, now 14.4, 25.7, 33.8 and 139.  Two pixels of a column per
// thread, each staged depth read once for both, measured 16, 37 and 72 us from
// 320x240 on: the shared-memory reads are not what it waits for.  (They are in the
// mixed form, whose taps are six operations and an exponential: bilateral_pair.)
constexpr int BTX = 32;

__device__ __host__ inline int bil_pitch(int D) { return BTX + D - 1; }
// Floats before the spatial weights (a multiple of four: they are read as
// vectors).
__device__ __host__ inline int bil_tile_floats(int D, int rows) {
  return (bil_pitch(D) * (rows + D - 1) + 3) / 4 * 4;
}

// exp(x) of dyn_expf for |x log2(e)| <= 1/2, where its k is 0: p * 2^0.
__device__ inline float expf_k0(float r) {
  float p = 1.98412698412698413e-4f;   // the terms of dyn_expf
  p = __fmaf_rn(p, r, 1.38888888888888889e-3f);
  p = __fmaf_rn(p, r, 8.33333333333333333e-3f);
  p = __fmaf_rn(p, r, 4.16666666666666667e-2f);
  p = __fmaf_rn(p, r, 1.66666666666666667e-1f);
  p = __fmaf_rn(p, r, 0.5f);
  p = __fmaf_rn(p, r, 1.0f);
  return __fmaf_rn(p, r, 1.0f);
}

template <bool FAST, bool SMALL, bool MASK, int DT>
__device__ inline float bilateral_sum(const float* __restrict__ t, const float* __restrict__ gs,
                                      int pitch, int D_, float inv2s2, float norm, float c) {
  const int D = DT ? DT : D_;
  const float c2 = inv2s2 * 1.4426950408889634f;  // FAST: log2(e) / (2 s^2)
  float acc = 0.0f, wp = 0.0f;
  auto tap = [&](float nv, float g) {
    const float dn = nv - c;
    float w;
    if (FAST) {
      asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(__fmaf_rn(-(dn * dn), c2, g)));
      if (MASK) w = nv > 0.0f ? w : 0.0f;
      acc = __fmaf_rn(nv, w, acc);
    } else {
      w = (SMALL ? expf_k0(-(dn * dn) * inv2s2) * norm : range_weight(dn, inv2s2, norm)) * g;
      if (MASK) w = nv > 0.0f ? w : 0.0f;
      acc += nv * w;
    }
    wp += w;
  };
#pragma unroll 1
  for (int i = 0; i < D; ++i) {
    const float* tr = t + i * pitch;
    const float* gr = gs + i * D;
    if (DT) {
#pragma unroll
      for (int j = 0; j < DT; j += 4) {
        const float4 g = *reinterpret_cast<const float4*>(gr + j);
        tap(tr[j], g.x);
        tap(tr[j + 1], g.y);
        tap(tr[j + 2], g.z);
        tap(tr[j + 3], g.w);
      }
    } else {
#pragma unroll 2
      for (int j = 0; j < D; ++j) tap(tr[j], gr[j]);
    }
  }
  return acc / wp;
}

// The mixed form's sums of two pixels of a column, each staged depth read once
// for both (window 16 only; each pixel's taps in the same order as above).
template <bool MASK>
__device__ inline void bilateral_pair(const float* __restrict__ t, const float* __restrict__ gs,
                                      int pitch, float inv2s2, const float (&c)[2],
                                      float (&out)[2]) {
  constexpr int D = 16;
  const float c2 = inv2s2 * 1.4426950408889634f;
  float acc[2] = {0.0f, 0.0f}, wp[2] = {0.0f, 0.0f};
  auto tap = [&](float nv, float g, int n) {
    const float dn = nv - c[n];
    float w;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(__fmaf_rn(-(dn * dn), c2, g)));
    if (MASK) w = nv > 0.0f ? w : 0.0f;
    acc[n] = __fmaf_rn(nv, w, acc[n]);
    wp[n] += w;
  };
  // tile row r holds window row r of the first pixel and r - 1 of the second
#pragma unroll 4
  for (int j = 0; j < D; ++j) tap(t[j], gs[j], 0);
#pragma unroll 1
  for (int r = 1; r < D; ++r) {
    const float* tr = t + r * pitch;
    const float* gr = gs + r * D;
#pragma unroll
    for (int j = 0; j < D; j += 4) {
      const float4 g0 = *reinterpret_cast<const float4*>(gr + j);
      const float4 g1 = *reinterpret_cast<const float4*>(gr - D + j);
      const float v[4] = {tr[j], tr[j + 1], tr[j + 2], tr[j + 3]};
      tap(v[0], g0.x, 0);
      tap(v[0], g1.x, 1);
      tap(v[1], g0.y, 0);
      tap(v[1], g1.y, 1);
      tap(v[2], g0.z, 0);
      tap(v[2], g1.z, 1);
      tap(v[3], g0.w, 0);
      tap(v[3], g1.w, 1);
    }
  }
#pragma unroll 4
  for (int j = 0; j < D; ++j) tap(t[D * pitch + j], gs[(D - 1) * D + j], 1);
#pragma unroll
  for (int n = 0; n < 2; ++n) out[n] = acc[n] / wp[n];
}

// One tile of 32 x (blockDim.y * NR) pixels, tile column bx and row by.
template <bool FAST, int NR>
__device__ inline void bilateral_tile(const float* __restrict__ src, float* __restrict__ dst,
                                      int rows, int cols, const BilateralTable& tb, int bx,
                                      int by, float* tile) {
  __shared__ unsigned lo_s, hi_s;
  const int D = 2 * tb.radius, half = tb.radius, TY = blockDim.y * NR;
  const int TW = bil_pitch(D), TH = TY + D - 1;
  float* gs = tile + bil_tile_floats(D, TY);  // the spatial weights, staged once per CTA
  const int tid = threadIdx.y * BTX + threadIdx.x, threads = blockDim.y * BTX;
  if (tid == 0) {
    lo_s = 0xffffffffu;
    hi_s = 0u;
  }
  __syncthreads();
  const int row0 = by * TY - half, col0 = bx * BTX - half;
  unsigned lo = 0xffffffffu, hi = 0u;  // valid depths as bits (positive floats order as theirs)
  bool hole = false;
  for (int tr = threadIdx.y; tr < TH; tr += blockDim.y) {
    const int gr = row0 + tr;
    const bool in = gr >= 0 && gr < rows;
    for (int tc = threadIdx.x; tc < TW; tc += BTX) {
      const int gc = col0 + tc;
      float d = (in && gc >= 0 && gc < cols) ? src[gr * cols + gc] : 0.0f;
      if (!(d > 0.0f)) {
        d = 0.0f;
        hole = true;
      } else {
        lo = min(lo, __float_as_uint(d));
        hi = max(hi, __float_as_uint(d));
      }
      tile[tr * TW + tc] = d;
    }
  }
  for (int k = tid; k < D * D; k += threads) gs[k] = FAST ? __log2f(tb.gs[k]) : tb.gs[k];
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (threadIdx.x == 0 && hi) {
    atomicMin(&lo_s, lo);
    atomicMax(&hi_s, hi);
  }
  const bool mask = __syncthreads_or(hole) != 0;
  const int y = bx * BTX + threadIdx.x;  // column
  if (y >= cols) return;
  if (NR == 2 && D == 16) {
    const int x = by * TY + 2 * threadIdx.y;
    const float* t = tile + 2 * (int)threadIdx.y * TW + threadIdx.x;
    const float c[2] = {t[half * TW + half], t[(half + 1) * TW + half]};
    float out[2] = {0.0f, 0.0f};
    if (c[0] > 0.0f || c[1] > 0.0f) {
      if (mask)
        bilateral_pair<true>(t, gs, TW, tb.inv2s2, c, out);
      else
        bilateral_pair<false>(t, gs, TW, tb.inv2s2, c, out);
    }
    if (x < rows) dst[x * cols + y] = c[0] > 0.0f ? out[0] : 0.0f;
    if (x + 1 < rows) dst[(x + 1) * cols + y] = c[1] > 0.0f ? out[1] : 0.0f;
    return;
  }
#pragma unroll 1
  for (int n = 0; n < NR; ++n) {
    const int row = (int)threadIdx.y + n * blockDim.y;
    const int x = by * TY + row;  // row (the reference's x)
    if (x >= rows) return;
    const float* t = tile + row * TW + threadIdx.x;
    const float c = t[half * TW + half];
    float out = 0.0f;
    if (c > 0.0f) {
      // the largest |exponent| of the tile's taps, by the taps' own (monotone)
      // operations
      const float span = __uint_as_float(hi_s) - __uint_as_float(lo_s);
      const float i2 = tb.inv2s2, nm = tb.norm;
      if (!FAST && !(span * span * i2 * 1.44269504088896341f <= 0.5f))
        out = bilateral_sum<FAST, false, true, 0>(t, gs, TW, D, i2, nm, c);
      else if (D != 16)
        out = bilateral_sum<FAST, true, true, 0>(t, gs, TW, D, i2, nm, c);
      else if (mask)
        out = bilateral_sum<FAST, true, true, 16>(t, gs, TW, D, i2, nm, c);
      else
        out = bilateral_sum<FAST, true, false, 16>(t, gs, TW, D, i2, nm, c);
    }
    dst[x * cols + y] = out;
  }
}

__global__ void bilateral_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                 int rows, int cols, const __grid_constant__ BilateralTable tb) {
  extern __shared__ float4 smem4[];
  bilateral_tile<false, 1>(src, dst, rows, cols, tb, blockIdx.x, blockIdx.y,
                        reinterpret_cast<float*>(smem4));
}

// One 2x pyramid step: mean of the valid depths of each 2x2 cell (fix of
// pyramid.cu:49-82, which scatters into a fixed 640x480 window).
__device__ inline float mean_valid(float a, float b, float c, float d) {
  const float v[4] = {a, b, c, d};
  float s = 0.0f;
  int n = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (v[k] > 0.0f) {
      s += v[k];
      n++;
    }
  // s / n: a half and a quarter are exact as products, a third by its reciprocal
  if (n == 3) {
    const float yh = 1.0f / 3.0f;
    return moderate(s) ? div_by(s, 3.0f, yh, fmaf(-3.0f, yh, 1.0f) * yh) : s / 3.0f;
  }
  return s * (n == 4 ? 0.25f : (n == 2 ? 0.5f : 1.0f));
}
__device__ inline float mean4(float a, float b, float c, float d) {
  return (((a + b) + c) + d) * 0.25f;
}

// creatPointCloudKernel (rgbdImage.cu:23-38) and vertextoNormal
// (rgbdImage.cu:126-145): n = normalize(cross(V(u+2)-V(u-2), V(v+1)-V(v-1))).
// Vertices are recomputed from depth, so neighbours need no vertex map.  A
// normal is 0 when the centre or a neighbour is invalid or outside the
// row/image.
//
// The quotients by the focal lengths go through their reciprocals with an exact
// correction (div_by) where no step can leave the normal range, else through
// IEEE division.
// (LevelCamera::ok: an offset u - cx is 0 or at least 2^-24 then.)
__device__ inline F3 camera_point(const LevelCamera& c, int u, int v, float d, bool fast) {
  if (!fast) return point3d_uv(u, v, d, c.s);
  const float a = ((float)u - c.s.cx) * d, b = ((float)v - c.s.cy) * d;
  return f3(div_by(a, c.s.fx, c.yhx, c.ylx), div_by(b, c.s.fy, c.yhy, c.yly), d);
}

// The normal of pixel (x, y), whose depth is d[0] in rows of 'pitch' floats
// (neighbours are read only inside the level).
__device__ inline float4 normal_at(const float* d, int pitch, const LevelCamera& c, int x, int y) {
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!(d[0] > 0.0f) || x < 2 || x + 2 >= c.s.cols || y < 1 || y + 1 >= c.s.rows) return none;
  const float dl = d[-2], dr = d[2], du = d[-pitch], dd = d[pitch];
  if (!(dl > 0.0f && dr > 0.0f && du > 0.0f && dd > 0.0f)) return none;
  const bool fast = c.ok && fminf(fminf(dl, dr), fminf(du, dd)) >= kModerateMin &&
                    fmaxf(fmaxf(dl, dr), fmaxf(du, dd)) <= kModerateMax;
  const F3 left = camera_point(c, x - 2, y, dl, fast), right = camera_point(c, x + 2, y, dr, fast);
  const F3 up = camera_point(c, x, y - 1, du, fast), down = camera_point(c, x, y + 1, dd, fast);
  const F3 k = cross3(right - left, down - up);
  const float k2 = dot3(k, k);
  if (!(k2 > 0.0f)) return none;
  const F3 n = k * (1.0f / sqrtf(k2));
  return make_float4(n.x, n.y, n.z, 0.0f);
}

// one level, a tile of 256 pixels per CTA (launch_maps; the stage entry points:
// little more than a launch, 6.1 us at 640x480 as without the tiles)
constexpr int kMapThreads = 256;
__global__ void __launch_bounds__(kMapThreads)
    maps_kernel(const float* __restrict__ depth, float4* __restrict__ normal,
                float4* __restrict__ vertex, const LevelCamera c) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= c.s.cols || y >= c.s.rows) return;
  const int i = y * c.s.cols + x;
  if (vertex) {
    const float d = depth[i];
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (d > 0.0f) {
      const F3 p = camera_point(c, x, y, d, c.ok && moderate(d));
      v = make_float4(p.x, p.y, p.z, 1.0f);
    }
    vertex[i] = v;
  }
  normal[i] = normal_at(depth + i, c.s.cols, c, x, y);
}

// raycast depth with its misses invalid
__global__ void miss_to_zero_kernel(const float* __restrict__ ray, float* __restrict__ d0,
                                    float dmax, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float d = ray[i];
  d0[i] = (d < dmax) ? d : 0.0f;
}

// ---------------------------------------------------------------- fused
// ingest: u16 sensor units -> metres (builder.cu:111, utils_Dataset.cpp:233-235;
// + the unfiltered copy when the bilateral filter is off), and what
// integration reads per voxel that projects to a pixel: the distance from the
// camera centre to the pixel's back-projected point (IntegrateScanKernel's
// |getPoint3d(pixel, depth)|, tsdf.cu:316-317 -- it depends only on the pixel,
// the same operations so the same bits; by the band form's approximate
// operations for band sessions), NaN where the depth is outside the sensor
// range (every comparison then fails, as the reference's range test does) and
// negative where it is the range's end (the reference's band test excludes it);
// and the packed colour.
__device__ inline float pixel_distance(int x, int y, float d, const DSensor& s, const DTsdf& t) {
  if (d < t.dmin || d > t.dmax) return __int_as_float(0x7fffffff);
  float sd;
  if (t.band) {
    const F3 p = f3(__fdividef(((float)x - s.cx) * d, s.fx), __fdividef(((float)y - s.cy) * d, s.fy), d);
    const float q = __fmaf_rn(p.x, p.x, __fmaf_rn(p.y, p.y, p.z * p.z));
    sd = q > 0.0f ? q * rsqrtf(q) : 0.0f;
  } else {
    sd = norm3(point3d_uv(x, y, d, s));
  }
  return d < t.dmax ? sd : -sd;
}

// A 32x8 pixel tile per CTA (four fine tiles of the ray bounds), which also
//  * resets the frame's counters, its visible list and its ray depth bounds
//    (near: no block, or 0 where unused; far: no block);
//  * builds the free-space tile map of a depth-only frame of a carving session:
//    per fine tile the least (sdist - truncation), 0 where a pixel's depth is
//    outside the sensor range, and its minimum per coarse tile.  The coarse map
//    is one of two by the frame's parity; each frame empties the other one.
// Bound by latency (the pointers, a pixel's load, a division).  As three
// kernels, the map's with a thread per tile, this took 31 us of a 320x240
// frame, now 12-15; 19.4 -> 15 of a 640x480 one with colours.
__global__ void __launch_bounds__(256) fused_ingest_kernel(const SessDev* __restrict__ tab,
                                                           int* __restrict__ gcount) {
  const SessDev& S = tab[blockIdx.z];
  const DSensor& s0 = S.ls[0];
  const DTsdf& t = S.vol.t;
  if ((int)blockIdx.x * 32 >= s0.cols || (int)blockIdx.y * 8 >= s0.rows) return;
  __shared__ unsigned least[4];
  const int lane = threadIdx.x & 31, tid = threadIdx.x;
  const int x = blockIdx.x * 32 + lane, y = blockIdx.y * 8 + (tid >> 5);
  const bool in = x < s0.cols && y < s0.rows;
  const int i = y * s0.cols + x;
  const unsigned raw = in ? S.u16[i] : 0u;
  const uint8_t* rgb = *S.rgb_flag ? S.rgb : nullptr;
  const bool free_map = S.ftile && !t.band && !rgb;
  const int parity = S.pose->frame & 1;
  if (tid < 4) least[tid] = 0x7f7f7f7fu;
  unsigned word = 0x7f7f7f7fu;
  if (in) {
    const float d = (float)raw / S.depth_scaler;
    const float sd = pixel_distance(x, y, d, s0, t);
    if (S.use_color) S.sint[0][i] = rgb ? intensity_u8(rgb + 3 * (size_t)i) : 0.0f;
    if (rgb) {
      const uint8_t* c = rgb + 3 * (size_t)i;
      S.rgb4[i] = (unsigned)c[0] | ((unsigned)c[1] << 8) | ((unsigned)c[2] << 16);
    }
    S.raw[i] = d;
    if (!S.bil_enabled) S.filt[i] = d;
    S.sdist[i] = sd;
    const float room = fabsf(sd) - t.trunc;  // NaN: outside the range
    word = room > 0.0f ? __float_as_uint(room) : 0u;
  }
  const int tx0 = blockIdx.x * 4, ty = blockIdx.y;
  const int cx = (S.rb_tx + kRbCoarse - 1) / kRbCoarse, cy = (S.rb_ty + kRbCoarse - 1) / kRbCoarse;
  unsigned* const coarse = S.ftile ? S.ftile + S.rb_tx * S.rb_ty : nullptr;
  if (free_map) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) word = min(word, __shfl_xor_sync(0xffffffffu, word, o));
    __syncthreads();
    if ((lane & 7) == 0) atomicMin(&least[lane >> 3], word);
    __syncthreads();
  }
  if (tid < 4 && tx0 + tid < S.rb_tx) {
    const int tx = tx0 + tid, i = ty * S.rb_tx + tx;
    const bool near_used = t.band || (S.vol.nonsat && S.vol.free_ok);
    const unsigned nb = near_used ? 0x7f7f7f7fu : 0u;
    const int c = (ty / kRbCoarse) * cx + tx / kRbCoarse;
    const bool first = tx % kRbCoarse == 0 && ty % kRbCoarse == 0;
    if (S.rbound) {
      unsigned* const n8 = S.rbound;
      unsigned* const n64 = n8 + 2 * S.rb_tx * S.rb_ty;
      n8[i] = nb;
      n8[S.rb_tx * S.rb_ty + i] = 0u;
      if (first) {
        n64[c] = nb;
        n64[cx * cy + c] = 0u;
      }
    }
    if (free_map) {
      S.ftile[i] = least[tid];
      atomicMin(coarse + parity * cx * cy + c, least[tid]);
    }
    if (coarse && first) coarse[(parity ^ 1) * cx * cy + c] = 0x7f7f7f7fu;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 4) {
    if (blockIdx.z == 0) *gcount = 0;
    Counters* c = S.vol.cnt;  // all but nalloc, the heap top
    c->new_blocks = 0;
    c->bucket_full = 0;
    c->heap_exhausted = 0;
    c->dda_overruns = 0;
    c->raycast_overruns = 0;
    c->visible = 0;
    c->unique_probed = 0;
    c->icp_timeout = 0;
  }
}

template <int NR>  // rows a thread of the mixed form
__global__ void fused_bilateral_kernel(const SessDev* __restrict__ tab) {
  extern __shared__ float4 smem4[];
  float* tile = reinterpret_cast<float*>(smem4);
  const SessDev& S = tab[blockIdx.z];
  if (!S.bil_enabled) return;
  const int rows = S.ls[0].rows, cols = S.ls[0].cols;
  const int ty = blockDim.y * (S.vol.fp16 ? NR : 1);
  if ((int)blockIdx.x * BTX >= cols || (int)blockIdx.y * ty >= rows) return;
  if (S.vol.fp16)  // mixed-precision session
    bilateral_tile<true, NR>(S.raw, S.filt, rows, cols, *S.btab, blockIdx.x, blockIdx.y, tile);
  else
    bilateral_tile<false, 1>(S.raw, S.filt, rows, cols, *S.btab, blockIdx.x, blockIdx.y, tile);
}

// ---- pyramid and normals of an image in one launch
// A CTA owns 32x16 pixels of level 0 and what lies over them on levels 1 and 2.
// It stages the level-0 depths with the halo that the level-2 normals need (8
// columns, 4 rows), computes the upper levels of the halo again in shared
// memory, and writes its own part of every level and its normals.  A tile this
// small, because the chain of a CTA (loads, three levels, normals) is what a
// frame waits for; six CTAs an SM hide each other's.  With a launch per level
// and one for the normals (four or five per image) a 640x480 frame took 16.4 us
// for the source and 20.6 for the target, now 12.3 and 15; a batch of 32 (8 of
// 160x120, 16 of 320x240, 8 of 640x480) 80 and 110 us, now 62 and 67.  A fourth level (scale 8) is
// made from level 2 by the two kernels below.
//
// what: 0 the frame's source (filtered depth and intensity are there); 1 the
// frame's target: the raycast, misses invalid (mode 1), or the source (mode 0);
// 2, 3 dyn_solver_solve's source (S.raw, colours S.rgb) and target (S.ray,
// S.trgb), colours only with has_rgb.
constexpr int kPyrX = 32, kPyrY = 16, kPyrHX = 8, kPyrHY = 4;
constexpr int kP0W = kPyrX + 2 * kPyrHX, kP0H = kPyrY + 2 * kPyrHY;
constexpr int kP1W = kP0W / 2, kP1H = kP0H / 2, kP2W = kP0W / 4, kP2H = kP0H / 4;
__global__ void __launch_bounds__(256, 6)
    fused_pyramid_kernel(const SessDev* __restrict__ tab, int what, int has_rgb) {
  const SessDev& S = tab[blockIdx.z];
  const DSensor& s0 = S.ls[0];
  const int X0 = blockIdx.x * kPyrX, Y0 = blockIdx.y * kPyrY;
  if (X0 >= s0.cols || Y0 >= s0.rows) return;
  __shared__ float d0[kP0H * kP0W], d1[kP1H * kP1W], d2[kP2H * kP2W];
  __shared__ float i0[kPyrY * kPyrX], i1[kPyrY * kPyrX / 4];
  const int tid = threadIdx.x;
  const bool target = (what & 1) != 0, frame = what < 2;
  const bool copy = what == 1 && S.mode != 1;  // frame-to-frame: the source is the target
  const float* in = what == 0 ? S.sdep[0] : (what == 1 ? (copy ? S.sdep[0] : S.ray)
                                                       : (what == 2 ? S.raw : S.ray));
  const float limit = what == 1 && !copy ? S.vol.t.dmax : 3.402823466e+38f;
  float* const out0 = what == 0 ? nullptr : (target ? S.tdep[0] : S.sdep[0]);
  const int nlev = min(S.nlev, 3);
  if (target && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) S.icp->have_target = 1;
  // all loads before the first store (a store could be to what they read)
  // (a warp per row of the staged depths: 24 rows of 48)
  constexpr int kOwn = kPyrY * kPyrX / 256, kRows = kP0H / 8;
  static_assert(kP0H % 8 == 0 && kP0W > 32 && kP0W <= 64 && kPyrX == 32, "row mapping");
  const int lane = tid & 31, warp = tid >> 5;
  const bool colour = S.use_color != 0, gray = what == 0 || copy;
  const uint8_t* rgb = colour && !gray && (frame || has_rgb) ? (target ? S.trgb : S.rgb) : nullptr;
  float dv[kRows][2], iv[kOwn];
  const int xa = X0 - kPyrHX + lane, xb = xa + 32;
  const bool ina = xa >= 0 && xa < s0.cols, inb = lane < kP0W - 32 && xb < s0.cols;
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    const int y = Y0 - kPyrHY + warp + j * 8;
    const bool iny = y >= 0 && y < s0.rows;
    const float* a = in + y * s0.cols + xa;
    dv[j][0] = ina && iny ? a[0] : 0.0f;
    dv[j][1] = inb && iny ? a[32] : 0.0f;
  }
#pragma unroll
  for (int j = 0; j < kOwn; ++j) {
    const int y = Y0 + warp + j * 8, x = X0 + lane, i = y * s0.cols + x;
    iv[j] = 0.0f;
    if (colour && x < s0.cols && y < s0.rows)
      iv[j] = gray ? S.sint[0][i] : (rgb ? intensity_u8(rgb + 3 * (size_t)i) : 0.0f);
  }
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    const int r = warp + j * 8, y = Y0 - kPyrHY + r;
    float a = dv[j][0], b = dv[j][1];
    if (what != 0 && !copy) {
      a = a < limit ? a : 0.0f;
      b = b < limit ? b : 0.0f;
    }
    d0[r * kP0W + lane] = a;
    if (lane < kP0W - 32) d0[r * kP0W + 32 + lane] = b;
    if (out0 && r >= kPyrHY && r < kPyrHY + kPyrY && y < s0.rows) {
      if (lane >= kPyrHX && xa < s0.cols) out0[y * s0.cols + xa] = a;
      if (lane < kPyrHX && xb < s0.cols) out0[y * s0.cols + xb] = b;
    }
  }
  if (colour) {
#pragma unroll
    for (int j = 0; j < kOwn; ++j) {
      const int k = tid + j * 256, y = Y0 + k / kPyrX, x = X0 + k % kPyrX;
      i0[k] = iv[j];
      if (what != 0 && x < s0.cols && y < s0.rows)
        (target ? S.tint[0] : S.sint[0])[y * s0.cols + x] = iv[j];
    }
  }
  __syncthreads();
  if (nlev > 1) {
    const DSensor& s = S.ls[1];
    for (int r = warp, c = lane; r < kP1H && c < kP1W; r += 8) {
      const int y = Y0 / 2 - kPyrHY / 2 + r, x = X0 / 2 - kPyrHX / 2 + c;
      float d = 0.0f;
      if (x >= 0 && y >= 0 && x < s.cols && y < s.rows) {
        const float* a = d0 + 2 * r * kP0W + 2 * c;
        d = mean_valid(a[0], a[1], a[kP0W], a[kP0W + 1]);
        if (r >= kPyrHY / 2 && r < (kPyrHY + kPyrY) / 2 && c >= kPyrHX / 2 && c < (kPyrHX + kPyrX) / 2)
          (target ? S.tdep[1] : S.sdep[1])[y * s.cols + x] = d;
      }
      d1[r * kP1W + c] = d;
    }
    if (colour && tid < kPyrY * kPyrX / 4) {
      const int r = tid / (kPyrX / 2), c = tid % (kPyrX / 2), y = Y0 / 2 + r, x = X0 / 2 + c;
      const float* a = i0 + 2 * r * kPyrX + 2 * c;
      const float v = mean4(a[0], a[1], a[kPyrX], a[kPyrX + 1]);
      i1[tid] = v;
      if (x < s.cols && y < s.rows) (target ? S.tint[1] : S.sint[1])[y * s.cols + x] = v;
    }
    __syncthreads();
  }
  if (nlev > 2) {
    const DSensor& s = S.ls[2];
    if (tid < kP2H * kP2W) {
      const int r = tid / kP2W, c = tid - r * kP2W;
      const int y = Y0 / 4 - kPyrHY / 4 + r, x = X0 / 4 - kPyrHX / 4 + c;
      float d = 0.0f;
      if (x >= 0 && y >= 0 && x < s.cols && y < s.rows) {
        const float* a = d1 + 2 * r * kP1W + 2 * c;
        d = mean_valid(a[0], a[1], a[kP1W], a[kP1W + 1]);
        if (r >= kPyrHY / 4 && r < (kPyrHY + kPyrY) / 4 && c >= kPyrHX / 4 && c < (kPyrHX + kPyrX) / 4)
          (target ? S.tdep[2] : S.sdep[2])[y * s.cols + x] = d;
      }
      d2[tid] = d;
    } else if (colour && tid >= 128 && tid < 128 + kPyrY * kPyrX / 16) {
      const int k = tid - 128, r = k / (kPyrX / 4), c = k % (kPyrX / 4);
      const int y = Y0 / 4 + r, x = X0 / 4 + c;
      const float* a = i1 + 2 * r * (kPyrX / 2) + 2 * c;
      if (x < s.cols && y < s.rows)
        (target ? S.tint[2] : S.sint[2])[y * s.cols + x] =
            mean4(a[0], a[1], a[kPyrX / 2], a[kPyrX / 2 + 1]);
    }
    __syncthreads();
  }
  // normals: level 0, then the upper levels by the threads it leaves
  float4* const* nrm = target ? S.tnrm : S.snrm;
  {
    const LevelCamera& c = S.cam[0];
#pragma unroll
    for (int k = 0; k < kPyrY * kPyrX; k += 256) {
      const int r = (k + tid) / kPyrX, q = (k + tid) % kPyrX, y = Y0 + r, x = X0 + q;
      if (x < s0.cols && y < s0.rows)
        nrm[0][y * s0.cols + x] =
            normal_at(d0 + (r + kPyrHY) * kP0W + q + kPyrHX, kP0W, c, x, y);
    }
  }
  if (nlev > 1 && tid < kPyrY * kPyrX / 4) {
    const LevelCamera& c = S.cam[1];
    const int r = tid / (kPyrX / 2), q = tid % (kPyrX / 2), y = Y0 / 2 + r, x = X0 / 2 + q;
    if (x < c.s.cols && y < c.s.rows)
      nrm[1][y * c.s.cols + x] =
          normal_at(d1 + (r + kPyrHY / 2) * kP1W + q + kPyrHX / 2, kP1W, c, x, y);
  } else if (nlev > 2 && tid >= 128 && tid < 128 + kPyrY * kPyrX / 16) {
    const LevelCamera& c = S.cam[2];
    const int k = tid - 128, r = k / (kPyrX / 4), q = k % (kPyrX / 4);
    const int y = Y0 / 4 + r, x = X0 / 4 + q;
    if (x < c.s.cols && y < c.s.rows)
      nrm[2][y * c.s.cols + x] =
          normal_at(d2 + (r + kPyrHY / 4) * kP2W + q + kPyrHX / 4, kP2W, c, x, y);
  }
}

// level 3 of the sessions that have it, from level 2; then its normals
__global__ void fused_level3_kernel(const SessDev* __restrict__ tab, int target) {
  const SessDev& S = tab[blockIdx.z];
  if (S.nlev < 4) return;
  const DSensor &s = S.ls[3], &p = S.ls[2];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.rows * s.cols) return;
  const int y = i / s.cols, x = i - y * s.cols, j = 2 * y * p.cols + 2 * x;
  const float* a = (target ? S.tdep[2] : S.sdep[2]) + j;
  (target ? S.tdep[3] : S.sdep[3])[i] = mean_valid(a[0], a[1], a[p.cols], a[p.cols + 1]);
  if (S.use_color) {
    const float* b = (target ? S.tint[2] : S.sint[2]) + j;
    (target ? S.tint[3] : S.sint[3])[i] = mean4(b[0], b[1], b[p.cols], b[p.cols + 1]);
  }
}
__global__ void fused_level3_normals_kernel(const SessDev* __restrict__ tab, int target) {
  const SessDev& S = tab[blockIdx.z];
  if (S.nlev < 4) return;
  const LevelCamera& c = S.cam[3];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.s.rows * c.s.cols) return;
  const int y = i / c.s.cols, x = i - y * c.s.cols;
  (target ? S.tnrm[3] : S.snrm[3])[i] =
      normal_at((target ? S.tdep[3] : S.sdep[3]) + i, c.s.cols, c, x, y);
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

// pyramid::gaussian, pyramid.cu:208-211, in double.
static double gaussian_d(double x, double sigma) {
  return std::exp(-(std::pow(x, 2)) / (2 * std::pow(sigma, 2))) /
         (2 * 3.14159265358979323846 * std::pow(sigma, 2));
}

BilateralTable make_bilateral_table(int radius, float sigma_i, float sigma_s) {
  BilateralTable tb;
  tb.radius = radius;
  const int D = 2 * radius, half = radius;
  // vertexDistance (pyramid.cu:201-206) in float, gaussian in double; a
  // weight depends on the offsets' magnitudes alone, in either order: 45
  // exponentials instead of 256 at radius 8 (the table is made per call:
  // 8.0 -> 2.0 us of host time there)
  float w[17][17];
  for (int i = 0; i <= half; ++i)
    for (int j = 0; j <= i; ++j) {
      const float dx = (float)i, dy = (float)j;
      const float dd = std::sqrt(dx * dx + dy * dy + 0.0f * 0.0f);
      w[i][j] = w[j][i] = (float)gaussian_d((double)dd, (double)sigma_s);
    }
  for (int i = 0; i < D; ++i)
    for (int j = 0; j < D; ++j) tb.gs[i * D + j] = w[std::abs(half - i)][std::abs(half - j)];
  double si = (double)sigma_i;
  tb.inv2s2 = (float)(1.0 / (2.0 * si * si));
  tb.norm = (float)(1.0 / (2.0 * 3.14159265358979323846 * si * si));
  return tb;
}

// depth tile with its halo, then the D x D spatial weights
static size_t bilateral_smem(int radius, int rows) {
  const int D = 2 * radius;
  return sizeof(float) * ((size_t)bil_tile_floats(D, rows) + (size_t)D * D);
}
// Rows of a CTA's tile: 8 stage less halo per pixel, 4 balance small images
// over the SMs (453x340: 20.2 us with 4, 23.4 with 8; 640x480: 35.1 and 32.6).
static int bilateral_rows(long long cols, long long rows, int n) {
  return (cols + BTX - 1) / BTX * ((rows + 7) / 8) * n >= 6 * 148 ? 8 : 4;
}

void launch_bilateral(const float* src, float* dst, int rows, int cols, const BilateralTable& tb,
                      cudaStream_t st) {
  const int ty = bilateral_rows(cols, rows, 1);
  bilateral_kernel<<<dim3(nblk(cols, BTX), nblk(rows, ty)), dim3(BTX, ty),
                     bilateral_smem(tb.radius, ty), st>>>(src, dst, rows, cols, tb);
}

// Tiles as wide as leave at most a quarter of the threads' columns outside the
// image: 128x2 (a row's vectors in one piece), 32x8 or 8x32.
void launch_maps(const float* depth, const DSensor& s, float4* normal, float4* vertex,
                 cudaStream_t st) {
  int tx = 128;
  while (tx > 8 && 4 * (nblk(s.cols, tx) * tx - s.cols) > s.cols) tx /= 4;
  const int ty = kMapThreads / tx;
  maps_kernel<<<dim3(nblk(s.cols, tx), nblk(s.rows, ty)), dim3(tx, ty), 0, st>>>(
      depth, normal, vertex, level_camera(s));
}
void launch_miss_to_zero(const float* ray_depth, float* depth0, float dmax, int n,
                         cudaStream_t st) {
  miss_to_zero_kernel<<<nblk(n, 256), 256, 0, st>>>(ray_depth, depth0, dmax, n);
}

// ---- fused stages
void fused_ingest(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  fused_ingest_kernel<<<dim3(nblk(b.max_cols, 32), nblk(b.max_rows, 8), b.n), 256, 0, st>>>(
      tab, b.gcount);
}

void fused_bilateral(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  if (b.max_bil_radius <= 0) return;
  const int ty = bilateral_rows(b.max_cols, b.max_rows, b.n);
  // Two pixels a thread for tables of mixed sessions alone of that size (one frame,
  // with / without: 560x420 24.5 / 26.1 us, 592x444 26.4 / 27.9, 640x480 26.7 /
  // 28.6, 720x540 32.7 / 30.4, 1280x720 47.2 / 52.3; a batch of 32, 8 of 160x120, 16
  // of 320x240 and 8 of 640x480, 177 / 213, where the exponentials take 211 were
  // every pixel valid).  An FP32 session's tile has no use for it, so a table with
  // one keeps the rows of its own.
  const dim3 threads(BTX, ty);
  if (ty == 8 && b.fp16_mask == 2) {
    fused_bilateral_kernel<2><<<dim3(nblk(b.max_cols, BTX), nblk(b.max_rows, 2 * ty), b.n), threads,
                                bilateral_smem(b.max_bil_radius, 2 * ty), st>>>(tab);
    return;
  }
  fused_bilateral_kernel<1><<<dim3(nblk(b.max_cols, BTX), nblk(b.max_rows, ty), b.n), threads,
                              bilateral_smem(b.max_bil_radius, ty), st>>>(tab);
}

void fused_pyramid(const SessDev* tab, const BatchShape& b, int what, int has_rgb,
                   cudaStream_t st) {
  fused_pyramid_kernel<<<dim3(nblk(b.max_cols, kPyrX), nblk(b.max_rows, kPyrY), b.n), 256, 0,
                         st>>>(tab, what, has_rgb);
  if (b.max_nlev > 3 && b.max_level_px[3] > 0) {
    const dim3 grid(nblk(b.max_level_px[3], 256), 1, b.n);
    fused_level3_kernel<<<grid, 256, 0, st>>>(tab, what & 1);
    fused_level3_normals_kernel<<<grid, 256, 0, st>>>(tab, what & 1);
  }
}

}  // namespace dyn
