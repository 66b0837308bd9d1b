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
#include <cstring>

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

// u16 sensor units -> metres (builder.cu:111, utils_Dataset.cpp:233-235)
__device__ inline void ingest_px(const uint16_t* __restrict__ raw, const uint8_t* __restrict__ rgb,
                                 float scaler, float* __restrict__ depth,
                                 float* __restrict__ inten, int i) {
  depth[i] = (float)raw[i] / scaler;
  if (inten) inten[i] = rgb ? intensity_u8(rgb + 3 * (size_t)i) : 0.0f;
}

__global__ void ingest_kernel(const uint16_t* __restrict__ raw,
                              const uint8_t* __restrict__ rgb, int n, float scaler,
                              float* __restrict__ depth, float* __restrict__ inten) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ingest_px(raw, rgb, scaler, depth, inten, i);
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
// A call at diameter 8, before -> now: 160x120 43.3 -> 12.4 us (the kernel 8),
// 320x240 45 -> 14, 640x480 80 -> 33, 1280x720 146 -> 71.  Two pixels of a
// column per thread, each staged depth read once for both, measured 16, 37 and
// 72 us: the shared-memory reads are not what it waits for.
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

// One tile of 32 x blockDim.y pixels, tile column bx and row by.
template <bool FAST>
__device__ inline void bilateral_tile(const float* __restrict__ src, float* __restrict__ dst,
                                      int rows, int cols, const BilateralTable& tb, int bx,
                                      int by, float* tile) {
  __shared__ unsigned lo_s, hi_s;
  const int D = 2 * tb.radius, half = tb.radius, TY = blockDim.y;
  const int TW = bil_pitch(D), TH = TY + D - 1;
  float* gs = tile + bil_tile_floats(D, TY);  // the spatial weights, staged once per CTA
  const int tid = threadIdx.y * BTX + threadIdx.x, threads = TY * BTX;
  if (tid == 0) {
    lo_s = 0xffffffffu;
    hi_s = 0u;
  }
  __syncthreads();
  const int row0 = by * TY - half, col0 = bx * BTX - half;
  unsigned lo = 0xffffffffu, hi = 0u;  // valid depths as bits (positive floats order as theirs)
  bool hole = false;
  for (int tr = threadIdx.y; tr < TH; tr += TY) {
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
  const int x = by * TY + threadIdx.y;   // row (the reference's x)
  if (x >= rows || y >= cols) return;
  const float* t = tile + (int)threadIdx.y * TW + threadIdx.x;
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

__global__ void bilateral_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                 int rows, int cols, const __grid_constant__ BilateralTable tb) {
  extern __shared__ float4 smem4[];
  bilateral_tile<false>(src, dst, rows, cols, tb, blockIdx.x, blockIdx.y,
                        reinterpret_cast<float*>(smem4));
}

// One 2x pyramid step: mean of the valid depths of each 2x2 cell (fix of
// pyramid.cu:49-82, which scatters into a fixed 640x480 window).
__device__ inline void downsample_depth_px(const float* __restrict__ src, int cols, int c2,
                                           float* __restrict__ dst, int i) {
  int y = i / c2, x = i - (i / c2) * c2;
  const float* a = src + (2 * y) * cols + 2 * x;
  float v[4] = {a[0], a[1], a[cols], a[cols + 1]};
  float s = 0.0f;
  int n = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (v[k] > 0.0f) {
      s += v[k];
      n++;
    }
  dst[i] = n ? s / (float)n : 0.0f;
}
__device__ inline void downsample_intensity_px(const float* __restrict__ src, int cols, int c2,
                                               float* __restrict__ dst, int i) {
  int y = i / c2, x = i - (i / c2) * c2;
  const float* a = src + (2 * y) * cols + 2 * x;
  dst[i] = (((a[0] + a[1]) + a[cols]) + a[cols + 1]) * 0.25f;
}

__global__ void downsample_depth_kernel(const float* __restrict__ src, int rows, int cols,
                                        float* __restrict__ dst) {
  int c2 = cols / 2, r2 = rows / 2;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= r2 * c2) return;
  downsample_depth_px(src, cols, c2, dst, i);
}

__global__ void downsample_intensity_kernel(const float* __restrict__ src, int rows, int cols,
                                            float* __restrict__ dst) {
  int c2 = cols / 2, r2 = rows / 2;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= r2 * c2) return;
  downsample_intensity_px(src, cols, c2, dst, i);
}

// creatPointCloudKernel (rgbdImage.cu:23-38) and vertextoNormal
// (rgbdImage.cu:126-145): n = normalize(cross(V(u+2)-V(u-2), V(v+1)-V(v-1))).
// Vertices are recomputed from depth, so neighbours need no vertex map.  A
// normal is 0 when the centre or a neighbour is invalid or outside the
// row/image.
__device__ inline void maps_px(const float* __restrict__ depth, float4* __restrict__ normal,
                               float4* __restrict__ vertex, const DSensor& s, int i) {
  const int y = i / s.cols, x = i - y * s.cols;
  float d = depth[i];
  float4 nrm = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!(d > 0.0f)) {
    normal[i] = nrm;
    if (vertex) vertex[i] = nrm;
    return;
  }
  F3 p = point3d_uv(x, y, d, s);
  if (vertex) vertex[i] = make_float4(p.x, p.y, p.z, 1.0f);
  if (x - 2 >= 0 && x + 2 < s.cols && y - 1 >= 0 && y + 1 < s.rows) {
    int il = i - 2, ir = i + 2, iu = i - s.cols, id = i + s.cols;
    float dl = depth[il], dr = depth[ir], du = depth[iu], dd = depth[id];
    if (dl > 0.0f && dr > 0.0f && du > 0.0f && dd > 0.0f) {
      F3 left = point3d_uv(x - 2, y, dl, s), right = point3d_uv(x + 2, y, dr, s);
      F3 up = point3d_uv(x, y - 1, du, s), down = point3d_uv(x, y + 1, dd, s);
      F3 c = cross3(right - left, down - up);
      float dd2 = dot3(c, c);
      if (dd2 > 0.0f) {
        F3 n = c * (1.0f / sqrtf(dd2));
        nrm = make_float4(n.x, n.y, n.z, 0.0f);
      }
    }
  }
  normal[i] = nrm;
}

// all pyramid levels of one image in one launch
__global__ void maps_kernel(MapsArgs a) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= a.total) return;
  int l = 0;
#pragma unroll
  for (int k = 1; k < kLevels; ++k)
    if (k < a.nlev && g >= a.lv[k].offset) l = k;
  const LevelMaps& L = a.lv[l];
  maps_px(L.depth, L.normal, L.vertex, L.s, g - L.offset);
}

__device__ inline void target_prepare_px(const float* __restrict__ ray, float* __restrict__ d0,
                                         float dmax, const uint8_t* __restrict__ rgb,
                                         float* __restrict__ inten, int i) {
  float d = ray[i];
  d0[i] = (d < dmax) ? d : 0.0f;
  if (inten) inten[i] = rgb ? intensity_u8(rgb + 3 * (size_t)i) : 0.0f;
}

__global__ void target_prepare_kernel(const float* __restrict__ ray, float* __restrict__ d0,
                                      float dmax, const uint8_t* __restrict__ rgb,
                                      float* __restrict__ inten, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  target_prepare_px(ray, d0, dmax, rgb, inten, i);
}

// ---------------------------------------------------------------- fused
// ingest (+ the unfiltered copy when the bilateral filter is off), and what
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

__global__ void fused_ingest_kernel(const SessDev* __restrict__ tab) {
  const SessDev& S = tab[blockIdx.z];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.npx) return;
  const uint8_t* rgb = *S.rgb_flag ? S.rgb : nullptr;
  ingest_px(S.u16, rgb, S.depth_scaler, S.raw, S.use_color ? S.sint[0] : nullptr, i);
  if (rgb) {
    const uint8_t* c = rgb + 3 * (size_t)i;
    S.rgb4[i] = (unsigned)c[0] | ((unsigned)c[1] << 8) | ((unsigned)c[2] << 16);
  }
  const float d = S.raw[i];
  if (!S.bil_enabled) S.filt[i] = d;
  const DSensor& s0 = S.ls[0];
  const int y = i / s0.cols;
  S.sdist[i] = pixel_distance(i - y * s0.cols, y, d, s0, S.vol.t);
}

// The free-space tile map of a depth-only frame of a carving session (one
// thread per fine tile; its value also enters its coarse tile's minimum).
__global__ void fused_free_tiles_kernel(const SessDev* __restrict__ tab) {
  const SessDev& S = tab[blockIdx.z];
  if (!S.ftile || S.vol.t.band || *S.rgb_flag) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S.rb_tx * S.rb_ty) return;
  const DSensor& s = S.ls[0];
  const DTsdf& t = S.vol.t;
  const int tx = i % S.rb_tx, ty = i / S.rb_tx;
  const int x0 = tx * kRbTile, y0 = ty * kRbTile;
  const int x1 = min(x0 + kRbTile, s.cols), y1 = min(y0 + kRbTile, s.rows);
  float mn = 3.0e38f;
  bool ok = true;
  for (int y = y0; y < y1; ++y)
    for (int x = x0; x < x1; ++x) {
      const float d = S.raw[y * s.cols + x];
      if (!(d >= t.dmin && d <= t.dmax)) ok = false;
      else mn = fminf(mn, fabsf(S.sdist[y * s.cols + x]) - t.trunc);
    }
  const unsigned v = __float_as_uint(ok ? fmaxf(mn, 0.0f) : 0.0f);
  S.ftile[i] = v;
  const int cx = (S.rb_tx + kRbCoarse - 1) / kRbCoarse;
  atomicMin(S.ftile + S.rb_tx * S.rb_ty + (ty / kRbCoarse) * cx + tx / kRbCoarse, v);
}

__global__ void fused_bilateral_kernel(const SessDev* __restrict__ tab) {
  extern __shared__ float4 smem4[];
  float* tile = reinterpret_cast<float*>(smem4);
  const SessDev& S = tab[blockIdx.z];
  if (!S.bil_enabled) return;
  const int rows = S.ls[0].rows, cols = S.ls[0].cols;
  if ((int)blockIdx.x * BTX >= cols || (int)(blockIdx.y * blockDim.y) >= rows) return;
  if (S.vol.fp16)  // mixed-precision session
    bilateral_tile<true>(S.raw, S.filt, rows, cols, *S.btab, blockIdx.x, blockIdx.y, tile);
  else
    bilateral_tile<false>(S.raw, S.filt, rows, cols, *S.btab, blockIdx.x, blockIdx.y, tile);
}

// level l of the source (target == 0) or target pyramid from level l-1
__global__ void fused_downsample_kernel(const SessDev* __restrict__ tab, int l, int target) {
  const SessDev& S = tab[blockIdx.z];
  if (l >= S.nlev) return;
  const DSensor& sp = S.ls[l - 1];
  const int c2 = sp.cols / 2, n = (sp.rows / 2) * c2;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  downsample_depth_px(target ? S.tdep[l - 1] : S.sdep[l - 1], sp.cols, c2,
                      target ? S.tdep[l] : S.sdep[l], i);
  if (S.use_color)
    downsample_intensity_px(target ? S.tint[l - 1] : S.sint[l - 1], sp.cols, c2,
                            target ? S.tint[l] : S.sint[l], i);
}

__global__ void fused_maps_kernel(const SessDev* __restrict__ tab, int target) {
  const SessDev& S = tab[blockIdx.z];
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  for (int l = 0; l < S.nlev; ++l) {
    const int n = S.ls[l].rows * S.ls[l].cols;
    if (g < n) {
      float4* vtx = S.debug_maps ? (target ? S.tvtx[l] : S.svtx[l]) : nullptr;
      maps_px(target ? S.tdep[l] : S.sdep[l], target ? S.tnrm[l] : S.snrm[l], vtx, S.ls[l], g);
      return;
    }
    g -= n;
  }
}

// next frame's target level 0: the raycast (mode 1, misses -> 0) or the
// source itself (mode 0); flags the target as present
__global__ void fused_target_prepare_kernel(const SessDev* __restrict__ tab) {
  const SessDev& S = tab[blockIdx.z];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) S.icp->have_target = 1;
  if (i >= S.npx) return;
  if (S.mode == 1) {
    target_prepare_px(S.ray, S.tdep[0], S.vol.t.dmax, S.use_color ? S.trgb : nullptr,
                      S.use_color ? S.tint[0] : nullptr, i);
  } else {
    S.tdep[0][i] = S.sdep[0][i];
    if (S.use_color) S.tint[0][i] = S.sint[0][i];
  }
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

void launch_ingest(const uint16_t* raw, const uint8_t* rgb, int n, float scaler,
                   float* depth_out, float* intensity_out, cudaStream_t st) {
  ingest_kernel<<<nblk(n, 256), 256, 0, st>>>(raw, rgb, n, scaler, depth_out, intensity_out);
}

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

void launch_downsample_depth(const float* src, int rows, int cols, float* dst, cudaStream_t st) {
  int n = (rows / 2) * (cols / 2);
  if (n > 0) downsample_depth_kernel<<<nblk(n, 256), 256, 0, st>>>(src, rows, cols, dst);
}
void launch_downsample_intensity(const float* src, int rows, int cols, float* dst,
                                 cudaStream_t st) {
  int n = (rows / 2) * (cols / 2);
  if (n > 0) downsample_intensity_kernel<<<nblk(n, 256), 256, 0, st>>>(src, rows, cols, dst);
}
void launch_maps(const MapsArgs& a, cudaStream_t st) {
  if (a.total > 0) maps_kernel<<<nblk(a.total, 256), 256, 0, st>>>(a);
}
void launch_target_prepare(const float* ray_depth, float* depth0, float dmax, const uint8_t* rgb,
                           float* intensity0, int n, cudaStream_t st) {
  target_prepare_kernel<<<nblk(n, 256), 256, 0, st>>>(ray_depth, depth0, dmax, rgb, intensity0,
                                                      n);
}
void launch_copy_f(const float* src, float* dst, size_t n, cudaStream_t st) {
  if (n) cudaMemcpyAsync(dst, src, n * sizeof(float), cudaMemcpyDeviceToDevice, st);
}

// ---- fused stages
void fused_ingest(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  fused_ingest_kernel<<<dim3(nblk(b.max_npx, 256), 1, b.n), 256, 0, st>>>(tab);
  fused_free_tiles_kernel<<<dim3(nblk(b.max_rb_tiles, 128), 1, b.n), 128, 0, st>>>(tab);
}

void fused_bilateral(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  if (b.max_bil_radius <= 0) return;
  const int ty = bilateral_rows(b.max_cols, b.max_rows, b.n);
  fused_bilateral_kernel<<<dim3(nblk(b.max_cols, BTX), nblk(b.max_rows, ty), b.n), dim3(BTX, ty),
                           bilateral_smem(b.max_bil_radius, ty), st>>>(tab);
}

void fused_pyramid(const SessDev* tab, const BatchShape& b, int target, cudaStream_t st) {
  for (int l = 1; l < b.max_nlev; ++l)
    if (b.max_level_px[l] > 0)
      fused_downsample_kernel<<<dim3(nblk(b.max_level_px[l], 256), 1, b.n), 256, 0, st>>>(
          tab, l, target);
  int tot = 0;
  for (int l = 0; l < b.max_nlev; ++l) tot += b.max_level_px[l];
  fused_maps_kernel<<<dim3(nblk(tot, 256), 1, b.n), 256, 0, st>>>(tab, target);
}

void fused_target_prepare(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  fused_target_prepare_kernel<<<dim3(nblk(b.max_npx, 256), 1, b.n), 256, 0, st>>>(tab);
}

}  // namespace dyn
