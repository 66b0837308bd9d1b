// image.cuh -- depth ingest, bilateral filter, pyramid and normal maps.
#pragma once
#include "common.cuh"

namespace dyn {

// Bilateral filter constants: spatial weights per tap offset (row-major
// 2r x 2r, r <= 16) and the range-weight constants.
struct BilateralTable {
  float gs[32 * 32];
  int radius;
  float inv2s2;  // 1 / (2 sigma_i^2)
  float norm;    // 1 / (2 pi sigma_i^2)
};
BilateralTable make_bilateral_table(int radius, float sigma_i, float sigma_s);

// Launchers (all asynchronous on 'st').
void launch_bilateral(const float* src, float* dst, int rows, int cols,
                      const BilateralTable& tb, cudaStream_t st);
// Normals (and, unless null, vertices) of one level.
void launch_maps(const float* depth, const DSensor& s, float4* normal, float4* vertex,
                 cudaStream_t st);
// raycast output -> depth: misses (>= dmax) become 0
void launch_miss_to_zero(const float* ray_depth, float* depth0, float dmax, int n,
                         cudaStream_t st);

}  // namespace dyn
