// The raycast's choice between its block grid and the hash
// (dynamap_b200/csrc/ray_grid.cuh), on the CPU: every block that a ray taking
// the grid would look up must lie in the grid's box, since the march does not
// check its indices.
#include "cuda_emu.h"

#include <cstdint>

#include "../../dynamap_b200/csrc/ray_grid.cuh"

// pose: 16 floats; sensor: fx, fy, cx, cy; tsdf: voxel, truncation, range.
// Rays of every step-th pixel at 'samples' depths below the range.  out: rays
// of the exact form that take the grid, of the mixed form, lookups outside the
// box, whether the box is in use.
extern "C" void ray_grid_check(const float* pose, const float* sensor, int rows, int cols,
                               const float* tsdf, int cap, int step, int samples, int64_t* out) {
  using namespace dyn;
  DSensor s{};
  s.rows = rows;
  s.cols = cols;
  s.fx = sensor[0];
  s.fy = sensor[1];
  s.cx = sensor[2];
  s.cy = sensor[3];
  DTsdf t{};
  t.vs = tsdf[0];
  t.bsm = 8.0f * tsdf[0];
  t.trunc = tsdf[1];
  t.dmax = tsdf[2];
  t.num_blocks = 1 << 20;
  M4f T;
  std::memcpy(T.m, pose, sizeof(T.m));
  const GridBox b = grid_box(pose, s, t, cap);
  out[0] = out[1] = out[2] = 0;
  out[3] = b.ok;
  const float inv_vs = 1.0f / t.vs;
  const int lo[3] = {b.x0, b.y0, b.z0}, n[3] = {b.nx, b.ny, b.nz};
  for (int y = 0; y < rows; y += step)
    for (int x = 0; x < cols; x += step) {
      const float ax = (float)x - s.cx, ay = (float)y - s.cy;
      MarchRay R;
      const bool exact = b.ok && march_setup(t, s, T, ax, ay, inv_vs, R);
      const bool mixed =
          b.ok && march_bounded(t) && march_within(t, T, ax / s.fx, ay / s.fy, inv_vs);
      out[0] += exact;
      out[1] += mixed;
      if (!exact && !mixed) continue;
      for (int k = 0; k < samples; ++k) {
        const float cur = t.dmax * (float)k / (float)samples;
        const F3 p = xform(T, f3(ax * cur / s.fx, ay * cur / s.fy, cur));
        const float v[3] = {p.x * inv_vs, p.y * inv_vs, p.z * inv_vs};
        for (int a = 0; a < 3; ++a)
          for (const float c : {std::floor(v[a]), std::floor(v[a]) + 1.0f, std::rint(v[a])}) {
            const float block = std::floor(c / 8.0f);
            out[2] += !(block >= (float)lo[a] && block < (float)(lo[a] + n[a]));
          }
      }
    }
}
