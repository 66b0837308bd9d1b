// icp.cu -- normal equations of projective point-to-plane (+photometric) ICP
// and the Gauss-Newton step, on the device.
//
// Reference: buildNLSKernel (include/solver/gnSolver/gnSolver.cu:26-196) and
// gnSolver::solve (:317-438).  The reference adds 42 FP32 atomics per
// correspondence into one 6x6 system and round-trips to the host (Eigen LDLT)
// every iteration.  Here each thread accumulates its pixels' 21 upper-
// triangle JtJ terms, 6 Jtr terms, r^2 and a count in registers (FP64 sums of
// the FP32 terms; in the mixed form FP32 sums of a few pixels, from there on
// compensated FP32 pairs), warps and blocks reduce them with shuffles into a
// partial per pixel tile, and the tiles' partials are added in a fixed order:
// rows w, w + 16, ... by warp w, then the 16 warps' sums (level_total).  So
// results are run-to-run deterministic and do not depend on the grid.  The GN
// update (scale by 1/max(A), damping, 6x6 LDL^T, convergence test) and the SE(3)
// exponential for the next iteration follow in FP64, with no host round trip.
// Per frame this runs either as one chained launch per iteration (the last block
// to finish a level's tiles updates the solver) or as one persistent cooperative
// launch for all levels and iterations (below); both give the same bits.
#include "icp.cuh"

#include <algorithm>
#include <mutex>

#include "last_block.cuh"
#include "sessdev.cuh"

namespace dyn {

namespace {

// A level as the per-frame kernels keep it in shared memory, with its tiles'
// shape and the session's parameters (read again and again while a thread's
// registers hold sums).
struct FrameLevel : IcpLevel {
  int n, group, slots, tile, ntiles;  // pixels; icp_group, icp_slots, icp_tile_slots, icp_tiles
  int parts_log2;                     // a tile's parts, one per warp: 16 or 8
  IcpParams P;
};

__device__ inline bool normal_ok(float4 n) {
  if (isnan(n.x) || isnan(n.y) || isnan(n.z)) return false;
  return !(n.x == 0.0f && n.y == 0.0f && n.z == 0.0f);
}

// Per-thread sums of the per-pixel terms.  The FP32 form adds each pixel's
// FP32 terms in FP64 (as the oracle does), so that its normal equations
// differ from the oracle's only by the order of FP64 additions.  The mixed
// form (KAHAN) sums a thread's few pixels in FP32 by fused multiply-adds;
// from the warp sums on, its sums are compensated pairs (block_reduce).
struct Acc {
  double d[kIcpVals];  // FP64 sums (kahan == 0)
  float v[kIcpVals];   // FP32 sums (kahan != 0)
};

__device__ inline void acc_add(Acc& a, int k, float x) { a.d[k] += (double)x; }

// Per-pixel terms of buildNLSKernel (gnSolver.cu:55-194) for source pixel
// idx; the reference's unchecked projection is bounded (z > 0, inside the
// image) and photometric gradient taps outside the image read the centre.
// Three steps, so that a thread can issue the loads of several pixels
// before it waits on any: the source pixel's depth and normal, its
// projection into the target, the target's depth, normal and intensities.
struct PixSrc {
  float d;
  float4 n;
};
struct PixProj {
  F3 p;        // source point in the target frame
  float4 sn;   // source normal
  int index;   // target pixel
  int px, py;
};
struct PixTgt {
  float td;
  float4 tn;
  float ic, il, iu, si;  // photometric taps (colour weight != 0)
};

__device__ inline PixSrc load_src(const IcpLevel& L, int idx) {
  PixSrc a;
  a.d = L.sd[idx];
  a.n = L.sn[idx];
  return a;
}

// Pixel (u, v) of index idx in an image of 'cols' columns, exactly: a
// reciprocal estimate of the row (relative error a few 2^-24, so under one
// row off for images of up to 2^26 pixels) corrected by one step.
__device__ inline void pixel_uv(int idx, int cols, int& u, int& v) {
  v = __float2int_rz(__int2float_rn(idx) * __fdividef(1.0f, (float)cols));
  u = idx - v * cols;
  if (u < 0) {
    --v;
    u += cols;
  } else if (u >= cols) {
    ++v;
    u -= cols;
  }
}

// getPoint3d and Project (utils.h:104-119) by fused multiply-adds and
// approximate division: the mixed form's projective association.
__device__ inline F3 point3d_fast(int u, int v, float d, const DSensor& s) {
  return f3(__fdividef(((float)u - s.cx) * d, s.fx), __fdividef(((float)v - s.cy) * d, s.fy), d);
}
__device__ inline bool project_fast(F3 p, const DSensor& s, int* px, int* py) {
  const float rz = __fdividef(1.0f, p.z);
  const float x = __fmaf_rn(s.fx * p.x, rz, s.cx), y = __fmaf_rn(s.fy * p.y, rz, s.cy);
  if (!(fabsf(x) < 2e9f) || !(fabsf(y) < 2e9f)) return false;
  *px = (int)roundf(x);
  *py = (int)roundf(y);
  return true;
}
__device__ inline F3 xform_fma_icp(const M4f& T, F3 v) {
  return f3(__fmaf_rn(T.m[0], v.x, __fmaf_rn(T.m[1], v.y, __fmaf_rn(T.m[2], v.z, T.m[3]))),
            __fmaf_rn(T.m[4], v.x, __fmaf_rn(T.m[5], v.y, __fmaf_rn(T.m[6], v.z, T.m[7]))),
            __fmaf_rn(T.m[8], v.x, __fmaf_rn(T.m[9], v.y, __fmaf_rn(T.m[10], v.z, T.m[11]))));
}

// FAST: the mixed form (fused multiply-adds, approximate division); else
// the reference's expressions with IEEE rounding.
template <bool FAST>
__device__ inline bool project_src(const IcpLevel& L, const IcpParams& P, const M4f& T, int idx,
                                   const PixSrc& a, PixProj& q) {
  const DSensor& s = L.s;
  if (a.d < P.dmin || a.d > P.dmax) return false;
  if (!normal_ok(a.n)) return false;
  int u, v;
  pixel_uv(idx, s.cols, u, v);
  F3 p = FAST ? xform_fma_icp(T, point3d_fast(u, v, a.d, s)) : xform(T, point3d_uv(u, v, a.d, s));
  if (!(p.z > 0.0f)) return false;
  int px, py;
  if (!(FAST ? project_fast(p, s, &px, &py) : project(p, s, &px, &py))) return false;
  if (px < 0 || py < 0 || px >= s.cols || py >= s.rows) return false;
  q.p = p;
  q.sn = a.n;
  q.index = py * s.cols + px;
  q.px = px;
  q.py = py;
  return true;
}

__device__ inline PixTgt load_tgt(const IcpLevel& L, const IcpParams& P, const PixProj& q,
                                  int idx) {
  PixTgt t;
  t.td = L.td[q.index];
  t.tn = L.tn[q.index];
  if (P.cw != 0.0f) {
    const int il = q.px >= 1 ? q.index - 1 : q.index;
    const int iu = q.py >= 1 ? q.index - L.s.cols : q.index;
    t.ic = L.ti[q.index];
    t.il = L.ti[il];
    t.iu = L.ti[iu];
    t.si = L.si[idx];
  }
  return t;
}

// The mixed form's terms of one pixel (the same terms as below, by fused
// multiply-adds: b_k = cn_k (pq . n), the reference's three-product sum in
// exact arithmetic) added into FP32 per-thread sums.
__device__ inline void accumulate_mixed(const IcpParams& P, const F3 p, const F3 n, const F3 pq,
                                        const PixTgt& t, float count, Acc& a) {
  const F3 c = cross3(p, n);
  const float cn[6] = {c.x, c.y, c.z, n.x, n.y, n.z};
  const float r = __fmaf_rn(pq.x, n.x, __fmaf_rn(pq.y, n.y, __fmul_rn(pq.z, n.z)));
  if (P.cw != 0.0f) {
    const float gx = (t.ic - t.il) * 0.5f, gy = (t.ic - t.iu) * 0.5f;
    const float Jc[6] = {-gy * p.z, gx * p.z, __fmaf_rn(gy, p.x, -gx * p.y), gx, gy, 0.0f};
    const float e = t.ic - t.si;
    const float w1 = 1.0f - P.cw;
    float wcn[6], cj[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      wcn[i] = w1 * cn[i];
      cj[i] = P.cw * Jc[i];
    }
    int u = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = i; j < 6; ++j, ++u)
        a.v[u] = __fmaf_rn(wcn[i], cn[j], __fmaf_rn(cj[i], Jc[j], a.v[u]));
#pragma unroll
    for (int k = 0; k < 6; ++k)
      a.v[21 + k] = __fmaf_rn(-wcn[k], r, __fmaf_rn(-cj[k], e, a.v[21 + k]));
  } else {
    int u = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = i; j < 6; ++j, ++u) a.v[u] = __fmaf_rn(cn[i], cn[j], a.v[u]);
#pragma unroll
    for (int k = 0; k < 6; ++k) a.v[21 + k] = __fmaf_rn(-cn[k], r, a.v[21 + k]);
  }
  a.v[27] = __fmaf_rn(r, r, a.v[27]);
  a.v[28] = __fadd_rn(a.v[28], count);
}

template <bool KAHAN>
__device__ inline void accumulate(const IcpLevel& L, const IcpParams& P, const PixProj& q,
                                  const PixTgt& t, Acc& a) {
  const DSensor& s = L.s;
  if (t.td < P.dmin || t.td > P.dmax) return;
  if (!normal_ok(t.tn)) return;
  const F3 p = q.p;
  F3 n = f3(t.tn.x, t.tn.y, t.tn.z);
  float cosT = dot3(n, f3(q.sn.x, q.sn.y, q.sn.z));
  F3 qq = KAHAN ? point3d_fast(q.px, q.py, t.td, s) : point3d_uv(q.px, q.py, t.td, s);
  if (!(fabsf(cosT) > P.cos_thr)) return;
  F3 pq = p - qq;
  if (KAHAN) {
    accumulate_mixed(P, p, n, pq, t, 1.0f, a);
    return;
  }
  F3 c = cross3(p, n);
  float cn[6] = {c.x, c.y, c.z, n.x, n.y, n.z};
  float b[6];
#pragma unroll
  for (int k = 0; k < 6; ++k)
    b[k] = pq.x * (cn[k] * n.x) + pq.y * (cn[k] * n.y) + pq.z * (cn[k] * n.z);
  float r = dot3(pq, n);
  if (P.cw != 0.0f) {
    // gnSolver.cu:137-190: J_c = grad(I_t)(1x3) * [-p^ | I](3x6)
    float gx = (t.ic - t.il) / 2.0f;
    float gy = (t.ic - t.iu) / 2.0f;
    float Jc[6] = {gx * 0.0f + gy * (-p.z), gx * p.z + gy * 0.0f, gx * (-p.y) + gy * p.x,
                   gx, gy, 0.0f};
    float e = t.ic - t.si;
    float w1 = 1.0f - P.cw;
    int u = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = i; j < 6; ++j) acc_add(a, u++, w1 * (cn[i] * cn[j]) + (P.cw * Jc[i]) * Jc[j]);
#pragma unroll
    for (int k = 0; k < 6; ++k) acc_add(a, 21 + k, -(w1 * b[k] + (P.cw * Jc[k]) * e));
  } else {
    int u = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = i; j < 6; ++j) acc_add(a, u++, cn[i] * cn[j]);
#pragma unroll
    for (int k = 0; k < 6; ++k) acc_add(a, 21 + k, -b[k]);
  }
  acc_add(a, 27, r * r);
  acc_add(a, 28, 1.0f);
}

template <bool KAHAN>
__device__ inline void pixel_terms(const IcpLevel& L, const IcpParams& P, const M4f& T,
                                   int idx, Acc& a) {
  PixProj q;
  if (!project_src<KAHAN>(L, P, T, idx, load_src(L, idx), q)) return;
  accumulate<KAHAN>(L, P, q, load_tgt(L, P, q, idx), a);
}

// N pixels i, i + stride, ... below n of the mixed form, added in order: the
// terms of pixel_terms on one after the other, without branches, so that the
// pixels' latencies overlap (at 16 warps per SM nothing else hides them).  A
// pixel without a correspondence loads pixel 0, counts 0, and its vectors are
// zero: its terms are zeros, which change no sum.
template <int N>
__device__ inline void pixel_group(const FrameLevel& L, const M4f& T, int i, int stride, int n,
                                   Acc& a) {
  const IcpParams& P = L.P;
  PixSrc src[N];
  PixProj q[N];
  PixTgt t[N];
  bool ok[N];
#pragma unroll
  for (int m = 0; m < N; ++m) {
    ok[m] = i + m * stride < n;
    src[m] = load_src(L, ok[m] ? i + m * stride : 0);
  }
#pragma unroll
  for (int m = 0; m < N; ++m) {
    const bool in = project_src<true>(L, P, T, i + m * stride, src[m], q[m]);
    ok[m] = ok[m] && in;
    q[m].index = ok[m] ? q[m].index : 0;
    q[m].px = ok[m] ? q[m].px : 0;
    q[m].py = ok[m] ? q[m].py : 0;
  }
#pragma unroll
  for (int m = 0; m < N; ++m) t[m] = load_tgt(L, P, q[m], ok[m] ? i + m * stride : 0);
#pragma unroll
  for (int m = 0; m < N; ++m) {
    const F3 n = f3(t[m].tn.x, t[m].tn.y, t[m].tn.z);
    const float cosT = dot3(n, f3(q[m].sn.x, q[m].sn.y, q[m].sn.z));
    const bool in = ok[m] && !(t[m].td < P.dmin || t[m].td > P.dmax) && normal_ok(t[m].tn) &&
                    fabsf(cosT) > P.cos_thr;
    const F3 pq = q[m].p - point3d_fast(q[m].px, q[m].py, t[m].td, L.s);
    auto sel = [in](F3 v) { return f3(in ? v.x : 0.0f, in ? v.y : 0.0f, in ? v.z : 0.0f); };
    PixTgt u = t[m];
    u.ic = in ? u.ic : 0.0f;
    u.il = in ? u.il : 0.0f;
    u.iu = in ? u.iu : 0.0f;
    u.si = in ? u.si : 0.0f;
    accumulate_mixed(P, sel(q[m].p), sel(n), sel(pq), u, in ? 1.0f : 0.0f, a);
  }
}

// ---- block and tile sums
// The FP32 form adds in FP64 throughout.  The mixed form keeps the normal
// equations in FP32 up to the solve: a compensated pair (s, c) -- value
// s + c, c the rounding error carried along -- is added with Knuth's
// two-sum at every step (thread, warp shuffles, warps of a block, tiles),
// and only the level's total becomes FP64 for the 6x6 solve.  A pair is
// stored in a double-sized slot as two floats.
__device__ inline void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float ap = __fsub_rn(s, b), bp = __fsub_rn(s, ap);
  e = __fadd_rn(__fsub_rn(a, ap), __fsub_rn(b, bp));
}
__device__ inline void pair_add(float& s, float& c, float s2, float c2) {
  float e;
  two_sum(s, s2, s, e);
  c = __fadd_rn(__fadd_rn(c, c2), e);
}
__device__ inline double pack_pair(float s, float c) {
  return __longlong_as_double((long long)(((unsigned long long)__float_as_uint(c) << 32) |
                                          (unsigned long long)__float_as_uint(s)));
}
__device__ inline void unpack_pair(double d, float& s, float& c) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(d);
  s = __uint_as_float((unsigned)(u & 0xffffffffull));
  c = __uint_as_float((unsigned)(u >> 32));
}

// Warp sum of the 29 accumulators in a fixed order: lane l < 29 gets the total
// of value l (FP64, or a compensated pair).
// The warp sum is a halving exchange over 32 slots (values 29..31 zero):
// at offset o every lane keeps the half of its remaining slots that its
// bit o selects, sends the other half to lane ^ o and adds what that lane
// sent; after offsets 16, 8, 4, 2, 1 lane l holds the warp's total of value
// l.  31 exchanges per lane instead of 29 x 5 for a butterfly per value.
struct LaneSum {
  double d;    // plain
  float s, c;  // compensated
};
template <bool KAHAN>
__device__ inline LaneSum warp_reduce(const Acc& a) {
  const int lane = threadIdx.x & 31;
  LaneSum out;
  if (KAHAN) {
    float s[32], c[16];
#pragma unroll
    for (int k = 0; k < kIcpVals; ++k) s[k] = a.v[k];
#pragma unroll
    for (int k = kIcpVals; k < 32; ++k) s[k] = 0.0f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {  // the first exchange: no corrections yet
      const bool up = (lane & 16) != 0;
      const float ks = up ? s[k + 16] : s[k], gs = up ? s[k] : s[k + 16];
      two_sum(ks, __shfl_xor_sync(0xffffffffu, gs, 16), s[k], c[k]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < o; ++k) {
        const float ks = up ? s[k + o] : s[k], kc = up ? c[k + o] : c[k];
        const float gs = up ? s[k] : s[k + o], gc = up ? c[k] : c[k + o];
        const float rs = __shfl_xor_sync(0xffffffffu, gs, o);
        const float rc = __shfl_xor_sync(0xffffffffu, gc, o);
        s[k] = ks;
        c[k] = kc;
        pair_add(s[k], c[k], rs, rc);
      }
    }
    out.s = s[0];
    out.c = c[0];
  } else {
    double s[32];
#pragma unroll
    for (int k = 0; k < kIcpVals; ++k) s[k] = a.d[k];
#pragma unroll
    for (int k = kIcpVals; k < 32; ++k) s[k] = 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < o; ++k) {
        const double keep = up ? s[k + o] : s[k], give = up ? s[k] : s[k + o];
        s[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    out.d = s[0];
  }
  return out;
}

// One value of the first nw of NW warps (red[0], red[29], ...: shared) added in
// warp order.
template <bool KAHAN, int NW>
__device__ inline double add_warps(const double* red, int nw = NW) {
  if (KAHAN) {
    float sv = 0.0f, sc = 0.0f;
#pragma unroll
    for (int w = 0; w < NW; ++w)
      if (w < nw) {
        float s2, c2;
        unpack_pair(red[w * kIcpVals], s2, c2);
        pair_add(sv, sc, s2, c2);
      }
    return pack_pair(sv, sc);
  }
  double sum = 0.0;
#pragma unroll
  for (int w = 0; w < NW; ++w)
    if (w < nw) sum += red[w * kIcpVals];
  return sum;
}

// Block sum in red[0..28] (shared, NW x 29) after the call.
template <bool KAHAN, int NW>
__device__ inline void block_reduce(const Acc& a, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LaneSum l = warp_reduce<KAHAN>(a);
  if (lane < kIcpVals) red[warp * kIcpVals + lane] = KAHAN ? pack_pair(l.s, l.c) : l.d;
  __syncthreads();
  // (row 0 reused: each thread its own column)
  if (threadIdx.x < kIcpVals) red[threadIdx.x] = add_warps<KAHAN, NW>(red + threadIdx.x);
  __syncthreads();
}

// Sum of the stage kernel's per-block partials in a fixed order: thread
// (g, k) of 8 x 29 sums value k of rows g, g + 8, g + 16, ... (all 29
// values' loads in flight at once, coalesced along k), then thread k adds
// the 8 group sums in group order.  'scratch' is 8 x 29 doubles of shared
// memory; out[29] (shared).
__device__ inline void final_reduce(const double* __restrict__ partials, int nblocks,
                                    double* out, double* scratch) {
  constexpr int kGroups = kIcpThreads / 32;  // 8: scratch is the block-reduce array
  static_assert(kGroups * kIcpVals <= kIcpThreads, "one thread per (group, value)");
  const int t = threadIdx.x;
  if (t < kGroups * kIcpVals) {
    const int g = t / kIcpVals, k = t - g * kIcpVals;
    double sum = 0.0;
#pragma unroll 4
    for (int b = g; b < nblocks; b += kGroups) sum += __ldcg(partials + (size_t)b * kIcpVals + k);
    scratch[g * kIcpVals + k] = sum;
  }
  __syncthreads();
  if (t < kIcpVals) {
    double sum = 0.0;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) sum += scratch[g * kIcpVals + t];
    out[t] = sum;
  }
  __syncthreads();
}

// The level's total of its tiles' partials, in a fixed order: warp w sums rows
// w, w + 16, ... (v[i] lane k's value k of row w + 16 i, zero past the last
// tile), then lane k of warp 0 adds the 16 warps' sums.  'red' is 16 x 29
// doubles of shared memory; out[29] (shared) is there for warp 0 after the
// call: FP64 values (a compensated pair's s + c in the KAHAN form).
constexpr int kFrameWarps = kIcpFrameThreads / 32;
constexpr int kWarpRows = (kIcpMaxTiles + kFrameWarps - 1) / kFrameWarps;
template <bool KAHAN>
__device__ inline void level_total(const double (&v)[kWarpRows], double* out, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane < kIcpVals) {
    if (KAHAN) {
      float sv = 0.0f, sc = 0.0f;
#pragma unroll
      for (int i = 0; i < kWarpRows; ++i) {  // (rows that are not there add zero pairs)
        float s2, c2;
        unpack_pair(v[i], s2, c2);
        pair_add(sv, sc, s2, c2);
      }
      red[w * kIcpVals + lane] = pack_pair(sv, sc);
    } else {
      double sum = 0.0;
#pragma unroll
      for (int i = 0; i < kWarpRows; ++i) sum += v[i];
      red[w * kIcpVals + lane] = sum;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    if (lane < kIcpVals) {
      const double t = add_warps<KAHAN, kFrameWarps>(red + lane);
      if (KAHAN) {
        float s2, c2;
        unpack_pair(t, s2, c2);
        out[lane] = (double)s2 + (double)c2;  // FP64 from here on: the 6x6 solve
      } else {
        out[lane] = t;
      }
    }
    __syncwarp();
  }
}

// ---- FP64 6x6 algebra (one thread) --------------------------------------
// The 6x6 system lives in registers: every loop below has compile-time
// bounds and is unrolled, so no array is indexed at run time (a run-time
// index would put the arrays in local memory and make each dependent step
// of the one-thread solve wait on an L1 round trip).  The lower triangle is
// kept packed, row i at tri(i, 0) (the system is symmetric; the
// factorisation reads only the lower triangle).
__host__ __device__ constexpr int tri(int i, int j) { return i * (i + 1) / 2 + j; }

// LDL^T of a symmetric positive definite 6x6 in place (stands in for
// Eigen's A.ldlt().solve(b), gnSolver.cu:439-442), column by column: with
// D[j] = A[j][j], L[i][j] = A[i][j] / D[j], then A[i][k] -= L[i][j] A[k][j]
// for the columns behind -- so that only a reciprocal, a product and a fused
// multiply-add lie between two pivots (this one thread sits between every two
// ICP iterations); then forward substitution, division by D, back
// substitution.  L overwrites the strict lower triangle of a, D its diagonal.
// Returns false on a zero pivot.
__device__ __forceinline__ bool ldlt6(double (&a)[21], const double (&b)[6], double (&x)[6]) {
  double rd[6];  // 1 / D[j]
  // triangular bounds are written as guards on fixed-length loops, so that
  // every loop has a constant trip count and unrolls completely
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    if (!(fabs(a[tri(j, j)]) > 0.0)) return false;
    rd[j] = 1.0 / a[tri(j, j)];
    double l[6];
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (i > j) l[i] = a[tri(i, j)] * rd[j];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int k = 0; k < 6; ++k)
        if (k > j && k <= i) a[tri(i, k)] = fma(-l[i], a[tri(k, j)], a[tri(i, k)]);
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (i > j) a[tri(i, j)] = l[i];
  }
  double y[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    double t = b[i];
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (k < i) t = fma(-a[tri(i, k)], y[k], t);
    y[i] = t;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) y[i] *= rd[i];
#pragma unroll
  for (int i = 5; i >= 0; --i) {
    double t = y[i];
#pragma unroll
    for (int k = 5; k >= 0; --k)
      if (k > i) t = fma(-a[tri(k, i)], x[k], t);
    x[i] = t;
  }
  return true;
}

// exp of the twist matrix v2t(xi) (gnSolver.cu:443-455): rotation by
// Rodrigues' formula and translation through the SE(3) left Jacobian,
// R = I + a W + b W^2, t = (I + b W + c W^2) v, with a = sin t / t,
// b = (1 - cos t)/t^2, c = (t - sin t)/t^3.  Up to half a radian they are
// their Taylor series in t^2 to the eighth term (the rest is below 1e-19 of
// the value; the closed forms lose digits to cancellation there, and their
// square root, sine, cosine and divisions are a serial chain between every two
// ICP iterations).
__device__ __forceinline__ void se3_exp(const double* xi, double* T) {
  double w0 = xi[0], w1 = xi[1], w2 = xi[2];
  double th2 = w0 * w0 + w1 * w1 + w2 * w2;
  double a, b, c;
  if (th2 < 0.25) {
    // 1 / n! for n = 1 .. 17
    const double f[18] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040,
                          1.0 / 40320, 1.0 / 362880, 1.0 / 3628800, 1.0 / 39916800,
                          1.0 / 479001600, 1.0 / 6227020800.0, 1.0 / 87178291200.0,
                          1.0 / 1307674368000.0, 1.0 / 20922789888000.0,
                          1.0 / 355687428096000.0};
    a = f[15];
    b = f[16];
    c = f[17];
#pragma unroll
    for (int k = 6; k >= 0; --k) {
      a = fma(-a, th2, f[2 * k + 1]);
      b = fma(-b, th2, f[2 * k + 2]);
      c = fma(-c, th2, f[2 * k + 3]);
    }
  } else {
    double sn, cs;
    const double th = sqrt(th2);
    sincos(th, &sn, &cs);
    a = sn / th;
    b = (1.0 - cs) / th2;
    c = (th - sn) / (th2 * th);
  }
  double W[9] = {0, -w2, w1, w2, 0, -w0, -w1, w0, 0};
  double W2[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double s = 0;
      for (int k = 0; k < 3; ++k) s += W[i * 3 + k] * W[k * 3 + j];
      W2[i * 3 + j] = s;
    }
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 3; ++j) {
      double I = (i == j) ? 1.0 : 0.0;
      T[i * 4 + j] = I + a * W[i * 3 + j] + b * W2[i * 3 + j];
    }
    double V0 = (i == 0 ? 1.0 : 0.0) + b * W[i * 3 + 0] + c * W2[i * 3 + 0];
    double V1 = (i == 1 ? 1.0 : 0.0) + b * W[i * 3 + 1] + c * W2[i * 3 + 1];
    double V2 = (i == 2 ? 1.0 : 0.0) + b * W[i * 3 + 2] + c * W2[i * 3 + 2];
    T[i * 4 + 3] = V0 * xi[3] + V1 * xi[4] + V2 * xi[5];
  }
  T[12] = T[13] = T[14] = 0.0;
  T[15] = 1.0;
}

__device__ void matmul4d(const double* A, const double* B, double* C) {
  double t[16];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      double s = 0;
      for (int k = 0; k < 4; ++k) s += A[i * 4 + k] * B[k * 4 + j];
      t[i * 4 + j] = s;
    }
  for (int k = 0; k < 16; ++k) C[k] = t[k];
}

// float4x4::getInverse, utils_matrix.h:970-1086: cofactors summed in the
// reference's order, determinant from row 0, times 1/det.
__device__ void inverse4f(const float* e, float* out) {
  float inv[16];
  inv[0] = e[5] * e[10] * e[15] - e[5] * e[11] * e[14] - e[9] * e[6] * e[15] +
           e[9] * e[7] * e[14] + e[13] * e[6] * e[11] - e[13] * e[7] * e[10];
  inv[4] = -e[4] * e[10] * e[15] + e[4] * e[11] * e[14] + e[8] * e[6] * e[15] -
           e[8] * e[7] * e[14] - e[12] * e[6] * e[11] + e[12] * e[7] * e[10];
  inv[8] = e[4] * e[9] * e[15] - e[4] * e[11] * e[13] - e[8] * e[5] * e[15] +
           e[8] * e[7] * e[13] + e[12] * e[5] * e[11] - e[12] * e[7] * e[9];
  inv[12] = -e[4] * e[9] * e[14] + e[4] * e[10] * e[13] + e[8] * e[5] * e[14] -
            e[8] * e[6] * e[13] - e[12] * e[5] * e[10] + e[12] * e[6] * e[9];
  inv[1] = -e[1] * e[10] * e[15] + e[1] * e[11] * e[14] + e[9] * e[2] * e[15] -
           e[9] * e[3] * e[14] - e[13] * e[2] * e[11] + e[13] * e[3] * e[10];
  inv[5] = e[0] * e[10] * e[15] - e[0] * e[11] * e[14] - e[8] * e[2] * e[15] +
           e[8] * e[3] * e[14] + e[12] * e[2] * e[11] - e[12] * e[3] * e[10];
  inv[9] = -e[0] * e[9] * e[15] + e[0] * e[11] * e[13] + e[8] * e[1] * e[15] -
           e[8] * e[3] * e[13] - e[12] * e[1] * e[11] + e[12] * e[3] * e[9];
  inv[13] = e[0] * e[9] * e[14] - e[0] * e[10] * e[13] - e[8] * e[1] * e[14] +
            e[8] * e[2] * e[13] + e[12] * e[1] * e[10] - e[12] * e[2] * e[9];
  inv[2] = e[1] * e[6] * e[15] - e[1] * e[7] * e[14] - e[5] * e[2] * e[15] +
           e[5] * e[3] * e[14] + e[13] * e[2] * e[7] - e[13] * e[3] * e[6];
  inv[6] = -e[0] * e[6] * e[15] + e[0] * e[7] * e[14] + e[4] * e[2] * e[15] -
           e[4] * e[3] * e[14] - e[12] * e[2] * e[7] + e[12] * e[3] * e[6];
  inv[10] = e[0] * e[5] * e[15] - e[0] * e[7] * e[13] - e[4] * e[1] * e[15] +
            e[4] * e[3] * e[13] + e[12] * e[1] * e[7] - e[12] * e[3] * e[5];
  inv[14] = -e[0] * e[5] * e[14] + e[0] * e[6] * e[13] + e[4] * e[1] * e[14] -
            e[4] * e[2] * e[13] - e[12] * e[1] * e[6] + e[12] * e[2] * e[5];
  inv[3] = -e[1] * e[6] * e[11] + e[1] * e[7] * e[10] + e[5] * e[2] * e[11] -
           e[5] * e[3] * e[10] - e[9] * e[2] * e[7] + e[9] * e[3] * e[6];
  inv[7] = e[0] * e[6] * e[11] - e[0] * e[7] * e[10] - e[4] * e[2] * e[11] +
           e[4] * e[3] * e[10] + e[8] * e[2] * e[7] - e[8] * e[3] * e[6];
  inv[11] = -e[0] * e[5] * e[11] + e[0] * e[7] * e[9] + e[4] * e[1] * e[11] -
            e[4] * e[3] * e[9] - e[8] * e[1] * e[7] + e[8] * e[3] * e[5];
  inv[15] = e[0] * e[5] * e[10] - e[0] * e[6] * e[9] - e[4] * e[1] * e[10] +
            e[4] * e[2] * e[9] + e[8] * e[1] * e[6] - e[8] * e[2] * e[5];
  float det = e[0] * inv[0] + e[1] * inv[4] + e[2] * inv[8] + e[3] * inv[12];
  float detr = 1.0f / det;
  for (int i = 0; i < 16; ++i) out[i] = inv[i] * detr;
}

// gnSolver::solve's per-iteration host block (gnSolver.cu:389-415) for the
// summed system 'acc' (upper triangle row by row, then the 6 right-hand
// sides): scale by 1 / max(A), add reg * max(scaled A) / it to the
// diagonal, solve, accumulate.  The maxima run over all 36 entries in
// row-major order, as over the full symmetric matrix.  Updates inc/prev
// (the solver state's, in global or shared memory); returns true when
// converged.
__device__ __forceinline__ double max21(const double (&a)[21]) {
  double m[11];
#pragma unroll
  for (int k = 0; k < 10; ++k) m[k] = fmax(a[2 * k], a[2 * k + 1]);
  m[10] = a[20];
#pragma unroll
  for (int w = 1; w < 11; w *= 2)
#pragma unroll
    for (int k = 0; k + w < 11; k += 2 * w) m[k] = fmax(m[k], m[k + w]);
  return m[0];
}
__device__ bool gn_update(const double* acc, const IcpParams& P, int it, double* st_inc,
                          double* st_prev) {
  double a[21], b[6];
  {  // acc holds the upper triangle row by row
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = 0; j < 6; ++j)
        if (j >= i) a[tri(j, i)] = acc[i * 6 - i * (i - 1) / 2 + (j - i)];
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) b[k] = acc[21 + k];
  // the maxima over all 36 entries are the maxima over the 21 stored ones
  // (fmax ignores NaNs in any order), taken as a tree
  const double mx = max21(a);
  const double scaling = 1.0 / mx;
#pragma unroll
  for (int k = 0; k < 6; ++k) b[k] *= scaling;
#pragma unroll
  for (int k = 0; k < 21; ++k) a[k] *= scaling;
  const double mx2 = mx * scaling;  // the scaled entries' maximum (rounding is monotone)
  const double alpha = (double)P.reg * mx2;
#pragma unroll
  for (int k = 0; k < 6; ++k) a[tri(k, k)] += alpha / (double)it;
  double d[6] = {0, 0, 0, 0, 0, 0};
  if (!ldlt6(a, b, d)) {
#pragma unroll
    for (int k = 0; k < 6; ++k) d[k] = __longlong_as_double(0x7ff8000000000000LL);
  }
  double inc[6], ch = 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    inc[k] = st_inc[k] + d[k];
    st_inc[k] = inc[k];
    double c = inc[k] - st_prev[k];
    ch += c * c;
  }
  bool conv = fabs(sqrt(ch)) <= (double)P.min_inc;
  if (!conv) {
#pragma unroll
    for (int k = 0; k < 6; ++k) st_prev[k] = inc[k];
  }
  return conv;
}

// Blocks of the stage entry points' reduction: about 256, 512 or 1024 pixels
// each, at most kIcpMaxBlocks (a block then strides).
inline __host__ __device__ int icp_stage_grid(int n) {
  const int t = n <= 8192 ? 256 : (n <= 65536 ? 512 : 1024);
  int g = (n + t - 1) / t;
  if (g > kIcpMaxBlocks) g = kIcpMaxBlocks;
  if (g < 1) g = 1;
  return g;
}

// Part 'part' (of nw) of tile 'tile' of level L, slots part * 32 + lane + m * 512
// of the tile, by one warp, added in a fixed order into red[0..28] (shared).  The
// compensated form's warp totals move into compensated pairs, one value per
// lane, after every slot's pixels.
template <bool KAHAN>
__device__ inline void tile_warp_sum(const FrameLevel& L, const M4f& T, int tile, int part,
                                     double* red) {
  const int lane = threadIdx.x & 31;
  const int end = min(L.slots, (tile + 1) * L.tile), first = tile * L.tile + part * 32 + lane;
  Acc a;
  if (KAHAN) {
    const int group = L.group;
    LaneSum l;
    l.s = l.c = 0.0f;
    // (whole warps: slots come in runs of 256)
    for (int g = first; g < end; g += kIcpFrameThreads) {
      const int i = (g >> 8) * group * 256 + (g & 255);
#pragma unroll
      for (int k = 0; k < kIcpVals; ++k) a.v[k] = 0.0f;
#pragma unroll 1
      for (int m = 0; m < group; m += 2)  // (a group of one: its second pixel is out)
        pixel_group<2>(L, T, i + m * 256, 256, group > 1 ? L.n : min(L.n, i + 1), a);
      const LaneSum w = warp_reduce<KAHAN>(a);
      pair_add(l.s, l.c, w.s, w.c);
    }
    if (lane < kIcpVals) red[lane] = pack_pair(l.s, l.c);
  } else {  // FP64 sums hold most registers: one pixel at a time
#pragma unroll
    for (int k = 0; k < kIcpVals; ++k) a.d[k] = 0.0;
    for (int i = first; i < end; i += kIcpFrameThreads) pixel_terms<KAHAN>(L, L.P, T, i, a);
    __syncwarp();
    const LaneSum w = warp_reduce<KAHAN>(a);
    if (lane < kIcpVals) red[lane] = w.d;
  }
}

// The partial sums of the block's tiles first, first + step, ... of level L,
// each value handed to put(tile, k, value).  The warps go through up to
// kTileBatch tiles on their own (their loads' latencies overlap: a block of
// few warps and many tiles waits on nothing else) before the block adds their
// parts, in warp order.  Every thread of the block calls it; red: kTileBatch x
// 16 x 29.
constexpr int kTileBatch = 8;
template <bool KAHAN, class Put>
__device__ inline void tile_partials(const FrameLevel& L, const M4f& T, int first, int step,
                                     double* red, Put&& put) {
  const int warp = threadIdx.x >> 5, lg = L.parts_log2, ntiles = L.ntiles;
  for (int t0 = first; t0 < ntiles; t0 += kTileBatch * step) {
    int m = 1;  // tiles of this batch
    while (m < kTileBatch && t0 + m * step < ntiles) ++m;
#pragma unroll 1
    for (int p = warp; p < m << lg; p += kFrameWarps) {  // each tile's parts in order
      const int u = p >> lg, part = p - (u << lg);
      tile_warp_sum<KAHAN>(L, T, t0 + u * step, part, red + (u * kFrameWarps + part) * kIcpVals);
    }
    __syncthreads();
    // (a value per thread, a tile per warp)
    const int k = threadIdx.x & 31;
    if (warp < m && k < kIcpVals)
      put(t0 + warp * step, k,
          add_warps<KAHAN, kFrameWarps>(red + warp * kFrameWarps * kIcpVals + k, 1 << lg));
    if (t0 + kTileBatch * step < ntiles) __syncthreads();  // red is reused
  }
}

// The iteration's GN update and the next transform from the rows' values v
// (level_total), for a solver state held at st_* (global memory in the chained
// kernels, shared memory in the persistent one), and its statistics.  tot[]
// must be shared; the update runs on thread 0, then the statistics on another
// warp.
template <bool KAHAN>
__device__ inline void level_update(const double (&v)[kWarpRows], const IcpParams& P, int pl,
                                    int it, double* tot, double* red, double* st_inc,
                                    double* st_prev, float* st_T, int* st_converged,
                                    int* st_iters, int* st_inliers, float* st_rms) {
  level_total<KAHAN>(v, tot, red);
  if (threadIdx.x == 0) {
    const bool conv = gn_update(tot, P, it, st_inc, st_prev);
    *st_converged = conv ? 1 : 0;
    double Td[16];
    se3_exp(st_inc, Td);
    for (int k = 0; k < 16; ++k) st_T[k] = (float)Td[k];
  }
  __syncthreads();
  if (threadIdx.x == 32) {
    st_iters[pl] = it;
    st_inliers[pl] = (int)tot[28];
    st_rms[pl] = tot[28] > 0 ? (float)sqrt(tot[27] / tot[28]) : 0.0f;
  }
}

// One GN iteration of level slot pl, iteration it (1-based), block 'bid' of
// 'nb' blocks: the partial sums of the block's tiles, then -- in the last
// block to finish -- the FP64 total and the GN update (gnSolver.cu:379-415).
template <bool KAHAN>
__device__ inline void icp_iteration_body(const FrameLevel& L, int pl, int it, IcpState* st,
                                          double* __restrict__ partials, int bid,
                                          int nb) {
  __shared__ double red[kTileBatch * kFrameWarps * kIcpVals];
  __shared__ M4f Ts;
  __shared__ int skip;
  if (threadIdx.x == 0) {
    int sk = (st->have_target == 0) || (it > 1 && st->converged);
    skip = sk;
  }
  if (threadIdx.x < 16) Ts.m[threadIdx.x] = st->T[threadIdx.x];
  __syncthreads();
  if (skip) return;
  // the transform stays in shared memory (registers go to the sums)
  tile_partials<KAHAN>(L, Ts, bid, nb, red, [&](int tile, int k, double x) {
    partials[(size_t)tile * kIcpVals + k] = x;
  });
  if (!last_block(&st->ticket, (unsigned)nb)) return;
  __shared__ double tot[kIcpVals];
  double v[kWarpRows];
#pragma unroll
  for (int i = 0; i < kWarpRows; ++i) {  // every row's load in flight at once
    const int b = (threadIdx.x >> 5) + i * kFrameWarps, k = threadIdx.x & 31;
    v[i] = (b < L.ntiles && k < kIcpVals) ? __ldcg(partials + (size_t)b * kIcpVals + k) : 0.0;
  }
  level_update<KAHAN>(v, L.P, pl, it, tot, red, st->inc, st->prev, st->T, &st->converged, st->iters,
                      st->inliers, st->rms);
  if (threadIdx.x == 0) st->ticket = 0;
}

// Programmatic dependent launch: an iteration kernel launched with the
// programmatic-serialization attribute may start while its predecessor
// still runs.  It reads only data that no kernel of the ICP chain writes
// (the session table, the level maps) before griddepcontrol.wait, which
// returns once the predecessor grid has completed and its writes are
// visible; it then lets its own successor launch.  Without the attribute
// both instructions are no-ops.
__device__ inline void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ inline void release_successor() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ inline FrameLevel level_of(const SessDev& S, int l) {
  FrameLevel L;
  L.sd = S.sdep[l];
  L.sn = S.snrm[l];
  L.si = S.sint[l];
  L.td = S.tdep[l];
  L.tn = S.tnrm[l];
  L.ti = S.tint[l];
  L.s = S.ls[l];
  L.n = L.s.rows * L.s.cols;
  const int kahan = S.icpp.kahan;
  L.group = icp_group(L.n);
  L.slots = icp_slots(L.n, kahan);
  L.tile = icp_tile_slots(L.n, kahan);
  L.ntiles = icp_tiles(L.n, kahan);
  L.parts_log2 = L.tile >= kIcpFrameThreads ? 4 : 3;
  L.P = S.icpp;
  return L;
}

// Every session of the frame in one launch (blockIdx.z); a session uses
// only the blocks of its own grid.  One instantiation per summation kind;
// sessions of the other kind return.
template <bool KAHAN>
__global__ void __launch_bounds__(kIcpFrameThreads, 1)
    fused_icp_iteration_kernel(const SessDev* __restrict__ tab, int pl, int it) {
  const SessDev& S = tab[blockIdx.z];
  const int l = S.slot_level[pl];
  const int nb = icp_tiles(S.ls[l].rows * S.ls[l].cols, KAHAN);
  // (the reference runs iterations 1 .. N-1)
  const bool mine = (S.icpp.kahan != 0) == KAHAN && it < S.slot_iters[pl] && (int)blockIdx.x < nb;
  __shared__ FrameLevel L;  // shared: registers go to the sums
  if (mine && threadIdx.x == 0) L = level_of(S, l);
  // The solver state and partials of the previous iteration.  Every block waits,
  // those without work too: a launch waits for the one before it alone, so one
  // whose blocks all left at once (no session of its kind has that many
  // iterations) would let the next start beside the last but one.
  wait_predecessor();
  release_successor();
  if (!mine) return;
  icp_iteration_body<KAHAN>(L, pl, it, S.icp, S.partials, blockIdx.x, nb);
}

// ---- the persistent form: one launch walks every level and iteration
//
// A cooperative launch (all blocks resident at once, one per SM) over the
// table: each session owns a run of blocks (icp_share: its share of the
// work), every block keeps its session's solver state in shared memory, sums
// its tiles, and then waits for the rows of the level's other tiles, adds them
// (the same sums, in the same order, so every block holds the same state) and
// runs the GN update itself.
//
// There is no barrier: a row is 29 doubles as tagged words {32 data bits, tag},
// written and read as single 64-bit accesses, and a reader polls the rows
// themselves until they carry the iteration's tag -- one store's and one
// load's way through L2 between two blocks, with no fence (whose acquire side
// also empties L1, where the images stay from iteration to iteration).
// A level's iterations alternate between two rows per tile: a block writes its
// row of an iteration only after reading every row of the one before, which the
// others wrote after reading the rows that it overwrites.  Each level has its own
// rows (icp_row).  Blocks without a tile of a level wait for the state that the
// session's first block leaves at the level's end; those without a tile of a
// later level return.
//
// The coarse levels are a chain of latencies, about six iterations of a
// frame's nine: the block's sums 2,500 (sky) to 6,000 cycles, the rows 2,000,
// the 6x6 solve 3,000; a finest iteration of 640x480 is 22,000 and 8,000.
// Live ICP stage, before (256-thread blocks, 300 rows that every block read, a
// hub block's barrier over the whole table, a square root, sine and cosine per
// update) -> now: 640x480 FP32 132 -> 85 us, mixed 112 -> 94, 1280x720 band
// 123 -> 101, 320x240 FP32 97 -> 66, 32-session band batch in one group 460 ->
// 408.  A barrier of one counter instead of the tagged rows measured 88, 91,
// 96, 68 and 396; finishing the pose in this kernel 4 us more than in its own.

// Current value of the GPU's nanosecond timer.
__device__ inline unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A wait's bound: expired() after kWaitNs, or once the abort word is raised
// (looked at every 64th try); it raises the word.
constexpr unsigned long long kWaitNs = 500000000ull;  // half a second
struct BoundedWait {
  unsigned n = 0;
  unsigned long long t0 = 0;
  __device__ bool expired(unsigned* abort_word) {
    if ((++n & 63u) != 0) return false;
    const unsigned long long t = global_ns();
    if (t0 == 0) t0 = t;
    if (*(volatile unsigned*)abort_word == 0 && t - t0 <= kWaitNs) return false;
    atomicExch(abort_word, 1u);
    return true;
  }
};

__device__ inline uint2 load_word(const uint2* p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return make_uint2((unsigned)w, (unsigned)(w >> 32));
}
__device__ inline void store_word(uint2* p, unsigned data, unsigned tag) {
  const unsigned long long w = ((unsigned long long)tag << 32) | data;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
// Value k of a row: words k and 32 + k.
__device__ inline void put_value(uint2* row, int k, double x, unsigned tag) {
  store_word(row + k, (unsigned)__double2loint(x), tag);
  store_word(row + 32 + k, (unsigned)__double2hiint(x), tag);
}

// Lane k's values of this warp's rows (w, w + 16, ... below ntiles) once they
// carry 'tag'; false when the wait ran out.  All rows are asked for at once,
// then those that are not there yet again.
__device__ inline bool wait_rows(const uint2* rows, int ntiles, unsigned tag,
                                 unsigned* abort_word, double (&v)[kWarpRows]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned missing = 0;
#pragma unroll
  for (int i = 0; i < kWarpRows; ++i) {
    v[i] = 0.0;
    if (w + i * kFrameWarps < ntiles) missing |= 1u << i;
  }
  BoundedWait wait;
  while (missing) {
    uint2 lo[kWarpRows], hi[kWarpRows];
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i)
      if (missing >> i & 1u) {
        const uint2* r = rows + (size_t)(w + i * kFrameWarps) * kIcpRowWords + lane;
        lo[i] = load_word(r);
        hi[i] = load_word(r + 32);
      }
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i)
      if (missing >> i & 1u) {
        const bool here = lane >= kIcpVals || (lo[i].y == tag && hi[i].y == tag);
        if (__all_sync(0xffffffffu, here)) {
          missing &= ~(1u << i);
          if (lane < kIcpVals) v[i] = __hiloint2double((int)hi[i].x, (int)lo[i].x);
        }
      }
    if (missing && __any_sync(0xffffffffu, lane == 0 && wait.expired(abort_word))) return false;
  }
  return true;
}

// The persistent kernel's per-block solver state.
struct FrameState {
  double tot[kIcpVals];
  double inc[6], prev[6];
  M4f T;  // the transform of the iteration
  int conv, have, iters[3], inliers[3];
  float rms[3];
  unsigned epoch;
};

// The rows of the level, then the iteration's update; false when the wait ran
// out (block-uniform).  Out of line: its registers are not the sums'.
template <bool KAHAN>
__device__ __noinline__ bool finish_iteration(const uint2* rows, const FrameLevel& L,
                                              unsigned tag, unsigned* abort_word, int pl, int it,
                                              FrameState& F, double* red) {
  double v[kWarpRows];
  const bool good = wait_rows(rows, L.ntiles, tag, abort_word, v);
  if (!__syncthreads_and(good)) return false;
  level_update<KAHAN>(v, L.P, pl, it, F.tot, red, F.inc, F.prev, F.T.m, &F.conv, F.iters,
                      F.inliers, F.rms);
  return true;
}

// This block's session among the table's sessions of its kind, its index
// among the session's blocks and their number, in shared memory (out[3]).
template <bool KAHAN>
__device__ inline void find_session(const SessDev* __restrict__ tab, int n, int pool, int base,
                                    int* out) {
  __shared__ long long sum_s;
  __shared__ int part[kFrameWarps], carry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    sum_s = 0;
    carry = 0;
    out[0] = out[1] = out[2] = 0;
  }
  __syncthreads();
  long long mine = 0;
  for (int j = tid; j < n; j += kIcpFrameThreads)
    if ((tab[j].icpp.kahan != 0) == KAHAN) mine += icp_weight(tab[j].npx, KAHAN);
  if (mine) atomicAdd(reinterpret_cast<unsigned long long*>(&sum_s), (unsigned long long)mine);
  __syncthreads();
  for (int j0 = 0; j0 < n; j0 += kIcpFrameThreads) {
    const int j = j0 + tid;
    int b = 0;
    if (j < n && (tab[j].icpp.kahan != 0) == KAHAN)
      b = icp_share(tab[j].npx, KAHAN, sum_s, pool, base);
    int sum = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += u;
    }
    if (lane == 31) part[warp] = sum;
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; ++w) before += part[w];
    const int first = before + sum - b;
    if (b > 0 && (int)blockIdx.x >= first && (int)blockIdx.x < first + b) {
      out[0] = j;
      out[1] = (int)blockIdx.x - first;
      out[2] = b;
    }
    __syncthreads();
    if (tid == kIcpFrameThreads - 1) carry = before + sum;
    __syncthreads();
  }
}

// One instantiation per summation kind: a table whose sessions sum both
// ways gets one launch per kind, each over that kind's sessions only.
template <bool KAHAN>
__global__ void __launch_bounds__(kIcpFrameThreads, 1)
    fused_icp_persistent_kernel(const SessDev* __restrict__ tab, int n, int pool, int base,
                                int it0, int it1, int it2) {
  // this block's session, its index among the session's blocks, their number
  __shared__ int who[3];
  if (n == 1) {
    if (threadIdx.x == 0) {
      who[0] = 0;
      who[1] = blockIdx.x;
      who[2] = gridDim.x;
    }
    __syncthreads();
  } else {
    find_session<KAHAN>(tab, n, pool, base, who);
  }
  const SessDev& S = tab[who[0]];
  const int local = who[1], nblk = who[2];
  if (nblk == 0) return;  // (the grid is the sum of the shares)
  // the session's solver state, one copy per block
  __shared__ double red[kTileBatch * kFrameWarps * kIcpVals];
  __shared__ FrameState F;
  __shared__ FrameLevel Ls;  // the iteration's level
  float* const Tf = F.T.m;
  if (threadIdx.x < 6) {
    F.inc[threadIdx.x] = S.icp->inc[threadIdx.x];
    F.prev[threadIdx.x] = S.icp->prev[threadIdx.x];
  }
  if (threadIdx.x < 16) Tf[threadIdx.x] = S.icp->T[threadIdx.x];
  if (threadIdx.x < 3) {
    F.iters[threadIdx.x] = S.icp->iters[threadIdx.x];
    F.inliers[threadIdx.x] = S.icp->inliers[threadIdx.x];
    F.rms[threadIdx.x] = S.icp->rms[threadIdx.x];
  }
  if (threadIdx.x == 0) {
    F.conv = S.icp->converged;
    F.have = S.icp->have_target;
    F.epoch = S.icp_bar[0];
  }
  __syncthreads();
  const int maxit[3] = {it0, it1, it2};
  const unsigned epoch = F.epoch;
  unsigned* const abort_word = S.icp_bar + kIcpAbort;
  uint2* const rows =
      reinterpret_cast<uint2*>(reinterpret_cast<char*>(S.partials) + icp_rows_offset());
  // the last level this block has a tile of
  int last = -1;
  for (int pl = 0; pl < 3; ++pl)
    if (min(maxit[pl], S.slot_iters[pl]) > 1 &&
        local < icp_tiles(S.ls[S.slot_level[pl]].rows * S.ls[S.slot_level[pl]].cols, KAHAN))
      last = pl;
  if (local == 0) last = 2;
  bool good = true;
  for (int pl = 0; pl <= last; ++pl) {
    const int l = S.slot_level[pl], iters_pl = min(maxit[pl], S.slot_iters[pl]);
    if (!F.have || iters_pl <= 1) continue;  // (alike in every block of the session)
    const int ntiles = icp_tiles(S.ls[l].rows * S.ls[l].cols, KAHAN);
    const unsigned tag0 = epoch + (unsigned)pl * 1024u;  // iterations 1 .. 999, then the state
    uint2* const state = rows + (size_t)icp_state_row(pl) * kIcpRowWords;
    if (local < ntiles) {
      // level and transform stay in shared memory (registers go to the sums)
      if (threadIdx.x == 0) Ls = level_of(S, l);
      __syncthreads();
      for (int it = 1; it < iters_pl; ++it) {
        // every block at the level holds the state: they leave it together
        if (it > 1 && F.conv) break;
        uint2* const part = rows + (size_t)icp_row(pl, it, 0) * kIcpRowWords;
        const unsigned tag = tag0 + (unsigned)it;
        tile_partials<KAHAN>(Ls, F.T, local, nblk, red,
                             [&](int tile, int k, double x) {
                               put_value(part + (size_t)tile * kIcpRowWords, k, x, tag);
                             });
        good = finish_iteration<KAHAN>(part, Ls, tag, abort_word, pl, it, F, red);
        if (!good) break;
      }
      if (!good) break;  // (block-uniform)
      __syncthreads();
      if (local == 0 && nblk > ntiles) {  // for the blocks without a tile here
        const unsigned tag = tag0 + 1023u;
        const int k = threadIdx.x;
        if (k < 12) put_value(state, k, k < 6 ? F.inc[k] : F.prev[k - 6], tag);
        else if (k < 28) store_word(state + k, __float_as_uint(Tf[k - 12]), tag);
      }
      __syncthreads();
    } else {
      if (threadIdx.x < 32) {
        const unsigned tag = tag0 + 1023u;
        const int k = threadIdx.x;
        uint2 a = make_uint2(0u, 0u), b = a;
        BoundedWait wait;
        for (;;) {
          bool here = true;
          if (k < 28) {
            a = load_word(state + k);
            here = a.y == tag;
          }
          if (k < 12) {
            b = load_word(state + 32 + k);
            here = here && b.y == tag;
          }
          if (__all_sync(0xffffffffu, here)) break;
          if (__any_sync(0xffffffffu, k == 0 && wait.expired(abort_word))) {
            good = false;
            break;
          }
          __nanosleep(200);  // (leave L2 to the level's blocks)
        }
        if (k < 12) (k < 6 ? F.inc[k] : F.prev[k - 6]) = __hiloint2double((int)b.x, (int)a.x);
        else if (k < 28) Tf[k - 12] = __uint_as_float(a.x);
      }
      if (!__syncthreads_and(good)) {
        good = false;
        break;
      }
    }
  }
  if (!good && threadIdx.x == 0) atomicExch(&S.vol.cnt->icp_timeout, 1);
  __syncthreads();
  // the session's first block hands the state on to the pose finalisation
  // (after a timeout it stays as the frame found it)
  if (local == 0 && good) {
    if (threadIdx.x < 6) {
      S.icp->inc[threadIdx.x] = F.inc[threadIdx.x];
      S.icp->prev[threadIdx.x] = F.prev[threadIdx.x];
    }
    if (threadIdx.x < 16) S.icp->T[threadIdx.x] = Tf[threadIdx.x];
    if (threadIdx.x < 3) {
      S.icp->iters[threadIdx.x] = F.iters[threadIdx.x];
      S.icp->inliers[threadIdx.x] = F.inliers[threadIdx.x];
      S.icp->rms[threadIdx.x] = F.rms[threadIdx.x];
    }
    if (threadIdx.x == 0) S.icp->converged = F.conv;
  }
}

// The bounded wait run alone: each block adds one to the counter and waits
// until it holds 'expect' (more than were launched: a wait that cannot
// complete, which must end in the timeout).
__global__ void barrier_selftest_kernel(unsigned* bar, unsigned expect) {
  if (threadIdx.x != 0) return;
  atomicAdd(bar, 1u);
  BoundedWait wait;
  while (*(volatile unsigned*)bar < expect)
    if (wait.expired(bar + kIcpAbort)) return;
}

// Normal equations only (stage entry point): no solver state.  The transform
// comes by value (Tdev null) and 'out' may be pinned host memory: a call is then
// one launch and a wait, without a copy each way (640x480 with colours: 36.4 us
// with both copies, now 28.6).
__global__ void __launch_bounds__(kIcpThreads)
    icp_reduce_kernel(const __grid_constant__ IcpLevel L, const __grid_constant__ IcpParams P,
                      const float* __restrict__ Tdev, const __grid_constant__ M4f Tval,
                      double* __restrict__ partials, unsigned int* ticket_ctr,
                      double* __restrict__ out) {
  __shared__ double red[(kIcpThreads / 32) * kIcpVals];
  __shared__ M4f Ts;
  if (threadIdx.x < 16) Ts.m[threadIdx.x] = Tdev ? Tdev[threadIdx.x] : Tval.m[threadIdx.x];
  __syncthreads();
  const M4f T = Ts;
  Acc a;
#pragma unroll
  for (int k = 0; k < kIcpVals; ++k) {
    a.v[k] = 0.0f;
    a.d[k] = 0.0;
  }
  const int n = L.s.rows * L.s.cols;
  for (int idx = blockIdx.x * kIcpThreads + threadIdx.x; idx < n;
       idx += gridDim.x * kIcpThreads)
    pixel_terms<false>(L, P, T, idx, a);
  block_reduce<false, kIcpThreads / 32>(a, red);
  if (threadIdx.x < kIcpVals) partials[(size_t)blockIdx.x * kIcpVals + threadIdx.x] = red[threadIdx.x];
  if (!last_block(ticket_ctr, gridDim.x)) return;
  __shared__ double tot[kIcpVals];
  final_reduce(partials, gridDim.x, tot, red);
  if (threadIdx.x < kIcpVals) out[threadIdx.x] = tot[threadIdx.x];
  if (threadIdx.x == 0) *ticket_ctr = 0;
}

__device__ void finish_pose(PoseState* ps) {
  for (int k = 0; k < 16; ++k) ps->posef[k] = (float)ps->pose[k];
  inverse4f(ps->posef, ps->invf);
}

// gnSolver.cu:426-430 + builder pose bookkeeping (one thread).
__device__ void pose_finalize_body(const IcpParams& P, IcpState* st, PoseState* ps) {
  ps->reset = 0;
  if (st->have_target) {
    double s = 0.0;
    for (int k = 0; k < 6; ++k) s += st->inc[k];
    bool reset = isnan(s) || isinf(s) || s >= (double)P.max_inc;
    if (reset)
      for (int k = 0; k < 6; ++k) st->inc[k] = 0.0;
    double E[16];
    se3_exp(st->inc, E);
    if (P.compose_left) matmul4d(E, ps->pose, ps->pose);
    else matmul4d(ps->pose, E, ps->pose);
    ps->reset = reset ? 1 : 0;
  } else {
    for (int k = 0; k < 3; ++k) {
      st->iters[k] = 0;
      st->inliers[k] = 0;
      st->rms[k] = 0.0f;
    }
  }
  for (int k = 0; k < 6; ++k) {
    ps->last_inc[k] = st->inc[k];
    st->inc[k] = 0.0;
    st->prev[k] = 0.0;
  }
  for (int k = 0; k < 16; ++k) st->T[k] = (k % 5 == 0) ? 1.0f : 0.0f;
  st->converged = 0;
  st->ticket = 0;
  finish_pose(ps);
}

__global__ void pose_finalize_kernel(IcpParams P, IcpState* st, PoseState* ps) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  pose_finalize_body(P, st, ps);
}

// one thread per session; bump != 0 also advances the frame counter (within the
// persistent kernel it measured 4 us slower)
__global__ void fused_pose_finalize_kernel(const SessDev* __restrict__ tab, int n, int bump) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const SessDev& S = tab[s];
  pose_finalize_body(S.icpp, S.icp, S.pose);
  advance_epoch(S.icp_bar, S.partials);  // the next launch's tags
  S.icp_bar[kIcpAbort] = 0;
  if (bump) S.pose->frame += 1;
}

// SE(3) logarithm of a rigid transform T (row-major 4x4), the inverse of
// se3_exp: w from the rotation angle and axis, t = V^-1 translation with
// V^-1 = I - W/2 + (1 - a / (2 b)) / th^2 W^2 (a = sin th / th,
// b = (1 - cos th) / th^2; series below th = 1e-4).
__device__ void se3_log(const double* T, double* xi) {
  const double tr = T[0] + T[5] + T[10];
  double c = 0.5 * (tr - 1.0);
  c = c > 1.0 ? 1.0 : (c < -1.0 ? -1.0 : c);
  const double th = acos(c);
  const double vx = T[9] - T[6], vy = T[2] - T[8], vz = T[4] - T[1];
  double f;  // th / (2 sin th)
  if (th < 1e-4) f = 0.5 + th * th / 12.0;
  else f = th / (2.0 * sin(th));
  const double w0 = f * vx, w1 = f * vy, w2 = f * vz;
  double g;  // (1 - a / (2 b)) / th^2
  if (th < 1e-4) g = 1.0 / 12.0 + th * th / 720.0;
  else g = (1.0 - (sin(th) / th) / (2.0 * (1.0 - cos(th)) / (th * th))) / (th * th);
  const double W[9] = {0, -w2, w1, w2, 0, -w0, -w1, w0, 0};
  double W2[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double s = 0;
      for (int k = 0; k < 3; ++k) s += W[i * 3 + k] * W[k * 3 + j];
      W2[i * 3 + j] = s;
    }
  const double t[3] = {T[3], T[7], T[11]};
  xi[0] = w0;
  xi[1] = w1;
  xi[2] = w2;
  for (int i = 0; i < 3; ++i) {
    double s = 0;
    for (int j = 0; j < 3; ++j) {
      const double Vi = (i == j ? 1.0 : 0.0) - 0.5 * W[i * 3 + j] + g * W2[i * 3 + j];
      s += Vi * t[j];
    }
    xi[3 + i] = s;
  }
}

// rel = pose^-1 * hint (hint * pose^-1 when increments compose on the
// left); the solver starts at log(rel).  Before the first target exists
// the hint becomes the pose.
__global__ void pose_hint_kernel(PoseState* ps, IcpState* st, const double* hint,
                                 int compose_left) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (!st->have_target) {
    for (int k = 0; k < 16; ++k) ps->pose[k] = hint[k];
    finish_pose(ps);
    return;
  }
  const double* P = ps->pose;
  double inv[16];
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 3; ++j) inv[i * 4 + j] = P[j * 4 + i];
    inv[i * 4 + 3] = -(P[0 * 4 + i] * P[3] + P[1 * 4 + i] * P[7] + P[2 * 4 + i] * P[11]);
  }
  inv[12] = inv[13] = inv[14] = 0.0;
  inv[15] = 1.0;
  double rel[16];
  if (compose_left) matmul4d(hint, inv, rel);
  else matmul4d(inv, hint, rel);
  double xi[6];
  se3_log(rel, xi);
  for (int k = 0; k < 6; ++k) {
    st->inc[k] = xi[k];
    st->prev[k] = xi[k];
  }
  double Td[16];
  se3_exp(xi, Td);
  for (int k = 0; k < 16; ++k) st->T[k] = (float)Td[k];
}

__global__ void pose_set_kernel(PoseState* ps, const double* pose) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  for (int k = 0; k < 16; ++k) ps->pose[k] = pose[k];
  finish_pose(ps);
}

}  // namespace

size_t icp_scratch_bytes() { return sizeof(double) * (size_t)kIcpMaxBlocks * kIcpVals; }

int icp_persistent_capacity(int device) {
  static std::mutex mu;
  static int cap[64] = {};
  if (device < 0 || device >= 64) return 0;
  std::lock_guard<std::mutex> lk(mu);
  if (cap[device] == 0) {
    int coop = 0, sms = 0, per_sm = 0, per_k = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_icp_persistent_kernel<false>,
                                                      kIcpFrameThreads, 0) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_k, fused_icp_persistent_kernel<true>,
                                                      kIcpFrameThreads, 0) != cudaSuccess) {
      cudaGetLastError();
      coop = 0;
    }
    per_sm = std::min(per_sm, per_k);
    cap[device] = coop ? std::max(1, per_sm * sms) : -1;
  }
  return cap[device] > 0 ? cap[device] : 0;
}

template <bool KAHAN>
static void launch_persistent(const SessDev* tab, const BatchShape& b, int part, cudaStream_t st) {
  const int grid = b.icp.grid[part][KAHAN];
  if (grid == 0) return;
  const int first = icp_part_first(b.n, b.icp.parts, part);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kIcpFrameThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, fused_icp_persistent_kernel<KAHAN>, tab + first,
                     icp_part_first(b.n, b.icp.parts, part + 1) - first, b.icp.pool[part][KAHAN],
                     b.icp.base[part][KAHAN], b.max_slot_iters[0], b.max_slot_iters[1],
                     b.max_slot_iters[2]);
}

void fused_icp_persistent(const SessDev* tab, const BatchShape& b, cudaStream_t st) {
  for (int part = 0; part < b.icp.parts; ++part) {
    launch_persistent<false>(tab, b, part, st);
    launch_persistent<true>(tab, b, part, st);
  }
}

dyn_status icp_barrier_selftest(int blocks, int missing, unsigned* bar_dev, cudaStream_t st) {
  if (blocks < 1 || missing < 0) return DYN_ERR_INVALID_ARG;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, barrier_selftest_kernel, 32, 0) !=
          cudaSuccess) {
    cudaGetLastError();
    return DYN_ERR_CUDA;
  }
  if (blocks > per_sm * sms) return DYN_ERR_INVALID_ARG;  // not all resident at once
  if (cudaMemsetAsync(bar_dev, 0, kIcpBarWords * sizeof(unsigned), st) != cudaSuccess)
    return DYN_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(32);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e =
      cudaLaunchKernelEx(&cfg, barrier_selftest_kernel, bar_dev, (unsigned)(blocks + missing));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e == cudaErrorCooperativeLaunchTooLarge ? DYN_ERR_INVALID_ARG : DYN_ERR_CUDA;
  }
  int abort_h = 0;
  if (cudaMemcpyAsync(&abort_h, bar_dev + kIcpAbort, sizeof(int),
                      cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return DYN_ERR_CUDA;
  return abort_h ? DYN_ERR_TIMEOUT : DYN_OK;
}

void launch_pose_finalize(const IcpParams& P, IcpState* st, PoseState* ps, cudaStream_t stream) {
  pose_finalize_kernel<<<1, 32, 0, stream>>>(P, st, ps);
}

void launch_pose_hint(PoseState* ps, IcpState* st, const double* hint_dev, int compose_left,
                      cudaStream_t stream) {
  pose_hint_kernel<<<1, 32, 0, stream>>>(ps, st, hint_dev, compose_left);
}

void launch_pose_set(PoseState* ps, const double* pose_dev, cudaStream_t stream) {
  pose_set_kernel<<<1, 32, 0, stream>>>(ps, pose_dev);
}

void launch_icp_reduce_only(const IcpLevel& L, const IcpParams& P, const M4f& T,
                            double* partials, unsigned int* ticket, double* out,
                            cudaStream_t stream) {
  icp_reduce_kernel<<<icp_stage_grid(L.s.rows * L.s.cols), kIcpThreads, 0, stream>>>(
      L, P, nullptr, T, partials, ticket, out);
}

void launch_icp_reduce_grid(const IcpLevel& L, const IcpParams& P, const float* T_dev,
                            double* partials, unsigned int* ticket, double* out_dev, int grid,
                            cudaStream_t stream) {
  icp_reduce_kernel<<<grid, kIcpThreads, 0, stream>>>(L, P, T_dev, M4f{}, partials, ticket,
                                                      out_dev);
}

// 'chained': launched with programmatic stream serialization, so that the
// kernel's launch and prologue overlap its predecessor (an earlier ICP
// iteration kernel, never the first of the frame, whose predecessor writes
// the level maps).
void fused_icp_iteration(const SessDev* tab, const BatchShape& b, int slot, int it, bool chained,
                         cudaStream_t st) {
  if (it >= b.max_slot_iters[slot]) return;
  cudaLaunchConfig_t cfg = {};
  // (the table's most tiles, not its largest level's: a smaller level may have more)
  cfg.gridDim = dim3(b.max_slot_tiles[slot], 1, b.n);
  cfg.blockDim = dim3(kIcpFrameThreads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  if (b.kahan_mask & 1) {
    cfg.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, fused_icp_iteration_kernel<false>, tab, slot, it);
    chained = true;
  }
  if (b.kahan_mask & 2) {
    cfg.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, fused_icp_iteration_kernel<true>, tab, slot, it);
  }
}

void fused_pose_finalize(const SessDev* tab, const BatchShape& b, int bump, cudaStream_t st) {
  fused_pose_finalize_kernel<<<(b.n + 31) / 32, 32, 0, st>>>(tab, b.n, bump);
}

}  // namespace dyn
