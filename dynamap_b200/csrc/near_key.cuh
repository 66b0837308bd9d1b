// near_key.cuh -- the keys of allocation's CTA-local block set.
#pragma once
#include "common.cuh"

namespace dyn {

namespace {

constexpr int kSetBits = 11, kSetSlots = 1 << kSetBits;  // the set's slots

// A block in a CTA's set: its offset from the camera's block, biased fields of
// kBits bits an axis, so that a step is one addition and the 32-bit form of it
// (10 bits) one multiplication away from its slot.  The 64-bit form (21 bits,
// as wide as the volume's own keys) serves sessions whose rays may take more
// steps than 10 bits hold.
template <class K>
struct NearKey;
template <>
struct NearKey<unsigned> {
  static constexpr int kBits = 10;
  static __device__ unsigned slot(unsigned k) { return (k * 0x9E3779B1u) >> (32 - kSetBits); }
};
template <>
struct NearKey<unsigned long long> {
  static constexpr int kBits = 21;
  static __device__ unsigned slot(unsigned long long k) {
    return (unsigned)((k * 0x9E3779B97F4A7C15ull) >> (64 - kSetBits));
  }
};
template <class K>
__device__ inline K near_key(int dx, int dy, int dz) {
  constexpr int B = NearKey<K>::kBits, half = 1 << (B - 1);
  return ((K)(unsigned)(dx + half) << (2 * B)) + ((K)(unsigned)(dy + half) << B) +
         (K)(unsigned)(dz + half);
}
template <class K>
__device__ inline unsigned long long volume_key(K k, const int (&cam)[3]) {
  constexpr int B = NearKey<K>::kBits, half = 1 << (B - 1), mask = (1 << B) - 1;
  return pack_key((int)((k >> (2 * B)) & mask) - half + cam[0],
                  (int)((k >> B) & mask) - half + cam[1], (int)(k & mask) - half + cam[2]);
}
__device__ inline int apart_of(int a, int b) { return (int)((unsigned)a - (unsigned)b); }
// Whether a walk of up to 'left' steps (and the pre-step) from offset (ox, oy,
// oz) stays inside the fields, so that no key carries from one into another or
// is the empty slot's value.
template <class K>
__device__ inline bool near_walk(int ox, int oy, int oz, int left) {
  constexpr unsigned half = 1u << (NearKey<K>::kBits - 1);
  const unsigned far = half - 2u - (unsigned)left;  // the farthest start
  return (unsigned)left <= half - 2u && (unsigned)ox + far <= 2u * far &&
         (unsigned)oy + far <= 2u * far && (unsigned)oz + far <= 2u * far;
}

}  // namespace

}  // namespace dyn
