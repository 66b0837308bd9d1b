// The tile-local keys of allocation (dynamap_b200/csrc/near_key.cuh) on the CPU.
#include "cuda_emu.h"

#include <cstdint>

#include "../../dynamap_b200/csrc/near_key.cuh"

// A walk from offset o of camera block cam, 'left' steps along the sign s of one
// axis after a pre-step along -s on all of them, its keys stepped as
// allocation steps them.  Returns -1 where the walk is refused, else the number
// of keys that are the empty slot's or name another block.
template <class K>
static int walk(const int* o, const int* cam, int left, int axis, int s) {
  using namespace dyn;
  if (!near_walk<K>(o[0], o[1], o[2], left)) return -1;
  constexpr int B = NearKey<K>::kBits;
  const int c[3] = {cam[0], cam[1], cam[2]};
  int p[3] = {o[0] - s, o[1] - s, o[2] - s}, bad = 0;
  K key = near_key<K>(p[0], p[1], p[2]);
  const K step = (K)(long long)s << (axis == 0 ? 2 * B : (axis == 1 ? B : 0));
  for (int k = 0; k <= left; ++k) {
    if (k) {
      key += step;
      p[axis] += s;
    }
    bad += key == ~(K)0;
    bad += volume_key(key, c) != pack_key(p[0] + c[0], p[1] + c[1], p[2] + c[2]);
  }
  return bad;
}

extern "C" int near_walk_check(int wide, const int* o, const int* cam, int left, int axis, int s) {
  return wide ? walk<unsigned long long>(o, cam, left, axis, s)
              : walk<unsigned>(o, cam, left, axis, s);
}
