// The division by a hoisted reciprocal of the raycast's march (div_by in
// dynamap_b200/csrc/tsdf.cu), the same operations on the CPU: how many of the
// dividends of two binades (every significand, both signs) differ from the
// IEEE quotient.
#include <cmath>
#include <cstdint>
#include <cstring>

extern "C" int64_t march_div_mismatches(float b, float lo) {
  const float yh = 1.0f / b;
  const float yl = std::fmaf(-b, yh, 1.0f) * yh;
  uint32_t u;
  std::memcpy(&u, &lo, 4);
  int64_t bad = 0;
  for (uint32_t k = 0; k < (1u << 24); ++k) {
    const uint32_t w = u + k;
    float a;
    std::memcpy(&a, &w, 4);
    const float q = std::fmaf(a, yh, a * yl);
    const float r = std::fmaf(std::fmaf(-b, q, a), yh, q);
    bad += r != a / b;
    const float an = -a;
    const float qn = std::fmaf(an, yh, an * yl);
    bad += std::fmaf(std::fmaf(-b, qn, an), yh, qn) != an / b;
  }
  return bad;
}
