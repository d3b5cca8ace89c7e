// Host side: the integers a seeded CPU generator draws, straight into a 32-bit array.
//
// The shortlist head's random negatives are what torch.randint(0, V, shape, generator=torch.Generator().manual_seed(s))
// returns (the reference draws them per step, output.py:86-94): the 32-bit Mersenne Twister of Matsumoto and Nishimura
// (MT19937, ACM TOMACS 8(1), 1998), one output per element, modulo the range.  Through torch that is an int64 tensor and a
// conversion of it: 1.7 ms for the 128 x 128 x 32 negatives of a step, as long as half the step takes on the device; this
// writes the int32 array in 0.9 ms.

#include <stdint.h>

#include "rte_b200.h"

namespace {

constexpr int MT_N = 624, MT_M = 397;

inline uint32_t mix(uint32_t hi, uint32_t lo, uint32_t far) {
  const uint32_t y = (hi & 0x80000000u) | (lo & 0x7fffffffu);
  return far ^ (y >> 1) ^ ((0u - (lo & 1u)) & 0x9908b0dfu);
}

}  // namespace

extern "C" int rte_host_randint(uint64_t seed, int64_t n, int32_t range, int32_t* out) {
  if (out == nullptr || n < 0 || range <= 0 || range >= (1 << 28)) return RTE_ERR_BAD_ARG;
  uint32_t mt[MT_N];
  mt[0] = static_cast<uint32_t>(seed);
  for (int i = 1; i < MT_N; ++i) mt[i] = 1812433253u * (mt[i - 1] ^ (mt[i - 1] >> 30)) + static_cast<uint32_t>(i);
  const uint32_t r = static_cast<uint32_t>(range);
  const bool pow2 = (r & (r - 1)) == 0;
  for (int64_t at = 0; at < n; at += MT_N) {
    for (int i = 0; i < MT_N - MT_M; ++i) mt[i] = mix(mt[i], mt[i + 1], mt[i + MT_M]);
    for (int i = MT_N - MT_M; i < MT_N - 1; ++i) mt[i] = mix(mt[i], mt[i + 1], mt[i + MT_M - MT_N]);
    mt[MT_N - 1] = mix(mt[MT_N - 1], mt[0], mt[MT_M - 1]);
    const int count = n - at < MT_N ? static_cast<int>(n - at) : MT_N;
    int32_t* o = out + at;
    uint32_t y[MT_N];                      // (loops of their own: the first vectorises)
    for (int i = 0; i < count; ++i) {
      uint32_t v = mt[i];
      v ^= v >> 11; v ^= (v << 7) & 0x9d2c5680u; v ^= (v << 15) & 0xefc60000u; v ^= v >> 18;
      y[i] = v;
    }
    if (pow2) {
      for (int i = 0; i < count; ++i) o[i] = static_cast<int32_t>(y[i] & (r - 1));
    } else {
      // y mod r without a division: one off in the quotient at most, put right by the comparisons
      const double inv = 1.0 / r;
      for (int i = 0; i < count; ++i) {
        int32_t rem = static_cast<int32_t>(y[i] - static_cast<uint32_t>(static_cast<int64_t>(y[i] * inv)) * r);
        rem += rem < 0 ? static_cast<int32_t>(r) : 0;
        rem -= rem >= static_cast<int32_t>(r) ? static_cast<int32_t>(r) : 0;
        o[i] = rem;
      }
    }
  }
  return RTE_OK;
}
