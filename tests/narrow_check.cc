// Test harness of csrc/narrow.h: how many of the given doubles it covers, and how many of those differ from the
// conversion of the language.
#include <cstring>

#include "narrow.h"

extern "C" long long narrow_check(const double* x, long long n, long long* covered) {
  long long wrong = 0;
  *covered = 0;
  for (long long i = 0; i < n; ++i) {
    uint64_t b;
    std::memcpy(&b, x + i, 8);
    const uint32_t hi = static_cast<uint32_t>(b >> 32), lo = static_cast<uint32_t>(b);
    if (!leapgb::narrow_covers(hi, lo)) continue;
    ++*covered;
    const float f = static_cast<float>(x[i]);
    uint32_t want;
    std::memcpy(&want, &f, 4);
    wrong += leapgb::narrow_bits(hi, lo) != want;
  }
  return wrong;
}
