// Conversion of a double to float on the integer pipe, for the device and for the host.
//
// The conversion instruction runs at the FP64 rate (2 lanes per clock and SM), so that a 2-pol complex<double> sample
// of a warp's rows costs 64 clocks of the SM, as much as 16 directions' arithmetic on it; the nine integer operations
// here cost an eighth of that.
#pragma once

#include <cstdint>

#ifndef LEAP_HD
#ifdef __CUDACC__
#define LEAP_HD __host__ __device__ __forceinline__
#else
#define LEAP_HD inline
#endif
#endif

namespace leapgb {

// Whether narrow_bits covers the double (hi : lo): zero, or a magnitude in [2^-126, 2^128), which rounds to a normal
// float or to infinity.
LEAP_HD bool narrow_covers(uint32_t hi, uint32_t lo) {
  return (hi << 1) - (897u << 21) < (254u << 21) || ((hi << 1) | lo) == 0;
}

// The bits of the nearest float, ties to even.
LEAP_HD uint32_t narrow_bits(uint32_t hi, uint32_t lo) {
  if (((hi << 1) | lo) == 0) return hi;
  uint32_t t = (hi << 3) | (lo >> 29);                        // low bits of the exponent, 23 bits
  t += ((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (t & 1)) >> 29;    // the 29 bits below, rounded
  return ((t + 0x40000000u) & 0x7FFFFFFFu) | (hi & 0x80000000u);
}

#ifdef __CUDACC__
__device__ __forceinline__ float narrow(double x) {
  const uint32_t hi = static_cast<uint32_t>(__double2hiint(x)), lo = static_cast<uint32_t>(__double2loint(x));
  return narrow_covers(hi, lo) ? __uint_as_float(narrow_bits(hi, lo)) : static_cast<float>(x);
}
__device__ __forceinline__ float narrow(float x) { return x; }
#endif

}  // namespace leapgb
