// Fixed-point phasors of the all-FP64 rotate + average (kernels_fixed.cuh), as plain C++ for the
// device and for the host.
//
// For one row and direction the reference's argument at channel c is arg_c = fl(sf / lambda_c),
// sf = -2 pi (w_rot - w), lambda_c = fl(c / fl(f0 + fl(c df))) (LA/algorithm/cpu/CpuLeapCalibrator.cc:190-198,
// LA/model/cpu/MetaData.h:95-98).  Here sf / lambda_c is carried as a fixed-point number of radians with
// the unit ("LSB") 2^(E-63), |arg| < 2^E for every channel, i.e. 2^-10 of the unit in the last place that an
// FP64 argument in [2^(E-1), 2^E) has:
//   * its linear part sf (f0 + c df) / c_light is a 96-bit accumulator (32 bits below the LSB), advanced
//     by one addition per channel from 128-bit products formed once per (row, direction, timestep);
//   * lambda_c's own rounding enters as a per-channel correction rho_c, 2^-82 relative, from the host;
//   * rounding that sum, taken to 2^-18 LSB, to the argument's 53 bits gives the reference's argument (up to
//     one unit in its last place where sf / lambda_c is within a few 2^-18 LSB of a tie: one sample in 10^7).
//     Taken to an LSB only, one argument in 700 came out a unit off, and for arguments of thousands of radians
//     the averages had 8 times the error of the direct FP64 form.
// e_c, the rounded argument minus the linear part, is small, and z_c = exp(i arg_c) follows from z_{c-1} by one
// complex multiplication with exp(i step) turned by the small angle e_c - e_{c-1}: the errors of the
// recurrence are those of 60-bit fixed-point products, far below those of an FP64 one.
//
// Numbers in [-1, 1] are 60-bit fixed point in two limbs of radix 2^30: x = (h 2^30 + l) 2^-60, l in
// [0, 2^30).  Products of limbs go to 64-bit sums (IMAD.WIDE: 32 lanes per clock and SM measured, where
// FP64 FMAs run at 2); the product of the two low limbs is dropped.  60 bits, not
// fewer, because the rounding of the channel step's phasor adds up over the channels of a block: with
// 56 bits the phasors were up to 50 units of 2^-56 off after 32 channels.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LEAP_HD __host__ __device__ __forceinline__
#else
#define LEAP_HD inline
#endif

namespace leapgb {

constexpr int kFxMaxExp = 19;         // |arg| < 2^19 rad; beyond it the FP64 path takes the row
constexpr int kFxMinExp = 4;          // smaller arguments keep the LSB 2^-59 rad
constexpr uint32_t kFxLimb = 1u << 30;
constexpr int kFxFrac = 18;           // bits below the LSB in a residual
constexpr int32_t kFxMaxRho = 6400;   // three roundings of 2^-53 in lambda_c: 6144 2^-64
constexpr int kFxTable = 1024;        // entries of each of the two phasor tables

// (hi : lo) 2^(exp - 128) with the top bit of hi set, or 0 (hi == 0).
struct FxRatio {
  uint64_t hi, lo;
  int32_t exp, pad;
};

// The spectral window of a call.
struct FxSpectrum {
  FxRatio k0;     // f0 / c_light
  FxRatio k1;     // |df| / c_light
  FxRatio kt;     // |df| / (2 pi c_light)
  double kmax;    // at least max_c 1 / lambda_c
  int32_t s1;     // sign of df (+1 or -1)
  int32_t pad;
};

struct FxLimbs {  // a complex number in [-1, 1]^2
  int32_t rh, rl, ih, il;
};

// Phase of one (row, direction) at the current channel.
struct FxPhase {
  uint64_t v, q;         // integer part of the phase and of the channel step, in LSBs (signed)
  uint32_t vf, qf;       // fractions of an LSB
  int32_t E;             // |arg| < 2^E
  uint32_t sign;         // ~0 where sf is negative, else 0
  int32_t e;             // rounded argument minus phase, in 2^-kFxFrac LSB
};

// (m * (hi : lo)) >> 64, to within one unit.
LEAP_HD unsigned __int128 fx_mul(uint64_t m, uint64_t hi, uint64_t lo) {
  const unsigned __int128 low = (static_cast<unsigned __int128>(m) * lo) >> 64;
  return static_cast<unsigned __int128>(m) * hi + low;
}

LEAP_HD unsigned __int128 fx_shift(unsigned __int128 x, int s) { return s >= 128 ? 0 : x >> s; }

LEAP_HD int32_t fx_clz(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __clz(static_cast<int>(x));
#else
  return x ? __builtin_clz(x) : 32;
#endif
}

// a * b + c.  On the device as a carry pair, which the assembler fuses to one IMAD.WIDE: from mad.wide it
// makes a product and a two-instruction addition where a sum gets several products in a row, and from the
// plain expression 64-bit products of limbs that were cut out of 64-bit numbers.  (A constant c keeps the pair
// from being fused: a sum starts with fx_mul.)
LEAP_HD int64_t fx_mad(int32_t a, int32_t b, int64_t c) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("{\n\t.reg .u32 l, h;\n\tmov.b64 {l, h}, %3;\n\tmad.lo.cc.s32 l, %1, %2, l;\n\tmadc.hi.s32 h, %1, %2, h;\n\t"
      "mov.b64 %0, {l, h};\n\t}"
      : "=l"(r)
      : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return c + static_cast<int64_t>(a) * b;
#endif
}

LEAP_HD void fx_mad(int64_t& acc, int32_t a, int32_t b) { acc = fx_mad(a, b, acc); }

LEAP_HD int64_t fx_mul(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
#else
  return static_cast<int64_t>(a) * b;
#endif
}

// (a * b >> 32) + c
LEAP_HD int32_t fx_mad_hi(int32_t a, int32_t b, int32_t c) {
#ifdef __CUDA_ARCH__
  int32_t r;
  asm("mad.hi.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
#else
  return static_cast<int32_t>((static_cast<int64_t>(a) * b) >> 32) + c;
#endif
}

LEAP_HD FxLimbs fx_limbs(int64_t re, int64_t im) {
  return FxLimbs{static_cast<int32_t>(re >> 30), static_cast<int32_t>(static_cast<uint32_t>(re) & (kFxLimb - 1)),
                 static_cast<int32_t>(im >> 30), static_cast<int32_t>(static_cast<uint32_t>(im) & (kFxLimb - 1))};
}

// x * y as 60-bit integers, rounded down.  (nih, nil): the limbs of -im(x), not the negated ones: of a plainly
// negated operand the assembler makes an IMAD and an IMAD.HI instead of an IMAD.WIDE.
LEAP_HD void fx_product(const FxLimbs& x, int32_t nih, int32_t nil, const FxLimbs& y, int64_t& re, int64_t& im) {
  int64_t hr = fx_mul(x.rh, y.rh), hi = fx_mul(x.rh, y.ih), mr = fx_mul(x.rh, y.rl), mi = fx_mul(x.rh, y.il);
  fx_mad(hr, nih, y.ih);
  fx_mad(hi, x.ih, y.rh);
  fx_mad(mr, x.rl, y.rh);
  fx_mad(mi, x.rl, y.ih);
  fx_mad(mr, nih, y.il);
  fx_mad(mi, x.ih, y.rl);
  fx_mad(mr, nil, y.ih);
  fx_mad(mi, x.il, y.rh);
  re = hr + (mr >> 30);
  im = hi + (mi >> 30);
}

LEAP_HD FxLimbs fx_cmul(const FxLimbs& x, const FxLimbs& y) {
  int64_t re, im;
  fx_product(x, -x.ih, -x.il, y, re, im);
  return fx_limbs(re, im);
}

// exp(2 pi i t / 2^64): a and b are exp(2 pi i j / 2^10) for the top 10 bits of t and exp(2 pi i j / 2^20) for
// the next 10; the remaining angle d, below 6e-6, has cos d = 1 - d^2/2 and sin d = d - d^3/6 to 2^-74.
LEAP_HD FxLimbs fx_turn(uint64_t t, const FxLimbs& a, const FxLimbs& b) {
  const uint64_t u = t & ((uint64_t(1) << 44) - 1);
  // d 2^60 = u 2 pi / 2^4, with 2 pi 2^61 as a 64-bit constant
  const uint64_t p = static_cast<uint64_t>((static_cast<unsigned __int128>(u << 20) * 0xC90FDAA22168C234ull) >> 64);
  const uint32_t x = static_cast<uint32_t>(u >> 12);  // d / (2 pi 2^-20) as a 2^-32 fraction
  const uint32_t x2 = static_cast<uint32_t>((static_cast<uint64_t>(x) * x) >> 32);
  const uint32_t x3 = static_cast<uint32_t>((static_cast<uint64_t>(x2) * x) >> 32);
  // (2 pi 2^-20)^2 / 2 2^66 = 1324675878.8, (2 pi 2^-20)^3 / 6 2^80 = 43349916.8
  const uint32_t half_sq = static_cast<uint32_t>((static_cast<uint64_t>(x2) * 1324675879u + (uint64_t(1) << 37)) >> 38);
  const uint32_t cube = static_cast<uint32_t>((static_cast<uint64_t>(x3) * 43349917u) >> 32);  // d^3/6 in 2^-80
  const int64_t s = static_cast<int64_t>((p + (uint64_t(1) << 20)) >> 21) - ((cube + (1u << 19)) >> 20);
  return fx_cmul(fx_cmul(a, b), fx_limbs((int64_t(1) << 60) - half_sq, s));
}

// Whether sf (any double) can take the fixed-point path with this spectral window.
LEAP_HD bool fx_in_range(double sf, const FxSpectrum& sp) {
  const double m = (sf < 0 ? -sf : sf) * sp.kmax;
  return m < static_cast<double>(1 << kFxMaxExp);  // false for NaN and infinity
}

LEAP_HD uint64_t fx_bits(double x) {
#ifdef __CUDA_ARCH__
  return static_cast<uint64_t>(__double_as_longlong(x));
#else
  union { double d; uint64_t u; } v;
  v.d = x;
  return v.u;
#endif
}

// The rounded argument's distance from the linear phase at the current channel, in 2^-kFxFrac LSB (rho: that of
// lambda_c).  At most (512 + kFxMaxRho / 2) LSB: below 2^30.
LEAP_HD int32_t fx_residual(const FxPhase& ph, int32_t rho) {
  const int32_t hi = static_cast<int32_t>(ph.v >> 32);
  // The low 32 - kFxFrac bits of the phase and kFxFrac bits of its fraction.
  const uint32_t x = (static_cast<uint32_t>(ph.v) << kFxFrac) | (ph.vf >> (32 - kFxFrac));
  const uint32_t y = static_cast<uint32_t>(fx_mad_hi(hi, rho, static_cast<int32_t>(x)));
  const int lz = fx_clz(static_cast<uint32_t>(hi) ^ ph.sign) - 1;  // 0 .. 31: the argument is below 2^(E - lz)
  const int32_t mask = -(1 << (10 + kFxFrac)) >> lz;               // its last place is 2^(10 - lz) LSBs
  const uint32_t half = (1u << (9 + kFxFrac)) >> lz;
  return static_cast<int32_t>(((y + half) & static_cast<uint32_t>(mask)) - x);
}

// Phase of (row, direction) at channel c0, and `turn`, the phase step of a channel as a 2^-64 fraction of a
// turn.  sf must be in range (fx_in_range).
LEAP_HD void fx_setup(FxPhase& ph, double sf, const FxSpectrum& sp, int32_t c0, uint64_t& turn) {
  const uint64_t b = fx_bits(sf);
  const int ex = static_cast<int>((b >> 52) & 0x7FF);
  const uint64_t m = ex ? ((b << 11) | (uint64_t(1) << 63)) : 0;  // |sf| = m 2^(es - 64); denormals are 0
  const int es = ex - 1022;
  const bool neg = (b >> 63) != 0;
  const int eb = static_cast<int>((fx_bits((sf < 0 ? -sf : sf) * sp.kmax) >> 52) & 0x7FF) - 1022;
  ph.E = eb > kFxMinExp ? eb : kFxMinExp;
  ph.sign = neg ? ~0u : 0u;
  unsigned __int128 p = fx_shift(fx_mul(m, sp.k0.hi, sp.k0.lo), 33 + ph.E - es - sp.k0.exp);
  unsigned __int128 q = fx_shift(fx_mul(m, sp.k1.hi, sp.k1.lo), 33 + ph.E - es - sp.k1.exp);
  if (sp.s1 < 0) q = -q;
  p += q * static_cast<uint32_t>(c0);
  if (neg) {
    p = -p;
    q = -q;
  }
  ph.v = static_cast<uint64_t>(p >> 32);
  ph.vf = static_cast<uint32_t>(p);
  ph.q = static_cast<uint64_t>(q >> 32);
  ph.qf = static_cast<uint32_t>(q);
  turn = static_cast<uint64_t>(fx_shift(fx_mul(m, sp.kt.hi, sp.kt.lo), 64 - es - sp.kt.exp));
  if (neg != (sp.s1 < 0)) turn = ~turn + 1;
}

// The rounded argument at the current channel as a 2^-64 fraction of a turn (ph.e must be current).
LEAP_HD uint64_t fx_turns(const FxPhase& ph) {
  const int32_t up = (ph.e + static_cast<int32_t>(ph.vf >> (32 - kFxFrac))) >> kFxFrac;
  uint64_t r = ph.v + static_cast<uint64_t>(static_cast<int64_t>(up));
  const bool neg = static_cast<int64_t>(r) < 0;
  if (neg) r = ~r + 1;
  // r 2^E / pi mod 2^64; the constant is floor(2^128 / pi)
  const uint64_t t = static_cast<uint64_t>(fx_mul(r, 0x517CC1B727220A94ull, 0xFE13ABE8FA9A6EE0ull) >> (64 - ph.E));
  return neg ? ~t + 1 : t;
}

// One channel on: the phase, its residual, and the step's small turn d in units of 2^-62 rad, below 2^31 as
// residuals are below 2^30 (an LSB is 2^(E-1) of these units, E - 1 <= kFxFrac); nd = -d to a unit.
LEAP_HD void fx_advance(FxPhase& ph, int32_t rho, int32_t& d, int32_t& nd) {
#ifdef __CUDA_ARCH__
  uint32_t lo = static_cast<uint32_t>(ph.v), hi = static_cast<uint32_t>(ph.v >> 32);
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
      : "+r"(ph.vf), "+r"(lo), "+r"(hi)
      : "r"(ph.qf), "r"(static_cast<uint32_t>(ph.q)), "r"(static_cast<uint32_t>(ph.q >> 32)));
  ph.v = (static_cast<uint64_t>(hi) << 32) | lo;
#else
  const unsigned __int128 s = ((static_cast<unsigned __int128>(ph.v) << 32) | ph.vf) +
                              ((static_cast<unsigned __int128>(ph.q) << 32) | ph.qf);
  ph.v = static_cast<uint64_t>(s >> 32);
  ph.vf = static_cast<uint32_t>(s);
#endif
  const int32_t e = fx_residual(ph, rho);
  d = (e - ph.e) >> (kFxFrac + 1 - ph.E);
  nd = (ph.e - e) >> (kFxFrac + 1 - ph.E);
  ph.e = e;
}
static_assert(kFxMaxExp <= kFxFrac + 1, "the shift of a residual's difference");

// The phasor z = (re, im) of one channel times the step w turned by the small angle d (2^-62 rad, nd = -d), which
// changes the low limbs of w by less than 2^30.
LEAP_HD void fx_step(int64_t& re, int64_t& im, const FxLimbs& w, int32_t d, int32_t nd) {
  FxLimbs turned = w;
  turned.rl = fx_mad_hi(nd, w.ih, w.rl);
  turned.il = fx_mad_hi(d, w.rh, w.il);
  const int64_t n = -im;
  fx_product(fx_limbs(re, im), static_cast<int32_t>(n >> 30), static_cast<int32_t>(static_cast<uint32_t>(n) & (kFxLimb - 1)),
             turned, re, im);
}

// A component in [-1, 1] (to a scale) as (h + l 2^-32) 2^-28: h at most 2^28, l a signed 32-bit remainder.
struct FxPart {
  int32_t h, l;
};

// Of a 60-bit fixed-point number.
LEAP_HD FxPart fx_part(int64_t z) {
  const int32_t l = static_cast<int32_t>(static_cast<uint32_t>(z));
  return FxPart{static_cast<int32_t>((z + (int64_t(1) << 31)) >> 32), l};
}

// Of x, at most 2^28 in absolute value, to 2^-32.  (-l is one too.)
LEAP_HD FxPart fx_part(double x) {
  FxPart r;
#ifdef __CUDA_ARCH__
  r.h = __double2int_rn(x);
  r.l = __double2int_rn((x - r.h) * 4294967296.0);  // 2^31 saturates
#else
  r.h = static_cast<int32_t>(__builtin_nearbyint(x));
  const double l = __builtin_nearbyint((x - r.h) * 4294967296.0);
  r.l = l > 2147483647.0 ? 2147483647 : static_cast<int32_t>(l);
#endif
  if (r.l < -2147483647) r.l = -2147483647;
  return r;
}

// sum += a x + b y in units of 2^-56: the products of the high parts exactly, those of a high and a low part rounded
// together to the unit, those of the low parts (below half a unit) dropped.
LEAP_HD void fx_add_products(int64_t& sum, const FxPart& a, const FxPart& x, const FxPart& b, const FxPart& y) {
  int64_t mid = fx_mul(a.h, x.l);
  fx_mad(sum, a.h, x.h);
  fx_mad(mid, a.l, x.h);
  fx_mad(sum, b.h, y.h);
  fx_mad(mid, b.h, y.l);
  fx_mad(mid, b.l, y.h);
  sum += static_cast<int32_t>((mid + (int64_t(1) << 31)) >> 32);
}

}  // namespace leapgb
