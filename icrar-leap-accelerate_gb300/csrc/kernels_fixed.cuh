// All-FP64 rotate + average in fixed point.
//
// Same sums as rotate_average_fp64 (kernels_rotate.cuh): avg[b, p] = sum over timesteps and channels of
// V[p, r, c] exp(i arg), arg = fl(sf / lambda_c) as the reference rounds it.  GB300 runs FP64 FMAs at 2
// lanes per clock and SM and 32-bit integer multiply-adds into 64-bit sums (IMAD.WIDE) at 32, so the phasors
// come from fixed_phase.h and the products are split into whole numbers:
//   * a row's visibilities of one pol are scaled by a power of two that puts the largest of its channels
//     just below 2^28 (complex<float>) or 2^26 (complex<double>) and split into a whole number h and a rest l,
//     |l| <= 1/2: exactly for complex<float>, to 27 bits (2^-54 of the largest) for complex<double>;
//   * phasors are split likewise, h with 28 or 29 bits and the rest;
//   * h h adds up exactly in 64-bit sums, and h l + l h in FP32 (complex<float>: at most 2^-29 of it) or in
//     64-bit sums (complex<double>); l l, below 2^-56 of the largest product, is dropped;
//   * every 64 or 128 channels the two go to an FP64 sum.
// So an average has fewer and smaller roundings than FP64 FMAs give it: one FP64 addition per 64 channels,
// and phasors good to 2^-53 where the direct form's recurrence is off by up to 2^-49 after 16 channels.
// Rows that do not fit (a visibility that is not finite or beyond the exponent range, an argument of 2^19 rad
// or more, a UVW that is not finite) are left out of the integer sums and added in FP64 by fx_plain_row.
//
// What bounds it: issue slots.  An IMAD.WIDE takes 4 of a scheduler's slots and nothing else issues beside it;
// per (row, channel, direction) there are 16 for h h of 4 pols, 12 for the phasor's recurrence and 4 for its
// argument, then 32 FP32 FMAs and about 60 other instructions.  128 antennas, 14 timesteps, 384 channels, 64
// directions: 222 -> 20.9 ms a call (the direct form has 27 FP64 FMAs there, 16 cycles of the SM each).
#pragma once

#include "fixed_phase.h"
#include "kernels_rotate.cuh"

namespace leapgb {

constexpr int kFxStage = 16;    // channels whose integer visibilities a block holds at a time
constexpr int kFxSeed = 32;     // channels from one seeded phasor to the next: a multiple of kFxStage
constexpr int kFxDirs = 2;      // directions per warp (1 at 16 warps per SM: 25.8 against 22.0 ms with plain negations)
constexpr int kFxWarps = 12;    // warps per SM (168 registers; 8 warps with 226: 22.2 against 21.0 ms)
constexpr int kFxPlain = 32767; // exponent of a row that fx_plain_row takes

static_assert(kFxSeed % kFxStage == 0, "seeds at stage starts");

struct FxArgs {
  RotateArgs r;
  FxSpectrum sp;
  const int4* tab;        // [2 * kFxTable] phasors (fx_tables)
  const int32_t* rho;     // [channels]
  const int16_t* vexp;    // [rows][pols]: the largest component of the row is below 2^vexp
};

// A component's magnitude by its bits (the high word of a double, whose lowest bit also tells a low word that is not 0 from
// an exact zero): ordered as the magnitudes are, NaN above all.
__device__ __forceinline__ uint32_t fx_magnitude(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }
__device__ __forceinline__ uint32_t fx_magnitude(double x) {
  return (static_cast<uint32_t>(__double2hiint(x)) & 0x7FFFFFFFu) | (__double2loint(x) != 0 ? 1u : 0u);
}

// Exponent of the largest magnitude m: it is below 2^e.  kFxPlain where the integer sums do not apply.  m == 0: a
// row of zeros, which adds nothing.
template <typename VisT>
__device__ __forceinline__ int16_t fx_exponent(uint32_t m) {
  int e;
  if (sizeof(VisT) == 8) {
    const int x = static_cast<int>(m >> 23);
    e = x == 255 || x < 37 ? kFxPlain : x - 126;  // 2^(28 - e) must be a float
  } else {
    const int x = static_cast<int>(m >> 20);
    e = x == 2047 || x - 1022 > 900 || x - 1022 < -850 ? kFxPlain : x - 1022;  // 2^(e - 56) and its multiples must be doubles
  }
  return static_cast<int16_t>(m == 0 ? 0 : e);
}

// Exponent of each (row, pol): block of 32 elements x 8 channel lanes, reading the cube once.
template <typename VisT>
__global__ void __launch_bounds__(256) fx_exponents(const VisT* __restrict__ vis, int64_t elems, int channels,
                                                    int16_t* __restrict__ out) {
  __shared__ uint32_t part[8][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int64_t i = blockIdx.x * 32ll + lane;
  uint32_t m = 0;
  if (i < elems)
#pragma unroll 8
    for (int c = g; c < channels; c += 8) {
      const VisT v = __ldg(vis + static_cast<int64_t>(c) * elems + i);
      m = max(m, max(fx_magnitude(v.x), fx_magnitude(v.y)));
    }
  part[g][lane] = m;
  __syncthreads();
  if (g == 0 && i < elems) {
#pragma unroll
    for (int k = 1; k < 8; ++k) m = max(m, part[k][lane]);
    out[i] = fx_exponent<VisT>(m);
  }
}

// A component with the row exponent e, as a whole number h and a remainder.  complex<float>: x 2^(28-e) = h + l
// exactly, |l| <= 1/2.
__device__ __forceinline__ void fx_split(float x, float scale, int& h, float& l) {
  const float y = x * scale;  // scale = 2^(28 - e): |y| < 2^28, exact
  h = __float2int_rn(y);
  l = y - static_cast<float>(h);
}

// complex<double>: rint(x 2^(53 - e)) = h 2^27 + l.
__device__ __forceinline__ void fx_split(double x, int e, int& h, int& l) {
  const uint64_t b = static_cast<uint64_t>(__double_as_longlong(x));
  const int ex = static_cast<int>((b >> 52) & 0x7FF);
  const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | (ex ? 0x10000000000000ull : 0);
  const int s = e + 1022 - max(ex, 1);  // x 2^(53 - e) = m 2^-s, s >= 0
  int64_t v = s > 54 ? 0 : static_cast<int64_t>(s > 0 ? (m + (uint64_t(1) << (s - 1))) >> s : m);
  if (static_cast<int64_t>(b) < 0) v = -v;
  h = static_cast<int>((v + (1 << 26)) >> 27);
  l = static_cast<int>(v - (static_cast<int64_t>(h) << 27));
}

// The sums of one row and direction over channels [c_lo, c_hi) in FP64, as rotate_average_fp64 forms them
// but with a sincos per channel: for the rare rows that the integer sums leave out.
template <typename VisT, int P>
__device__ __noinline__ void fx_plain_row(const RotateArgs& a, int64_t r, double sf, int c_lo, int c_hi, double2* out) {
  for (int p = 0; p < P; ++p) out[p] = make_double2(0.0, 0.0);
  for (int c = c_lo; c < c_hi; ++c) {
    const double lam = __ldg(a.lambda + c);
    double zi, zr;
    sincos(sf / lam, &zi, &zr);
    const VisT* src = static_cast<const VisT*>(a.vis) + (static_cast<int64_t>(c) * a.rows + r) * P;
    for (int p = 0; p < P; ++p) {
      double vr, vi;
      load_sample(src + p, vr, vi);
      out[p].x += vr * zr - vi * zi;
      out[p].y += vr * zi + vi * zr;
    }
  }
}

__device__ __forceinline__ void fx_copy_async(void* dst, const void* src, bool valid, int bytes) {
  const uint32_t n = valid ? static_cast<uint32_t>(bytes) : 0u;
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}

template <typename VisT, int P>
__host__ __device__ constexpr int fx_raw_bytes() { return kFxStage * 32 * P * static_cast<int>(sizeof(VisT)); }
// 16-byte rows per lane of a channel after the split.
template <typename VisT, int P>
__host__ __device__ constexpr int fx_rows() { return sizeof(VisT) == 8 ? P + (P + 1) / 2 : P; }
template <typename VisT, int P>
__host__ __device__ constexpr int fx_smem_bytes() {
  return fx_raw_bytes<VisT, P>() + kFxStage * 32 * 16 * fx_rows<VisT, P>();
}

// One channel's products for one direction.  Int: complex<double>, V = h 2^27 + l, |h| <= 2^26; Z likewise with
// |h| <= 2^29; h h and h l + l h in 64-bit sums over 128 channels: |mid| grows by at most 2 2^26 2^27 (h l) +
// 2^26 sqrt(2) 2^29 (l h; |z| <= 1) = 1.914 2^55 a channel.
template <int P>
struct FxSumInt {
  static constexpr int kFlush = 128;
  int64_t hh[P][2], mid[P][2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int p = 0; p < P; ++p) hh[p][0] = hh[p][1] = mid[p][0] = mid[p][1] = 0;
  }
  struct Phasor {
    int32_t rh, rl, ih, il, nih, nil;  // (nih, nil): the negated imaginary part
  };
  // 56 bits of a 60-bit phasor, rounded, in limbs of radix 2^27.
  static __device__ __forceinline__ void limbs(int64_t x, int32_t& h, int32_t& l) {
    h = static_cast<int32_t>(x >> 31);
    l = static_cast<int32_t>((static_cast<uint32_t>(x) >> 4) & 0x7FFFFFFu);
  }
  static __device__ __forceinline__ Phasor phasor(int64_t zr, int64_t zi) {
    Phasor z;
    limbs(zr + 8, z.rh, z.rl);
    limbs(zi + 8, z.ih, z.il);
    limbs(8 - zi, z.nih, z.nil);
    return z;
  }
  struct Vis {
    int4 v[P];  // (re h, re l, im h, im l)
  };
  static __device__ __forceinline__ void store(unsigned char* limb, int k, int lane, const double2 (&x)[P], const int (&e)[P],
                                              bool keep) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      int4 o = make_int4(0, 0, 0, 0);
      if (keep) {
        fx_split(x[p].x, e[p], o.x, o.y);
        fx_split(x[p].y, e[p], o.z, o.w);
      }
      reinterpret_cast<int4*>(limb)[(k * P + p) * 32 + lane] = o;
    }
  }
  static __device__ __forceinline__ Vis load(const unsigned char* limb, int k, int lane) {
    Vis r;
#pragma unroll
    for (int p = 0; p < P; ++p) r.v[p] = reinterpret_cast<const int4*>(limb)[(k * P + p) * 32 + lane];
    return r;
  }
  __device__ __forceinline__ void add(const Vis& x, const Phasor& z) {
    const int32_t nih = z.nih, nil = z.nil;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int4 v = x.v[p];
      fx_mad(hh[p][0], v.x, z.rh);
      fx_mad(hh[p][1], v.x, z.ih);
      fx_mad(mid[p][0], v.x, z.rl);
      fx_mad(mid[p][1], v.x, z.il);
      fx_mad(hh[p][0], v.z, nih);
      fx_mad(hh[p][1], v.z, z.rh);
      fx_mad(mid[p][0], v.z, nil);
      fx_mad(mid[p][1], v.z, z.rl);
      fx_mad(mid[p][0], v.y, z.rh);
      fx_mad(mid[p][1], v.y, z.ih);
      fx_mad(mid[p][0], v.w, nih);
      fx_mad(mid[p][1], v.w, z.rh);
    }
  }
  static constexpr int kUnitExp = -55;  // sums are in 2^(e - 55): (hh 2^54 + mid 2^27) 2^(e - 53) 2^-56
  __device__ __forceinline__ void flush(double (&sum)[P][2], const double (&scale)[P]) const {
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int c = 0; c < 2; ++c)
        sum[p][c] = fma(static_cast<double>(hh[p][c] + (mid[p][c] >> 27)), scale[p], sum[p][c]);
  }
};

// Float: complex<float>.  V = h + l exactly, |h| < 2^28; Z = h 2^32 + l, |h| <= 2^28; h h in a 64-bit sum, h l and
// l h, at most 2^-29 of the largest product, in FP32.  Both over 64 channels: |hh| grows by at most sqrt(2) 2^56
// a channel.  (With 26 and 29 bits the FP32 sums' roundings were 4 times larger, and an average's error 1.1 to
// 2.5 times that of FP64 FMAs.)
template <int P>
struct FxSumFloat {
  static constexpr int kFlush = 64;
  int64_t hh[P][2];
  float ra[P], im[P];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      hh[p][0] = hh[p][1] = 0;
      ra[p] = im[p] = 0.f;
    }
  }
  struct Phasor {
    int32_t rh, ih, nih;  // nih = -ih
    float rhf, rlf, ihf, ilf;
  };
  static __device__ __forceinline__ Phasor phasor(int64_t zr, int64_t zi) {
    Phasor z;
    z.rh = static_cast<int32_t>((zr + (int64_t(1) << 31)) >> 32);
    z.ih = static_cast<int32_t>((zi + (int64_t(1) << 31)) >> 32);
    z.nih = static_cast<int32_t>(((int64_t(1) << 31) - 1 - zi) >> 32);  // as such: see fx_product
    z.rlf = static_cast<float>(static_cast<int32_t>(zr));
    z.ilf = static_cast<float>(static_cast<int32_t>(zi));
    z.rhf = static_cast<float>(z.rh);
    z.ihf = static_cast<float>(z.ih);
    return z;
  }
  struct Vis {
    int h[P][2];
    float hf[P][2], l[P][2];  // h as floats times 2^-32, and l
  };
  // Rows of 16 bytes per lane: (h re, h im, l re, l im) per pol, then h as floats, two pols a row.
  static __device__ __forceinline__ void store(unsigned char* limb, int k, int lane, const float2 (&x)[P], const int (&e)[P],
                                              bool keep) {
    float4* o = reinterpret_cast<float4*>(limb) + k * kRows * 32 + lane;
    float hf[P + 1][2];
    hf[P][0] = hf[P][1] = 0.f;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      int h0 = 0, h1 = 0;
      float l0 = 0.f, l1 = 0.f;
      if (keep) {
        const float scale = __int_as_float((28 - e[p] + 127) << 23);
        fx_split(x[p].x, scale, h0, l0);
        fx_split(x[p].y, scale, h1, l1);
      }
      o[p * 32] = make_float4(__int_as_float(h0), __int_as_float(h1), l0, l1);
      hf[p][0] = h0 * kUnit;
      hf[p][1] = h1 * kUnit;
    }
#pragma unroll
    for (int p = 0; p < P; p += 2) o[(P + p / 2) * 32] = make_float4(hf[p][0], hf[p][1], hf[p + 1][0], hf[p + 1][1]);
  }
  static __device__ __forceinline__ Vis load(const unsigned char* limb, int k, int lane) {
    Vis r;
    const float4* o = reinterpret_cast<const float4*>(limb) + k * kRows * 32 + lane;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const float4 a = o[p * 32];
      r.h[p][0] = __float_as_int(a.x);
      r.h[p][1] = __float_as_int(a.y);
      r.l[p][0] = a.z;
      r.l[p][1] = a.w;
    }
#pragma unroll
    for (int p = 0; p < P; p += 2) {
      const float4 a = o[(P + p / 2) * 32];
      r.hf[p][0] = a.x;
      r.hf[p][1] = a.y;
      if (p + 1 < P) {
        r.hf[p + 1][0] = a.z;
        r.hf[p + 1][1] = a.w;
      }
    }
    return r;
  }
  __device__ __forceinline__ void add(const Vis& x, const Phasor& z) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      fx_mad(hh[p][0], x.h[p][0], z.rh);
      fx_mad(hh[p][1], x.h[p][0], z.ih);
      fx_mad(hh[p][0], x.h[p][1], z.nih);
      fx_mad(hh[p][1], x.h[p][1], z.rh);
      ra[p] = fmaf(x.l[p][0], z.rhf, fmaf(x.hf[p][0], z.rlf, ra[p]));
      ra[p] = fmaf(x.l[p][1], -z.ihf, fmaf(x.hf[p][1], -z.ilf, ra[p]));
      im[p] = fmaf(x.l[p][0], z.ihf, fmaf(x.hf[p][0], z.ilf, im[p]));
      im[p] = fmaf(x.l[p][1], z.rhf, fmaf(x.hf[p][1], z.rlf, im[p]));
    }
  }
  static constexpr int kUnitExp = -56;  // sums are in 2^(e - 56): V's h in 2^(e - 28), Z's h in 2^-28
  __device__ __forceinline__ void flush(double (&sum)[P][2], const double (&scale)[P]) const {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      sum[p][0] = fma(static_cast<double>(hh[p][0]) + static_cast<double>(ra[p]), scale[p], sum[p][0]);
      sum[p][1] = fma(static_cast<double>(hh[p][1]) + static_cast<double>(im[p]), scale[p], sum[p][1]);
    }
  }
  static constexpr int kRows = P + (P + 1) / 2;
  static constexpr float kUnit = 2.3283064365386963e-10f;  // 2^-32
};

template <typename VisT, int P> struct FxSumOf;
template <int P> struct FxSumOf<float2, P> { using type = FxSumFloat<P>; };
template <int P> struct FxSumOf<double2, P> { using type = FxSumInt<P>; };

__device__ __forceinline__ FxLimbs fx_lookup(const int4* tab, uint64_t t) {
  const int4 a = __ldg(tab + (t >> 54)), b = __ldg(tab + kFxTable + ((t >> 44) & (kFxTable - 1)));
  return fx_turn(t, FxLimbs{a.x, a.y, a.z, a.w}, FxLimbs{b.x, b.y, b.z, b.w});
}

// The phasor of one (row, direction), channel by channel.
struct FxRay {
  FxPhase ph;
  FxLimbs w;        // channel step; 0 for a row that does not fit
  int64_t zr, zi;   // 60-bit phasor

  // At channel c0 of a row.  Returns whether sf fits; if not, the phasor is 0.
  __device__ __forceinline__ bool begin(double sf, const FxSpectrum& sp, int c0, const int4* tab) {
    const bool fits = fx_in_range(sf, sp);
    uint64_t step;
    fx_setup(ph, fits ? sf : 0.0, sp, c0, step);
    w = fx_lookup(tab, step);
    if (!fits) w = FxLimbs{0, 0, 0, 0};
    return fits;
  }
  __device__ __forceinline__ void seed(int32_t rho, const int4* tab) {
    ph.e = fx_residual(ph, rho);
    const FxLimbs z = fx_lookup(tab, fx_turns(ph));
    const bool fits = w.rh != 0 || w.ih != 0;  // a phasor's high limbs are not both 0
    zr = fits ? (static_cast<int64_t>(z.rh) << 30) + z.rl : 0;
    zi = fits ? (static_cast<int64_t>(z.ih) << 30) + z.il : 0;
  }
  __device__ __forceinline__ void next(int32_t rho) {
    int32_t d, nd;
    fx_advance(ph, rho, d, nd);
    fx_step(zr, zi, w, d, nd);
  }
};

// sf = -2 pi (w_rot - w) of a row, without fused operations, as the reference forms it.
__device__ __forceinline__ double fx_shift_factor(const double* dd2, double u, double v, double w) {
  const double wrot = __dadd_rn(__dadd_rn(__dmul_rn(__ldg(dd2), u), __dmul_rn(__ldg(dd2 + 1), v)), __dmul_rn(__ldg(dd2 + 2), w));
  return __dmul_rn(-kTwoPi, __dadd_rn(wrot, -w));
}

// Fetch of channels [c0, c0 + n) of the 32 rows from r0 (rows >= nrows of them are zero) to raw, by all threads of
// the block: pieces of 16 bytes (8 for a single complex<float>), lanes along a channel's rows.
template <typename VisT, int P>
__device__ __forceinline__ void fx_fetch(unsigned char* raw, const void* vis, int64_t rows, int64_t r0, int nrows, int c0, int n) {
  constexpr int kGroup = P * static_cast<int>(sizeof(VisT));
  constexpr int kPiece = kGroup >= 16 ? 16 : 8;
  constexpr int kPieces = kGroup * 32 / kPiece;  // per channel
  const char* base = static_cast<const char*>(vis);
  for (int i = threadIdx.x; i < n * kPieces; i += blockDim.x) {
    const int k = i / kPieces, q = i % kPieces;
    const bool ok = q * kPiece / kGroup < nrows;
    const int64_t off = (static_cast<int64_t>(c0 + k) * rows + r0) * kGroup + q * kPiece;
    fx_copy_async(raw + (k * kPieces + q) * kPiece, base + (ok ? off : 0), ok, kPiece);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// A block is NW warps of kFxDirs directions each, over 32 baselines (one per lane) and a slab of timesteps
// and channels.  The raw visibilities of a stage (kFxStage channels) arrive by cp.async while the previous
// stage computes; all warps split them into limbs once, and every warp reads the limbs.
template <typename VisT, int P, int NW>
__global__ void __launch_bounds__(NW * 32, kFxWarps / NW) rotate_average_fixed(const FxArgs a) {
  extern __shared__ __align__(128) unsigned char fx_smem[];
  VisT* raw = reinterpret_cast<VisT*>(fx_smem);
  unsigned char* limb = fx_smem + fx_raw_bytes<VisT, P>();  // the split stage, laid out by Sum::store
  using Sum = typename FxSumOf<VisT, P>::type;
  const RotateArgs& ra = a.r;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dgroups = (ra.ndir + NW * kFxDirs - 1) / (NW * kFxDirs);
  const int tile = blockIdx.x / dgroups, dg = blockIdx.x % dgroups;  // direction groups of a tile side by side: one read
  const int slab = blockIdx.y;
  const int ts = slab / ra.n_cslab, cs = slab % ra.n_cslab;
  const int t_lo = ts * ra.t_per_slab, t_hi = min(ra.timesteps, t_lo + ra.t_per_slab);
  const int c_lo = cs * ra.c_per_slab, c_hi = min(ra.channels, c_lo + ra.c_per_slab);
  const int b0 = tile * 32, b = b0 + lane;
  const bool valid = b < ra.nbl;
  const int d0 = (dg * NW + warp) * kFxDirs;
  const bool active = d0 < ra.ndir;
  const int nst = (c_hi - c_lo + kFxStage - 1) / kFxStage;  // stages per timestep
  const int total = (t_hi - t_lo) * nst;

  auto fetch = [&](int s) {
    const int t = t_lo + s / nst, c0 = c_lo + (s % nst) * kFxStage;
    fx_fetch<VisT, P>(fx_smem, ra.vis, ra.rows, static_cast<int64_t>(t) * ra.nbl + b0, ra.nbl - b0, c0, min(kFxStage, c_hi - c0));
  };

  double sum[kFxDirs][P][2];
  Sum acc[kFxDirs];
  FxRay ray[kFxDirs];
  int ve[P];
#pragma unroll
  for (int j = 0; j < kFxDirs; ++j)
#pragma unroll
    for (int p = 0; p < P; ++p) sum[j][p][0] = sum[j][p][1] = 0.0;

  if (total > 0) fetch(0);
  for (int s = 0; s < total; ++s) {
    const int t = t_lo + s / nst, cb = c_lo + (s % nst) * kFxStage, cf = cb - c_lo;
    const int n = min(kFxStage, c_hi - cb);
    const int64_t r = static_cast<int64_t>(t) * ra.nbl + (valid ? b : 0);
    bool plain_row = false;
    if (cf == 0) {
#pragma unroll
      for (int p = 0; p < P; ++p) ve[p] = __ldg(a.vexp + r * P + p);
    }
#pragma unroll
    for (int p = 0; p < P; ++p) plain_row |= ve[p] == kFxPlain;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the raw stage has landed, and the limbs of the previous one are no longer read
    for (int k = warp; k < n; k += NW) {
      VisT x[P];
#pragma unroll
      for (int p = 0; p < P; ++p) x[p] = raw[(k * 32 + lane) * P + p];
      Sum::store(limb, k, lane, x, ve, valid && !plain_row);
    }
    __syncthreads();
    if (s + 1 < total) fetch(s + 1);
    if (!active) continue;

    if (cf == 0) {
      const double u = __ldg(ra.uvw + 3 * r), v = __ldg(ra.uvw + 3 * r + 1), x = __ldg(ra.uvw + 3 * r + 2);
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) {
        const double sf = fx_shift_factor(ra.dd + 9 * min(d0 + j, ra.ndir - 1) + 6, u, v, x);
        const bool fits = ray[j].begin(sf, a.sp, c_lo, a.tab);
        if (valid && (plain_row || !fits)) {
          double2 add[P];
          fx_plain_row<VisT, P>(ra, r, sf, c_lo, c_hi, add);
#pragma unroll
          for (int p = 0; p < P; ++p) {
            sum[j][p][0] += add[p].x;
            sum[j][p][1] += add[p].y;
          }
        }
      }
    }
    if (cf % kFxSeed == 0) {
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) ray[j].seed(__ldg(a.rho + cb), a.tab);
    }
    if (cf % Sum::kFlush == 0) {
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) acc[j].clear();
    }
#pragma unroll 2
    for (int k = 0; k < n; ++k) {
      const int32_t rho = __ldg(a.rho + min(cb + k + 1, ra.channels - 1));
      const typename Sum::Vis v = Sum::load(limb, k, lane);
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) {
        acc[j].add(v, Sum::phasor(ray[j].zr, ray[j].zi));
        ray[j].next(rho);
      }
    }
    if ((cf + kFxStage) % Sum::kFlush == 0 || cb + kFxStage >= c_hi) {
      double scale[P];
#pragma unroll
      for (int p = 0; p < P; ++p) scale[p] = __hiloint2double((plain_row ? 0 : ve[p] + Sum::kUnitExp + 1023) << 20, 0);
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) acc[j].flush(sum[j], scale);
    }
  }
  if (!active || !valid) return;
  const int64_t off = static_cast<int64_t>(slab) * ra.ndir * P * ra.nbl;
#pragma unroll
  for (int j = 0; j < kFxDirs; ++j)
    if (d0 + j < ra.ndir) {
#pragma unroll
      for (int p = 0; p < P; ++p)
        ra.out[off + (static_cast<int64_t>(d0 + j) * P + p) * ra.nbl + b] = make_double2(sum[j][p][0], sum[j][p][1]);
    }
}

}  // namespace leapgb
