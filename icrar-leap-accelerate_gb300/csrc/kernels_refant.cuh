// Reference-antenna baselines of the mixed form, complex<float> visibilities: pol 0 of the |I1| baselines through
// the reference antenna, averaged to about 1e-9 of the terms (kernels_rotate.cuh, refant_average_fp64, says why
// these rows need more than FP32).
//
// The sum over the channels c of v_c exp(2 pi i (A + c B)) (LA/algorithm/cpu/CpuLeapCalibrator.cc:181-217) is taken in
// blocks of 16 channels,
//   exp(2 pi i (A + c0 B)) sum_{i<16} v_{c0+i} w_i,   w_i = exp(2 pi i i B),
// where the w_i are the same for all blocks of a row, so that a lane (one row) keeps them in registers and a channel
// costs four integer multiply-adds per direction, without a phasor of its own:
//  * w_i in units of 1 / kRefUnit (31 bits);
//  * v in units of a power of two per row and block, at which sum |re| + |im| over the block is between 2^29 and 2^30, so
//    that no 64-bit sum of products overflows.  A component of 2^-6 of that sum or more is exact (24 bits); of a smaller
//    one the remainder, below a unit, is kept to 2^-8 and multiplied by the top 7 bits of w_i, four channels per
//    instruction (without, the error is 18 times as large);
//  * a block's sum, 45 bits of it as two floats, is multiplied by the block's phasor, held as (hi, lo) float pairs, and
//    added to a TwoSum pair: the product with the phasor's high part is exact (TwoProd), so the running sum carries no
//    FP32 rounding.
// Times and errors stand at the kernel.
#pragma once

#include "fixed_phase.h"
#include "leap_common.cuh"

namespace leapgb {

constexpr int kRefChannels = 16;     // channels per block
constexpr int kRefWarps = 8;         // warps per thread block, a direction each
constexpr int kRefRound = 64;        // channels staged at a time
constexpr int kRefStage = kRefRound / kRefWarps;  // of them by one warp
constexpr int32_t kRefUnit = 2147483520;  // 2^31 - 128 (a float): 1.0 as a fixed-point factor
static_assert(kRefStage == 8 && kRefChannels == 2 * kRefStage, "two warps stage a block of channels");

struct DfAcc {
  float s, c;  // value = s + c
};

// acc += (x + xl) * (yh + yl) (xl yl is dropped): x*yh = p + e exactly (TwoProd), TwoSum of acc.s and p, and
// err + (x*yl + xl*yh + e) into acc.c.
__device__ __forceinline__ void df_add_product(DfAcc& acc, float x, float xl, float yh, float yl) {
  const float p = __fmul_rn(x, yh);
  const float e = __fmaf_rn(x, yh, -p);
  float sum, err;
  two_sum(acc.s, p, sum, err);
  acc.s = sum;
  acc.c = __fadd_rn(acc.c, __fadd_rn(err, __fmaf_rn(x, yl, __fmaf_rn(xl, yh, e))));
}

// exp(2 pi i t / 2^64) as (hi, lo) pairs.  The nearest of 1024 table entries (cos_hi, cos_lo, sin_hi, sin_lo) is turned
// by the remaining angle d, at most pi / 1024, of which 25 bits are kept: cos d - 1 = -d^2/2 (d^4/24 < 4e-12) and
// sin d = d - d^3/6.
__device__ __forceinline__ void df_twiddle(uint64_t t, const float4* __restrict__ tab, float& zrh, float& zrl,
                                           float& zih, float& zil) {
  t += (uint64_t(1) << 53) + (uint64_t(1) << 28);
  const float4 a = tab[t >> 54];
  const float d = __int2float_rn(static_cast<int32_t>(static_cast<uint32_t>(t >> 29) & 0x1FFFFFFu) - (1 << 24)) *
                  1.8286475990841e-10f;  // 2 pi / 2^35
  const float d2 = d * d, c2 = -0.5f * d2, sd = d * fmaf(d2, -0.16666667f, 1.f);
  two_sum(a.x, fmaf(a.x, c2, fmaf(a.z, -sd, a.y)), zrh, zrl);
  two_sum(a.z, fmaf(a.z, c2, fmaf(a.x, sd, a.w)), zih, zil);
}

// hi + lo (|hi + lo| <= 1) in units of 1 / kRefUnit.
__device__ __forceinline__ int32_t refant_unit(float hi, float lo) {
  constexpr float k = static_cast<float>(kRefUnit);
  const float x = __fmul_rn(hi, k);
  const int32_t i = __float2int_rn(x);
  return i + __float2int_rn((x - __int2float_rn(i)) + fmaf(lo, k, fmaf(hi, k, -x)));
}

// Four small integers as the bytes of a word.
__device__ __forceinline__ int32_t refant_pack(int32_t a, int32_t b, int32_t c, int32_t d) {
  return static_cast<int32_t>(__byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410));
}

// x (below 2^30) to an integer, and 2^7 times the remainder, up to 64, as the low byte of the second.
__device__ __forceinline__ int32_t refant_round(float x, int32_t& rest) {
  // Above 2^23 x is an integer; below, adding and subtracting 2^23 rounds it as the conversion does.
  const float s = copysignf(8388608.f, x);
  const float r = fabsf(x) < 8388608.f ? __fsub_rn(x, __fsub_rn(__fadd_rn(x, s), s)) : 0.f;
  rest = __float_as_int(__fmaf_rn(r, 128.f, 12582912.f));
  return __float2int_rn(x);
}

// Fractional part of x (turns) as a 2^-64 fixed-point value.
__device__ __forceinline__ uint64_t frac_turns_u64(double x) {
  const double f = x - rint(x);  // in [-0.5, 0.5]
  return static_cast<uint64_t>(static_cast<long long>(rint(f * 9223372036854775808.0))) << 1;
}

// One work item of the pass (batched calls: one per integration chunk).  Blocks are numbered across items.
struct RefantItem {
  const float2* vis;       // [C][rows][pols]
  const double* uvw;       // [rows][3]
  const double* dd;        // the item's first direction matrix
  double2* out;            // [nslab][ndir][nI1]
  int64_t rows;
  int32_t T, C, pols, ndir;
  int32_t t_per_slab, c_per_slab, n_tslab, n_cslab;
  int32_t dgroups, block_begin, pad_[2];
};

struct RefantParams {
  const RefantItem* items;
  const int32_t* I1;
  double f0, df;
  int32_t nitems, nbl, nI1;
};

constexpr int kRefTabBytes = kTwiddleSize * 16;
constexpr int kRefRawBytes = kRefRound * 32 * 8;
constexpr int kRefRestBytes = kRefRound / 4 * 32 * 8;
constexpr int refant_smem_bytes() {
  return kRefTabBytes + 2 * kRefRawBytes + kRefRestBytes + kRefWarps * 32 * 4 + kRefRound / kRefChannels * 32 * 4;
}

__device__ __forceinline__ void refant_copy8(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid ? 8 : 0) : "memory");
}

// (A sum of products below 2^61 in absolute value) 2^-31 as two floats, without the low 18 of its bits.
__device__ __forceinline__ void refant_split(int64_t s, float& hi, float& lo) {
  const uint32_t h = static_cast<uint32_t>(static_cast<uint64_t>(s) >> 32), l = static_cast<uint32_t>(s);
  const float a = __int_as_float(0x4B400000 + (static_cast<int32_t>(h) >> 9));          // 1.5 2^23 + (s >> 41)
  const float b = __int_as_float(0x4B000000 | (__funnelshift_r(l, h, 18) & 0x7FFFFF));  // 2^23 + 23 bits
  hi = fmaf(a, 1024.f, -12582912.f * 1024.f);
  lo = fmaf(b, 0x1p-13f, -8388608.f * 0x1p-13f);
}

// A thread block takes 32 rows (reference baselines, one per lane), 8 directions (one per warp) and one (timestep,
// channel) slab.  Its warps stage 8 channels each, copied asynchronously a round ahead and converted once for all
// directions.
//
// Bound by the issue slots: 45 per row, channel and direction of a warp's 32, 16 of them for the four wide multiply-adds,
// which take 4 each (one direction per warp, 24 warps per SM; two directions in 12 warps: no faster, and spills).  128
// antennas, 14 timesteps, 384 channels, 64 directions: 134 -> 57 us, where a phasor per channel, its product and a TwoSum
// in FP32 pairs took 112 slots.  Error of the averages against 64 bits, relative to sqrt(sum |v|^2): 2.5e-10 rms, 8e-10 at
// most (before: 2.6e-10, 8e-10); with a bright source, 256 antennas over 40 km, 4.2e-10 and 2.9e-9 (5.0e-10, 4.9e-9).
static __global__ void __launch_bounds__(kRefWarps * 32, 3)
    refant_average_items(const RefantParams rp, const float4* __restrict__ df_tab) {
  extern __shared__ __align__(16) unsigned char refant_smem[];
  float4* tab = reinterpret_cast<float4*>(refant_smem);
  float2* raw = reinterpret_cast<float2*>(refant_smem + kRefTabBytes);               // [kRefRound][32]
  int2* fix = reinterpret_cast<int2*>(refant_smem + kRefTabBytes + kRefRawBytes);    // [kRefRound][32]
  int2* rest = fix + kRefRound * 32;                                                 // [kRefRound / 4][32]
  float* part = reinterpret_cast<float*>(rest + kRefRound / 4 * 32);                 // [kRefWarps][32]
  float* unit = part + kRefWarps * 32;                                               // [kRefRound / kRefChannels][32]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kTwiddleSize; i += blockDim.x) tab[i] = __ldg(df_tab + i);
  // The last item that begins at or before this block, 32 of them at a time.
  int ii = -1;
  for (int i = lane; i - lane < rp.nitems; i += 32)
    ii += __popc(__ballot_sync(0xffffffffu, i < rp.nitems && rp.items[i].block_begin <= static_cast<int>(blockIdx.x)));
  const RefantItem& it = rp.items[ii];
  const int nslab = it.n_tslab * it.n_cslab;
  const int local = static_cast<int>(blockIdx.x) - it.block_begin;
  const int ktile = local / (it.dgroups * nslab);
  const int j = (local / nslab) % it.dgroups * kRefWarps + warp;
  const int slab = local % nslab;
  const int k = ktile * 32 + lane;
  const int ts = slab / it.n_cslab, cs = slab % it.n_cslab;
  const int t_lo = ts * it.t_per_slab, t_hi = min(it.T, t_lo + it.t_per_slab);
  const int c_lo = cs * it.c_per_slab, c_hi = min(it.C, c_lo + it.c_per_slab);
  const bool valid = k < rp.nI1, active = j < it.ndir;  // active: the same in the whole warp
  int b = valid ? __ldg(rp.I1 + k) : 0;
  if (b < 0) b += rp.nbl;  // VectorRangeSelect wrap-around (LA/math/cpu/vector.h:97-104)
  const int64_t cstride = it.rows * it.pols;
  const float2* src = it.vis + static_cast<int64_t>(b) * it.pols;
  const int64_t tstride = static_cast<int64_t>(rp.nbl) * it.pols;
  float2* raw_col = raw + warp * kRefStage * 32 + lane;
  const uint32_t raw_dst = static_cast<uint32_t>(__cvta_generic_to_shared(raw_col));

  // This warp's channels of the round at (t, cb) on their way to raw; channels past the slab and lanes without a
  // baseline give zeros.
  auto fetch = [&](int t, int cb) {
    const int c0 = cb + warp * kRefStage;
    const float2* s = src + t * tstride + c0 * cstride;
#pragma unroll
    for (int i = 0; i < kRefStage; ++i) {
      const bool in = valid && c0 + i < c_hi;
      refant_copy8(raw_dst + i * 256, in ? s + i * cstride : it.vis, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  DfAcc re{0.f, 0.f}, im = re;
  fetch(t_lo, c_lo);
  __syncthreads();  // the table is written
  for (int t = t_lo; t < t_hi; ++t) {
    int32_t wr[kRefChannels], wi[kRefChannels];          // w_i
    int32_t tr[kRefChannels / 4], ti[kRefChannels / 4];  // their top 7 bits
    uint64_t pa = 0, pb = 0;                             // phase at the next block of channels, and its step
    if (active) {  // while the first round is on its way
      const int64_t r = static_cast<int64_t>(t) * rp.nbl + b;
      const double uu = __ldg(it.uvw + 3 * r), vv = __ldg(it.uvw + 3 * r + 1), ww = __ldg(it.uvw + 3 * r + 2);
      const double wrot =
          __ldg(it.dd + 9 * j + 6) * uu + __ldg(it.dd + 9 * j + 7) * vv + __ldg(it.dd + 9 * j + 8) * ww;
      const double dw = wrot - ww;
      pb = frac_turns_u64(-dw * (rp.df / kSpeedOfLight));
      pa = frac_turns_u64(-dw * (rp.f0 / kSpeedOfLight)) + static_cast<uint64_t>(c_lo) * pb;
      wr[0] = kRefUnit;
      wi[0] = 0;
#pragma unroll
      for (int i = 1; i < kRefChannels; ++i) {
        float zrh, zrl, zih, zil;
        df_twiddle(i * pb, tab, zrh, zrl, zih, zil);
        wr[i] = refant_unit(zrh, zrl);
        wi[i] = refant_unit(zih, zil);
      }
      auto top = [](int32_t w) { return (w >> 25) + ((w >> 24) & 1); };
#pragma unroll
      for (int g = 0; g < kRefChannels / 4; ++g) {
        tr[g] = refant_pack(top(wr[4 * g]), top(wr[4 * g + 1]), top(wr[4 * g + 2]), top(wr[4 * g + 3]));
        ti[g] = refant_pack(top(wi[4 * g]), top(wi[4 * g + 1]), top(wi[4 * g + 2]), top(wi[4 * g + 3]));
      }
      pb *= kRefChannels;
    }
    for (int cb = c_lo; cb < c_hi; cb += kRefRound) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      float2 v[kRefStage];
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < kRefStage; ++i) {
        v[i] = raw_col[i * 32];  // this lane's own copies
        sum += fabsf(v[i].x) * 0x1p-6f;  // (scaled: 32 of the largest floats do not overflow)
        sum += fabsf(v[i].y) * 0x1p-6f;
      }
      part[warp * 32 + lane] = sum;
      __syncthreads();  // the round before has been read
      {
        sum += part[(warp ^ 1) * 32 + lane];
        // sum |v| 2^ex < 2^30; 2^ex as two factors, since ex reaches 148
        const uint32_t be = __float_as_uint(sum) >> 23;
        const int ex = 23 - max(static_cast<int>(be) - 127, -125);
        const int k1 = ex >> 1, k2 = ex - k1;
        const float f1 = __int_as_float((k1 + 127) << 23), f2 = __int_as_float((k2 + 127) << 23);
        // An infinite or NaN sample makes the row's average NaN, as its products would.
        if (!(warp & 1))
          unit[(warp >> 1) * 32 + lane] =
              be == 255 ? __int_as_float(0x7FC00000)
                        : __int_as_float((127 - k1) << 23) * __int_as_float((127 - k2) << 23);
#pragma unroll
        for (int g = 0; g < kRefStage; g += 4) {
          int32_t rr[4], ri[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int32_t x = refant_round(v[g + i].x * f1 * f2, rr[i]);
            const int32_t y = refant_round(v[g + i].y * f1 * f2, ri[i]);
            fix[(warp * kRefStage + g + i) * 32 + lane] = make_int2(x, y);
          }
          rest[(warp * kRefStage + g) / 4 * 32 + lane] =
              make_int2(refant_pack(rr[0], rr[1], rr[2], rr[3]), refant_pack(ri[0], ri[1], ri[2], ri[3]));
        }
      }
      if (cb + kRefRound < c_hi)
        fetch(t, cb + kRefRound);
      else if (t + 1 < t_hi)
        fetch(t + 1, c_lo);
      __syncthreads();
      if (!active) continue;
      const int nq = min(kRefRound / kRefChannels, (c_hi - cb + kRefChannels - 1) / kRefChannels);
#pragma unroll 1
      for (int q = 0; q < nq; ++q) {
        const int2* vq = fix + q * kRefChannels * 32 + lane;
        const int2* rq = rest + q * (kRefChannels / 4) * 32 + lane;
        // Sums of v_re w_re, v_im w_im and of the imaginary part, and of the remainders with the top bits of w.
        const int2 v0 = vq[0];
        int64_t sr = fx_mul(v0.x, kRefUnit), si = 0, sx = fx_mul(v0.y, kRefUnit);
        int32_t er = 0, ex = 0;
#pragma unroll
        for (int i = 1; i < kRefChannels; ++i) {
          const int2 v = vq[i * 32];
          fx_mad(sr, v.x, wr[i]);
          fx_mad(si, v.y, wi[i]);
          fx_mad(sx, v.x, wi[i]);
          fx_mad(sx, v.y, wr[i]);
        }
        int32_t ei = 0;
#pragma unroll
        for (int g = 0; g < kRefChannels / 4; ++g) {
          const int2 r = rq[g * 32];
          er = __dp4a(r.x, tr[g], er);
          ei = __dp4a(r.y, ti[g], ei);
          ex = __dp4a(r.x, ti[g], ex);
          ex = __dp4a(r.y, tr[g], ex);
        }
        const float u = unit[q * 32 + lane];
        float xr, xrl, xi, xil;
        refant_split(sr - si + (static_cast<int64_t>(er - ei) << 18), xr, xrl);
        refant_split(sx + (static_cast<int64_t>(ex) << 18), xi, xil);
        xr *= u;
        xrl *= u;
        xi *= u;
        xil *= u;
        float zrh, zrl, zih, zil;
        df_twiddle(pa, tab, zrh, zrl, zih, zil);
        pa += pb;
        df_add_product(re, xr, xrl, zrh, zrl);  // re += x_re z_re - x_im z_im
        df_add_product(re, -xi, -xil, zih, zil);
        df_add_product(im, xr, xrl, zih, zil);  // im += x_re z_im + x_im z_re
        df_add_product(im, xi, xil, zrh, zrl);
      }
    }
  }
  if (!active || !valid) return;
  constexpr double scale = 2147483648.0 / kRefUnit;
  it.out[(static_cast<int64_t>(slab) * it.ndir + j) * rp.nI1 + k] =
      make_double2((static_cast<double>(re.s) + static_cast<double>(re.c)) * scale,
                   (static_cast<double>(im.s) + static_cast<double>(im.c)) * scale);
}

}  // namespace leapgb
