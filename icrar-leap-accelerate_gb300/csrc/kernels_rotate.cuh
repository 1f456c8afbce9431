// Rotate + average kernels (the hot path).
//
// Reference semantics (CpuLeapCalibrator::RotateVisibilities,
// LA/algorithm/cpu/CpuLeapCalibrator.cc:181-217; g_RotateVisibilities,
// LA/algorithm/cuda/CudaLeapCalibrator.cu:305-400): for every row r of the
// integration and channel c
//     shift  = -2*pi*(w_rot[r] - w[r]) / lambda_c,   w_rot = (dd * uvw[r]).z
//     avg[r % nbl, p] += V[p, r, c] * exp(i*shift)   for every pol p
// where samples with a NaN in any pol are skipped.  Here NaN groups were
// zeroed when the integration was ingested, so they add exactly nothing.
//
// Differences in structure from the reference (same sums, new schedule):
//  * the visibilities are read-only and resident; nothing is written back;
//  * one launch handles many directions, so every visibility load is reused
//    by all the directions of a warp;
//  * lanes own baselines, loops run over (timestep, channel) in the
//    reference's order, and partial sums over (timestep, channel) slabs are
//    combined in a fixed order, so results are deterministic (no atomics).
#pragma once

#include "leap_common.cuh"
#include "narrow.h"
#include "kernels_pipe.cuh"

namespace leapgb {

struct RotateArgs {
  const void* vis;          // [channels][rows][pols] complex (float2 or double2)
  const double* uvw;        // [rows][3]
  const double* dd;         // [ndir][9] row-major direction matrices
  const double* lambda;     // [channels] c / (f0 + ch*df), as the reference computes it
  const double* inv_lambda; // [channels] 1 / lambda, rounded (all-FP64 form)
  const float2* twiddle;    // [kTwiddleSize] (cos, sin) table for the mixed form
  const float* uvw_f;       // [rows][6] (u, v, w) as (hi, lo) float pairs
  const float* dirk;        // [ndir][12] phase constants as (hi, lo) pairs: -(l, m, n-1)*f0/c, -(l, m, n-1)*df/c
  int64_t rows;
  int32_t channels, pols, nbl, timesteps, ndir;
  double f0, df;
  int32_t t_per_slab, c_per_slab, n_tslab, n_cslab;
  double2* out;             // nslab == 1: avg [ndir][pols][nbl]; else partial [nslab][ndir][pols][nbl]
  int* err;
};

template <typename T> struct VisScalar;
template <> struct VisScalar<float2> { using type = float; };
template <> struct VisScalar<double2> { using type = double; };

template <typename VisT>
__device__ __forceinline__ void load_sample(const VisT* __restrict__ p, double& re, double& im) {
  const VisT v = __ldg(p);
  re = static_cast<double>(v.x);
  im = static_cast<double>(v.y);
}

// ---------------------------------------------------------------------------
// All-FP64 form.  Lanes own baselines, a warp owns DPW directions, a block's
// warps share one baseline tile (so the visibility loads of one warp hit L1
// for the others).  The reference phase is shiftRad(c) = fl(shiftFactor /
// lambda_c) (CpuLeapCalibrator.cc:190-198), nearly linear in the channel index,
// so exp(i*shiftRad) is advanced channel to channel by one complex multiply with
// exp(i*shiftFactor*df/c_light) and re-seeded with an FP64 sincos every kSeed
// channels.  FP64 sincos runs at about 1/25 of the DFMA rate on GB300, so this
// removes it from the inner loop.
//
// The reference's own rounding matters here.  Its argument reaches thousands of
// radians for directions ~1 rad from the phase centre, where one unit in the last
// place is ~1e-12 rad, and lambda_c's rounding is the same for every row; the
// solve then moves the cal phases by ~5e-11 rad between two equally valid FP64
// roundings of the argument (shiftFactor * (1 / lambda_c) against shiftFactor /
// lambda_c).  So each channel's twiddle is corrected to the reference's own
// argument: fl(shiftFactor / lambda_c) from the rounded reciprocal and one
// FMA-exact remainder step (the correctly rounded quotient), minus the
// recurrence's phase seed + k * step, applied to first order (the difference is
// below 1e-11 rad, so its square is far below rounding).  shiftFactor itself is
// formed without fused operations, as the reference's expression is.
// ---------------------------------------------------------------------------
// kCheckNan: skip (row, channel) groups with a NaN in any pol inside the kernel
// (for callers whose visibilities did not go through the ingestion sanitiser).
template <typename VisT, int P, int DPW, bool kCheckNan = false>
__global__ void __launch_bounds__(128) rotate_average_fp64(RotateArgs a) {
  constexpr int NW = 4;
  constexpr int kSeed = 16;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int b = blockIdx.x * 32 + lane;
  const int d0 = (blockIdx.y * NW + warp) * DPW;
  const int slab = blockIdx.z;
  const int ts = slab / a.n_cslab, cs = slab % a.n_cslab;
  const int t_lo = ts * a.t_per_slab, t_hi = min(a.timesteps, t_lo + a.t_per_slab);
  const int c_lo = cs * a.c_per_slab, c_hi = min(a.channels, c_lo + a.c_per_slab);
  if (d0 >= a.ndir) return;
  const bool valid = b < a.nbl;

  double dd2[DPW][3];
#pragma unroll
  for (int j = 0; j < DPW; ++j) {
    const int d = min(d0 + j, a.ndir - 1);
    dd2[j][0] = __ldg(a.dd + 9 * d + 6);
    dd2[j][1] = __ldg(a.dd + 9 * d + 7);
    dd2[j][2] = __ldg(a.dd + 9 * d + 8);
  }
  double accr[DPW][P], acci[DPW][P];
#pragma unroll
  for (int j = 0; j < DPW; ++j)
#pragma unroll
    for (int p = 0; p < P; ++p) accr[j][p] = acci[j][p] = 0.0;

  const double inv_c = 1.0 / kSpeedOfLight;
  const VisT* vis = static_cast<const VisT*>(a.vis);
  if (valid) {
    for (int t = t_lo; t < t_hi; ++t) {
      const int64_t r = static_cast<int64_t>(t) * a.nbl + b;
      const double u = __ldg(a.uvw + 3 * r), v = __ldg(a.uvw + 3 * r + 1), w = __ldg(a.uvw + 3 * r + 2);
      double sf[DPW], st[DPW], wr[DPW], wi[DPW];
#pragma unroll
      for (int j = 0; j < DPW; ++j) {
        const double wrot =
            __dadd_rn(__dadd_rn(__dmul_rn(dd2[j][0], u), __dmul_rn(dd2[j][1], v)), __dmul_rn(dd2[j][2], w));
        sf[j] = __dmul_rn(-kTwoPi, __dadd_rn(wrot, -w));
        st[j] = sf[j] * (a.df * inv_c);
        sincos(st[j], &wi[j], &wr[j]);
      }
      for (int cb = c_lo; cb < c_hi; cb += kSeed) {
        const int ce = min(c_hi, cb + kSeed);
        double zr[DPW], zi[DPW], seed[DPW];
#pragma unroll
        for (int j = 0; j < DPW; ++j) {
          seed[j] = sf[j] / __ldg(a.lambda + cb);
          sincos(seed[j], &zi[j], &zr[j]);
        }
        for (int c = cb; c < ce; ++c) {
          const double lam = __ldg(a.lambda + c), rlam = __ldg(a.inv_lambda + c);
          const double k = static_cast<double>(c - cb);
          const VisT* src = vis + (static_cast<int64_t>(c) * a.rows + r) * P;
          double vr[P], vi[P];
#pragma unroll
          for (int p = 0; p < P; ++p) load_sample(src + p, vr[p], vi[p]);
          if (kCheckNan) {
            bool nan = false;
#pragma unroll
            for (int p = 0; p < P; ++p) nan |= isnan(vr[p]) || isnan(vi[p]);
            if (nan) {
#pragma unroll
              for (int p = 0; p < P; ++p) vr[p] = vi[p] = 0.0;
            }
          }
#pragma unroll
          for (int j = 0; j < DPW; ++j) {
            // The reference's argument fl(sf / lambda_c), and its difference from seed + k * step.
            const double q = sf[j] * rlam;
            const double arg = fma(fma(-q, lam, sf[j]), rlam, q);
            const double dlt = fma(-k, st[j], arg - seed[j]);
            const double tr = fma(-dlt, zi[j], zr[j]), ti = fma(dlt, zr[j], zi[j]);
#pragma unroll
            for (int p = 0; p < P; ++p) {
              accr[j][p] += vr[p] * tr - vi[p] * ti;
              acci[j][p] += vr[p] * ti + vi[p] * tr;
            }
            const double nr = zr[j] * wr[j] - zi[j] * wi[j];
            zi[j] = zr[j] * wi[j] + zi[j] * wr[j];
            zr[j] = nr;
          }
        }
      }
    }
  }
  if (!valid) return;
  const int64_t slab_off = static_cast<int64_t>(slab) * a.ndir * P * a.nbl;
#pragma unroll
  for (int j = 0; j < DPW; ++j) {
    const int d = d0 + j;
    if (d < a.ndir) {
#pragma unroll
      for (int p = 0; p < P; ++p)
        a.out[slab_off + (static_cast<int64_t>(d) * P + p) * a.nbl + b] = make_double2(accr[j][p], acci[j][p]);
    }
  }
}

// ---------------------------------------------------------------------------
// Mixed-precision form (direct loads).  Per (row, direction) the phase
//     turns(c) = -(w_rot - w) * (f0 + c*df) / c_light = A + c*B
// is formed in FP64 once per timestep and reduced to 32-bit fixed-point
// fractions of a turn; each channel then costs one integer multiply-add, the
// table twiddle of twiddle_turns (about 1e-7 absolute; the hardware sin/cos
// approximations, about 5e-7, are not accurate enough for nearly cancelling
// sums) and FP32 complex MACs.
// Sums run in FP32 over blocks of KB channels and are folded into Kahan
// (sum, compensation) pairs, written out as sum - compensation in FP64.
//
// Bound by latency (the loads' and the table's) and by the issue slots: 7 blocks per SM (72 registers) and the loads of
// one or two groups of samples ahead do better than more of either; complex<double> samples are converted on the
// integer pipe (narrow.h).  128 antennas, 4 timesteps, 96 channels, 16 directions, two complex<double> pols: a call
// 365 -> 231 us with the FP64 pass over the reference baselines above (4 or 8 samples ahead: 282 and 333; 8 or 10
// blocks: 231 and 245; converted by the conversion instruction: 269).
// ---------------------------------------------------------------------------
template <typename VisT, int P, int DPW>
__global__ void __launch_bounds__(128, P == 4 ? 4 : 7) rotate_average_mixed(RotateArgs a) {
  constexpr int NW = 4;
  constexpr int KB = 16;
  constexpr int KU = 4 / P;  // channels whose loads are on their way together
  __shared__ float2 tab[kTwiddleSize];
  for (int i = threadIdx.x; i < kTwiddleSize; i += blockDim.x) tab[i] = __ldg(a.twiddle + i);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int b = blockIdx.x * 32 + lane;
  const int d0 = (blockIdx.y * NW + warp) * DPW;
  const int slab = blockIdx.z;
  const int ts = slab / a.n_cslab, cs = slab % a.n_cslab;
  const int t_lo = ts * a.t_per_slab, t_hi = min(a.timesteps, t_lo + a.t_per_slab);
  const int c_lo = cs * a.c_per_slab, c_hi = min(a.channels, c_lo + a.c_per_slab);
  if (d0 >= a.ndir) return;
  const bool valid = b < a.nbl;

  const double kA = a.f0 / kSpeedOfLight, kB = a.df / kSpeedOfLight;
  float sr[DPW][P], si[DPW][P], cr[DPW][P], ci[DPW][P];
#pragma unroll
  for (int j = 0; j < DPW; ++j)
#pragma unroll
    for (int p = 0; p < P; ++p) sr[j][p] = si[j][p] = cr[j][p] = ci[j][p] = 0.f;

  const VisT* vis = static_cast<const VisT*>(a.vis);
  if (valid) {
    for (int t = t_lo; t < t_hi; ++t) {
      const int64_t r = static_cast<int64_t>(t) * a.nbl + b;
      const double u = __ldg(a.uvw + 3 * r), v = __ldg(a.uvw + 3 * r + 1), w = __ldg(a.uvw + 3 * r + 2);
      uint32_t pa[DPW], pb[DPW];
#pragma unroll
      for (int j = 0; j < DPW; ++j) {
        const int d = min(d0 + j, a.ndir - 1);
        const double wrot = __ldg(a.dd + 9 * d + 6) * u + __ldg(a.dd + 9 * d + 7) * v + __ldg(a.dd + 9 * d + 8) * w;
        const double dw = wrot - w;
        pa[j] = frac_turns_u32(-dw * kA);
        pb[j] = frac_turns_u32(-dw * kB);
      }
      for (int cb = c_lo; cb < c_hi; cb += KB) {
        const int ce = min(c_hi, cb + KB);
        float pr[DPW][P], pi[DPW][P];
#pragma unroll
        for (int j = 0; j < DPW; ++j)
#pragma unroll
          for (int p = 0; p < P; ++p) pr[j][p] = pi[j][p] = 0.f;
        for (int c0 = cb; c0 < ce; c0 += KU) {
          VisT raw[KU][P];
#pragma unroll
          for (int k = 0; k < KU; ++k)
#pragma unroll
            for (int p = 0; p < P; ++p)
              raw[k][p] = __ldg(vis + (static_cast<int64_t>(min(c0 + k, ce - 1)) * a.rows + r) * P + p);
#pragma unroll
          for (int k = 0; k < KU; ++k) {
            const int c = c0 + k;
            if (c >= ce) break;
            float vr[P], vi[P];
#pragma unroll
            for (int p = 0; p < P; ++p) {
              vr[p] = narrow(raw[k][p].x);
              vi[p] = narrow(raw[k][p].y);
            }
#pragma unroll
            for (int j = 0; j < DPW; ++j) {
              float s, co;
              twiddle_turns(pa[j] + static_cast<uint32_t>(c) * pb[j], tab, co, s);
#pragma unroll
              for (int p = 0; p < P; ++p) {
                pr[j][p] = fmaf(vr[p], co, fmaf(-vi[p], s, pr[j][p]));
                pi[j][p] = fmaf(vr[p], s, fmaf(vi[p], co, pi[j][p]));
              }
            }
          }
        }
#pragma unroll
        for (int j = 0; j < DPW; ++j)
#pragma unroll
          for (int p = 0; p < P; ++p) {
            float y = pr[j][p] - cr[j][p];
            float tt = sr[j][p] + y;
            cr[j][p] = (tt - sr[j][p]) - y;
            sr[j][p] = tt;
            y = pi[j][p] - ci[j][p];
            tt = si[j][p] + y;
            ci[j][p] = (tt - si[j][p]) - y;
            si[j][p] = tt;
          }
      }
    }
  }
  if (!valid) return;
  const int64_t slab_off = static_cast<int64_t>(slab) * a.ndir * P * a.nbl;
#pragma unroll
  for (int j = 0; j < DPW; ++j) {
    const int d = d0 + j;
    if (d < a.ndir) {
#pragma unroll
      for (int p = 0; p < P; ++p)
        a.out[slab_off + (static_cast<int64_t>(d) * P + p) * a.nbl + b] =
            make_double2(static_cast<double>(sr[j][p]) - static_cast<double>(cr[j][p]),
                         static_cast<double>(si[j][p]) - static_cast<double>(ci[j][p]));
    }
  }
}

// ---------------------------------------------------------------------------
// Reference-antenna baselines in FP64 (mixed form).  The solve reads pol 0 of
// the |I1| baselines through the reference antenna with weight one (cal1 =
// Ad1 * arg(avg[I1, 0])) and then multiplies cal1 by 2*pi, so an FP32 phase
// error on one of them reaches every antenna's cal phase ~7x amplified; on
// nearly cancelling sums FP32 products leave errors of 1e-6..1e-5 rad there.
// These rows are therefore accumulated in FP64 (the all-FP64 recurrence of
// rotate_average_fp64, pol 0 only), gathered by I1.  They are 1-2% of the rows
// and use the FP64 pipe, which the FP32 bulk kernel leaves idle, so the call
// launches this kernel on a second stream to overlap the two.
// (128 antennas, 4 timesteps, 96 channels, 16 directions, alone: 70 -> 35 us with Horner's rule, and slabs of 16 channels
// where longer ones leave SMs without a block.)
// Output: [nslab][ndir][nI1] double2 (nslab == 1: final).
// ---------------------------------------------------------------------------
template <typename VisT, int DPW>
__global__ void __launch_bounds__(128) refant_average_fp64(RotateArgs a, const int32_t* __restrict__ I1, int nI1,
                                                          double2* __restrict__ out) {
  constexpr int NW = 4;
  constexpr int kSeed = 16;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  const int d0 = (blockIdx.y * NW + warp) * DPW;
  const int slab = blockIdx.z;
  const int ts = slab / a.n_cslab, cs = slab % a.n_cslab;
  const int t_lo = ts * a.t_per_slab, t_hi = min(a.timesteps, t_lo + a.t_per_slab);
  const int c_lo = cs * a.c_per_slab, c_hi = min(a.channels, c_lo + a.c_per_slab);
  if (d0 >= a.ndir || k >= nI1) return;
  int b = __ldg(I1 + k);
  if (b < 0) b += a.nbl;  // VectorRangeSelect wrap-around (LA/math/cpu/vector.h:97-104)

  double dd2[DPW][3];
#pragma unroll
  for (int j = 0; j < DPW; ++j) {
    const int d = min(d0 + j, a.ndir - 1);
    dd2[j][0] = __ldg(a.dd + 9 * d + 6);
    dd2[j][1] = __ldg(a.dd + 9 * d + 7);
    dd2[j][2] = __ldg(a.dd + 9 * d + 8);
  }
  double accr[DPW], acci[DPW];
#pragma unroll
  for (int j = 0; j < DPW; ++j) accr[j] = acci[j] = 0.0;
  const double inv_c = 1.0 / kSpeedOfLight;
  const VisT* vis = static_cast<const VisT*>(a.vis);
  for (int t = t_lo; t < t_hi; ++t) {
    const int64_t r = static_cast<int64_t>(t) * a.nbl + b;
    const double u = __ldg(a.uvw + 3 * r), v = __ldg(a.uvw + 3 * r + 1), w = __ldg(a.uvw + 3 * r + 2);
    double sf[DPW], wr[DPW], wi[DPW];
#pragma unroll
    for (int j = 0; j < DPW; ++j) {
      const double wrot = dd2[j][0] * u + dd2[j][1] * v + dd2[j][2] * w;
      sf[j] = -kTwoPi * (wrot - w);
      sincos(sf[j] * (a.df * inv_c), &wi[j], &wr[j]);
    }
    for (int cb = c_lo; cb < c_hi; cb += kSeed) {
      const int ce = min(c_hi, cb + kSeed);
      // Horner's rule in the step's phasor from the block's last channel on, then the first channel's phasor: four FMAs
      // per channel and direction instead of the eight that advance a phasor and add its product.
      double hr[DPW], hi[DPW];
#pragma unroll
      for (int j = 0; j < DPW; ++j) hr[j] = hi[j] = 0.0;
      const VisT* src = vis + (static_cast<int64_t>(cb) * a.rows + r) * a.pols;
#pragma unroll 8
      for (int c = ce - cb - 1; c >= 0; --c) {
        double vr, vi;
        load_sample(src + c * a.rows * a.pols, vr, vi);
#pragma unroll
        for (int j = 0; j < DPW; ++j) {
          const double nr = fma(-hi[j], wi[j], fma(hr[j], wr[j], vr));
          hi[j] = fma(hi[j], wr[j], fma(hr[j], wi[j], vi));
          hr[j] = nr;
        }
      }
#pragma unroll
      for (int j = 0; j < DPW; ++j) {
        double zr, zi;
        sincos(sf[j] / __ldg(a.lambda + cb), &zi, &zr);
        accr[j] += hr[j] * zr - hi[j] * zi;
        acci[j] += hr[j] * zi + hi[j] * zr;
      }
    }
  }
  const int64_t slab_off = static_cast<int64_t>(slab) * a.ndir * nI1;
#pragma unroll
  for (int j = 0; j < DPW; ++j) {
    const int d = d0 + j;
    if (d < a.ndir) out[slab_off + static_cast<int64_t>(d) * nI1 + k] = make_double2(accr[j], acci[j]);
  }
}

// UVWs as (hi, lo) float pairs for the double-float phase set-up.
static __global__ void split_uvw(const double* __restrict__ uvw, int64_t rows, float* __restrict__ out) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < 3 * rows;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double x = uvw[i];
    const float hi = static_cast<float>(x);
    out[2 * i] = hi;
    out[2 * i + 1] = static_cast<float>(x - static_cast<double>(hi));
  }
}

// Per-direction phase constants: -(l, m, n-1) * f0/c and -(l, m, n-1) * df/c as
// (hi, lo) float pairs, from the third row of each direction matrix.  n-1 is
// exact in FP64 (Sterbenz), which removes the reference's w_rot - w cancellation.
static __global__ void direction_constants(const double* __restrict__ dd, int ndir, double f0, double df,
                                           float* __restrict__ out) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= ndir) return;
  const double kA = f0 / kSpeedOfLight, kB = df / kSpeedOfLight;
  const double lmn[3] = {dd[9 * d + 6], dd[9 * d + 7], dd[9 * d + 8] - 1.0};
  for (int s = 0; s < 2; ++s) {
    const double k = s == 0 ? kA : kB;
    for (int i = 0; i < 3; ++i) {
      const double x = -lmn[i] * k;
      const float hi = static_cast<float>(x);
      out[12 * d + 6 * s + 2 * i] = hi;
      out[12 * d + 6 * s + 2 * i + 1] = static_cast<float>(x - static_cast<double>(hi));
    }
  }
}

// Sum of slab partials in slab order: avg[i] = sum_s partial[s][i].
static __global__ void reduce_slabs(const double2* __restrict__ partial, int nslab, int64_t n, double2* __restrict__ avg) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double re = 0.0, im = 0.0;
    for (int s = 0; s < nslab; ++s) {
      const double2 v = partial[static_cast<int64_t>(s) * n + i];
      re += v.x;
      im += v.y;
    }
    avg[i] = make_double2(re, im);
  }
}

// Zero every (row, channel) group of P samples that holds a NaN in any pol,
// copying src -> dst (dst may equal src).  This applies the reference's
// per-sample NaN skip (CpuLeapCalibrator.cc:201-214) once, at ingestion.
template <typename VisT, int P>
__global__ void sanitize_nan_groups(const VisT* src, VisT* dst, int64_t groups) {  // src may equal dst
  using S = typename VisScalar<VisT>::type;
  for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; g < groups;
       g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    VisT v[P];
    bool nan = false;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      v[p] = src[g * P + p];
      nan |= isnan(v[p].x) || isnan(v[p].y);
    }
    if (!nan && src == dst) continue;  // in place: a clean group stays as it is
#pragma unroll
    for (int p = 0; p < P; ++p) {
      VisT o = v[p];
      if (nan) { o.x = S(0); o.y = S(0); }
      dst[g * P + p] = o;
    }
  }
}

// Runtime-P variant of the NaN sanitiser for pol counts without a template instance.
template <typename VisT>
__global__ void sanitize_nan_groups_generic(const VisT* src, VisT* dst, int64_t groups, int P) {
  using S = typename VisScalar<VisT>::type;
  for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; g < groups;
       g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    bool nan = false;
    for (int p = 0; p < P; ++p) {
      const VisT v = src[g * P + p];
      nan |= isnan(v.x) || isnan(v.y);
    }
    if (!nan && src == dst) continue;
    for (int p = 0; p < P; ++p) {
      VisT o = src[g * P + p];
      if (nan) { o.x = S(0); o.y = S(0); }
      dst[g * P + p] = o;
    }
  }
}

// K1: rotated[d][r] = dd[d] * uvw[r]  (MetaData::CalcUVW, LA/model/cpu/MetaData.cc:220-229;
// g_RotateUVW, LA/algorithm/cuda/CudaLeapCalibrator.cu:271-282).
static __global__ void rotate_uvw(const double* __restrict__ dd, const double* __restrict__ uvw, int64_t rows, int ndir,
                           double* __restrict__ out) {
  const int64_t total = rows * ndir;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t d = i / rows, r = i % rows;
    const double* m = dd + 9 * d;
    const double x = uvw[3 * r], y = uvw[3 * r + 1], z = uvw[3 * r + 2];
#pragma unroll
    for (int k = 0; k < 3; ++k) out[3 * i + k] = m[3 * k] * x + m[3 * k + 1] * y + m[3 * k + 2] * z;
  }
}

}  // namespace leapgb
