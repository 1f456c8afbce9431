// Adjoint of the calibration chain rotate -> average -> arg -> solve, to FP64 accuracy.
//
// Forward, per direction (LA/algorithm/cpu/CpuLeapCalibrator.cc:159-217):
//   phase[r][c] = -2*pi*(l*u_r + m*v_r + (n-1)*w_r) / lambda_c,   (l, m, n) = row 2 of dd
//   avg[b]      = sum_{t, c} V[0][t*nbl + b][c] * exp(i*phase)    (pol 0; NaN groups skipped)
//   phi1[k]     = arg(avg[I1[k]]),  phi1[|I1|] = 0
//   cal1        = Ad1 * phi1
//   dInt[n]     = arg(exp(-2*pi*i*(A*cal1)[n]) * avg[n]),  n < |I|   (row n, not I[n])
//   cal         = Ad * (dInt ++ [0]) + cal1
//
// Gradients follow the convention of complex autograd: for a real loss L and a
// complex quantity z = x + iy, gz = dL/dx + i*dL/dy (so y = a*z gives
// gz = conj(a)*gy, and arg(z) has gradient i*z/|z|^2).  Given g_cal:
//   g_dphi  = Ad^T g_cal                               (entries n < |I|)
//   g_cal1  = g_cal + A^T (-2*pi * g_dphi)             (rows n < |I| of A)
//   g_phi1  = Ad1^T g_cal1                             (entries k < |I1|)
//   g_avg[b] = [b < |I|] g_dphi[b] i avg[b]/|avg[b]|^2 + sum_{k: I1[k] = b} g_phi1[k] i avg[b]/|avg[b]|^2
//   g_V[0][r][c] = g_avg[r mod nbl] * exp(-i*phase[r][c])  (zero for other pols and NaN groups)
//   dL/d(l, m, n) = sum_{r, c} Re(conj(g_avg[b]) * i * V[0][r][c] * exp(i*phase)) * (-2*pi/lambda_c) * (u, v, w)_r
// The rotated samples are recomputed here, not stored by the forward pass.
// Sums over (row, channel) go to per-block partials that one kernel adds in a
// fixed order: results do not depend on scheduling.
//
// Two forms of the (row, channel, direction) work, as in the forward pass: fixed point (adjoint_lmn_fixed,
// adjoint_vis_fixed: the phasors of fixed_phase.h, hence of the reference's rounded arguments, and integer sums)
// and FP64 FMAs (adjoint_lmn, adjoint_vis) for spectral windows that the first does not take.
#pragma once

#include "leap_common.cuh"
#include "kernels_fixed.cuh"

namespace leapgb {

constexpr int kAdjChannels = 16;  // channels per thread item (phase re-seeded with sincos per item)

struct AdjointArgs {
  const void* vis;         // [C][rows][P], float2 (vis_c64) or double2
  int vis_c64;
  int check_nan;           // skip (row, channel) groups holding a NaN in any pol
  const double* uvw;       // [rows][3]
  const double* dd;        // [D][9]
  const double2* gavg;     // [D][nbl]
  int64_t rows;
  int32_t C, P, nbl, D;
  double f0, df;
  double* partial;         // [gridDim.x][D][3]
  void* gvis;              // [C][rows][P] same element type as vis, pol 0 written
};

__device__ __forceinline__ double2 adj_load(const AdjointArgs& a, int64_t idx) {
  if (a.vis_c64) {
    const float2 v = __ldg(static_cast<const float2*>(a.vis) + idx);
    return make_double2(v.x, v.y);
  }
  return __ldg(static_cast<const double2*>(a.vis) + idx);
}

// Pol-0 samples of one (row, 16-channel) item; zero where the group has a NaN or c >= C.
__device__ __forceinline__ void adj_item_samples(const AdjointArgs& a, int64_t r, int c0, double2 (&x)[kAdjChannels]) {
#pragma unroll
  for (int k = 0; k < kAdjChannels; ++k) {
    const int c = c0 + k;
    x[k] = make_double2(0.0, 0.0);
    if (c < a.C) {
      const int64_t base = (static_cast<int64_t>(c) * a.rows + r) * a.P;
      const double2 v0 = adj_load(a, base);
      bool nan = isnan(v0.x) || isnan(v0.y);
      if (a.check_nan)
        for (int p = 1; p < a.P; ++p) {
          const double2 v = adj_load(a, base + p);
          nan |= isnan(v.x) || isnan(v.y);
        }
      if (!nan) x[k] = v0;
    }
  }
}

// exp(i*phase) at channel c0 and the per-channel step exp(i*sf*df/c_light), sf = -2*pi*(w_rot - w).
__device__ __forceinline__ void adj_phasor(const AdjointArgs& a, int d, double u, double v, double w, int c0,
                                           double& zr, double& zi, double& wr, double& wi) {
  const double wrot = __ldg(a.dd + 9 * d + 6) * u + __ldg(a.dd + 9 * d + 7) * v + __ldg(a.dd + 9 * d + 8) * w;
  const double sf = -kTwoPi * (wrot - w);
  const double lambda0 = kSpeedOfLight / (a.f0 + c0 * a.df);
  sincos(sf / lambda0, &zi, &zr);
  sincos(sf * (a.df / kSpeedOfLight), &wi, &wr);
}

// dL/d(l, m, n) partial sums: blockIdx.y selects DPB directions, threads stride over (row, channel item).
template <int DPB>
__global__ void __launch_bounds__(256) adjoint_lmn(AdjointArgs a) {
  const int d0 = blockIdx.y * DPB;
  const int nitem = (a.C + kAdjChannels - 1) / kAdjChannels;
  const int64_t items = a.rows * nitem;
  double acc[DPB][3];
#pragma unroll
  for (int j = 0; j < DPB; ++j) acc[j][0] = acc[j][1] = acc[j][2] = 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < items;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i % a.rows;
    const int c0 = static_cast<int>(i / a.rows) * kAdjChannels;
    const int b = static_cast<int>(r % a.nbl);
    double2 g[DPB];
    bool any = false;
#pragma unroll
    for (int j = 0; j < DPB; ++j) {
      g[j] = d0 + j < a.D ? a.gavg[static_cast<int64_t>(d0 + j) * a.nbl + b] : make_double2(0.0, 0.0);
      any |= g[j].x != 0.0 || g[j].y != 0.0;
    }
    if (!any) continue;
    double2 x[kAdjChannels];
    adj_item_samples(a, r, c0, x);
    const double u = __ldg(a.uvw + 3 * r), v = __ldg(a.uvw + 3 * r + 1), w = __ldg(a.uvw + 3 * r + 2);
#pragma unroll
    for (int j = 0; j < DPB; ++j) {
      if (g[j].x == 0.0 && g[j].y == 0.0) continue;
      double zr, zi, wr, wi;
      adj_phasor(a, d0 + j, u, v, w, c0, zr, zi, wr, wi);
      double s = 0.0;  // sum_c Re(conj(g) * i * x_c * z_c) / lambda_c
#pragma unroll
      for (int k = 0; k < kAdjChannels; ++k) {
        const double yr = x[k].x * zr - x[k].y * zi, yi = x[k].x * zi + x[k].y * zr;
        s += (g[j].y * yr - g[j].x * yi) * ((a.f0 + (c0 + k) * a.df) / kSpeedOfLight);
        const double nr = zr * wr - zi * wi;
        zi = zr * wi + zi * wr;
        zr = nr;
      }
      acc[j][0] += -kTwoPi * s * u;
      acc[j][1] += -kTwoPi * s * v;
      acc[j][2] += -kTwoPi * s * w;
    }
  }
  // Block reduction: warp tree, then warps in order.
  __shared__ double red[8][DPB * 3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < DPB; ++j)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double x = acc[j][q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) red[warp][j * 3 + q] = x;
    }
  __syncthreads();
  if (threadIdx.x < DPB * 3) {
    double x = 0.0;
    for (int wi = 0; wi < static_cast<int>(blockDim.x >> 5); ++wi) x += red[wi][threadIdx.x];
    const int j = threadIdx.x / 3, q = threadIdx.x % 3;
    if (d0 + j < a.D) a.partial[(static_cast<int64_t>(blockIdx.x) * a.D + d0 + j) * 3 + q] = x;
  }
}

// out[d][q] = sum over blocks of partial[blk][d][q], one warp per (d, q): lanes take blocks in order, then a
// fixed tree.
static __global__ void adjoint_lmn_reduce(const double* __restrict__ partial, int nblk, int D, double* __restrict__ out) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= 3 * D) return;
  double x = 0.0;
  for (int k = lane; k < nblk; k += 32) x += partial[static_cast<int64_t>(k) * 3 * D + i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (lane == 0) out[i] = x;
}

// ---- fixed point ----

// Exponent of each row: the largest component of pol 0 over the groups that are not dropped is below 2^out.
template <typename VisT, int P>
__global__ void __launch_bounds__(256) adjoint_exponents(const VisT* __restrict__ vis, int64_t rows, int channels, int check_nan,
                                                         int16_t* __restrict__ out) {
  __shared__ uint32_t part[8][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int64_t r = blockIdx.x * 32ll + lane;
  uint32_t m = 0;
  if (r < rows)
#pragma unroll 4
    for (int c = g; c < channels; c += 8) {
      const VisT* src = vis + (static_cast<int64_t>(c) * rows + r) * P;
      const VisT v = __ldg(src);
      bool drop = isnan(v.x) || isnan(v.y);
      if (check_nan) {
#pragma unroll
        for (int p = 1; p < P; ++p) {
          const VisT x = __ldg(src + p);
          drop |= isnan(x.x) || isnan(x.y);
        }
      }
      if (!drop) m = max(m, max(fx_magnitude(v.x), fx_magnitude(v.y)));
    }
  part[g][lane] = m;
  __syncthreads();
  if (g == 0 && r < rows) {
#pragma unroll
    for (int k = 1; k < 8; ++k) m = max(m, part[k][lane]);
    out[r] = fx_exponent<VisT>(m);
  }
}

struct AdjointFixedArgs {
  AdjointArgs a;
  FxSpectrum sp;
  const int4* tab;           // phasor tables
  const int32_t* rho;        // [C]
  const double* lambda;      // [C]
  const double* inv_lambda;  // [C]
  const int16_t* vexp;       // [rows] (adjoint_exponents)
  int32_t kexp;              // 1 / lambda < 2^kexp
  int32_t T, t_per_slab, n_tslab, c_per_slab, n_cslab;
  const int4* g;             // [D][nbl][2] split g_avg (adjoint_split_g)
  const int16_t* gexp;       // [nbl]
};

__device__ __forceinline__ double2 adj_double(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 adj_double(double2 v) { return v; }

// sum_c V[0] z / lambda over channels [c_lo, c_hi) of a row, in FP64 with a sincos per channel: for the rows that
// the integer sums leave out.
template <typename VisT, int P>
__device__ __noinline__ double2 adj_plain_row(const AdjointFixedArgs& f, int64_t r, double sf, int c_lo, int c_hi) {
  double2 s = make_double2(0.0, 0.0);
  for (int c = c_lo; c < c_hi; ++c) {
    const VisT* src = static_cast<const VisT*>(f.a.vis) + (static_cast<int64_t>(c) * f.a.rows + r) * P;
    const double2 v = adj_double(__ldg(src));
    bool drop = isnan(v.x) || isnan(v.y);
    if (f.a.check_nan)
      for (int p = 1; p < P; ++p) drop |= isnan(__ldg(src + p).x) || isnan(__ldg(src + p).y);
    if (drop) continue;
    double zi, zr;
    sincos(sf / __ldg(f.lambda + c), &zi, &zr);
    const double k = __ldg(f.inv_lambda + c);
    s.x += (v.x * zr - v.y * zi) * k;
    s.y += (v.x * zi + v.y * zr) * k;
  }
  return s;
}

template <typename VisT, int P>
__host__ __device__ constexpr int adjoint_lmn_smem_bytes() { return fx_raw_bytes<VisT, P>() + kFxStage * 32 * 16; }

// dL/d(l, m, n) partial sums.  The forward kernel's structure (kernels_fixed.cuh) for pol 0 times 1 / lambda, with
// the sums of a row (timestep, baseline) taken to -2 pi Re(conj(g) i S) (u, v, w) at the row's end.  Bound by issue
// slots as that one is, the recurrence of the phasors above all.  128 antennas, 8 timesteps, 96 channels, 16
// directions: 5.46 -> 0.59 ms (FP64 FMAs: 15 per (row, channel, direction) and two sincos per 16 channels).
template <typename VisT, int P, int NW>
__global__ void __launch_bounds__(NW * 32, 16 / NW) adjoint_lmn_fixed(const AdjointFixedArgs f) {
  extern __shared__ __align__(128) unsigned char fx_smem[];
  using Sum = FxSumInt<1>;
  const VisT* raw = reinterpret_cast<const VisT*>(fx_smem);
  unsigned char* limb = fx_smem + fx_raw_bytes<VisT, P>();
  const AdjointArgs& a = f.a;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dgroups = (a.D + NW * kFxDirs - 1) / (NW * kFxDirs);
  const int tile = blockIdx.x / dgroups, dg = blockIdx.x % dgroups;
  const int slab = blockIdx.y, ts = slab / f.n_cslab, cs = slab % f.n_cslab;
  const int t_lo = ts * f.t_per_slab, t_hi = min(f.T, t_lo + f.t_per_slab);
  const int c_lo = cs * f.c_per_slab, c_hi = min(a.C, c_lo + f.c_per_slab);
  const int b0 = tile * 32, b = b0 + lane;
  const bool valid = b < a.nbl;
  const int d0 = (dg * NW + warp) * kFxDirs;
  const bool active = d0 < a.D;
  const int nst = (c_hi - c_lo + kFxStage - 1) / kFxStage;
  const int total = (t_hi - t_lo) * nst;
  auto fetch = [&](int s) {
    const int t = t_lo + s / nst, c0 = c_lo + (s % nst) * kFxStage;
    fx_fetch<VisT, P>(fx_smem, a.vis, a.rows, static_cast<int64_t>(t) * a.nbl + b0, a.nbl - b0, c0, min(kFxStage, c_hi - c0));
  };
  double2 g[kFxDirs];
  double out[kFxDirs][3], sum[kFxDirs][1][2];
  Sum acc[kFxDirs];
  FxRay ray[kFxDirs];
  double2 plain[kFxDirs];
#pragma unroll
  for (int j = 0; j < kFxDirs; ++j) {
    out[j][0] = out[j][1] = out[j][2] = 0.0;
    g[j] = valid && d0 + j < a.D ? a.gavg[static_cast<int64_t>(d0 + j) * a.nbl + b] : make_double2(0.0, 0.0);
  }
  int ve[1] = {0};
  if (total > 0) fetch(0);
  for (int s = 0; s < total; ++s) {
    const int t = t_lo + s / nst, cb = c_lo + (s % nst) * kFxStage, cf = cb - c_lo;
    const int n = min(kFxStage, c_hi - cb);
    const int64_t r = static_cast<int64_t>(t) * a.nbl + (valid ? b : 0);
    if (cf == 0) ve[0] = __ldg(f.vexp + r);
    const bool plain_row = ve[0] == kFxPlain;
    const int e[1] = {plain_row ? 0 : ve[0] + f.kexp};
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int k = warp; k < n; k += NW) {
      const VisT* src = raw + (k * 32 + lane) * P;
      double2 x[1] = {adj_double(src[0])};
      bool drop = isnan(x[0].x) || isnan(x[0].y);
      if (a.check_nan) {
#pragma unroll
        for (int p = 1; p < P; ++p) drop |= isnan(src[p].x) || isnan(src[p].y);
      }
      const double w = __ldg(f.inv_lambda + cb + k);
      x[0].x *= w;
      x[0].y *= w;
      Sum::store(limb, k, lane, x, e, valid && !plain_row && !drop);
    }
    __syncthreads();
    if (s + 1 < total) fetch(s + 1);
    if (!active) continue;
    const double u = __ldg(a.uvw + 3 * r), v = __ldg(a.uvw + 3 * r + 1), w = __ldg(a.uvw + 3 * r + 2);
    if (cf == 0) {
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) {
        const double sf = fx_shift_factor(a.dd + 9 * min(d0 + j, a.D - 1) + 6, u, v, w);
        const bool fits = ray[j].begin(sf, f.sp, c_lo, f.tab);
        plain[j] = make_double2(0.0, 0.0);
        if (valid && (plain_row || !fits)) plain[j] = adj_plain_row<VisT, P>(f, r, sf, c_lo, c_hi);
        sum[j][0][0] = plain[j].x;
        sum[j][0][1] = plain[j].y;
      }
    }
    if (cf % kFxSeed == 0) {
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) ray[j].seed(__ldg(f.rho + cb), f.tab);
    }
    if (cf % Sum::kFlush == 0) {
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) acc[j].clear();
    }
#pragma unroll 2
    for (int k = 0; k < n; ++k) {
      const int32_t rho = __ldg(f.rho + min(cb + k + 1, a.C - 1));
      const typename Sum::Vis x = Sum::load(limb, k, lane);
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) {
        acc[j].add(x, Sum::phasor(ray[j].zr, ray[j].zi));
        ray[j].next(rho);
      }
    }
    const bool last = cb + kFxStage >= c_hi;
    if ((cf + kFxStage) % Sum::kFlush == 0 || last) {
      const double scale[1] = {__hiloint2double((e[0] + Sum::kUnitExp + 1023) << 20, 0)};
#pragma unroll
      for (int j = 0; j < kFxDirs; ++j) {
        acc[j].flush(sum[j], scale);
        if (last && (g[j].x != 0.0 || g[j].y != 0.0)) {
          const double q = -kTwoPi * (g[j].y * sum[j][0][0] - g[j].x * sum[j][0][1]);  // -2 pi Re(conj(g) i S)
          out[j][0] += q * u;
          out[j][1] += q * v;
          out[j][2] += q * w;
        }
      }
    }
  }
  if (!active) return;
#pragma unroll
  for (int j = 0; j < kFxDirs; ++j)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double x = out[j][q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0 && d0 + j < a.D)
        a.partial[((static_cast<int64_t>(slab) * gridDim.x / dgroups + tile) * a.D + d0 + j) * 3 + q] = x;
    }
}

// g_avg for adjoint_vis_fixed: two words of four per (direction, baseline), g 2^(28 - e) in parts (re, im), then -re.
// e = kFxPlain: a gradient that is not finite, or out of range.
static __global__ void adjoint_split_g(const double2* __restrict__ gavg, int nbl, int D, int4* __restrict__ out,
                                       int16_t* __restrict__ gexp) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbl) return;
  uint32_t m = 0;
  for (int d = 0; d < D; ++d) {
    const double2 g = gavg[static_cast<int64_t>(d) * nbl + b];
    m = max(m, max(fx_magnitude(g.x), fx_magnitude(g.y)));
  }
  const int e = fx_exponent<double2>(m);
  const bool plain = e == kFxPlain;
  gexp[b] = static_cast<int16_t>(e);
  const double scale = plain ? 0.0 : scalbn(1.0, 28 - e);
  for (int d = 0; d < D; ++d) {
    const int64_t i = static_cast<int64_t>(d) * nbl + b;
    const double2 g = gavg[i];
    const FxPart x = fx_part(plain ? 0.0 : g.x * scale), y = fx_part(plain ? 0.0 : g.y * scale);
    out[2 * i] = make_int4(x.h, x.l, y.h, y.l);
    out[2 * i + 1] = make_int4(-x.h, -x.l, 0, 0);
  }
}

// One channel's gradient in FP64: for rows that the integer sums leave out.
__device__ __noinline__ double2 adj_plain_vis(const AdjointFixedArgs& f, int64_t r, int b, int c) {
  const AdjointArgs& a = f.a;
  double2 s = make_double2(0.0, 0.0);
  const double u = a.uvw[3 * r], v = a.uvw[3 * r + 1], w = a.uvw[3 * r + 2];
  for (int d = 0; d < a.D; ++d) {
    const double2 g = a.gavg[static_cast<int64_t>(d) * a.nbl + b];
    if (g.x == 0.0 && g.y == 0.0) continue;
    double zi, zr;
    sincos(fx_shift_factor(a.dd + 9 * d + 6, u, v, w) / f.lambda[c], &zi, &zr);
    s.x += g.x * zr + g.y * zi;
    s.y += g.y * zr - g.x * zi;
  }
  return s;
}

__device__ __forceinline__ void adj_write(float2* dst, double re, double im) { *dst = make_float2(static_cast<float>(re), static_cast<float>(im)); }
__device__ __forceinline__ void adj_write(double2* dst, double re, double im) { *dst = make_double2(re, im); }

// g_V[0][r][c] = sum_d g_avg[d][b] exp(-i phase_d[r][c]) and zeros for the other pols, zero at dropped groups.  A
// warp takes 32 rows (lanes) and kVisChannels channels, whose sums over the directions it keeps in 64-bit integers
// (fx_add_products), added to FP64 sums in shared memory every kVisFlush directions where there are more.  128
// antennas, 8 timesteps, 96 channels, 16 directions: 3.04 -> 0.64 ms (FP64 FMAs: 8 per (row, channel, direction) and
// two sincos per 16 channels).
constexpr int kVisChannels = 16;
constexpr int kVisFlush = 64;  // sqrt(2) 2^56 units a direction at most: below 2^63
constexpr int kVisThreads = 128;
constexpr int kVisSumBytes = kVisChannels * kVisThreads * 16;
template <typename VisT, int P>
__global__ void __launch_bounds__(kVisThreads, 3) adjoint_vis_fixed(const AdjointFixedArgs f) {
  extern __shared__ __align__(128) unsigned char fx_smem[];
  double2* sums = reinterpret_cast<double2*>(fx_smem) + threadIdx.x;  // [kVisChannels][kVisThreads]: with more than kVisFlush directions
  const AdjointArgs& a = f.a;
  const int lane = threadIdx.x & 31;
  const int ncb = (a.C + kVisChannels - 1) / kVisChannels;
  const int64_t rtiles = (a.rows + 31) / 32;
  const int64_t unit = blockIdx.x * static_cast<int64_t>(kVisThreads / 32) + (threadIdx.x >> 5);
  if (unit >= rtiles * ncb) return;
  const int c0 = static_cast<int>(unit % ncb) * kVisChannels, n = min(kVisChannels, a.C - c0);
  const int64_t r = (unit / ncb) * 32 + lane;
  const bool valid = r < a.rows;
  const int64_t rr = valid ? r : 0;
  const int b = static_cast<int>(rr % a.nbl);
  const int ge = __ldg(f.gexp + b);
  bool plain = ge == kFxPlain;
  int64_t hr[kVisChannels], hi[kVisChannels];
#pragma unroll
  for (int k = 0; k < kVisChannels; ++k) hr[k] = hi[k] = 0;
  const double u = __ldg(a.uvw + 3 * rr), v = __ldg(a.uvw + 3 * rr + 1), w = __ldg(a.uvw + 3 * rr + 2);
  for (int d = 0; d < a.D; ++d) {
    if (d > 0 && d % kVisFlush == 0) {
#pragma unroll
      for (int k = 0; k < kVisChannels; ++k) {
        double2 s = make_double2(static_cast<double>(hr[k]), static_cast<double>(hi[k]));
        if (d > kVisFlush) {
          s.x += sums[k * kVisThreads].x;
          s.y += sums[k * kVisThreads].y;
        }
        sums[k * kVisThreads] = s;
        hr[k] = hi[k] = 0;
      }
    }
    const int4* g = f.g + 2 * (static_cast<int64_t>(d) * a.nbl + b);
    const int4 g0 = __ldg(g), g1 = __ldg(g + 1);
    const FxPart gx{g0.x, g0.y}, gy{g0.z, g0.w}, ngx{g1.x, g1.y};
    FxRay ray;
    plain |= !ray.begin(fx_shift_factor(a.dd + 9 * d + 6, u, v, w), f.sp, c0, f.tab);
    ray.seed(__ldg(f.rho + c0), f.tab);
#pragma unroll
    for (int k = 0; k < kVisChannels; ++k) {
      const FxPart zr = fx_part(ray.zr), zi = fx_part(ray.zi);
      fx_add_products(hr[k], gx, zr, gy, zi);   // re: g.x z.r + g.y z.i
      fx_add_products(hi[k], gy, zr, ngx, zi);  // im: g.y z.r - g.x z.i
      if (k + 1 < kVisChannels) ray.next(__ldg(f.rho + min(c0 + k + 1, a.C - 1)));
    }
  }
  if (!valid) return;
  const double scale = plain ? 0.0 : __hiloint2double((ge - 56 + 1023) << 20, 0);
#pragma unroll
  for (int k = 0; k < kVisChannels; ++k) {
    if (k >= n) break;
    const int64_t base = (static_cast<int64_t>(c0 + k) * a.rows + r) * P;
    const VisT* src = static_cast<const VisT*>(a.vis) + base;
    bool drop = false;
    if (a.check_nan) {
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const VisT x = __ldg(src + p);
        drop |= isnan(x.x) || isnan(x.y);
      }
    }
    double2 o = make_double2(static_cast<double>(hr[k]), static_cast<double>(hi[k]));
    if (a.D > kVisFlush) {
      o.x += sums[k * kVisThreads].x;
      o.y += sums[k * kVisThreads].y;
    }
    o = make_double2(o.x * scale, o.y * scale);
    if (plain) o = adj_plain_vis(f, r, b, c0 + k);
    if (drop) o = make_double2(0.0, 0.0);
    VisT* dst = static_cast<VisT*>(a.gvis) + base;
    alignas(16) VisT group[P];
    adj_write(&group[0], o.x, o.y);
#pragma unroll
    for (int p = 1; p < P; ++p) adj_write(&group[p], 0.0, 0.0);
    if (P * sizeof(VisT) % 16 == 0) {
#pragma unroll
      for (int i = 0; i < static_cast<int>(P * sizeof(VisT) / 16); ++i)
        reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(group)[i];
    } else {
      dst[0] = group[0];
    }
  }
}

// g_V[0][r][c] = sum_d g_avg[d][b] * exp(-i*phase_d[r][c]); zero at NaN groups.
// The other pols' gradients are zero (the caller clears the array first).
static __global__ void __launch_bounds__(256) adjoint_vis(AdjointArgs a) {
  const int nitem = (a.C + kAdjChannels - 1) / kAdjChannels;
  const int64_t items = a.rows * nitem;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < items;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i % a.rows;
    const int c0 = static_cast<int>(i / a.rows) * kAdjChannels;
    const int b = static_cast<int>(r % a.nbl);
    const double u = __ldg(a.uvw + 3 * r), v = __ldg(a.uvw + 3 * r + 1), w = __ldg(a.uvw + 3 * r + 2);
    double gr[kAdjChannels], gi[kAdjChannels];
#pragma unroll
    for (int k = 0; k < kAdjChannels; ++k) gr[k] = gi[k] = 0.0;
    for (int d = 0; d < a.D; ++d) {
      const double2 g = a.gavg[static_cast<int64_t>(d) * a.nbl + b];
      if (g.x == 0.0 && g.y == 0.0) continue;
      double zr, zi, wr, wi;
      adj_phasor(a, d, u, v, w, c0, zr, zi, wr, wi);
#pragma unroll
      for (int k = 0; k < kAdjChannels; ++k) {
        gr[k] += g.x * zr + g.y * zi;  // g * conj(z)
        gi[k] += g.y * zr - g.x * zi;
        const double nr = zr * wr - zi * wi;
        zi = zr * wi + zi * wr;
        zr = nr;
      }
    }
#pragma unroll
    for (int k = 0; k < kAdjChannels; ++k) {
      const int c = c0 + k;
      if (c >= a.C) break;
      const int64_t base = (static_cast<int64_t>(c) * a.rows + r) * a.P;
      bool nan = false;
      if (a.check_nan)
        for (int p = 0; p < a.P; ++p) {
          const double2 x = adj_load(a, base + p);
          nan |= isnan(x.x) || isnan(x.y);
        }
      const double outr = nan ? 0.0 : gr[k], outi = nan ? 0.0 : gi[k];
      if (a.vis_c64)
        static_cast<float2*>(a.gvis)[base] = make_float2(static_cast<float>(outr), static_cast<float>(outi));
      else
        static_cast<double2*>(a.gvis)[base] = make_double2(outr, outi);
    }
  }
}

// out[d * ldo + k] = sum_s M[s + S*k] * G[d*S + s] for k < kmax: one warp per k.
static __global__ void adjoint_contract_t(const double* __restrict__ M, int S, int kmax, const double* __restrict__ G,
                                          int D, double* __restrict__ out, int ldo) {
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (k >= kmax) return;
  const double* col = M + static_cast<int64_t>(S) * k;
  // 16 directions at a time are summed over the lanes together, halving the directions that a lane holds with each
  // exchange: 16 additions instead of 80, which with the 64 products (128 stations) are bound by the FP64 pipe (128
  // stations, 16 directions, 8128 rows: 73 -> 48 us).  Up to 3 directions, fewer additions one by one.
  int d_lo = 0;
  for (; D - d_lo > 3; d_lo += 16) {
    double x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = 0.0;
    for (int s = lane; s < S; s += 32) {
      const double c = col[s];
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (d_lo + i < D) x[i] += c * G[static_cast<int64_t>(d_lo + i) * S + s];
    }
#pragma unroll
    for (int n = 8; n > 0; n >>= 1) {
      const bool up = lane & (2 * n);
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const double y = __shfl_xor_sync(0xffffffffu, up ? x[i] : x[i + n], 2 * n);
        x[i] = (up ? x[i + n] : x[i]) + y;
      }
    }
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
    const int d = d_lo + (lane >> 1);
    if (!(lane & 1) && d < D) out[static_cast<int64_t>(d) * ldo + k] = x[0];
  }
  for (int d = d_lo; d < D; ++d) {
    double x = 0.0;
    for (int s = lane; s < S; s += 32) x += col[s] * G[static_cast<int64_t>(d) * S + s];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) out[static_cast<int64_t>(d) * ldo + k] = x;
  }
}

// g_cal1[d][s] = g_cal[d][s] - 2*pi * sum_{rows n of A with a non-zero in column s, n < |I|} A[n][s] * g_dphi[d][n].
// (at_ptr, at_idx, at_val) is A^T in compressed-row form over the first |I| rows.  One warp per output (a thread
// each walked the ~S entries one after another: 44 us for 128 stations and 16 directions).
static __global__ void adjoint_cal1(const double* __restrict__ gcal, const double* __restrict__ gdphi, int ld_dphi,
                                    const int32_t* __restrict__ at_ptr, const int32_t* __restrict__ at_idx,
                                    const double* __restrict__ at_val, int S, int D, double* __restrict__ gcal1) {
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= static_cast<int64_t>(S) * D) return;
  const int d = static_cast<int>(i / S), s = static_cast<int>(i % S);
  double x = 0.0;
  for (int j = at_ptr[s] + lane; j < at_ptr[s + 1]; j += 32) x += at_val[j] * gdphi[static_cast<int64_t>(d) * ld_dphi + at_idx[j]];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (lane == 0) gcal1[i] = gcal[i] - kTwoPi * x;
}

__device__ __forceinline__ double2 grad_arg(double2 z, double g) {
  const double n2 = z.x * z.x + z.y * z.y;
  if (n2 == 0.0) return make_double2(0.0, 0.0);
  return make_double2(-g * z.y / n2, g * z.x / n2);  // g * i * z / |z|^2
}

// g_avg[d][b] from the dInt term (b < |I|).
static __global__ void adjoint_avg_dint(const double2* __restrict__ avg0, const double* __restrict__ gdphi, int ld_dphi,
                                        int nI, int nbl, int D, double2* __restrict__ gavg) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < static_cast<int64_t>(nbl) * D;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int d = static_cast<int>(i / nbl), b = static_cast<int>(i % nbl);
    gavg[i] = b < nI ? grad_arg(avg0[i], gdphi[static_cast<int64_t>(d) * ld_dphi + b]) : make_double2(0.0, 0.0);
  }
}

// Adds the phi1 term: block per direction, thread per entry of I1.  Entries may repeat: the first of them adds the
// others too, in order.  (One thread per direction walking I1: 264 us for 127 entries.)
static __global__ void __launch_bounds__(256) adjoint_avg_phi1(const double2* __restrict__ avg0, const double* __restrict__ gphi1,
                                                               const int32_t* __restrict__ I1, int nI1, int nbl, int D,
                                                               double2* __restrict__ gavg) {
  const int d = blockIdx.x;
  for (int k = threadIdx.x; k < nI1; k += blockDim.x) {
    const int mine = I1[k];
    const int idx = mine < 0 ? mine + nbl : mine;
    bool first = true;
    for (int j = 0; j < k && first; ++j) first = (I1[j] < 0 ? I1[j] + nbl : I1[j]) != idx;
    if (!first) continue;
    const int64_t o = static_cast<int64_t>(d) * nbl + idx;
    double2 s = gavg[o];
    const double2 z = avg0[o];
    for (int j = k; j < nI1; ++j) {
      if ((I1[j] < 0 ? I1[j] + nbl : I1[j]) != idx) continue;
      const double2 gz = grad_arg(z, gphi1[static_cast<int64_t>(d) * nI1 + j]);
      s.x += gz.x;
      s.y += gz.y;
    }
    gavg[o] = s;
  }
}

}  // namespace leapgb
