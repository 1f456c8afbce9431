// C ABI: leap_backward, the adjoint of one calibrate call to FP64 accuracy (differentiable form).
#include "leap_internal.h"
#include "kernels_solve.cuh"
#include "kernels_adjoint.cuh"

namespace leapabi {

// Blocks of a variant of the dL/d(l, m, n) kernel that an SM runs at a time: 16 warps by registers (more are not counted),
// fewer blocks of 1 or 2 warps by shared memory.
template <typename VisT, int P, int NW>
int adjoint_blocks_nw(leap_ctx* ctx, int& blocks) {
  constexpr int smem = adjoint_lmn_smem_bytes<VisT, P>();
  int& n = ctx->adj_blocks[sizeof(VisT) == 8 ? 0 : 1][P / 2][NW == 8 ? 3 : NW / 2];
  if (n == 0) {
    LEAP_CUDA(cudaFuncSetAttribute(adjoint_lmn_fixed<VisT, P, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
              "set shared memory size");
    LEAP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, adjoint_lmn_fixed<VisT, P, NW>, NW * 32, smem),
              "query resident blocks");
    n = std::max(1, std::min(n, 16 / NW));
  }
  blocks = n;
  return LEAP_OK;
}

template <typename VisT, int P, int NW>
void launch_adjoint_lmn(const AdjointFixedArgs& fa, dim3 grid, cudaStream_t s) {
  adjoint_lmn_fixed<VisT, P, NW><<<grid, NW * 32, adjoint_lmn_smem_bytes<VisT, P>(), s>>>(fa);
}

// Rotate + average adjoint in fixed point: dL/d(l, m, n) to d_grad_lmn and, with aa.gvis, dL/dV.
template <typename VisT, int P>
int adjoint_fixed(leap_ctx* ctx, AdjointFixedArgs fa, double* d_grad_lmn, cudaStream_t s) {
  const AdjointArgs& a = fa.a;
  const int nbl = a.nbl, D = a.D;
  // Up to 16 directions a block (the split of a stage into limbs is done once for them); fewer, and channel or
  // timestep slabs, as the forward kernel has them.
  int nw = D <= 2 ? 1 : D <= 4 ? 2 : D <= 8 ? 4 : 8;
  int resident = 1;
  if (nw == 1) {
    // 5 blocks of 1 warp (4 complex<double> pols) leave most of the issue slots free (128 antennas, 8 timesteps, 96
    // channels, 1 direction: 487 us, with 2 warps 434; complex<float>, 9 blocks: 260 and 291).
    if (const int rc = adjoint_blocks_nw<VisT, P, 1>(ctx, resident)) return rc;
    if (resident < 8) nw = 2;
  }
  {
    const int rc = nw == 1 ? adjoint_blocks_nw<VisT, P, 1>(ctx, resident) : nw == 2 ? adjoint_blocks_nw<VisT, P, 2>(ctx, resident)
                 : nw == 4 ? adjoint_blocks_nw<VisT, P, 4>(ctx, resident) : adjoint_blocks_nw<VisT, P, 8>(ctx, resident);
    if (rc != LEAP_OK) return rc;
  }
  const int tiles = (nbl + 31) / 32, dgroups = (D + nw * kFxDirs - 1) / (nw * kFxDirs);
  choose_fixed_slabs(fa.T, a.C, static_cast<int64_t>(tiles) * dgroups, static_cast<int64_t>(ctx->sms) * resident,
                     fa.t_per_slab, fa.c_per_slab,
                     fa.n_tslab, fa.n_cslab);
  const int nslab = fa.n_tslab * fa.n_cslab, nblk = tiles * nslab;
  LEAP_CUDA(ctx->adj_partial.ensure(sizeof(double) * 3 * static_cast<size_t>(nblk) * D), "alloc adjoint partials");
  fa.a.partial = ctx->adj_partial.as<double>();
  adjoint_exponents<VisT, P><<<static_cast<unsigned>((a.rows + 31) / 32), 256, 0, s>>>(
      static_cast<const VisT*>(a.vis), a.rows, a.C, a.check_nan, const_cast<int16_t*>(fa.vexp));
  const dim3 grid(tiles * dgroups, nslab);
  switch (nw) {
    case 1: launch_adjoint_lmn<VisT, P, 1>(fa, grid, s); break;
    case 2: launch_adjoint_lmn<VisT, P, 2>(fa, grid, s); break;
    case 4: launch_adjoint_lmn<VisT, P, 4>(fa, grid, s); break;
    default: launch_adjoint_lmn<VisT, P, 8>(fa, grid, s); break;
  }
  adjoint_lmn_reduce<<<(3 * D + 3) / 4, 128, 0, s>>>(fa.a.partial, nblk, D, d_grad_lmn);
  if (a.gvis) {
    adjoint_split_g<<<(nbl + 127) / 128, 128, 0, s>>>(a.gavg, nbl, D, const_cast<int4*>(fa.g), const_cast<int16_t*>(fa.gexp));
    const int64_t units = ((a.rows + 31) / 32) * ((a.C + kVisChannels - 1) / kVisChannels);
    constexpr int warps = kVisThreads / 32;
    adjoint_vis_fixed<VisT, P><<<static_cast<unsigned>((units + warps - 1) / warps), kVisThreads,
                                 D > kVisFlush ? kVisSumBytes : 0, s>>>(fa);
  }
  return LEAP_OK;
}

}  // namespace leapabi

extern "C" {

int32_t leap_backward(leap_ctx* ctx, int32_t slot, const double* d_dd, int32_t ndir, const double* d_avg0,
                      const double* d_grad_cal, const void* d_vis, double* d_grad_lmn, void* d_grad_vis,
                      void* stream) {
  if (!ctx || !d_dd || !d_avg0 || !d_grad_cal || !d_grad_lmn) return fail(ctx, LEAP_ERR_INVALID_ARGUMENT, "NULL argument");
  if (ndir <= 0) return fail(ctx, LEAP_ERR_INVALID_ARGUMENT, "ndirections must be positive");
  if (!ctx->md.set) return fail(ctx, LEAP_ERR_NOT_READY, "metadata not set");
  auto it = ctx->integ.find(slot);
  if (it == ctx->integ.end()) return fail(ctx, LEAP_ERR_NOT_READY, "integration slot not set");
  DeviceGuard g(ctx->device);
  Metadata& md = ctx->md;
  const Integration& in = it->second;
  const int nbl = static_cast<int>(md.k.nbaselines);
  const int S = md.S, D = ndir, nI = md.Arows - 1, nI1 = md.A1rows - 1;
  cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
  if (in.pending) cudaStreamWaitEvent(s, in.ready, 0);
  LEAP_CUDA(ctx->adj_dphi.ensure(sizeof(double) * std::max(nI, 1) * D), "alloc adjoint scratch");
  LEAP_CUDA(ctx->adj_cal1.ensure(sizeof(double) * S * D), "alloc adjoint scratch");
  LEAP_CUDA(ctx->adj_phi1.ensure(sizeof(double) * std::max(nI1, 1) * D), "alloc adjoint scratch");
  LEAP_CUDA(ctx->adj_gavg.ensure(sizeof(double2) * static_cast<size_t>(nbl) * D), "alloc adjoint scratch");
  // Solve adjoint: g_dphi, g_cal1, g_phi1, g_avg.
  if (nI > 0)
    adjoint_contract_t<<<(nI * 32 + 255) / 256, 256, 0, s>>>(md.Ad.as<double>(), S, nI, d_grad_cal, D,
                                                             ctx->adj_dphi.as<double>(), nI);
  else
    LEAP_CUDA(cudaMemsetAsync(ctx->adj_dphi.ptr, 0, sizeof(double) * D, s), "clear");
  adjoint_cal1<<<static_cast<unsigned>((static_cast<int64_t>(S) * D * 32 + 255) / 256), 256, 0, s>>>(
      d_grad_cal, ctx->adj_dphi.as<double>(), std::max(nI, 1), md.at_ptr.as<int32_t>(), md.at_idx.as<int32_t>(),
      md.at_val.as<double>(), S, D, ctx->adj_cal1.as<double>());
  if (nI1 > 0)
    adjoint_contract_t<<<(nI1 * 32 + 255) / 256, 256, 0, s>>>(md.Ad1.as<double>(), S, nI1, ctx->adj_cal1.as<double>(),
                                                              D, ctx->adj_phi1.as<double>(), nI1);
  const double2* avg0 = reinterpret_cast<const double2*>(d_avg0);
  adjoint_avg_dint<<<grid_1d(static_cast<int64_t>(nbl) * D, 256), 256, 0, s>>>(
      avg0, ctx->adj_dphi.as<double>(), std::max(nI, 1), nI, nbl, D, ctx->adj_gavg.as<double2>());
  if (nI1 > 0)
    adjoint_avg_phi1<<<D, 256, 0, s>>>(avg0, ctx->adj_phi1.as<double>(), md.I1.as<int32_t>(), nI1, nbl, D,
                                       ctx->adj_gavg.as<double2>());
  // Rotate + average adjoint over the integration, recomputing the rotated samples.
  AdjointArgs aa{};
  aa.vis = d_vis ? d_vis : in.vis.ptr;
  aa.vis_c64 = in.vis_type == LEAP_VIS_C64;
  aa.check_nan = d_vis != nullptr;
  aa.uvw = in.uvw.as<double>();
  aa.dd = d_dd;
  aa.gavg = ctx->adj_gavg.as<double2>();
  aa.rows = in.rows;
  aa.C = in.channels;
  aa.P = in.pols;
  aa.nbl = nbl;
  aa.D = D;
  aa.f0 = md.k.freq_start_hz;
  aa.df = md.k.freq_inc_hz;
  {
    const int rc = ensure_spectrum(ctx, aa.C, s);
    if (rc != LEAP_OK) return rc;
  }
  aa.gvis = d_grad_vis;
  // The fixed-point kernels read and write 16-byte pieces (8 for a single complex<float>); arrays that are not
  // aligned to that, and spectral windows that fixed_phase.h does not take, use the FP64 ones.
  const size_t esz = aa.vis_c64 ? sizeof(float2) : sizeof(double2);
  const uintptr_t align = esz * aa.P % 16 == 0 ? 16 : 8;
  if (ctx->tab->spectrum.fx_ok && in.rows % nbl == 0 && (reinterpret_cast<uintptr_t>(aa.vis) | reinterpret_cast<uintptr_t>(d_grad_vis)) % align == 0) {
    LEAP_CUDA(ctx->fx_exp.ensure(sizeof(int16_t) * in.rows), "alloc row exponents");
    LEAP_CUDA(ctx->adj_g.ensure(sizeof(int4) * 2 * static_cast<size_t>(nbl) * D), "alloc adjoint scratch");
    LEAP_CUDA(ctx->adj_gexp.ensure(sizeof(int16_t) * nbl), "alloc adjoint scratch");
    AdjointFixedArgs fa{};
    fa.a = aa;
    fa.sp = ctx->tab->spectrum.sp;
    fa.tab = ctx->fx_tab.as<int4>();
    fa.rho = ctx->tab->fx_rho.as<int32_t>();
    fa.lambda = ctx->tab->lambda.as<double>();
    fa.inv_lambda = ctx->tab->lambda.as<double>() + ctx->tab->spectrum.channels;
    fa.vexp = ctx->fx_exp.as<int16_t>();
    fa.kexp = std::ilogb(ctx->tab->spectrum.sp.kmax) + 1;
    fa.T = static_cast<int>(in.rows / nbl);
    fa.g = ctx->adj_g.as<int4>();
    fa.gexp = ctx->adj_gexp.as<int16_t>();
    int rc = LEAP_OK;
    if (aa.vis_c64)
      rc = aa.P == 1 ? adjoint_fixed<float2, 1>(ctx, fa, d_grad_lmn, s) : aa.P == 2 ? adjoint_fixed<float2, 2>(ctx, fa, d_grad_lmn, s)
                                                                                    : adjoint_fixed<float2, 4>(ctx, fa, d_grad_lmn, s);
    else
      rc = aa.P == 1 ? adjoint_fixed<double2, 1>(ctx, fa, d_grad_lmn, s) : aa.P == 2 ? adjoint_fixed<double2, 2>(ctx, fa, d_grad_lmn, s)
                                                                                     : adjoint_fixed<double2, 4>(ctx, fa, d_grad_lmn, s);
    if (rc != LEAP_OK) return rc;
    LEAP_CUDA(cudaGetLastError(), "adjoint launch");
    return LEAP_OK;
  }
  constexpr int kDPB = 4;
  const int64_t items = in.rows * ((in.channels + kAdjChannels - 1) / kAdjChannels);
  const int dgroups = (D + kDPB - 1) / kDPB;
  const int64_t want = (items + 255) / 256;
  const int bx = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(want, std::max(1, ctx->sms * 8 / dgroups))));
  LEAP_CUDA(ctx->adj_partial.ensure(sizeof(double) * 3 * static_cast<size_t>(bx) * D), "alloc adjoint partials");
  aa.partial = ctx->adj_partial.as<double>();
  adjoint_lmn<kDPB><<<dim3(bx, dgroups), 256, 0, s>>>(aa);
  adjoint_lmn_reduce<<<(3 * D + 3) / 4, 128, 0, s>>>(aa.partial, bx, D, d_grad_lmn);
  if (d_grad_vis) {
    LEAP_CUDA(cudaMemsetAsync(d_grad_vis, 0, esz * static_cast<size_t>(in.rows) * in.channels * in.pols, s),
              "clear vis gradient");
    adjoint_vis<<<grid_1d(items, 256), 256, 0, s>>>(aa);
  }
  LEAP_CUDA(cudaGetLastError(), "adjoint launch");
  return LEAP_OK;
}

}  // extern "C"
