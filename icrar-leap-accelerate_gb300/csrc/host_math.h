// Host-side FP64 set-up maths shared by the C ABI and the C++ calibrator.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "fixed_phase.h"

namespace leapgb {

// MetaData::GenerateDDMatrix (LA/model/cpu/MetaData.cc:166-203); dd is 3x3 row-major.
void dd_matrix(double phase_ra, double phase_dec, double ra, double dec, double* dd);

// PhaseMatrixFunction (LA/algorithm/cpu/PhaseMatrixFunction.cc:35-93).  ref_ant < 0 = none.
// A is returned column-major (rows x cols).  Returns a LEAP_* status.
int phase_matrix(const int32_t* a1, const int32_t* a2, const uint8_t* fg, int32_t n, int32_t ref_ant,
                 std::vector<double>& A, std::vector<int32_t>& I, int32_t& rows, int32_t& cols, std::string& err);

// One row of a phase matrix: the non-zeros (c0, v0), (c1, v1) in column order; a row with a
// single non-zero has c1 == c0 and v1 == 0.
struct SparseRow {
  int32_t c0, c1;
  double v0, v1;
};

// PhaseMatrixFunction in sparse row form (no dense rows x cols array).
int phase_matrix_sparse(const int32_t* a1, const int32_t* a2, const uint8_t* fg, int32_t n, int32_t ref_ant,
                        std::vector<SparseRow>& A, std::vector<int32_t>& I, int32_t& cols, std::string& err);

// SVDPseudoInverse (LA/math/cpu/matrix_invert.h:49-56): A (m x n, column-major) -> Ad (n x m, column-major).
int pseudo_inverse(const double* A, int32_t m, int32_t n, double* Ad, std::string& err);

// Grid matrix of the gridded rotate + average (kernels_grid.cuh) for C channels:
// E[l][c] = exp(2 pi i (c - C/2) l / (2C)) / Psi(c - C/2) for table rows r = l + lbase,
// r in [0, rows), with Psi the Fourier transform of the exponential-of-semicircle
// kernel of width `taps` and shape `beta` at frequency k / (2C).  Scaled by a power of
// two (its largest entry in [2^13, 2^14)) and written as FP16 (hi, lo) splits in the
// K-major layout the kernel copies from: [segment of 64 channels][row group of 8][chunk of 16
// channels][hi, lo][2 k-halves][8 rows x 8 k], rows 2 l + (0: re, 1: im), the last segment filled up
// with zeros.  Returns the inverse scale.
float grid_table(int32_t C, int32_t taps, double beta, int32_t lbase, int32_t rows, std::vector<uint16_t>& out);

// Interpolation weights of the gridded rotate + average as polynomials: for m = 0 .. taps-1,
// out[m * (degree + 1) + j] is the x^j coefficient (x = 2 f - 1, f in [0, 1)) of the degree
// `degree` Chebyshev interpolant of psi((f + taps/2 - 1 - m) * 2 / taps), psi the
// exponential-of-semicircle kernel of width `taps` and shape `beta` (the piecewise-polynomial
// kernel evaluation of Barnett, Magland & af Klinteberg, SIAM J. Sci. Comput. 41 (2019) C479).
void es_kernel_poly(int32_t taps, double beta, int32_t degree, float* out);

// Psi(k) = integral over |x| < taps/2 of psi(x) cos(2 pi x k / n), for k = 0..kmax.
std::vector<double> es_kernel_transform(int32_t taps, double beta, int32_t n, int32_t kmax);

// Spectral window of the fixed-point phasors (fixed_phase.h) for channel wavelengths lambda[c],
// c < channels, as the reference rounds them, and rho[c]: 2^(64 + kFxFrac) times the relative difference of
// 1 / lambda[c] from (f0 + c df) / c_light.  Returns false where the fixed-point path does not apply:
// a frequency that is not positive and finite, or wavelengths too far from their own formula.
bool fx_spectrum(double f0, double df, int32_t channels, const double* lambda, FxSpectrum& sp, int32_t* rho);

// Channel wavelengths of a spectral window and their reciprocals, and its fixed-point form: the host's copy of what the
// kernels read.
struct Spectrum {
  int32_t channels = 0;               // 0: the device tables hold nothing to rely on
  double f0 = 0.0, df = 0.0;
  std::vector<double> lambda;         // [wavelengths][their reciprocals]
  std::vector<int32_t> rho;           // corrections of the fixed-point phasors
  FxSpectrum sp{};
  bool fx_ok = false;                 // the fixed-point phasors apply to this window
};

// Wavelengths c / (f0 + ch*df) with each operation rounded on its own, as the reference's
// Constants::GetChannelWavelength (no fused multiply-add), and the rest of `t`.
void spectrum_tables(double f0, double df, int32_t channels, Spectrum& t);

// Makes `t` and the device tables those of a window: reserve() allocates them for `channels` channels, upload() copies
// them; both return 0 or an error, which leaves `t` empty, so that the next call starts over.
template <typename Reserve, typename Upload>
int update_spectrum(Spectrum& t, double f0, double df, int32_t channels, Reserve reserve, Upload upload) {
  if (channels > 0 && t.channels == channels && t.f0 == f0 && t.df == df) return 0;
  t.channels = 0;
  t.fx_ok = false;
  if (const int rc = reserve()) return rc;
  spectrum_tables(f0, df, channels, t);
  if (const int rc = upload()) {
    t.fx_ok = false;
    return rc;
  }
  t.channels = channels;
  t.f0 = f0;
  t.df = df;
  return 0;
}

// The two phasor tables: kFxTable entries exp(2 pi i j / 2^10), then kFxTable of exp(2 pi i j / 2^20).
void fx_tables(std::vector<FxLimbs>& out);

// `count` units of equal cost for schedule_units: numbers begin + (i / per) * stride + i % per, i < count.
struct UnitRun {
  int64_t cost;
  int32_t begin, count, per, stride;
};

// Unit schedule of a persistent kernel with `grid` blocks: longest unit first, each to the least loaded block.
// order[k * grid + b] is the k-th unit of block b, or -1 after its last; the last round is all -1.
void schedule_units(std::vector<UnitRun> runs, int32_t grid, std::vector<int32_t>& order);

// Slab split of (timestep, channel) space for the fixed-point kernels, `resident` of whose blocks run at a time: the
// fewest slabs whose blocks fill the last round of resident ones to 95%, of whole timesteps, then of 128-channel sums,
// and of 32-channel blocks (the seeding interval) or 16-channel ones (a stage) only where the call is too small to fill
// the GPU once (36 antennas, 48 channels, one direction: 145 us a call in 32s, 104 in 16s; in 8s 97, but another small
// call 8% slower).  t_per and c_per: timesteps and channels of a slab, nts and ncs: slabs.
void choose_fixed_slabs(int timesteps, int channels, int64_t base_blocks, int64_t resident, int& t_per, int& c_per, int& nts,
                        int& ncs);

}  // namespace leapgb
