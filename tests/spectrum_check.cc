// Test harness of update_spectrum (csrc/host_math.h): device tables faked by vectors, whose allocation or copies can be
// made to fail.  A window is (f0, df, channels); `fail` says which step of the call fails: 0 none, 1 the allocation of the
// wavelengths (whose old buffer is freed), 2 that of the corrections, 3 and 4 their copies.
#include "host_math.h"

using namespace leapgb;

namespace {
Spectrum spectrum;
std::vector<double> lambda;
std::vector<int32_t> rho;
}  // namespace

extern "C" void spectrum_reset() {
  spectrum = Spectrum{};
  lambda.clear();
  rho.clear();
}

extern "C" int spectrum_call(double f0, double df, int channels, int fail) {
  return update_spectrum(
      spectrum, f0, df, channels,
      [&]() -> int {
        if (lambda.size() < 2 * static_cast<size_t>(channels)) {
          lambda.clear();
          if (fail == 1) return 1;
          lambda.resize(2 * channels, -7.0);
        }
        if (rho.size() < static_cast<size_t>(channels)) {
          rho.clear();
          if (fail == 2) return 2;
          rho.resize(channels, -7);
        }
        return 0;
      },
      [&]() -> int {
        if (fail == 3) return 3;
        std::copy(spectrum.lambda.begin(), spectrum.lambda.end(), lambda.begin());
        if (fail == 4) return 4;
        std::copy(spectrum.rho.begin(), spectrum.rho.end(), rho.begin());
        return 0;
      });
}

// What a kernel of the last window would read: wavelengths, reciprocals and corrections.  Returns whether the tables are
// as long as it needs and the fixed-point form applies.
extern "C" int spectrum_read(int channels, double* lam, double* inv, int* corrections) {
  if (spectrum.channels != channels || !spectrum.fx_ok || lambda.size() < 2 * static_cast<size_t>(channels) ||
      rho.size() < static_cast<size_t>(channels))
    return 0;
  for (int c = 0; c < channels; ++c) {
    lam[c] = lambda[c];
    inv[c] = lambda[spectrum.channels + c];
    corrections[c] = rho[c];
  }
  return 1;
}
