// Test harness of csrc/fixed_phase.h: the phasors of one (row, direction), channel by channel, as the
// kernel forms them, returned as 60-bit integers.
#include "fixed_phase.h"
#include "host_math.h"

using namespace leapgb;

extern "C" int fx_check(double sf, double f0, double df, int channels, const double* lambda, int c0, int seed_every,
                        long long* zr, long long* zi) {
  FxSpectrum sp;
  std::vector<int32_t> rho(channels);
  std::vector<FxLimbs> tab;
  if (!fx_spectrum(f0, df, channels, lambda, sp, rho.data()) || !fx_in_range(sf, sp)) return 1;
  fx_tables(tab);
  auto phasor = [&](uint64_t t) { return fx_turn(t, tab[t >> 54], tab[kFxTable + ((t >> 44) & (kFxTable - 1))]); };
  FxPhase ph;
  uint64_t step;
  fx_setup(ph, sf, sp, c0, step);
  const FxLimbs w = phasor(step);
  int64_t re = 0, im = 0;
  for (int c = c0; c < channels; ++c) {
    if ((c - c0) % seed_every == 0) {
      ph.e = fx_residual(ph, rho[c]);
      const FxLimbs z = phasor(fx_turns(ph));
      re = (static_cast<int64_t>(z.rh) << 30) + z.rl;
      im = (static_cast<int64_t>(z.ih) << 30) + z.il;
    }
    zr[c - c0] = re;
    zi[c - c0] = im;
    if (c + 1 < channels) {
      int32_t d, nd;
      fx_advance(ph, rho[c + 1], d, nd);
      fx_step(re, im, w, d, nd);
    }
  }
  return 0;
}
