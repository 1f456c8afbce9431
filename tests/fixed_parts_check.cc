// Test harness of fx_part and fx_add_products (csrc/fixed_phase.h): the sum over n terms of a x + b y, in units of
// 2^-56, a and b given as doubles up to 2^28, x and y as 60-bit fixed-point numbers.
#include <cstdint>

#include "fixed_phase.h"

using namespace leapgb;

extern "C" long long fx_parts_check(int n, const double* a, const double* b, const long long* x, const long long* y) {
  int64_t sum = 0;
  for (int i = 0; i < n; ++i) fx_add_products(sum, fx_part(a[i]), fx_part(static_cast<int64_t>(x[i])), fx_part(b[i]), fx_part(static_cast<int64_t>(y[i])));
  return sum;
}
