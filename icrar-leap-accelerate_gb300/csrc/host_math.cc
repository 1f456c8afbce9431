// Host-side FP64 set-up maths behind the C ABI: the direction matrix, the
// phase matrix and the pseudoinverse.  These run once per observation (or once
// per direction for the 3x3 matrix), never per visibility.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>
#include <vector>

#include "leap_gb300.h"
#include "host_math.h"

namespace leapgb {

// dd = R3 * R2 * R1 with ang1 = pi/2 - dec0, ang2 = ra - ra0, ang3 = -pi/2 + dec
// (MetaData::GenerateDDMatrix, LA/model/cpu/MetaData.cc:166-203).  The three
// rotations are written out as the reference builds them and multiplied in the
// same order, so each element is formed from the same products.
void dd_matrix(double phase_ra, double phase_dec, double ra, double dec, double* dd) {
  const double pi = 3.141592653589793238462643383279502884;
  const double a1 = pi / 2.0 - phase_dec, a2 = ra - phase_ra, a3 = -pi / 2.0 + dec;
  const double r1[9] = {1, 0, 0, 0, std::cos(a1), -std::sin(a1), 0, std::sin(a1), std::cos(a1)};
  const double r2[9] = {std::cos(a2), std::sin(a2), 0, -std::sin(a2), std::cos(a2), 0, 0, 0, 1};
  const double r3[9] = {1, 0, 0, 0, std::cos(a3), -std::sin(a3), 0, std::sin(a3), std::cos(a3)};
  double t[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) t[3 * i + j] = r3[3 * i] * r2[j] + r3[3 * i + 1] * r2[3 + j] + r3[3 * i + 2] * r2[6 + j];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) dd[3 * i + j] = t[3 * i] * r1[j] + t[3 * i + 1] * r1[3 + j] + t[3 * i + 2] * r1[6 + j];
}

// PhaseMatrixFunction (LA/algorithm/cpu/PhaseMatrixFunction.cc:35-93): the checks, the
// number of antenna columns and the baselines kept (first-epoch cross baselines, not
// flagged, containing ref_ant when one is given), in baseline order.
static int phase_matrix_rows(const int32_t* a1, const int32_t* a2, const uint8_t* fg, int32_t n, int32_t ref_ant,
                             std::vector<int32_t>& keep, int32_t& cols, std::string& err) {
  if (ref_ant >= 0 && ref_ant >= n) {
    err = "refAnt " + std::to_string(ref_ant) + " is out of bounds";
    return LEAP_ERR_INVALID_ARGUMENT;
  }
  if (ref_ant >= 0 && fg[ref_ant]) {  // the reference indexes the baseline flags by antenna number
    err = "refAnt " + std::to_string(ref_ant) + " is flagged";
    return LEAP_ERR_INVALID_ARGUMENT;
  }
  if (n <= 0) {
    err = "a1 and a2 must not be empty";
    return LEAP_ERR_INVALID_ARGUMENT;
  }
  int32_t maxc = 0;
  for (int32_t i = 0; i < n; ++i) {
    if (a1[i] < 0 || a2[i] < 0) {
      err = "negative antenna index";
      return LEAP_ERR_INVALID_ARGUMENT;
    }
    maxc = std::max(maxc, std::max(a1[i], a2[i]));
  }
  cols = maxc + 1;
  keep.clear();
  keep.reserve(n);
  for (int32_t i = 0; i < n; ++i) {
    if (a1[i] == a2[i] || fg[i]) continue;
    if (ref_ant >= 0 && a1[i] != ref_ant && a2[i] != ref_ant) continue;
    keep.push_back(i);
  }
  return LEAP_OK;
}

int phase_matrix(const int32_t* a1, const int32_t* a2, const uint8_t* fg, int32_t n, int32_t ref_ant,
                 std::vector<double>& A, std::vector<int32_t>& I, int32_t& rows, int32_t& cols, std::string& err) {
  std::vector<int32_t> keep;
  const int rc = phase_matrix_rows(a1, a2, fg, n, ref_ant, keep, cols, err);
  if (rc != LEAP_OK) return rc;
  rows = static_cast<int32_t>(keep.size()) + 1;
  A.assign(static_cast<size_t>(rows) * cols, 0.0);
  I.assign(keep.begin(), keep.end());
  for (int32_t k = 0; k + 1 < rows; ++k) {
    A[k + static_cast<size_t>(rows) * a1[keep[k]]] = 1.0;
    A[k + static_cast<size_t>(rows) * a2[keep[k]]] = -1.0;
  }
  A[(rows - 1) + static_cast<size_t>(rows) * (ref_ant < 0 ? 0 : ref_ant)] = 1.0;
  return LEAP_OK;
}

int phase_matrix_sparse(const int32_t* a1, const int32_t* a2, const uint8_t* fg, int32_t n, int32_t ref_ant,
                        std::vector<SparseRow>& A, std::vector<int32_t>& I, int32_t& cols, std::string& err) {
  std::vector<int32_t> keep;
  const int rc = phase_matrix_rows(a1, a2, fg, n, ref_ant, keep, cols, err);
  if (rc != LEAP_OK) return rc;
  A.resize(keep.size() + 1);
  I.assign(keep.begin(), keep.end());
  for (size_t k = 0; k < keep.size(); ++k) {
    // column order, as the dense row of A lists its non-zeros
    const int32_t p = a1[keep[k]], q = a2[keep[k]];
    A[k] = p < q ? SparseRow{p, q, 1.0, -1.0} : SparseRow{q, p, -1.0, 1.0};
  }
  const int32_t r = ref_ant < 0 ? 0 : ref_ant;
  A[keep.size()] = SparseRow{r, r, 1.0, 0.0};
  return LEAP_OK;
}

// Pseudoinverse through the Gram matrix.
//
// A+ = (A^T A)+ A^T for any A.  G = A^T A is formed from the non-zeros of each
// row of A (two per row for a phase matrix, so G is an integer Laplacian plus
// the reference-antenna row and is formed exactly), diagonalised by cyclic
// Jacobi rotations (which keep exact zero rows and columns of G exact, so
// unobserved antennas get exactly zero weight), and applied to A^T row by row.
//
// Truncation: the reference drops singular values sigma <= max(m,n)*eps*sigma_0
// (LA/math/cpu/matrix_invert.h:54).  Eigenvalues of G are sigma^2 but are only
// resolved to about eps*lambda_0, so the rule is applied as
// lambda <= max(m,n)*eps*lambda_0; the two agree unless a singular value lies
// between max(m,n)*eps*sigma_0 and sqrt(max(m,n)*eps)*sigma_0, which the integer
// structure of phase matrices rules out.
int pseudo_inverse(const double* A, int32_t m, int32_t n, double* Ad, std::string& err) {
  if (m <= 0 || n <= 0) {
    err = "pseudo_inverse: empty matrix";
    return LEAP_ERR_INVALID_ARGUMENT;
  }
  // Row-wise non-zeros of A (column-major input).
  std::vector<int64_t> rowptr(static_cast<size_t>(m) + 1, 0);
  for (int32_t j = 0; j < n; ++j)
    for (int32_t i = 0; i < m; ++i)
      if (A[i + static_cast<size_t>(m) * j] != 0.0) rowptr[i + 1]++;
  for (int32_t i = 0; i < m; ++i) rowptr[i + 1] += rowptr[i];
  std::vector<int32_t> colidx(rowptr[m]);
  std::vector<double> val(rowptr[m]);
  {
    std::vector<int64_t> fill(rowptr.begin(), rowptr.end() - 1);
    for (int32_t j = 0; j < n; ++j)
      for (int32_t i = 0; i < m; ++i) {
        const double a = A[i + static_cast<size_t>(m) * j];
        if (a != 0.0) {
          colidx[fill[i]] = j;
          val[fill[i]] = a;
          fill[i]++;
        }
      }
  }
  // G = A^T A (row-major n x n, symmetric).
  std::vector<double> G(static_cast<size_t>(n) * n, 0.0);
  for (int32_t i = 0; i < m; ++i)
    for (int64_t p = rowptr[i]; p < rowptr[i + 1]; ++p)
      for (int64_t q = rowptr[i]; q < rowptr[i + 1]; ++q) G[static_cast<size_t>(colidx[p]) * n + colidx[q]] += val[p] * val[q];

  // Cyclic Jacobi: G <- J^T G J until the off-diagonal mass is negligible; V accumulates J.
  std::vector<double> V(static_cast<size_t>(n) * n, 0.0);
  for (int32_t i = 0; i < n; ++i) V[static_cast<size_t>(i) * n + i] = 1.0;
  auto g = [&](int32_t i, int32_t j) -> double& { return G[static_cast<size_t>(i) * n + j]; };
  const double eps = std::numeric_limits<double>::epsilon();
  for (int sweep = 0; sweep < 60; ++sweep) {
    double off = 0.0, diag = 0.0;
    for (int32_t i = 0; i < n; ++i) {
      diag += g(i, i) * g(i, i);
      for (int32_t j = i + 1; j < n; ++j) off += g(i, j) * g(i, j);
    }
    if (off <= eps * eps * diag * 1e-4 || off == 0.0) break;
    for (int32_t p = 0; p < n - 1; ++p) {
      for (int32_t q = p + 1; q < n; ++q) {
        const double apq = g(p, q);
        if (apq == 0.0) continue;
        const double app = g(p, p), aqq = g(q, q);
        // Skip rotations that cannot change the diagonal at working precision.
        if (std::fabs(apq) <= eps * 1e-3 * std::sqrt(std::fabs(app * aqq))) {
          g(p, q) = g(q, p) = 0.0;
          continue;
        }
        const double theta = (aqq - app) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int32_t k = 0; k < n; ++k) {
          const double gkp = g(k, p), gkq = g(k, q);
          g(k, p) = c * gkp - s * gkq;
          g(k, q) = s * gkp + c * gkq;
        }
        for (int32_t k = 0; k < n; ++k) {
          const double gpk = g(p, k), gqk = g(q, k);
          g(p, k) = c * gpk - s * gqk;
          g(q, k) = s * gpk + c * gqk;
        }
        g(p, q) = g(q, p) = 0.0;
        for (int32_t k = 0; k < n; ++k) {
          double* vr = &V[static_cast<size_t>(k) * n];
          const double vkp = vr[p], vkq = vr[q];
          vr[p] = c * vkp - s * vkq;
          vr[q] = s * vkp + c * vkq;
        }
      }
    }
  }
  std::vector<double> lam(n);
  double lmax = 0.0;
  for (int32_t i = 0; i < n; ++i) {
    lam[i] = g(i, i);
    lmax = std::max(lmax, std::fabs(lam[i]));
  }
  const double tol = static_cast<double>(std::max(m, n)) * eps * lmax;
  // Gplus = V diag(1/lambda) V^T  (row-major n x n)
  std::vector<double> Gp(static_cast<size_t>(n) * n, 0.0);
  for (int32_t e = 0; e < n; ++e) {
    if (!(std::fabs(lam[e]) > tol)) continue;
    const double inv = 1.0 / lam[e];
    for (int32_t i = 0; i < n; ++i) {
      const double vie = V[static_cast<size_t>(i) * n + e] * inv;
      if (vie == 0.0) continue;
      double* row = &Gp[static_cast<size_t>(i) * n];
      for (int32_t j = 0; j < n; ++j) row[j] += vie * V[static_cast<size_t>(j) * n + e];
    }
  }
  // Iterative refinement Gplus <- Gplus + R Gplus with R = I - Gplus G, where
  // R is accumulated in double-double (Ogita-Rump-Oishi Dot2: FMA TwoProduct
  // and Knuth TwoSum).  The eigenvalue errors (about eps * lambda_0 each) leave
  // Gplus with a relative error near eps * kappa(G) = eps * kappa(A)^2; with an
  // accurately computed residual each step multiplies that error by itself, so
  // two steps bring it to the eps * kappa(A) level of an SVD of A.  Exact zero
  // rows and columns of G stay exact zeros.
  {
    // G was overwritten by the rotations; rebuild it from the rows of A.
    std::vector<double> G0(static_cast<size_t>(n) * n, 0.0);
    for (int32_t i = 0; i < m; ++i)
      for (int64_t p = rowptr[i]; p < rowptr[i + 1]; ++p)
        for (int64_t q = rowptr[i]; q < rowptr[i + 1]; ++q)
          G0[static_cast<size_t>(colidx[p]) * n + colidx[q]] += val[p] * val[q];
    std::vector<double> R(static_cast<size_t>(n) * n), U(static_cast<size_t>(n) * n);
    std::vector<double> Gcol(n);
    for (int step = 0; step < 2; ++step) {
      for (int32_t j = 0; j < n; ++j) {
        for (int32_t l = 0; l < n; ++l) Gcol[l] = G0[static_cast<size_t>(l) * n + j];
        for (int32_t i = 0; i < n; ++i) {
          const double* mrow = &Gp[static_cast<size_t>(i) * n];
          double s = (i == j) ? 1.0 : 0.0, c = 0.0;
          for (int32_t l = 0; l < n; ++l) {
            const double g = Gcol[l];
            if (g == 0.0) continue;
            const double p = -mrow[l] * g;
            const double pe = std::fma(-mrow[l], g, -p);
            const double t = s + p;
            const double bb = t - s;
            const double se = (s - (t - bb)) + (p - bb);
            s = t;
            c += pe + se;
          }
          R[static_cast<size_t>(i) * n + j] = s + c;
        }
      }
      std::fill(U.begin(), U.end(), 0.0);  // U = R * Gplus
      for (int32_t i = 0; i < n; ++i) {
        double* urow = &U[static_cast<size_t>(i) * n];
        for (int32_t l = 0; l < n; ++l) {
          const double x = R[static_cast<size_t>(i) * n + l];
          if (x == 0.0) continue;
          const double* prow = &Gp[static_cast<size_t>(l) * n];
          for (int32_t j = 0; j < n; ++j) urow[j] += x * prow[j];
        }
      }
      for (size_t i = 0; i < Gp.size(); ++i) Gp[i] += U[i];
    }
  }
  // Ad = Gplus A^T : column k of Ad = sum over non-zeros (k, j) of A of A[k,j] * Gplus[:, j].
  for (int32_t k = 0; k < m; ++k) {
    double* out = Ad + static_cast<size_t>(n) * k;
    std::fill(out, out + n, 0.0);
    for (int64_t p = rowptr[k]; p < rowptr[k + 1]; ++p) {
      const int32_t j = colidx[p];
      const double a = val[p];
      for (int32_t i = 0; i < n; ++i) out[i] += a * Gp[static_cast<size_t>(i) * n + j];
    }
  }
  return LEAP_OK;
}

}  // namespace leapgb

namespace leapgb {

std::vector<double> es_kernel_transform(int32_t taps, double beta, int32_t n, int32_t kmax) {
  // psi and all its derivatives are ~exp(-beta) at the ends of the support, so the
  // trapezoidal rule converges spectrally; 8192 panels give full FP64 accuracy.
  const int panels = 8192;
  const double half = 0.5 * taps, h = 2.0 * half / panels;
  std::vector<double> psi(panels + 1);
  for (int i = 0; i <= panels; ++i) {
    const double x = -half + i * h, z = x / half;
    const double q = std::max(0.0, 1.0 - z * z);
    psi[i] = std::exp(beta * (std::sqrt(q) - 1.0)) * ((i == 0 || i == panels) ? 0.5 : 1.0);
  }
  std::vector<double> out(kmax + 1);
  const double kTwoPiD = 6.283185307179586476925286766559;
  for (int k = 0; k <= kmax; ++k) {
    double s = 0.0;
    const double w = kTwoPiD * k / n;
    for (int i = 0; i <= panels; ++i) s += psi[i] * std::cos(w * (-half + i * h));
    out[k] = s * h;
  }
  return out;
}

void es_kernel_poly(int32_t taps, double beta, int32_t degree, float* out) {
  // h_m(f) = psi((f + taps/2 - 1 - m) * 2 / taps) for f in [0, 1): interpolate at the
  // degree + 1 Chebyshev points of x = 2 f - 1, then expand the Chebyshev series into
  // monomials of x (the Chebyshev coefficients c_n; T_{n+1} = 2 x T_n - T_{n-1}).
  const int np = degree + 1;
  const double kPiD = 3.141592653589793238462643383279;
  std::vector<double> tm(static_cast<size_t>(np) * np, 0.0);  // tm[n * np + j]: x^j coefficient of T_n
  tm[0] = 1.0;
  if (np > 1) tm[1 * np + 1] = 1.0;
  for (int n = 1; n + 1 < np; ++n)
    for (int j = 0; j < np; ++j)
      tm[(n + 1) * np + j] = (j > 0 ? 2.0 * tm[n * np + j - 1] : 0.0) - tm[(n - 1) * np + j];
  for (int m = 0; m < taps; ++m) {
    std::vector<double> val(np), mono(np, 0.0);
    for (int k = 0; k < np; ++k) {
      const double x = std::cos(kPiD * (k + 0.5) / np);
      const double z = ((x + 1.0) * 0.5 + 0.5 * taps - 1.0 - m) * 2.0 / taps;
      const double q = 1.0 - z * z;
      val[k] = q > 0.0 ? std::exp(beta * (std::sqrt(q) - 1.0)) : 0.0;
    }
    for (int n = 0; n < np; ++n) {
      double c = 0.0;
      for (int k = 0; k < np; ++k) c += val[k] * std::cos(kPiD * n * (k + 0.5) / np);
      c *= (n == 0 ? 1.0 : 2.0) / np;
      for (int j = 0; j < np; ++j) mono[j] += c * tm[n * np + j];
    }
    for (int j = 0; j < np; ++j) out[m * np + j] = static_cast<float>(mono[j]);
  }
}

namespace {
// IEEE binary16 bits of x rounded to nearest, ties to even (|x| < 65504), and its value.
uint16_t to_f16_bits(double x) {
  const uint16_t sign = x < 0 ? 0x8000u : 0u;
  const double a = std::fabs(x);
  if (a == 0.0) return sign;
  int e = 0;
  const double f = std::frexp(a, &e);  // a = f 2^e, f in [0.5, 1)
  const int E = e + 14;                // biased exponent of 2 f 2^(e - 1)
  if (E < 1) return static_cast<uint16_t>(sign | static_cast<uint16_t>(std::nearbyint(std::ldexp(a, 24))));
  const int mant = static_cast<int>(std::nearbyint((2.0 * f - 1.0) * 1024.0));
  return static_cast<uint16_t>(sign | ((E << 10) + mant));  // mant == 1024 carries into the exponent
}
double from_f16_bits(uint16_t h) {
  const int E = (h >> 10) & 31, mant = h & 1023;
  const double v = E == 0 ? std::ldexp(static_cast<double>(mant), -24) : std::ldexp(1.0 + mant / 1024.0, E - 15);
  return (h & 0x8000u) ? -v : v;
}
}  // namespace

float grid_table(int32_t C, int32_t taps, double beta, int32_t lbase, int32_t rows, std::vector<uint16_t>& out) {
  const int n = 2 * C, c0 = C / 2;
  const int nchunk = (C + 15) / 16, nrg = rows / 8;
  const std::vector<double> psi_hat = es_kernel_transform(taps, beta, n, std::max(c0, C - 1 - c0));
  // One power of two for the table: the largest |E| = max 1 / Psi(k) goes into [2^13, 2^14).
  double emax = 0.0;
  for (int c = 0; c < C; ++c) emax = std::max(emax, 1.0 / psi_hat[std::abs(c - c0)]);
  int e = 0;
  (void)std::frexp(emax, &e);
  const double scale = std::ldexp(1.0, 14 - e);
  const int nseg = (nchunk + 3) / 4;
  out.assign(static_cast<size_t>(nseg) * 2 * nrg * 4 * 2 * 128, 0);
  const double kTwoPiD = 6.283185307179586476925286766559;
  for (int c = 0; c < C; ++c) {
    const int k = c - c0;
    const double inv = scale / psi_hat[std::abs(k)];
    const int q = c / 16, kk = c % 16;
    for (int r = 0; r < rows; ++r) {
      const long long l = static_cast<long long>(r) - lbase;
      long long m = (static_cast<long long>(k) * l) % n;  // exact phase index
      if (m < 0) m += n;
      const double ang = kTwoPiD * static_cast<double>(m) / n;
      const double v[2] = {std::cos(ang) * inv, std::sin(ang) * inv};
      for (int ri = 0; ri < 2; ++ri) {
        const uint16_t hi = to_f16_bits(v[ri]);
        const uint16_t lo = to_f16_bits(v[ri] - from_f16_bits(hi));
        const int rr = 2 * r + ri;  // re and im rows of a grid point are neighbours
        for (int hl = 0; hl < 2; ++hl) {
          // K-major core matrices of 8 rows x 16 bytes, in 2-byte units.
          const size_t block = (static_cast<size_t>(q / 4) * 2 * nrg + (rr >> 3)) * 8 + (q % 4) * 2 + hl;
          out[block * 128 + (kk >> 3) * 64 + (rr & 7) * 8 + (kk & 7)] = hl == 0 ? hi : lo;
        }
      }
    }
  }
  return static_cast<float>(1.0 / scale);
}

namespace {

// (hi : lo) with the top bit of hi set and the exponent that keeps the value.
FxRatio normalised(unsigned __int128 x, int exp) {
  FxRatio r{0, 0, 0, 0};
  if (x == 0) return r;
  while (!(x >> 127)) {
    x <<= 1;
    --exp;
  }
  r.hi = static_cast<uint64_t>(x >> 64);
  r.lo = static_cast<uint64_t>(x);
  r.exp = exp;
  return r;
}

// x / c_light to 2^-127 relative, x > 0 (the speed of light is a whole number of metres per second).
FxRatio over_c(double x) {
  int e = 0;
  const double f = std::frexp(x, &e);  // x = f 2^e
  const uint64_t m = static_cast<uint64_t>(std::ldexp(f, 53)) << 11;  // x = m 2^(e - 64)
  const uint64_t c = 299792458u;
  // m 2^160 / c by 32-bit digits: 7 of them, the first of which is 0 or small
  uint32_t q[7];
  uint64_t rem = 0;
  for (int i = 0; i < 7; ++i) {
    const uint32_t digit = i == 0 ? static_cast<uint32_t>(m >> 32) : i == 1 ? static_cast<uint32_t>(m) : 0u;
    const uint64_t cur = (rem << 32) | digit;
    q[i] = static_cast<uint32_t>(cur / c);
    rem = cur % c;
  }
  // x / c = (q[0] .. q[4]) 2^(e - 64 - 96): digits 1..4 as `top`, digit 0 above, digits 5 and 6 below
  unsigned __int128 top = 0;
  for (int i = 1; i < 5; ++i) top = (top << 32) | q[i];
  uint64_t above = q[0], below = (static_cast<uint64_t>(q[5]) << 32) | q[6];
  int exp = e - 64 - 96 + 128;
  while (above) {  // shift right until digit 0 is inside the 128 bits
    below = (below >> 1) | (static_cast<uint64_t>(top & 1) << 63);
    top = (top >> 1) | (static_cast<unsigned __int128>(above & 1) << 127);
    above >>= 1;
    ++exp;
  }
  while (top && !(top >> 127)) {
    top = (top << 1) | (below >> 63);
    below <<= 1;
    --exp;
  }
  return normalised(top, exp);
}

// x / (2 pi): the constant is floor(2^128 / pi).
FxRatio over_two_pi(const FxRatio& x) {
  if (x.hi == 0) return x;
  const uint64_t ph = 0x517CC1B727220A94ull, pl = 0xFE13ABE8FA9A6EE0ull;
  const unsigned __int128 hh = static_cast<unsigned __int128>(x.hi) * ph;
  const unsigned __int128 mid = (static_cast<unsigned __int128>(x.hi) * pl >> 1) + (static_cast<unsigned __int128>(x.lo) * ph >> 1);
  return normalised(hh + (mid >> 63), x.exp - 1);
}

}  // namespace

bool fx_spectrum(double f0, double df, int32_t channels, const double* lambda, FxSpectrum& sp, int32_t* rho) {
  if (!std::isfinite(f0) || !std::isfinite(df) || !(f0 > 1.0) || f0 > 1e18 || std::fabs(df) > 1e18) return false;
  double kmax = 0.0;
  for (int32_t c = 0; c < channels; ++c) {
    // f0 + c df as an unevaluated sum nh + nl
    const double p = static_cast<double>(c) * df, pe = std::fma(static_cast<double>(c), df, -p);
    const double nh = f0 + p, bb = nh - f0, nl = ((f0 - (nh - bb)) + (p - bb)) + pe;
    if (!(nh > 1.0) || !std::isfinite(nh) || !std::isfinite(lambda[c])) return false;
    kmax = std::max(kmax, 1.0 / lambda[c]);
    // lambda (f0 + c df) = c_light + r; 1 / lambda = (f0 + c df) / c_light (1 - r / c_light)
    const double h = lambda[c] * nh, he = std::fma(lambda[c], nh, -h);
    const double r = (h - 299792458.0) + he + lambda[c] * nl;
    const double x = std::nearbyint(std::ldexp(-r / 299792458.0, 64 + kFxFrac));
    if (!(std::fabs(x) <= static_cast<double>(kFxMaxRho) * (1 << kFxFrac))) return false;
    rho[c] = static_cast<int32_t>(x);
  }
  sp = FxSpectrum{};
  sp.k0 = over_c(f0);
  if (df != 0.0) {
    sp.k1 = over_c(std::fabs(df));
    sp.kt = over_two_pi(sp.k1);
  }
  sp.kmax = kmax * (1.0 + 1e-12);
  sp.s1 = df < 0 ? -1 : 1;
  return true;
}

void spectrum_tables(double f0, double df, int32_t channels, Spectrum& t) {
  t.lambda.resize(2 * static_cast<size_t>(channels));
  for (int32_t c = 0; c < channels; ++c) {
    volatile double prod = static_cast<double>(c) * df;
    const double lam = 299792458.0 / (f0 + prod);
    t.lambda[c] = lam;
    t.lambda[channels + c] = 1.0 / lam;
  }
  t.rho.resize(channels);
  t.fx_ok = fx_spectrum(f0, df, channels, t.lambda.data(), t.sp, t.rho.data());
}

// cos and sin of the angle x 2^-64 rad, x < 2^64 * pi / 4, in 60-bit fixed point: their Taylor series in whole
// numbers, each term to 2^-64: the same on every host (long double is software on aarch64: 1.4 ms a context).
static void fx_cos_sin(uint64_t x, int64_t& c, int64_t& s) {
  unsigned __int128 term = static_cast<unsigned __int128>(1) << 64;  // x^n / n! in 2^-64
  __int128 sum[2] = {0, 0};
  for (int n = 0; term != 0; ++n) {
    sum[n & 1] += (n & 2) ? -static_cast<__int128>(term) : static_cast<__int128>(term);
    term = ((term * x) >> 64) / static_cast<unsigned>(n + 1);
  }
  c = static_cast<int64_t>((sum[0] + 8) >> 4);
  s = static_cast<int64_t>((sum[1] + 8) >> 4);
}

void fx_tables(std::vector<FxLimbs>& out) {
  out.resize(2 * kFxTable);
  // 2 pi 2^108: j / 2^10 turns are j (two_pi / 2^10) 2^-108 rad, j / 2^20 turns the same 10 bits further down.
  const unsigned __int128 two_pi = (static_cast<unsigned __int128>(0x6487ED5110B4ull) << 64) | 0x611A62633145C06Eull;
  for (int j = 0; j < kFxTable; ++j) {
    // Quarter turns and the reflection about pi / 4 are exact.
    const int quad = j / (kFxTable / 4), k = j % (kFxTable / 4);
    const bool mirror = k > kFxTable / 8;
    int64_t c, s;
    fx_cos_sin(static_cast<uint64_t>((two_pi >> 10) * static_cast<unsigned>(mirror ? kFxTable / 4 - k : k) >> 44), c, s);
    if (mirror) std::swap(c, s);
    out[j] = quad == 0 ? fx_limbs(c, s) : quad == 1 ? fx_limbs(-s, c) : quad == 2 ? fx_limbs(-c, -s) : fx_limbs(s, -c);
    fx_cos_sin(static_cast<uint64_t>((two_pi >> 10) * static_cast<unsigned>(j) >> 54), c, s);
    out[kFxTable + j] = fx_limbs(c, s);
  }
}

// A run's units are dealt at once: block b takes those n_b of the costs load_b, load_b + cost, ... that are among the
// `count` least of all blocks, the numbers that taking the least loaded block for each unit in turn gives (a heap of
// blocks took 3.0 ms of the host for 65664 units and 102 us for 2064, this 78 and 8 us).
void schedule_units(std::vector<UnitRun> runs, int32_t grid, std::vector<int32_t>& order) {
  std::stable_sort(runs.begin(), runs.end(), [](const UnitRun& a, const UnitRun& b) { return a.cost > b.cost; });
  std::vector<int64_t> load(grid, 0);
  std::vector<int32_t> length(grid, 0), n(grid);
  order.clear();
  for (const UnitRun& r : runs) {
    if (r.count <= 0) continue;
    const int64_t cost = std::max<int64_t>(1, r.cost);
    auto below = [&](int64_t x, int64_t l) { return x > l ? (x - l + cost - 1) / cost : 0; };
    auto taken = [&](int64_t x) {
      int64_t s = 0;
      for (int64_t l : load) s += below(x, l);
      return s;
    };
    // The largest x with at most `count` costs below it.
    int64_t lo = *std::min_element(load.begin(), load.end()), hi = lo + (static_cast<int64_t>(r.count) + 1) * cost;
    while (hi - lo > 1) {
      const int64_t mid = lo + (hi - lo) / 2;
      (taken(mid) <= r.count ? lo : hi) = mid;
    }
    int64_t rest = r.count, most = 0;
    for (int32_t b = 0; b < grid; ++b) rest -= n[b] = static_cast<int32_t>(below(lo, load[b]));
    for (int32_t b = 0; b < grid && rest > 0; ++b)
      if (load[b] + n[b] * cost == lo) {
        ++n[b];
        --rest;
      }
    int64_t rounds = 0;
    for (int32_t b = 0; b < grid; ++b) {
      most = std::max<int64_t>(most, n[b]);
      rounds = std::max<int64_t>(rounds, length[b] + n[b]);
    }
    if (static_cast<int64_t>(order.size()) < rounds * grid) order.resize(rounds * grid, -1);
    // Neighbouring units to different blocks at the same time.
    int32_t base = r.begin, in = 0;
    for (int64_t k = 0; k < most; ++k)
      for (int32_t b = 0; b < grid; ++b) {
        if (n[b] <= k) continue;
        order[static_cast<int64_t>(length[b] + k) * grid + b] = base + in;
        if (++in == r.per) {
          in = 0;
          base += r.stride;
        }
      }
    for (int32_t b = 0; b < grid; ++b) {
      load[b] += n[b] * cost;
      length[b] += n[b];
    }
  }
  order.resize(order.size() + grid, -1);
}

// Timesteps may be cut as finely as the call has them, whatever their number: a limit of 32 slabs left 10 antennas, 1000
// timesteps and one direction with 64 blocks of one warp.  More slabs than 32 of a longer call go on to two rounds of
// resident blocks only, since their partial sums are added up one after another.
void choose_fixed_slabs(int timesteps, int channels, int64_t base_blocks, int64_t resident, int& t_per, int& c_per, int& nts,
                        int& ncs) {
  double best_eff = 0.0;
  t_per = timesteps; c_per = channels; nts = ncs = 1;
  for (int unit : {128, 32, 16}) {
    const int max_c = (channels + unit - 1) / unit;
    for (int c = 1; c <= max_c; ++c) {
      const int cp = ((channels + c - 1) / c + unit - 1) / unit * unit;
      const int cn = (channels + cp - 1) / cp;
      if (cn != c) continue;
      // Slabs of fewer and fewer timesteps; channels are cut only beside slabs of one timestep.
      for (int t = c == 1 ? 1 : timesteps; t <= timesteps;) {
        const int tp = (timesteps + t - 1) / t;
        const int tn = (timesteps + tp - 1) / tp;
        // Time of the call in blocks' lengths: rounds of resident blocks times a block's samples.
        const int64_t blocks = base_blocks * cn * tn;
        if (timesteps > 32 && static_cast<int64_t>(cn) * tn > 32 && blocks > 2 * resident) break;
        const double rounds = static_cast<double>((blocks + resident - 1) / resident);
        const double eff = static_cast<double>(base_blocks) * timesteps * channels /
                           (static_cast<double>(resident) * rounds * tp * std::min(cp, channels));
        if (eff > best_eff + std::min(0.02, 0.25 * best_eff)) {  // (the share of a small call is small however it is cut)
          best_eff = eff;
          t_per = tp; nts = tn; c_per = cp; ncs = cn;
        }
        if (best_eff >= 0.95) return;
        t = tp > 1 ? (timesteps + tp - 2) / (tp - 1) : timesteps + 1;  // the next smaller tp
      }
    }
    if (best_eff >= 0.5) return;
  }
}

}  // namespace leapgb
