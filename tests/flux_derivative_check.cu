// Checks roe_flux2_jvp against the flux on dual numbers, on the host, and prints
// one line of figures. Built and run by tests/test_flux_derivatives.py.
#include <cmath>
#include <cstdio>

#include "vt_adjoint.cuh"

namespace vt {
// A value, the sum of its terms' sizes, and likewise for its derivative: what a
// rounding anywhere in the formulas can be relative to.
struct Size {
  double v, a, d;
  Size(double x = 0.0) : v(x), a(std::fabs(x)), d(0.0) {}  // NOLINT: constants promote
  Size(double v_, double a_, double d_) : v(v_), a(a_), d(d_) {}
};
inline Size operator+(const Size& x, const Size& y) { return {x.v + y.v, x.a + y.a, x.d + y.d}; }
inline Size operator-(const Size& x, const Size& y) { return {x.v - y.v, x.a + y.a, x.d + y.d}; }
inline Size operator*(const Size& x, const Size& y) { return {x.v * y.v, x.a * y.a, x.d * y.a + x.a * y.d}; }
inline Size operator/(const Size& x, const Size& y) {
  const double i = 1.0 / std::fabs(y.v), q = y.a * i;
  return {x.v / y.v, x.a * i * q, (x.d + x.a * i * q * y.d) * i * q};
}
inline Size operator-(const Size& x) { return {-x.v, x.a, x.d}; }
inline Size dsqrt(const Size& x) {
  const double r = std::sqrt(x.v), q = x.a / x.v;
  return {r, r * q, 0.5 * x.d / r * q};
}
inline Size dabs(const Size& x) { return {std::fabs(x.v), x.a, x.d}; }
inline double val(const Size& x) { return x.v; }
}  // namespace vt

inline double uniform(unsigned long long i) {
  unsigned long long h = (i + 1) * 0x9E3779B97F4A7C15ull;  // splitmix64
  h ^= h >> 30;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 27;
  h *= 0x94D049BB133111EBull;
  h ^= h >> 31;
  return static_cast<double>(h >> 11) * (1.0 / 9007199254740992.0);
}

int main() {
  const int n = 1 << 17;
  double worst = 0.0;
  int count[6] = {0, 0, 0, 0, 0, 0}, used = 0;
  for (int i = 0; i < n; ++i) {
    const unsigned long long k = 32ull * i;
    const double angle = 6.283185307179586 * uniform(k), nx = std::cos(angle), ny = std::sin(angle);
    const double rho = std::exp2(-3.0 + 6.0 * uniform(k + 1)), T = std::exp2(-2.0 + 6.0 * uniform(k + 2));
    const double v[2] = {-3.0 + 6.0 * uniform(k + 3), -3.0 + 6.0 * uniform(k + 4)};
    double u[8], d[8];
    for (int s = 0; s < 2; ++s) {
      double* w = u + 4 * s;
      const unsigned long long j = k + 5 + 12 * s;
      w[0] = rho * (1.0 + 0.25 * (uniform(j) - 0.5));
      w[1] = w[0] * (v[0] + 0.25 * (uniform(j + 1) - 0.5));
      w[2] = w[0] * (v[1] + 0.25 * (uniform(j + 2) - 0.5));
      w[3] = w[0] * T * (1.0 + 0.25 * (uniform(j + 3) - 0.5)) / 0.4 + 0.5 * (w[1] * w[1] + w[2] * w[2]) / w[0];
      for (int c = 0; c < 4; ++c) d[4 * s + c] = (2.0 * uniform(j + 4 + c) - 1.0) * std::fabs(w[c == 1 || c == 2 ? 0 : c]);
    }
    vt::Dual<1> a[8], f[4];
    vt::Size b[8], m[4];
    for (int c = 0; c < 8; ++c) {
      a[c] = vt::Dual<1>(u[c]);
      a[c].d[0] = d[c];
      b[c] = vt::Size(u[c], std::fabs(u[c]), std::fabs(d[c]));
    }
    if (vt::roe_flux_t(a, a + 4, nx, ny, f)) continue;  // no physical state
    vt::roe_flux_t(b, b + 4, nx, ny, m);
    double df[4];
    vt::roe_flux2_jvp(u, u + 4, nx, ny, d, d + 4, df);
    ++used;
    for (int c = 0; c < 4; ++c) worst = std::fmax(worst, std::fabs(df[c] - 2.0 * f[c].d[0]) / (2.0 * m[c].d));
    // the branch, from averages formed here
    const double g = std::sqrt(u[4] / u[0]), q = 1.0 / (1.0 + g);
    auto H = [&](const double* w) { return (w[3] + 0.4 * (w[3] - 0.5 * (w[1] * w[1] + w[2] * w[2]) / w[0])) / w[0]; };
    const double x = (u[1] / u[0] + g * u[5] / u[4]) * q, y = (u[2] / u[0] + g * u[6] / u[4]) * q;
    const double c2 = 0.4 * ((H(u) + g * H(u + 4)) * q - 0.5 * (x * x + y * y)), t = (x * nx + y * ny) / (c2 * c2);
    const double e = std::fabs(t);
    ++count[e < 0.1 ? 0 : (e < 0.875 ? 1 : (e < 0.9 ? 2 : (e < 1.1 ? (t < 0 ? 3 : 4) : 5)))];
  }
  printf("used %d fixed %d usual %d between %d l0_fixed %d l1_fixed %d general %d worst %.3e\n", used, count[0], count[1],
         count[2], count[3], count[4], count[5], worst);
  return 0;
}
