// Checks the device formulas of the face phase on pseudo-random inputs and
// prints one line of figures. Built and run by tests/test_gpu_flux.py.
//   rsqrt_nr    against 1 / sqrt(x) in long double on the host (ulps);
//   roe_flux2   against twice roe_flux_t (IEEE division and square root, on the
//               host), relative to the sizes of the terms that the flux sums
//               times the condition of c2,
//               over states on both sides of the eigenvalue test and of the
//               entropy fix; and its error codes on planted bad states.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "vt_adjoint.cuh"
#include "vt_device.cuh"

inline double uniform(unsigned long long i) {
  unsigned long long h = (i + 1) * 0x9E3779B97F4A7C15ull;  // splitmix64
  h ^= h >> 30;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 27;
  h *= 0x94D049BB133111EBull;
  h ^= h >> 31;
  return static_cast<double>(h >> 11) * (1.0 / 9007199254740992.0);
}

// rho in [1/8, 8], velocities in [-3, 3], p over rho in [1/4, 16]; the two
// sides differ by up to a quarter; every 16th case plants a bad value
inline void states(int i, double* uL, double* uR, double* n) {
  const unsigned long long k = 16ull * i;
  const double r = exp2(-3.0 + 6.0 * uniform(k)), a = 6.283185307179586 * uniform(k + 1);
  const double v[2] = {-3.0 + 6.0 * uniform(k + 2), -3.0 + 6.0 * uniform(k + 3)};
  const double T = exp2(-2.0 + 6.0 * uniform(k + 4));
  for (int side = 0; side < 2; ++side) {
    double* u = side ? uR : uL;
    const double d = side ? 0.25 : 0.0;
    u[0] = r * (1.0 + d * (uniform(k + 5) - 0.5));
    u[1] = u[0] * (v[0] + d * (uniform(k + 6) - 0.5));
    u[2] = u[0] * (v[1] + d * (uniform(k + 7) - 0.5));
    u[3] = u[0] * T * (1.0 + d * (uniform(k + 8) - 0.5)) / 0.4 + 0.5 * (u[1] * u[1] + u[2] * u[2]) / u[0];
  }
  n[0] = cos(a), n[1] = sin(a);
  if (i % 16 == 15) {
    double* u = (i / 16) % 2 ? uR : uL;
    const int what = (i / 32) % 4;
    if (what == 0) u[0] = -u[0];
    if (what == 1) u[3] = 0.0;
    if (what == 2) u[0] = 0.0;
    if (what == 3) uL[3] = uR[3] = -1.0;
  }
}

// in: per case x for rsqrt_nr, uL (4), uR (4), the normal (2); the inputs come
// from the host, so that both sides see the same bits
constexpr int kIn = 11;
__global__ void run(int n, const double* in, double* root, double* flux, int* code) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* x = in + kIn * i;
  root[i] = vt::rsqrt_nr(x[0]);
  code[i] = 0;
  vt::roe_flux2(x + 1, x + 5, x[9], x[10], flux + 4 * i, [&](int c) { code[i] = c; });
}

int main() {
  const int n = 1 << 18;
  std::vector<double> in(kIn * n);
  for (int i = 0; i < n; ++i) {
    double* x = &in[kIn * i];
    x[0] = std::exp2(-20.0 + 40.0 * uniform(i + (1ull << 40)));
    states(i, x + 1, x + 5, x + 9);
  }
  double *din, *root, *flux;
  int* code;
  if (cudaMalloc(&din, in.size() * sizeof(double)) || cudaMalloc(&root, n * sizeof(double)) ||
      cudaMalloc(&flux, 4 * n * sizeof(double)) || cudaMalloc(&code, n * 4) ||
      cudaMemcpy(din, in.data(), in.size() * sizeof(double), cudaMemcpyHostToDevice))
    return 2;
  run<<<n / 256, 256>>>(n, din, root, flux, code);
  std::vector<double> hr(n), hf(4 * n);
  std::vector<int> hc(n);
  if (cudaMemcpy(hr.data(), root, n * sizeof(double), cudaMemcpyDeviceToHost) ||
      cudaMemcpy(hf.data(), flux, 4 * n * sizeof(double), cudaMemcpyDeviceToHost) ||
      cudaMemcpy(hc.data(), code, n * 4, cudaMemcpyDeviceToHost))
    return 2;
  double ulp = 0.0, rel = 0.0;
  int wrong = 0, bad = 0, general = 0, fixed = 0;
  for (int i = 0; i < n; ++i) {
    const long double want = 1.0L / std::sqrt(static_cast<long double>(in[kIn * i]));
    const double w = static_cast<double>(want);
    ulp = std::fmax(ulp, std::fabs(static_cast<double>(hr[i] - want)) / (std::nextafter(w, 2 * w) - w));
    const double *uL = &in[kIn * i + 1], *uR = uL + 4, *nn = uL + 8;
    double f[4];
    const int c = vt::roe_flux_t(uL, uR, nn[0], nn[1], f);
    if (c != hc[i]) ++wrong;
    if (c) {
      ++bad;
      continue;
    }
    // the sizes of the flux's terms: lam |u| of either side (lam the fastest
    // eigenvalue) and the acoustic dissipation |C1| (1, u, H), whose divisions
    // by ci enlarge them; c2 itself is a difference, with condition q
    double big = 0.0, u_n = 0.0, ci = 0.0, q = 1.0, H = 0.0, vel = 0.0, cmin = 1e300;
    for (const double* u : {uL, uR}) {
      const double un = (u[1] * nn[0] + u[2] * nn[1]) / u[0], v2 = (u[1] * u[1] + u[2] * u[2]) / (u[0] * u[0]);
      const double p = 0.4 * (u[3] - 0.5 * u[0] * v2), h = (u[3] + p) / u[0], c2 = 1.4 * p / u[0];
      u_n = std::fmax(u_n, std::fabs(un)), ci = std::fmax(ci, c2 * c2), cmin = std::fmin(cmin, c2 * c2);
      H = std::fmax(H, h), vel = std::fmax(vel, std::sqrt(v2));
      q = std::fmax(q, 0.4 * (h + 0.5 * v2) / c2);
      big = std::fmax(big, std::fabs(u[0]) + std::fabs(u[1]) + std::fabs(u[2]) + std::fabs(u[3]));
    }
    double du[4];
    for (int k = 0; k < 4; ++k) du[k] = std::fabs(uR[k] - uL[k]);
    const double lam = u_n + ci, G1 = 0.4 * (0.5 * vel * vel * du[0] + vel * (du[1] + du[2]) + du[3]);
    const double G2 = vel * du[0] + du[1] + du[2];
    const double C1 = (G1 / cmin + G2) * lam / cmin, C2 = (G1 / cmin + G2) * lam;
    const double size = q * (lam * big + C1 * (1.0 + vel + H) + C2 * (1.0 + vel));
    if (u_n > 0.9 * ci) ++general;
    if (u_n < 0.05 * ci) ++fixed;
    for (int k = 0; k < 4; ++k) rel = std::fmax(rel, std::fabs(hf[4 * i + k] - 2.0 * f[k]) / size);
  }
  printf("states %d bad %d wrong_codes %d general %d entropy_fixed %d rsqrt_ulp %.3f flux_rel %.3e\n", n, bad, wrong, general,
         fixed, ulp, rel);
  cudaFree(din), cudaFree(root), cudaFree(flux), cudaFree(code);
  return 0;
}
