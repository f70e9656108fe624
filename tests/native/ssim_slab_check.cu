// Host-side check of the bounds that let a slab of pairs take the factorised form. SSIM's: for
// random slabs (centres and half ranges of the weight argument a over many decades), the form's
// value against the exact one in 64 bits, in the slab's corners and along its edges. Prints
// the slabs tried, the slabs accepted, those with a wide range and the largest relative error of an
// accepted one. Weighted NRMSE's: no row factor is subnormal (exit code 1 otherwise). Built and run by
// tests/test_ssim_slab.py.
#include "../../sred_b200/csrc/global_tc.cu"

#include <cmath>
#include <cstdio>
#include <random>

int main() {
  using namespace sred;
  std::mt19937_64 rng(1);
  auto uni = [&](double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); };
  auto decades = [&](double lo, double hi) { return std::pow(10.0, uni(lo, hi)); };
  long long tried = 0, accepted = 0, wide = 0;
  double worst = 0.0;
  for (int i = 0; i < 3000000; i++) {
    const double iw = decades(-4, 1);  // sigma / a
    double a = decades(-3, 3), b = i % 2 ? a * uni(0.5, 2.0) : decades(-3, 3);
    const double ra = a * decades(-5, 0), rb = b * decades(-5, 0), c2 = 9e-4;
    if (std::fabs(a - b) - ra - rb > kZeroDist || std::fabs(a - b) * rb > 24.0) continue;
    const double x0 = a * iw, y0 = b * iw, S0 = x0 * x0 + y0 * y0 + c2;
    const double h = 4 * x0 * y0 * iw * iw / (S0 * S0), e = (1.3862944 + h) * ra * rb;
    tried++;
    if (e > kFirstTol) continue;
    auto group = [&](double c, double r) {  // centre and half range of a and of 1 / sigma, as the kernel keeps them
      const double lo = 1 / ((c + r) * iw), hi = 1 / ((c - r) * iw);
      return make_float4((float)c, (float)r, (float)(0.5 * (lo + hi)), (float)(0.5 * (hi - lo)));
    };
    if (!ssim_split_bounded(group(a, ra), group(b, rb), (float)(h * ra * rb))) continue;
    accepted++;
    wide += ra > 0.03 * a || rb > 0.03 * b;
    for (int u = 0; u < 25; u++) {
      const double dp = ra * (u % 5 - 2) / 2, dq = rb * (u / 5 - 2) / 2;
      const double x = (a + dp) * iw, y = (b + dq) * iw;
      const double split = S0 / ((x * x + y0 * y0 + c2) * (x0 * x0 + y * y + c2)) *
                           (e > kPureTol ? 1 + (1.3862944 + h) * dp * dq : 1.0);
      worst = std::fmax(worst, std::fabs(split * (x * x + y * y + c2) / std::exp2(2 * dp * dq) - 1));
    }
  }
  // Row factors of accepted slabs: the smallest one, in the FP32 arithmetic of the kernel.
  float least = 1.0f;
  for (int i = 0; i < 1000000; i++) {
    const float D = (float)uni(-13, 13), ra = (float)(i % 2 ? uni(0, 4) : decades(-6, 0));
    if (!row_factors_normal(D, ra)) continue;
    for (float d : {D - ra, D + ra}) least = std::fmin(least, std::exp2(-d * d));
  }
  if (!(least >= 1.17549435e-38f)) return 1;
  std::printf("%lld %lld %lld %.3e\n", tried, accepted, wide, worst);
  return 0;
}
