// Weights of the squared Hadamard coefficients in the adjoint's quadratic form
// (host only).
#pragma once
#include <cmath>

namespace ltm {

// d(lambda_k)/dK / 2^L, lambda_k = (2 cosh K)^(L-k) (2 sinh K)^k, for k = 0..L.
// 2 cosh K and 2 sinh K are taken with their roundings, which L powers would
// multiply.
inline void power_weights(double K, int L, double* w) {
  const long double ea = std::exp((long double)K), cl = ea + 1.0L / ea, sl = ea - 1.0L / ea;
  const double c2 = (double)cl, s2 = (double)sl;
  const double dc = (double)((cl - (long double)c2) / cl), ds = s2 == 0.0 ? 0.0 : (double)((sl - (long double)s2) / sl);
  auto term = [&](int n, int a, int b) { return n * std::pow(c2, a) * std::pow(s2, b) * (1.0 + (a * dc + b * ds)); };
  for (int k = 0; k <= L; ++k) {  // (s^(L-k) d^k)' with s' = d, d' = s
    double r = 0.0;
    if (k < L) r += term(L - k, L - k - 1, k + 1);
    if (k > 0) r += term(k, L - k + 1, k - 1);
    w[k] = r * std::ldexp(1.0, -L);
  }
}

}  // namespace ltm
