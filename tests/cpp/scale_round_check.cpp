// Reads lines "kind v_hi v_lo t S" (hexadecimal floats; kind 0: FP32 value,
// 1: double-float value) and prints scale_round(v, t, scale_factor(S)); kind 2:
// scale_round(v, t).
#include "scale_round_host.h"

#include <cstdio>
#include <cstdlib>

#include "tm_df.cuh"

int main() {
  char w[5][64];
  while (std::scanf("%63s %63s %63s %63s %63s", w[0], w[1], w[2], w[3], w[4]) == 5) {
    const float hi = std::strtof(w[1], nullptr), lo = std::strtof(w[2], nullptr);
    const double t = std::strtod(w[3], nullptr), S = std::strtod(w[4], nullptr);
    const ltm::ScaleF f = ltm::scale_factor(S);
    const int kind = std::atoi(w[0]);
    const float y = kind == 2   ? ltm::scale_round(hi, t)
                    : kind == 1 ? ltm::scale_round(ltm::dfloat(hi, lo), t, f)
                                : ltm::scale_round(hi, t, f);
    std::printf("%a\n", (double)y);
  }
  return 0;
}
