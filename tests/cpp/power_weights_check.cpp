// Prints power_weights(K, L) for lines "K L" (K a hexadecimal float).
#include <cstdio>
#include <cstdlib>

#include "tm_power.h"

int main() {
  char k[64];
  int L;
  double w[33];
  while (std::scanf("%63s %d", k, &L) == 2) {
    ltm::power_weights(std::strtod(k, nullptr), L, w);
    for (int i = 0; i <= L; ++i) std::printf("%a ", w[i]);
    std::printf("\n");
  }
  return 0;
}
