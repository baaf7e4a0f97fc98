// The chain tuning table's entries after a tuning that throws and one that ends.
#include "tm_tune.cu"

#include <cstdio>

namespace ltm {
void fail(tm_status code, const std::string& msg) { throw Failure{code, msg}; }
}  // namespace ltm

using namespace ltm;

static bool is(size_t elem, int tb, int th) {
  int a = 0, b = 0;
  chain_tuning(20, elem, true, a, b);
  if (a != tb || b != th) std::printf("elem %zu: %d, %d and not %d, %d\n", elem, a, b, tb, th);
  return a == tb && b == th;
}

int main() {
  int tb[2], th[2];
  for (int e = 0; e < 2; ++e) chain_tuning(20, e ? 8 : 4, true, tb[e], th[e]);
  bool ok = true;
  for (int e = 0; e < 2; ++e) {
    const size_t elem = e ? 8 : 4;
    // the defaults, then what a caller asked for (each block size, a default one among them)
    for (int want : {0, 64, 128, 256}) {
      for (int bits : {0, 11, tb[e]}) {
        chain_set_tuning(20, elem, true, bits, want);
        try {
          ChainTuneKeep tried(20, elem, true);
          chain_set_tuning(20, elem, true, 10, 64);
          fail(TM_ERR_CUDA, "a product failed");
        } catch (const Failure&) {
        }
        ok &= is(elem, bits ? bits : tb[e], want ? want : th[e]);
      }
    }
    {
      ChainTuneKeep tried(20, elem, true);
      chain_set_tuning(20, elem, true, 10, 64);
      tried.set(12, 128);
    }
    ok &= is(elem, 12, 128);
    chain_set_tuning(20, elem, true, 0, 0);
    ok &= is(elem, tb[e], th[e]);
  }
  if (ok) std::printf("ok\n");
  return ok ? 0 : 1;
}
