// Butterflies of the inter-layer factor [[a, b], [b, a]], applied as
// x0' = x0 + r x1, x1' = x1 + r x0 with r = min(a, b) / max(a, b) (outputs
// exchanged where b > a): one FMA per element and level.  The factor
// max(a, b) per level is applied to the result.
#pragma once
#include "tm_df.cuh"

namespace ltm {

// shared-memory slot with one pad element every 32 (strided butterflies)
__device__ __forceinline__ int spad(int e) { return e + (e >> 5); }

// r * x + y in the engine's arithmetic
__device__ __forceinline__ float fma_t(float r, float x, float y) { return fmaf(r, x, y); }
__device__ __forceinline__ double fma_t(double r, double x, double y) { return fma(r, x, y); }
__device__ __forceinline__ dfloat fma_t(dfloat r, dfloat x, dfloat y) { return df_fma_unnorm(r, x, y); }

// In-register butterflies on all NB levels of the 2^NB elements held by one
// thread.  Output pair of level lv: (x0 + r x1, x1 + r x0), or exchanged
// (swap).
template <class T, int NB>
__device__ __forceinline__ void reg_bfly(T (&v)[1 << NB], T r, int swap) {
  if (!swap) {
#pragma unroll
    for (int lv = 0; lv < NB; ++lv)
#pragma unroll
      for (int i = 0; i < (1 << NB); ++i)
        if (!(i & (1 << lv))) {
          const T x0 = v[i], x1 = v[i | (1 << lv)];
          v[i] = fma_t(r, x1, x0);
          v[i | (1 << lv)] = fma_t(r, x0, x1);
        }
  } else {
#pragma unroll
    for (int lv = 0; lv < NB; ++lv)
#pragma unroll
      for (int i = 0; i < (1 << NB); ++i)
        if (!(i & (1 << lv))) {
          const T x0 = v[i], x1 = v[i | (1 << lv)];
          v[i] = fma_t(r, x0, x1);
          v[i | (1 << lv)] = fma_t(r, x1, x0);
        }
  }
}

}  // namespace ltm
