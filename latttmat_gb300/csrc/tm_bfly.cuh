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

// Coefficients of a Kronecker factor.
template <class T>
struct Kron {
  T r;       // min(a, b) / max(a, b)
  int swap;  // b > a
};

// The Walsh-Hadamard transform (x0 + x1, x0 - x1), for the adjoint.
struct Had {};

template <class T, int NB>
__device__ __forceinline__ void bfly(T (&v)[1 << NB], const Kron<T>& c) {
  reg_bfly<T, NB>(v, c.r, c.swap);
}
template <class T, int NB>
__device__ __forceinline__ void bfly(T (&v)[1 << NB], const Had&) {
#pragma unroll
  for (int lv = 0; lv < NB; ++lv)
#pragma unroll
    for (int i = 0; i < (1 << NB); ++i)
      if (!(i & (1 << lv))) {
        const T x0 = v[i], x1 = v[i | (1 << lv)];
        v[i] = x0 + x1;
        v[i | (1 << lv)] = x0 - x1;
      }
}
// the two outputs of one butterfly (no exchange)
template <class T>
__device__ __forceinline__ T out0(const Kron<T>& c, T x0, T x1) { return fma_t(c.r, x1, x0); }
template <class T>
__device__ __forceinline__ T out1(const Kron<T>& c, T x0, T x1) { return fma_t(c.r, x0, x1); }
template <class T>
__device__ __forceinline__ T out0(const Had&, T x0, T x1) { return x0 + x1; }
template <class T>
__device__ __forceinline__ T out1(const Had&, T x0, T x1) { return x0 - x1; }
template <class T>
__device__ __forceinline__ bool swapped(const Kron<T>& c) { return c.swap; }
__device__ __forceinline__ bool swapped(const Had&) { return false; }

// ------------------------------------------------------------------ tiles
// One butterfly round on tile bits [G0, G0 + GS) of every row (a row is the
// 2^nb mixed positions of one chunk position).
template <class T, int G0, int GS, class C>
__device__ __forceinline__ void tile_round(T* sm, int nb, int cb, int pitch, const C& c) {
  const int fb = nb - GS;
  for (int f = threadIdx.x; f < (1 << (fb + cb)); f += blockDim.x) {
    const int g = f & ((1 << fb) - 1);
    T* b = sm + (f >> fb) * pitch + spad((g & ((1 << G0) - 1)) | ((g >> G0) << (G0 + GS)));
    T v[1 << GS];
#pragma unroll
    for (int i = 0; i < (1 << GS); ++i) v[i] = b[spad(i << G0)];
    bfly<T, GS>(v, c);
#pragma unroll
    for (int i = 0; i < (1 << GS); ++i) b[spad(i << G0)] = v[i];
  }
  __syncthreads();
}

constexpr int kTileMix = 14;  // most mixed bits of a tile

template <class T, int KB, class C, int R = 0>
__device__ __forceinline__ void tile_rounds(T* sm, int nb, int cb, int pitch, const C& c) {
  constexpr int G0 = R * KB;
  const int left = nb - G0;
  if (left <= 0) return;
  if (left >= KB) {
    tile_round<T, G0, KB>(sm, nb, cb, pitch, c);
  } else {
    if constexpr (KB > 3)
      if (left == 3) tile_round<T, G0, 3>(sm, nb, cb, pitch, c);
    if constexpr (KB > 2)
      if (left == 2) tile_round<T, G0, 2>(sm, nb, cb, pitch, c);
    if constexpr (KB > 1)
      if (left == 1) tile_round<T, G0, 1>(sm, nb, cb, pitch, c);
    return;
  }
  if constexpr ((R + 1) * KB < kTileMix) tile_rounds<T, KB, C, R + 1>(sm, nb, cb, pitch, c);
}

}  // namespace ltm
