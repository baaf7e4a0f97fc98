// One FP64 Gram-Schmidt step of a short Krylov vector in four launches.
//
// The general step (tm_blas.cu) is ten: two projections of a dot sweep, its
// final reduction and an update, then the norm with its reduction, the column
// of the projected matrix and the scaling.  For vectors of some thousand rows
// each of them takes a launch's 3-4 us and runs on a dozen SMs, whose FP64
// pipes (two lanes per clock) are then the limit.  Here a kernel takes one
// element per thread, so the multiply-adds spread over many blocks;
// the update of one projection is fused with the dots (or the norm) of the
// next; and the last block to finish reduces the block sums, in block order,
// so the result does not depend on which block that is.  At 16384 rows (L = 14
// full x-ANNNI) a solve with eigenvectors takes 1.25 ms, 1.83 kernel by kernel.
#include "tm_blas.cuh"
#include "tm_internal.h"

namespace ltm {

namespace {

constexpr int BT = 256;
constexpr int kMaxCols = 64;

// The warp sums of eight values per lane, lane group (lane >> 2) holding value
// 4 * bit 4 + 2 * bit 3 + bit 2: halves the values at each of three exchanges,
// nine additions where a sum per value would take forty.
__device__ __forceinline__ double warp_sum8(double (&a)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int half = 4, o = 16; half > 0; half >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const double give = up ? a[k] : a[k + half], keep = up ? a[k + half] : a[k];
      a[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  double v = a[0];
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

enum { kDots = 0, kUpdateDots = 1, kUpdateNorm = 2 };

// MODE kDots: hout = V^T w; kUpdateDots: w -= V hin, then hout = V^T w;
// kUpdateNorm: w -= V hin, then hout[0] = |w|^2 and column j of H from
// h1 + hin and |w| (sym: its mirror too).  ctr: zero between launches.
template <int MODE>
__global__ void __launch_bounds__(BT) cgs_kernel(const double* __restrict__ V, int64_t ldv, int nc, double* w,
                                                 int64_t n, const double* __restrict__ hin, double* hout,
                                                 double* part, unsigned* ctr, const double* __restrict__ h1, double* H,
                                                 int ldh, int sym) {
  __shared__ double hs[kMaxCols];
  __shared__ double ws[8][kMaxCols];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * BT + threadIdx.x;
  const bool on = i < n;
  const double* v = V + (on ? i : 0);
  double x = on ? w[i] : 0.0;
  const int nv = (MODE == kUpdateNorm) ? 1 : nc;  // values to sum
  if (MODE != kDots) {
    if ((int)threadIdx.x < nc) hs[threadIdx.x] = hin[threadIdx.x];
    __syncthreads();
    if (on) {
      for (int k = 0; k < nc; ++k) x = fma(-hs[k], v[k * ldv], x);
      w[i] = x;
    }
  }
  for (int k0 = 0; k0 < nv; k0 += 8) {
    double a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      a[k] = (k0 + k < nv) ? (MODE == kUpdateNorm ? x : v[(k0 + k) * ldv]) * x : 0.0;
    const double s = warp_sum8(a);
    const int k = k0 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    if ((lane & 3) == 0 && k < nv) ws[wid][k] = s;
  }
  __syncthreads();
  if ((int)threadIdx.x < nv) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += ws[q][threadIdx.x];
    part[(int64_t)blockIdx.x * nv + threadIdx.x] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ctr, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int k = wid; k < nv; k += 8) {
    double t = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) t += __ldcg(part + (int64_t)b * nv + k);
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) {
      hout[k] = t;
      if (MODE == kUpdateNorm) {
        const int j = nc - 1;
        const double b = sqrt(t);
        H[(j + 1) + (int64_t)j * ldh] = b;
        if (sym) H[j + (int64_t)(j + 1) * ldh] = b;
      }
    }
  }
  if (MODE == kUpdateNorm && (int)threadIdx.x < nc) {
    const int j = nc - 1, r = threadIdx.x;
    const double h = h1[r] + hs[r];
    H[r + (int64_t)j * ldh] = h;
    if (sym) H[j + (int64_t)r * ldh] = h;
  }
  if (threadIdx.x == 0) *ctr = 0u;
}

}  // namespace

void cgs_step(const double* V, int64_t ldv, int j, double* w, int64_t n, double* H, int ldh, bool sym,
              const CgsScratch& c, double* vnext, cudaStream_t s) {
  const int nc = j + 1;
  const unsigned nb = (unsigned)((n + BT - 1) / BT);
  if (nc > kMaxCols || n > kCgsRows) fail(TM_ERR_LIMIT, "short Gram-Schmidt step: too many rows or columns");
  cgs_kernel<kDots><<<nb, BT, 0, s>>>(V, ldv, nc, w, n, nullptr, c.h1, c.part, c.ctr, nullptr, nullptr, 0, 0);
  TM_CKK("cgs_dots");
  cgs_kernel<kUpdateDots><<<nb, BT, 0, s>>>(V, ldv, nc, w, n, c.h1, c.h2, c.part, c.ctr, nullptr, nullptr, 0, 0);
  TM_CKK("cgs_update_dots");
  cgs_kernel<kUpdateNorm><<<nb, BT, 0, s>>>(V, ldv, nc, w, n, c.h2, c.nsq, c.part, c.ctr, c.h1, H, ldh, sym ? 1 : 0);
  TM_CKK("cgs_update_norm");
  normalize(w, c.nsq, vnext, nullptr, n, s);
}

size_t cgs_scratch_bytes() { return ((size_t)(kCgsRows / BT) * kMaxCols + 2 * kMaxCols + 2) * 8; }
CgsScratch cgs_scratch(const DBuf& b, cudaStream_t s) {
  CgsScratch c;
  c.h1 = b.as<double>();
  c.h2 = c.h1 + kMaxCols;
  c.nsq = c.h2 + kMaxCols;
  c.ctr = reinterpret_cast<unsigned*>(c.nsq + 1);
  c.part = c.nsq + 2;
  TM_CK(cudaMemsetAsync(c.ctr, 0, 4, s));
  return c;
}

}  // namespace ltm
