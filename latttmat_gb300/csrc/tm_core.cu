// Full-space transfer-matrix cores and the generic reduced-basis path.
//
// Kronecker factor (x-ANNNI perpendicular TM, 3D ANNNI): the inter-layer
// factor Th = (x)_{i<L} t with t = [[e^K, e^-K], [e^-K, e^K]]
// (TMat/tmat.cpp:79-93, the L in-place butterflies of XATMatVecProd2D and of
// permute_mult_TL), applied as x0 + r x1 (tm_bfly.cuh).  FP64 products are
// bound by the FP64 pipe (two lanes per clock and SM on sm_103a: every FMA
// and conversion counts, memory does not), FP32 products by memory.
//
// Full operators: shared-memory tile passes of up to 11 bits
// (kron_tile_kernel), Tv^(1/2) fused into the first load and nf Tv^(1/2) into
// the last store.
//
// Reduced operators evaluate y = D^(1/2) Tv^(1/2) Th Tv^(1/2) P D^(-1/2) x
// (TMat/tmatreduce.cpp:406-529) at the representatives.  With a translation
// group the output bits are built from the top down and only prefixes that
// lead to a representative are kept (tm_tree.cu, kron_tree_kernel): about a
// third of the multiply-adds at L = 25.  Groups without translations (open
// boundary) expand to the full space, run the full passes and gather.
#include <algorithm>
#include <cmath>
#include <vector>

#include "tm_bfly.cuh"
#include "tm_internal.h"
#include "tm_power.h"

namespace ltm {

namespace {

template <class T>
Kron<T> kron_of(const Op& op) {
  return Kron<T>{(T)op.kron.r, op.mp.betaJ < 0 ? 1 : 0};
}

// Weights of the squared Hadamard coefficients by bit count (adjoint), and
// the sum of one block's terms.
struct PowerTab {
  double d[33];
};
__device__ __forceinline__ void block_sum(double acc, double* __restrict__ part) {
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  __shared__ double sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sh[q];
    part[blockIdx.x] = t;
  }
}

// ------------------------------------------------------------------ tile passes
// x * pre * fac (load) and v * sc * fac (store) in the vector's type
// (FP64 loads take no factor: it costs a slot on the FP64 pipe per element, and
// the output factor can hold it)
__device__ __forceinline__ double weigh(double v, double t, const ScaleF& f) { return v * t * f.f64; }
__device__ __forceinline__ double weigh_load(double v, double t, const ScaleF&) { return v * t; }
__device__ __forceinline__ float weigh_load(float v, double t, const ScaleF& f) { return scale_round(v, t, f); }
__device__ __forceinline__ float weigh(float v, double t, const ScaleF& f) { return scale_round(v, t, f); }

// One pass: 2^nb positions of bits [lo, lo + nb) times 2^cb contiguous
// positions of bits [0, cb) (only when lo > 0), for one value of the other
// bits per block.
//   load_mode 0: v = x[i]; 1: v = x[i]*pre[i] (FP32: *fin); 2: v = x[map[i]];
//             3: as 1 from the layer-swapped position of a two-layer state
//   store_mode 0: out[i] = v; 1: out[i] = v*scale[i]*fout;
//              2: v [* scale] to the layer-swapped position
// (swapped positions are contiguous along the mixed bits, which then start at
// bit half, the layer width, so those modes walk the tile along them)
template <class T, int KB>
__global__ void __launch_bounds__(512) kron_tile_kernel(const T* __restrict__ x, T* __restrict__ out, int lo, int nb,
                                                        int cb, Kron<T> c, int load_mode,
                                                        const double* __restrict__ pre, ScaleF fin,
                                                        const uint32_t* __restrict__ map, int store_mode,
                                                        const double* __restrict__ scale, ScaleF fout, int half) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  const int tile = 1 << (nb + cb);
  const int pitch = spad(1 << nb) | 1;  // odd: chunk neighbours fall into different banks
  // block index -> the bits not in [0, cb) U [lo, lo + nb)
  const uint64_t outer = blockIdx.x;
  const int low_outer = lo - cb;
  const uint64_t base = ((outer & ((1ull << low_outer) - 1)) << cb) | ((outer >> low_outer) << (lo + nb));
  const int kmask = (1 << cb) - 1, jmask = (1 << nb) - 1;
  const uint64_t hmask = (1ull << half) - 1;
  if (load_mode == 3) {
    for (int e = threadIdx.x; e < tile; e += blockDim.x) {
      const uint64_t i = base | (uint64_t)(e >> nb) | ((uint64_t)(e & jmask) << lo);
      const uint64_t o = (i >> half) | ((i & hmask) << half);
      sm[(e >> nb) * pitch + spad(e & jmask)] = weigh_load(x[o], pre[o], fin);
    }
  } else {
    for (int e = threadIdx.x; e < tile; e += blockDim.x) {
      const uint64_t i = base | (uint64_t)(e & kmask) | ((uint64_t)(e >> cb) << lo);
      T v;
      if (load_mode == 0)
        v = x[i];
      else if (load_mode == 1)
        v = weigh_load(x[i], pre[i], fin);
      else
        v = x[map[i]];
      sm[(e & kmask) * pitch + spad(e >> cb)] = v;
    }
  }
  __syncthreads();
  tile_rounds<T, KB, Kron<T>>(sm, nb, cb, pitch, c);
  if (store_mode == 2) {
    for (int e = threadIdx.x; e < tile; e += blockDim.x) {
      const uint64_t i = base | (uint64_t)(e >> nb) | ((uint64_t)(e & jmask) << lo);
      const uint64_t o = (i >> half) | ((i & hmask) << half);
      const T v = sm[(e >> nb) * pitch + spad(e & jmask)];
      out[o] = scale ? weigh_load(v, scale[o], fout) : v;
    }
    return;
  }
  for (int e = threadIdx.x; e < tile; e += blockDim.x) {
    const uint64_t i = base | (uint64_t)(e & kmask) | ((uint64_t)(e >> cb) << lo);
    T v = sm[(e & kmask) * pitch + spad(e >> cb)];
    if (store_mode == 1) v = weigh(v, scale[i], fout);
    out[i] = v;
  }
}

template <class T, int KB>
void launch_tile(int64_t nblocks, int threads, size_t shm, cudaStream_t s, const T* x, T* out, int lo, int nb, int cb,
                 const Kron<T>& c, int load_mode, const double* pre, const ScaleF& fin, const uint32_t* map,
                 int store_mode, const double* scale, const ScaleF& fout, int half = 1) {
  if (shm > 48 * 1024) raise_smem_limit((const void*)kron_tile_kernel<T, KB>, shm);
  kron_tile_kernel<T, KB><<<(unsigned)nblocks, threads, shm, s>>>(x, out, lo, nb, cb, c, load_mode, pre, fin, map,
                                                                  store_mode, scale, fout, half);
  TM_CKK("kron_tile");
}

// The passes of a full-space product.  Up to 10 bits (FP32: 11) go in one pass
// (one block; a second launch costs more than its levels, in time alone and in
// host time where several operators' products overlap), else the bits are spread
// over ceil(L / 9) passes of at most 9 (FP64), or passes of at most 10 and a
// first one, which has no chunk, of 11 (FP32: L = 21 in three passes 45.3 us, in
// two 39.1; the same in FP64 at L = 19 is slower, 42.6 for 39.0).  A block takes
// up to 16 contiguous positions beside the mixed ones, fewer where that would
// leave SMs without a block: at small L the FP64 pipe of one SM is the limit
// (L = 12 in one 4096-element block took 38 us).  Threads: 16 elements each
// (one round of four levels in registers) in large tiles, 2 or 4 in small
// ones, so that all four schedulers of an SM have a warp.
struct TilePass {
  int nb, cb, kb, threads;
  size_t shm;
  int64_t nblocks;
};
int tile_passes(int L, size_t elem) {
  if (elem == 8) return L <= 10 ? 1 : (L + 8) / 9;
  return std::max(1, (L + 8) / 10);
}
// the pass that starts at bit lo, with `left` passes to go
TilePass tile_pass(int L, int lo, int left, size_t elem) {
  TilePass t;
  t.nb = (L - lo + left - 1) / left;
  t.cb = std::min(std::min(4, lo), std::max(0, L - t.nb - 7));
  const int tb = t.nb + t.cb;
  t.kb = (tb >= 11 && t.nb < L) ? 4 : (tb >= 9 ? 2 : 1);  // (a block alone: more threads)
  t.threads = std::min(512, std::max(32, (1 << tb) >> t.kb));
  t.shm = ((size_t)(((1 << t.nb) + (1 << t.nb) / 32) | 1) << t.cb) * elem;
  t.nblocks = (int64_t)1 << (L - tb);
  return t;
}
template <class T>
void run_sweep(const Op& op, const T* x, T* out, int load_mode, const double* pre, double fin, const uint32_t* map,
               int store_mode, const double* scale, double fout, cudaStream_t s) {
  const int L = op.L;
  const Kron<T> c = kron_of<T>(op);
  const int npass = tile_passes(L, sizeof(T));
  // (FP64 takes the plain factors)
  const bool f64 = sizeof(T) == 8;
  const ScaleF fi = f64 ? ScaleF{fin, 1.f, dfloat(0)} : scale_factor(fin);
  const ScaleF fo = f64 ? ScaleF{fout, 1.f, dfloat(0)} : scale_factor(fout);
  int lo = 0;
  const T* src = x;
  for (int p = 0; p < npass; ++p) {
    const TilePass t = tile_pass(L, lo, npass - p, sizeof(T));
    const int nb = t.nb, cb = t.cb, kb = t.kb, threads = t.threads;
    const size_t shm = t.shm;
    const int64_t nblocks = t.nblocks;
    const bool first = (p == 0), last = (p == npass - 1);
    auto go = [&](auto k) {
      launch_tile<T, decltype(k)::value>(nblocks, threads, shm, s, src, out, lo, nb, cb, c, first ? load_mode : 0, pre,
                                         fi, map, last ? store_mode : 0, scale, fo);
    };
    if (kb == 4)
      go(std::integral_constant<int, 4>());
    else if (kb == 2)
      go(std::integral_constant<int, 2>());
    else
      go(std::integral_constant<int, 1>());
    src = out;
    lo += nb;
  }
}

// A pass of the Hadamard transform, as kron_tile_kernel: input x, through map
// or times pre where given; the last pass stores nothing but the block's sum
// of d[bit count] value^2.  Bound by the FP64 pipe (one addition per element
// and level).
template <int KB>
__global__ void __launch_bounds__(512) had_tile_kernel(const double* x, double* out, int lo, int nb, int cb,
                                                       const uint32_t* __restrict__ map,
                                                       const double* __restrict__ pre, double* __restrict__ part,
                                                       PowerTab pw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  const int tile = 1 << (nb + cb), kmask = (1 << cb) - 1;
  const int pitch = spad(1 << nb) | 1;
  const uint64_t outer = blockIdx.x;
  const int low_outer = lo - cb;
  const uint64_t base = ((outer & ((1ull << low_outer) - 1)) << cb) | ((outer >> low_outer) << (lo + nb));
  for (int e = threadIdx.x; e < tile; e += blockDim.x) {
    const uint64_t i = base | (uint64_t)(e & kmask) | ((uint64_t)(e >> cb) << lo);
    double v = map ? x[map[i]] : x[i];
    if (pre) v *= pre[i];
    sm[(e & kmask) * pitch + spad(e >> cb)] = v;
  }
  __syncthreads();
  tile_rounds<double, KB, Had>(sm, nb, cb, pitch, Had());
  double acc = 0.0;
  for (int e = threadIdx.x; e < tile; e += blockDim.x) {
    const uint64_t i = base | (uint64_t)(e & kmask) | ((uint64_t)(e >> cb) << lo);
    const double v = sm[(e & kmask) * pitch + spad(e >> cb)];
    if (part)
      acc = fma(pw.d[__popcll(i)], v * v, acc);
    else
      out[i] = v;
  }
  if (part) block_sum(acc, part);
}

}  // namespace

// The full two-layer y-ANNNI products (YATMatVecProd2D and _T): the Kronecker
// factor [[w0, w1], [w1, w0]], w0 = e^{-K kappa}, w1 = 1 / w0, on one layer's
// bits and the layer swap with its weights.  y = nf Tvec .* swap(K_high x) is
// top bits first and the swap in the last store; T^T x = nf swap(K_low (Tvec
// .* x)) = nf K_high swap(Tvec .* x) takes the swap in its first load.  Bound
// by the FP64 pipe (one FMA per bit and a multiply): at L = 12 two passes take
// 0.45 ms where separate mixing and swap kernels with two operations per bit
// took 0.94 ms.
void kron_swap_product(const Op& op, const double* x, double* y, double* ws, bool transposed, cudaStream_t s) {
  const int L = op.L;
  const double kk = op.mp.betaJ * op.mp.kappa;
  const Kron<double> c{std::exp(-2.0 * std::fabs(kk)), kk > 0 ? 1 : 0};
  const double* tv = op.tvec.as<double>();
  const ScaleF one = scale_factor(1.0);  // (Tvec holds the output factor)
  const int npass = std::max(2, (L + 7) / 8);
  int cut[8] = {0};  // pass boundaries within the layer's bits
  for (int p = 0; p < npass; ++p) cut[p + 1] = cut[p] + (L - cut[p] + npass - p - 1) / (npass - p);
  for (int q = 0; q < npass; ++q) {
    const int p = transposed ? q : npass - 1 - q;
    const bool first = (q == 0), last = (q == npass - 1);
    const int lo = L + cut[p], nb = cut[p + 1] - cut[p];
    const int cb = std::min(std::min(4, L), std::max(0, 2 * L - nb - 7)), tb = nb + cb;
    const int kb = (tb >= 11) ? 4 : (tb >= 9 ? 2 : 1);
    const int threads = std::min(512, std::max(32, (1 << tb) >> kb));
    const size_t shm = ((size_t)(((1 << nb) + (1 << nb) / 32) | 1) << cb) * 8;
    const double* src = first ? x : ws;
    double* dst = last ? y : ws;
    auto go = [&](auto k) {
      launch_tile<double, decltype(k)::value>((int64_t)1 << (2 * L - tb), threads, shm, s, src, dst, lo, nb, cb, c,
                                              first && transposed ? 3 : 0, tv, one, nullptr,
                                              last && !transposed ? 2 : 0, tv, one, L);
    };
    if (kb == 4)
      go(std::integral_constant<int, 4>());
    else if (kb == 2)
      go(std::integral_constant<int, 2>());
    else
      go(std::integral_constant<int, 1>());
  }
}

// ((1 + rl) / (1 + r))^n: the factor that the rounding of r adds to a constant
// vector, all n levels sharing it (the powers of their tiny difference end with
// the third; long double power functions took 3 of a small operator's 35 us)
static long double rounding_factor(long double rl, double r, int n) {
  const long double d = (rl - (long double)r) / (1.0L + (long double)r);
  return 1.0L + n * d * (1.0L + (n - 1) * d / 2.0L * (1.0L + (n - 2) * d / 3.0L));
}

// e^{|K'| L} of a Kronecker factor with coupling K' on L bits, with the factor
// that the rounding of its r adds to a constant vector taken out
double kron_out_factor(double coupling, int L, double r) {
  const long double a = std::fabs((long double)coupling);
  return (double)(std::exp(a * (long double)L) * rounding_factor(std::exp(-2.0L * a), r, L));
}

namespace {

// ------------------------------------------------------------------ prefix-tree passes
// The butterflies (x0 + r x1, x1 + r x0) on a thread's 2^KB values, top bit
// first, forming output blocks below which the mask has a child.  The mask is
// the same for the whole warp and each block of outputs is one branch: a
// predicated or selected FMA would take its slot on the FP64 pipe all the
// same.  The last two levels of a block of four outputs go together.
template <class T, int KB, class C, int B = KB - 1, int H = 0>
__device__ __forceinline__ void tree_bfly(T (&v)[1 << KB], uint32_t mask, const C& c) {
  constexpr uint32_t kSub = (1u << (1 << B)) - 1u;  // the 2^B leaves of one output block
  constexpr int J0 = (2 * H) << B, J1 = (2 * H + 1) << B;
  const bool a0 = (mask >> J0) & kSub, a1 = (mask >> J1) & kSub;
  if (B <= 1 ? (a0 || a1) : (a0 && a1)) {
#pragma unroll
    for (int i = 0; i < (1 << B); ++i) {
      const T x0 = v[J0 + i], x1 = v[J1 + i];
      v[J0 + i] = out0<T>(c, x0, x1);
      v[J1 + i] = out1<T>(c, x0, x1);
    }
    if constexpr (B > 0) {
      tree_bfly<T, KB, C, B - 1, 2 * H>(v, B == 1 ? 3u << J0 : mask, c);
      tree_bfly<T, KB, C, B - 1, 2 * H + 1>(v, B == 1 ? 3u << J1 : mask, c);
    }
  } else if constexpr (B > 1) {
    if (a0) {
#pragma unroll
      for (int i = 0; i < (1 << B); ++i) v[J0 + i] = out0<T>(c, v[J0 + i], v[J1 + i]);
      tree_bfly<T, KB, C, B - 1, 2 * H>(v, mask, c);
    } else if (a1) {
#pragma unroll
      for (int i = 0; i < (1 << B); ++i) v[J1 + i] = out1<T>(c, v[J0 + i], v[J1 + i]);
      tree_bfly<T, KB, C, B - 1, 2 * H + 1>(v, mask, c);
    }
  }
}

// One level of a reduced product: the KB next output bits.  Element (node,
// low): value of the vector whose top bits are the node's prefix (new bits)
// and whose low bits (`rest` of them, plus the KB mixed here) are still old.
// A thread holds the 2^KB values of one (node, low), mixes them and stores
// the node's children at (child, low).
//   FIRST: one node, values gathered from u through the state -> rank map,
//          at the complement of every state for K < 0 (t with a and b
//          exchanged is t after a spin flip, and the flip commutes with t);
//          with the input scaling (u = x tvec gin) folded in where tv is given
//          (few enough rows that gathering the weights too costs less than a
//          launch);
//   LAST:  the children are the representatives: y = post dup tvec value; of
//          the Hadamard transform (C = Had) the sum over the block's
//          representatives of dup d[bit count] value^2.
// Bound by the FP64 pipe in FP64 (busy 81, 78, 72 and 67% in the first four
// levels at L = 25, 58 to 66% in the short last ones), by the map gather in FP32.  FP64 products against three full-space tile passes
// with two FP64 operations per element and bit: x-ANNNI at L = 25 without
// flip 3.17 -> 0.465 ms, the 5x5 layer with flip 3.16 -> 0.142 ms.
template <class T, int KB, bool FIRST, bool LAST, class C>
__global__ void __launch_bounds__(256) kron_tree_kernel(const T* __restrict__ src, const uint32_t* __restrict__ smap,
                                                        const uint2* __restrict__ nodes, int64_t nnode, int rest,
                                                        C c, T* __restrict__ dst,
                                                        const uint16_t* __restrict__ dup,
                                                        const double* __restrict__ tv, ScaleF post,
                                                        const uint32_t* __restrict__ idx, PowerTab pw) {
  constexpr bool kPower = LAST && std::is_same<C, Had>::value;
  double acc = 0.0;
  const int64_t total = nnode << rest;
  const int64_t span = (total + 31) & ~(int64_t)31;  // whole warps (the mask is combined over the warp)
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < span; t += (int64_t)gridDim.x * blockDim.x) {
    const bool on = t < total;
    const int64_t node = on ? (t >> rest) : 0;
    const int64_t low = on ? (t & (((int64_t)1 << rest) - 1)) : 0;
    const uint2 nd = on ? __ldg(nodes + node) : make_uint2(0u, 0u);
    T v[1 << KB];
    if constexpr (FIRST) {
      uint32_t at[1 << KB];
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j) {
        const int64_t i = ((int64_t)j << rest) | low;
        at[j] = __ldcs(smap + (swapped(c) ? ((int64_t)1 << (rest + KB)) - 1 - i : i));
      }
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j) v[j] = __ldg(src + at[j]);
      if (tv) {
#pragma unroll
        for (int j = 0; j < (1 << KB); ++j) v[j] = weigh(v[j], tv[at[j]], post);
      }
    } else {
      const T* p = src + (node << (rest + KB)) + low;
#pragma unroll
      for (int j = 0; j < (1 << KB); ++j) v[j] = p[(int64_t)j << rest];
    }
    tree_bfly<T, KB, C>(v, __reduce_or_sync(0xffffffffu, nd.y), c);
    int64_t child = nd.x;
#pragma unroll
    for (int j = 0; j < (1 << KB); ++j) {
      if ((nd.y >> j) & 1u) {
        if constexpr (kPower)
          acc = fma((double)dup[child] * pw.d[__popc(idx[child])], (double)v[j] * (double)v[j], acc);
        else if constexpr (LAST)
          dst[child] = (T)((double)v[j] * post.f64 * (double)dup[child] * tv[child]);
        else
          dst[(child << rest) | low] = v[j];
        ++child;
      }
    }
  }
  if constexpr (kPower) block_sum(acc, dst);
}

int grid_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  int64_t cap = (int64_t)num_sms() * 16;
  return (int)std::max<int64_t>(1, std::min(b, cap));
}

// (small levels in blocks of two warps, so that more than a few SMs' FP64 pipes
// have work)
int tree_threads(int64_t nnode, int rest) { return (nnode << rest) < (int64_t)num_sms() * 256 ? 64 : 256; }
int tree_grid(int64_t nnode, int rest) {
  const int th = tree_threads(nnode, rest);
  return (int)std::min<int64_t>(((nnode << rest) + th - 1) / th, (int64_t)num_sms() * 64);
}

template <class T, bool FIRST, bool LAST, class C>
void launch_tree(int kb, const T* src, const uint32_t* smap, const uint2* nodes, int64_t nnode, int rest, const C& c,
                 T* dst, const uint16_t* dup, const double* tv, double post, cudaStream_t s,
                 const uint32_t* idx = nullptr, const PowerTab* pw = nullptr) {
  const int grid = tree_grid(nnode, rest), threads = tree_threads(nnode, rest);
  const PowerTab tab = pw ? *pw : PowerTab{};
  const ScaleF pf = scale_factor(post);
  auto go = [&](auto k) {
    kron_tree_kernel<T, decltype(k)::value, FIRST, LAST, C><<<grid, threads, 0, s>>>(src, smap, nodes, nnode, rest, c,
                                                                                     dst, dup, tv, pf, idx, tab);
  };
  switch (kb) {
    case 5: go(std::integral_constant<int, 5>()); break;
    case 4: go(std::integral_constant<int, 4>()); break;
    case 3: go(std::integral_constant<int, 3>()); break;
    case 2: go(std::integral_constant<int, 2>()); break;
    default: go(std::integral_constant<int, 1>()); break;
  }
  TM_CKK("kron_tree");
}

// y = post dup tvec (Th u) at the representatives; fold: u is x, to be
// scaled by tvec gin on the way in
template <class T>
void run_tree(const Op& op, const T* u, T* y, bool fold, double gin, double post, cudaStream_t s) {
  const PrefixTree& t = op.tree;
  const Kron<T> c = kron_of<T>(op);
  T* buf[2] = {op.ws_a.as<T>(), op.ws_b.as<T>()};
  const T* src = u;
  const uint16_t* dup = op.dup.as<uint16_t>();
  const double* tv = op.tvec.as<double>();
  for (int i = 0; i < t.nlev; ++i) {
    const int kb = t.b[i + 1] - t.b[i], rest = op.L - t.b[i + 1];
    const bool first = (i == 0), last = (i == t.nlev - 1);
    T* dst = last ? y : buf[i & 1];
    const uint32_t* smap = op.smap.as<uint32_t>();
    if (first)
      launch_tree<T, true, false, Kron<T>>(kb, src, smap, t.level(i), t.n[i], rest, c, dst, dup, fold ? tv : nullptr, gin, s);
    else if (!last)
      launch_tree<T, false, false, Kron<T>>(kb, src, smap, t.level(i), t.n[i], rest, c, dst, dup, tv, post, s);
    else
      launch_tree<T, false, true, Kron<T>>(kb, src, smap, t.level(i), t.n[i], rest, c, dst, dup, tv, post, s);
    src = dst;
  }
}

// ------------------------------------------------------------------ small operators
// A whole reduced product in one block: expand, mix, contract (y may be x:
// every read of x precedes the first barrier).  Launches are what a small
// product costs (about 2.5 us each).  In FP64 one SM's pipe takes 1.1 us at
// L = 9 and longer than the tree's launches from L = 12 on; FP32 has 64 times
// the rate and stays in one block up to 12 bits (at 13: 22.6 us, the open
// boundary's tile passes 16.4, a tree 20.5).
template <class T>
constexpr int small_bits() {
  return sizeof(T) == 4 ? 12 : 11;
}
template <class T, int KB>
__global__ void __launch_bounds__(1024) kron_small_kernel(const T* x, const uint32_t* __restrict__ smap,
                                                          const uint32_t* __restrict__ idx,
                                                          const uint16_t* __restrict__ dup,
                                                          const double* __restrict__ tv, int L, Kron<T> c, double gin,
                                                          double post, T* y, int n) {
  __shared__ T sm[(1 << small_bits<T>()) + (1 << small_bits<T>()) / 32 + 1];
  for (int i = threadIdx.x; i < (1 << L); i += blockDim.x) {
    const uint32_t q = smap[i];
    sm[spad(i)] = (T)((double)x[q] * tv[q] * gin);
  }
  __syncthreads();
  tile_rounds<T, KB, Kron<T>>(sm, L, 0, 0, c);
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    y[i] = (T)((double)sm[spad((int)idx[i])] * post * (double)dup[i] * tv[i]);
}

// ---- generic reduced path kernels
template <class T>
__global__ void scale_in_kernel(const T* __restrict__ x, const double* __restrict__ tv, double gin, T* __restrict__ u,
                                int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) u[i] = (T)((double)x[i] * tv[i] * gin);
}

// y[r] = post * dup[r] * tv[r] * z[idx[r]]
template <class T>
__global__ void contract_kernel(const T* __restrict__ z, const uint32_t* __restrict__ idx,
                                const uint16_t* __restrict__ dup, const double* __restrict__ tv,
                                double post, T* __restrict__ y, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) y[i] = (T)((double)z[idx[i]] * post * (double)dup[i] * tv[i]);
}

}  // namespace

// Four bits per level, the odd ones out in threes at the end.  Up to 20 bits,
// where launches are what a product costs, a single bit left over joins the
// first level (L = 13, 17; all levels of five bits were slower at L = 15 and 20).
static std::vector<int> tree_steps(int L) {
  std::vector<int> steps;
  const int nlev = (L + 3) / 4 - (L <= 20 && L % 4 == 1 ? 1 : 0);
  for (int i = 0, b = 0; i < nlev; ++i) {
    steps.push_back((L - b + nlev - i - 1) / (nlev - i));
    b += steps.back();
  }
  return steps;
}
// elements of the two buffers that the levels write in turn
static void tree_buffer_elems(const Op& op, int64_t most[2]) {
  most[0] = most[1] = 1;
  for (int i = 0; i + 1 < op.tree.nlev; ++i)
    most[i & 1] = std::max(most[i & 1], op.tree.n[i + 1] << (op.L - op.tree.b[i + 1]));
}

// Constants of a Kronecker-core operator, and the workspace of its generic
// reduced product: the prefix tree of the translation groups with its two
// level buffers, or the full-space vector.
void build_bfly(Op& op) {
  const double K = op.mp.betaJ, aK = std::fabs(K);
  KronConst& kc = op.kron;
  kc.r = std::exp(-2.0 * aK);
  kc.S = std::pow(std::exp(K) + std::exp(-K), (double)op.L);
  // gin keeps the magnitudes of the unnormalised butterflies those of the
  // normalised factor, (max(a, b) / (a + b))^L = (1 + r)^-L; out undoes it
  // (its rounding cancels) and applies max(a, b)^L = e^{|K| L}, with the
  // factor that the rounding of r adds to a constant vector taken out: all L
  // levels share that rounding, which would grow as L
  const long double rl = std::exp(-2.0L * (long double)aK);
  kc.gin = std::pow(1.0 + (double)rl, -(double)op.L);
  const long double emax = std::exp((long double)aK * (long double)op.L) / kc.gin;
  kc.out64 = (double)(emax * rounding_factor(rl, kron_of<double>(op).r, op.L));
  kc.out32 = (double)(emax * rounding_factor(rl, kron_of<float>(op).r, op.L));
  if (op.kind == K_XAT) return;
  const bool shifts = (op.kind == K_XAM && op.grp.periodic) || op.kind == K_XAM3;
  if (op.L <= small_bits<double>()) return;
  if (!shifts) {
    op.ws_a.alloc((size_t)op.nstate * 8);
    return;
  }
  build_prefix_tree(op, op.L, tree_steps(op.L), false, op.tree);
  int64_t most[2];
  tree_buffer_elems(op, most);
  op.ws_a.alloc((size_t)most[0] * 8);
  op.ws_b.alloc((size_t)most[1] * 8);
}

// v^T (dTh / dK) v of the Kronecker factor for v = Tvec x expanded to the full
// space (x: device, the operator's rows), as block sums in part; returns
// their number.  All 2 x 2 factors are diagonal in the Hadamard basis, so
//   v^T dTh v = 2^-L sum_w lambda'_{|w|} vhat(w)^2,
//   lambda_k = (2 cosh K)^(L-k) (2 sinh K)^k,
// one addition per element and level where tangent pairs (value, derivative)
// took eight FP64 operations per pair and level, and no cancellation that T
// itself does not have.  vhat has the symmetries of v: with translations and
// no spin flip only representatives' prefixes are formed (as in the
// products); a flip-symmetric v has vhat(w) = 0 at odd |w| and twice the
// transform of its lower half at even |w|.  A gradient of the reduced L = 24
// operator (no flip) took 4.79 ms with tangent pairs on all 2^24 states and
// takes 0.39 ms, its copies included.
int64_t kron_power(const Op& op, const double* x, DBuf& part, cudaStream_t s) {
  const int L = op.L;
  double dlam[33];
  power_weights(op.mp.betaJ, L, dlam);
  const double* tv = op.tvec.as<double>();
  const bool reduced = op.kind != K_XAT;
  const bool shifts = (op.kind == K_XAM && op.grp.periodic) || op.kind == K_XAM3;
  PowerTab pw{};
  DBuf u, a, b;
  if (reduced) {
    u.alloc((size_t)op.n * 8);
    scale_in_kernel<double><<<grid_for(op.n), 256, 0, s>>>(x, tv, 1.0, u.as<double>(), op.n);
    TM_CKK("scale_in");
  }
  const uint32_t* smap = op.smap.as<uint32_t>();
  if (reduced && shifts && !op.grp.flip && L > small_bits<double>()) {
    // (an even/odd operator has no tree of its own; it keeps this one)
    {
      Op& o = const_cast<Op&>(op);
      std::lock_guard<std::mutex> lock(o.lazy_mu);
      if (!o.tree.nlev) build_prefix_tree(op, L, tree_steps(L), false, o.tree);
    }
    const PrefixTree& t = op.tree;
    for (int k = 0; k <= L; ++k) pw.d[k] = dlam[k];
    int64_t most[2];
    tree_buffer_elems(op, most);
    a.alloc((size_t)most[0] * 8);
    b.alloc((size_t)most[1] * 8);
    const double* src = u.as<double>();
    const uint16_t* dup = op.dup.as<uint16_t>();
    const Had had;
    for (int i = 0; i < t.nlev; ++i) {
      const int kb = t.b[i + 1] - t.b[i], rest = L - t.b[i + 1];
      double* dst = (i & 1) ? b.as<double>() : a.as<double>();
      if (i == 0) {
        launch_tree<double, true, false, Had>(kb, src, smap, t.level(i), t.n[i], rest, had, dst, dup, nullptr, 1.0, s);
      } else if (i + 1 < t.nlev) {
        launch_tree<double, false, false, Had>(kb, src, smap, t.level(i), t.n[i], rest, had, dst, dup, nullptr, 1.0, s);
      } else {
        const int64_t np = tree_grid(t.n[i], rest);
        part.alloc((size_t)np * 8);
        launch_tree<double, false, true, Had>(kb, src, smap, t.level(i), t.n[i], rest, had, part.as<double>(), dup,
                                              nullptr, 1.0, s, op.idx.as<uint32_t>(), &pw);
        return np;
      }
      src = dst;
    }
  }
  const bool half = reduced && op.grp.flip;
  const int n = half ? L - 1 : L;
  for (int k = 0; k <= n; ++k) pw.d[k] = half ? 4.0 * dlam[k + (k & 1)] : dlam[k];
  a.alloc(((size_t)1 << n) * 8);
  int lo = 0;
  const int npass = tile_passes(n, 8);
  int64_t np = 0;
  for (int p = 0; p < npass; ++p) {
    const TilePass t = tile_pass(n, lo, npass - p, 8);
    const bool last = (p == npass - 1);
    np = t.nblocks;
    if (last) part.alloc((size_t)np * 8);
    const double* src = p ? a.as<double>() : (reduced ? u.as<double>() : x);
    auto go = [&](auto k) {
      constexpr int KB = decltype(k)::value;
      if (t.shm > 48 * 1024) raise_smem_limit((const void*)had_tile_kernel<KB>, t.shm);
      had_tile_kernel<KB><<<(unsigned)t.nblocks, t.threads, t.shm, s>>>(src, a.as<double>(), lo, t.nb, t.cb,
                                                                       (p || !reduced) ? nullptr : smap,
                                                                       (p || reduced) ? nullptr : tv,
                                                                       last ? part.as<double>() : nullptr, pw);
    };
    if (t.kb == 4)
      go(std::integral_constant<int, 4>());
    else if (t.kb == 2)
      go(std::integral_constant<int, 2>());
    else
      go(std::integral_constant<int, 1>());
    TM_CKK("had_tile");
    lo += t.nb;
  }
  return np;
}

// y = T x on the full space (K_XAT) or on the reduced basis through the full
// space (reduced kinds whose core is the Kronecker factor).  scaled=true:
// the result is divided by the returned factor, S = (e^K+e^-K)^L or, where
// what is left of the output factor would take FP32 results out of their
// range (scale_fits), the whole of it.
template <class T>
double matvec_bfly(const Op& op, const T* x, T* y, bool scaled, cudaStream_t s) {
  const KronConst& kc = op.kron;
  const double sf = ((sizeof(T) == 8) ? kc.out64 : kc.out32) / (scaled ? kc.S : 1.0);
  const double ret = scaled ? kc.S : 1.0;
  const double* tv = op.tvec.as<double>();
  if (op.kind == K_XAT) {
    // y = nf * Tv^(1/2) * Th * Tv^(1/2) * x   (TMat/tmat.cpp:71-102)
    const double gin = (sizeof(T) == 8) ? 1.0 : kc.gin;
    const double f = op.normfactor * sf * (kc.gin / gin);
    const bool whole = scaled && !scale_fits(f);
    run_sweep<T>(op, x, y, 1, tv, gin, nullptr, 1, tv, whole ? 1.0 : f, s);
    return whole ? ret * f : ret;
  }
  const uint32_t* smap = op.smap.as<uint32_t>();
  const uint32_t* idx = op.idx.as<uint32_t>();
  const uint16_t* dup = op.dup.as<uint16_t>();
  // reduced: u = Tvec .* x ; v = P u ; z = Th v ; y = dup .* Tvec .* z[idx]
  if (op.L <= small_bits<T>()) {
    if (op.L <= 11)
      kron_small_kernel<T, 2><<<1, 512, 0, s>>>(x, smap, idx, dup, tv, op.L, kron_of<T>(op), kc.gin, sf, y, (int)op.n);
    else
      kron_small_kernel<T, 3><<<1, 1024, 0, s>>>(x, smap, idx, dup, tv, op.L, kron_of<T>(op), kc.gin, sf, y, (int)op.n);
    TM_CKK("kron_small");
    return ret;
  }
  const bool fold = op.tree.nlev && op.L <= (sizeof(T) == 4 ? 20 : 16);
  T* u = static_cast<T*>(op.ws_c.p);
  if (!fold) {
    scale_in_kernel<T><<<grid_for(op.n), 256, 0, s>>>(x, tv, kc.gin, u, op.n);
    TM_CKK("scale_in");
  }
  if (op.tree.nlev) {
    run_tree<T>(op, fold ? x : u, y, fold, kc.gin, sf, s);
    return ret;
  }
  T* full = static_cast<T*>(op.ws_a.p);
  run_sweep<T>(op, u, full, 2, nullptr, 1.0, smap, 0, nullptr, 1.0, s);
  contract_kernel<T><<<grid_for(op.n), 256, 0, s>>>(full, idx, dup, tv, sf, y, op.n);
  TM_CKK("contract");
  return ret;
}

template double matvec_bfly<float>(const Op&, const float*, float*, bool, cudaStream_t);
template double matvec_bfly<double>(const Op&, const double*, double*, bool, cudaStream_t);

// ---- permutation helpers
namespace {
template <class T>
__global__ void gather_kernel(const T* __restrict__ src, const uint32_t* __restrict__ idx,
                              T* __restrict__ dst, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) dst[i] = src[idx[i]];
}
// dst[c*n + i] = src[c*lds + idx[i]] for nvec columns, two consecutive
// outputs per thread in one 16-byte store where dst allows it (the stores may
// go to host memory over the host link, where wide stores count)
__global__ void gather_cols_f64_kernel(const double* __restrict__ src, int64_t lds, const uint32_t* __restrict__ idx,
                                       double* __restrict__ dst, int64_t n, int nvec) {
  const int64_t half = (n + 1) >> 1;
  const int64_t total = half * nvec;
  const bool pairs = (n % 2 == 0) && ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = t / half, i = (t - c * half) * 2;
    const double* sc = src + c * lds;
    double* dc = dst + c * n;
    if (pairs) {
      const double a = sc[idx[i]], b = sc[idx[i + 1]];
      *reinterpret_cast<double2*>(dc + i) = make_double2(a, b);
    } else {
      dc[i] = sc[idx[i]];
      if (i + 1 < n) dc[i + 1] = sc[idx[i + 1]];
    }
  }
}

template <class T>
__global__ void scatter_kernel(const T* __restrict__ src, const uint32_t* __restrict__ idx,
                               T* __restrict__ dst, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) dst[idx[i]] = src[i];
}
}  // namespace

void gather_f64(const double* src, const uint32_t* idx, double* dst, int64_t n, cudaStream_t s) {
  gather_kernel<double><<<grid_for(n), 256, 0, s>>>(src, idx, dst, n);
  TM_CKK("gather");
}
void gather_cols_f64(const double* src, int64_t lds, const uint32_t* idx, double* dst, int64_t n, int nvec,
                     cudaStream_t s) {
  gather_cols_f64_kernel<<<grid_for(((n + 1) / 2) * nvec), 256, 0, s>>>(src, lds, idx, dst, n, nvec);
  TM_CKK("gather_cols");
}
void scatter_f64(const double* src, const uint32_t* idx, double* dst, int64_t n, cudaStream_t s) {
  scatter_kernel<double><<<grid_for(n), 256, 0, s>>>(src, idx, dst, n);
  TM_CKK("scatter");
}
}  // namespace ltm
