// Two-layer parallel transfer matrices: the y-direction TMs, whose state is a
// pair of adjacent layers (2L spins; the reference index puts one layer in the
// high L bits and the other in the low L bits).
//
//   YATMatVecProd2D / _T (TMat/tmat.cpp:106-242): L shift-and-mix steps on one
//     layer amount to the Kronecker factor (x)_i [[e^-Kk, e^Kk], [e^Kk, e^-Kk]]
//     on that layer's L bits, then a layer swap and the dense NN-only x-ANNNI
//     weight as a diagonal: y = nf * Tvec .* swap(K_high x); the transpose is
//     y = nf * swap(K_low (Tvec .* x)).
//   Y2ATMatVecProd2D (TMat/tmat.cpp:245-315): the L steps of permute_mult_T1
//     apply one 4x4 matrix to every bit pair (i, L+i); y = nf * Tv^(1/2) .*
//     P4 (Tv^(1/2) .* x).  The reference's get_t_instance is the operator itself.
//   YAMMatVecProd2D / _T, YBMMatVecProd2D (TMat/tmatreduce.cpp:661-1021):
//     representatives are grouped by their left (high) layer l; one CTA per
//     group fills the right-layer vector at g(r) for every g in the stabiliser
//     of l, applies the Kronecker factor on the L right bits in shared memory
//     and writes each representative's entry to its layer-swapped orbit.
//
// The full forms run as shared-memory tile passes over HBM: a pass gathers a
// tile of 2^nt states whose index bits are chosen per pass (a few contiguous
// low bits for coalescing plus the bits being mixed), applies the factor for
// those bits, and writes the tile back.  FP64 throughout (these operators are
// at most 4^14 states).
#include <algorithm>
#include <cmath>
#include <vector>

#include "tm_bfly.cuh"
#include "tm_bits.cuh"
#include "tm_group.cuh"
#include "tm_internal.h"

namespace ltm {

void kron_swap_product(const Op& op, const double* x, double* y, double* ws, bool transposed, cudaStream_t s);
double kron_out_factor(double coupling, int L, double r);

namespace {

constexpr int kMaxTileBits = 12;  // 4096 doubles = 32 KB per tile

// Y2ATMatVecProd2D's factor on one bit pair (low site p & 1, high site p >> 1):
//   out(p) = e1[j] (e2[0] in(p) + in(p^2)) + e1[j^1] (e2[1] in(p^3) + in(p^1)),
// j = low ^ high, e2[1] = 1 / e2[0].  With a(p) = e2[0] in(p) + in(p^2) the
// second bracket is e2[1] a(p^1), and the factor e1[j] of the output state can
// wait until all pairs are done (it is e^{K (L - 2 popc(low ^ high))} then):
//   out(p) = e1[j] (a(p) + rho_j a(p^1)), rho_j = e1[j^1] e2[1] / e1[j],
// two FMAs per element and pair where the 4 x 4 matrix takes four.
//   The L pairs grow the values by up to ((1 + e2) (1 + rho_j))^L before the
// output factor brings them back.  Where that comes near the end of the FP64
// range, a ratio above one is turned round, a(p^1) + a(p) / rho_j, and its power
// goes into the factor of the output state (e2 likewise: a(p) / e2 = in(p) +
// in(p^2) / e2), so that a pair grows them by four at most.  TURN: bit 0 for e2,
// bits 1 and 2 for rho_0 and rho_1.  The turned form of rho_1 alone takes 0.93
// ms at L = 12, the plain one 0.84.
struct PairCoef {
  double e2;
  double rho[2];
};
template <int TURN>
__device__ __forceinline__ void pair_step(double (&v)[4], const PairCoef& c) {
  double a[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) a[p] = fma(c.e2, (TURN & 1) ? v[p ^ 2] : v[p], (TURN & 1) ? v[p] : v[p ^ 2]);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int j = (p & 1) ^ (p >> 1);
    const bool turned = (TURN >> (j + 1)) & 1;
    v[p] = fma(c.rho[j], turned ? a[p] : a[p ^ 1], turned ? a[p ^ 1] : a[p]);
  }
}

struct PairTab {
  double d[16];  // e^{K (L - 2 q)} times the output factor, by q = popc(low ^ high)
};

// One tile pass: bit pairs (lo + j, L + lo + j), j < np, and cb contiguous low
// bits.  Tile index: chunk bits, then the low sites, then the high sites.
// pre / post_sc: per-state input / output weights (first / last pass).
// Bound by the FP64 pipe.
template <int TURN>
__global__ void __launch_bounds__(512) pair_kernel(const double* x, double* y, int L, int lo, int np, int cb,
                                                   PairCoef c, const double* __restrict__ pre,
                                                   const double* __restrict__ post_sc, PairTab tab) {
  extern __shared__ double sm[];
  const int tile = 1 << (cb + 2 * np);
  const int cmask = (1 << cb) - 1, nmask = (1 << np) - 1;
  // block index -> bits [cb, lo), [lo + np, L) and [L, L + lo), [L + lo + np, 2L)
  uint64_t o = blockIdx.x;
  uint64_t base = (o & ((1ull << (lo - cb)) - 1)) << cb;
  o >>= lo - cb;
  base |= (o & ((1ull << (L - lo - np)) - 1)) << (lo + np);
  o >>= L - lo - np;
  base |= (o & ((1ull << lo) - 1)) << L;
  o >>= lo;
  base |= o << (L + lo + np);
  auto state = [&](int e) -> uint64_t {
    return base | (uint64_t)(e & cmask) | ((uint64_t)((e >> cb) & nmask) << lo) | ((uint64_t)(e >> (cb + np)) << (L + lo));
  };
  for (int e = threadIdx.x; e < tile; e += blockDim.x) {
    const uint64_t g = state(e);
    sm[spad(e)] = pre ? x[g] * pre[g] : x[g];
  }
  __syncthreads();
  for (int j = 0; j < np; ++j) {
    const int ba = cb + j, bb = cb + np + j;  // ba < bb
    const int o1 = 1 << ba, o2 = 1 << bb;
    for (int q = threadIdx.x; q < (tile >> 2); q += blockDim.x) {
      // insert zeros at bits ba and bb
      int e = ((q >> ba) << (ba + 1)) | (q & (o1 - 1));
      e = ((e >> bb) << (bb + 1)) | (e & (o2 - 1));
      double v[4] = {sm[spad(e)], sm[spad(e | o1)], sm[spad(e | o2)], sm[spad(e | o1 | o2)]};
      pair_step<TURN>(v, c);
      sm[spad(e)] = v[0];
      sm[spad(e | o1)] = v[1];
      sm[spad(e | o2)] = v[2];
      sm[spad(e | o1 | o2)] = v[3];
    }
    __syncthreads();
  }
  const uint64_t lm = (1ull << L) - 1;
  for (int e = threadIdx.x; e < tile; e += blockDim.x) {
    const uint64_t g = state(e);
    const double v = sm[spad(e)];
    y[g] = post_sc ? v * (post_sc[g] * tab.d[__popcll((g ^ (g >> L)) & lm)]) : v;
  }
}

// --- Tvec of the full forms
// YATMatVecProd2D::genTvec (TMat/tmat.hpp:361-366, TMat/tmat.cpp:668-684):
// entry (row = low layer, col = high layer) of the dense NN-only x-ANNNI TM
// (times the product's output factor f)
__global__ void yat_tvec_kernel(double* __restrict__ tv, int L, double bj, double h, double f) {
  const int64_t n = 1ll << (2 * L);
  const uint64_t lm = (1ull << L) - 1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t row = (uint64_t)i & lm, col = (uint64_t)i >> L;
    const int n1 = popc64(row ^ rotr(row, L, 1)), n0 = popc64(row), nx = popc64(row ^ col);
    tv[i] = f * exp(-bj * (2 * n1 - L) - bj * h * (2 * n0 - L) - bj * (2 * nx - L));
  }
}

// Y2ATMatVecProd2D::genTvec (TMat/tmat.hpp:396-414) at betaJ/2: Tv^(1/2)
__global__ void y2at_tvec_kernel(double* __restrict__ tv, int L, double bj, double h) {
  const int64_t n = 1ll << (2 * L);
  const uint64_t lm = (1ull << L) - 1;
  const double J1 = -0.5 * bj, hJ = -0.5 * bj * h;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t lo = (uint64_t)i & lm, hi = (uint64_t)i >> L;
    const int n1 = popc64(lo ^ rotr(lo, L, 1)), n2 = popc64(hi ^ rotr(hi, L, 1)), n0 = popc64(lo ^ hi);
    const int fa = 2 * (n1 + n2 + n0) - 3 * L, fb = 2 * (popc64((uint64_t)i) - L);
    tv[i] = exp(J1 * fa + hJ * fb);
  }
}

// YAMMatVecProd2D::genTvec / genTvec1 (TMat/tmatreduce.cpp:725-797)
__global__ void yam_tvec_kernel(const uint32_t* __restrict__ idx, const uint16_t* __restrict__ dup,
                                double* __restrict__ tv, int64_t n, int L, int ltype, double bj, double k,
                                double k2, double h, double nfe) {
  const uint64_t lm = (1ull << L) - 1;
  const double hb = 0.5 * bj, J1 = -hb, hJ = -hb * h, Jn = hb * nfe, k1J = hb * k, k2J = hb * k2;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t s = idx[r], l = s >> L, rt = s & lm;
    const int n1 = popc64(l ^ rotr(l, L, 1)), n2 = popc64(l ^ rt), n0 = popc64(l);
    double bz = J1 * (2 * (n1 + n2 - L)) + hJ * (2 * n0 - L) + Jn;
    if (ltype) {
      const int b1 = popc64(l ^ rotr(l, L, 2)), d1 = popc64(l ^ rotr(rt, L, 1)), d2 = popc64(l ^ rotl(rt, L, 1));
      bz += k1J * (2 * b1 - L) + k2J * (2 * (d1 + d2 - L));
    }
    tv[r] = exp(bz) / sqrt((double)dup[r]);
  }
}

// swp[r] = rank of the orbit holding the layer-swapped states of orbit r
__global__ void yswap_kernel(GroupDev g, const uint32_t* __restrict__ idx, int64_t n,
                             const uint32_t* __restrict__ bits, const uint32_t* __restrict__ prefix,
                             uint32_t* __restrict__ swp) {
  const int L = g.L;
  const uint64_t lm = (1ull << L) - 1;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t s = idx[r];
    const uint64_t c = canon(g, (s & lm) << L | (s >> L));
    const uint32_t w = (uint32_t)(c >> 5);
    swp[r] = prefix[w] + __popc(bits[w] & ((1u << (c & 31)) - 1u));
  }
}

// one layer under group element gi of the two-layer group (translation,
// reflection, flip), the same element acting on both layers
__device__ __forceinline__ uint32_t layer_act(uint32_t x, int L, int gi) {
  const uint32_t lm = (1u << L) - 1;
  const int sh = gi % L, rf = (gi / L) & 1, f = gi / (2 * L);
  uint64_t v = x;
  if (rf) v = brev(v, L);
  if (f) v = ~v & lm;
  return (uint32_t)rotr(v, L, sh);
}

// YAMMatVecProd2D::perform_op (TMat/tmatreduce.cpp:827-876), transposed:
// YAMMatVecProd2D_T::perform_op (:953-1016).  One CTA per left-layer block,
// KB bits of the right layer per round in registers.
template <int KB>
__global__ void __launch_bounds__(512) yam_block_kernel(const double* __restrict__ x, double* __restrict__ y,
                                                        const uint32_t* __restrict__ idx,
                                                        const uint16_t* __restrict__ dup,
                                                        const double* __restrict__ tv,
                                                        const uint32_t* __restrict__ swp,
                                                        const uint32_t* __restrict__ bstart, int L, int ng,
                                                        int transposed, Kron<double> c, double post) {
  extern __shared__ double tmp[];
  __shared__ int stab[64];
  __shared__ int nstab;
  const uint32_t r0 = bstart[blockIdx.x], r1 = bstart[blockIdx.x + 1];
  const uint32_t lm = (1u << L) - 1;
  const uint32_t l = idx[r0] >> L;
  if (threadIdx.x == 0) nstab = 0;
  __syncthreads();
  if ((int)threadIdx.x < ng && layer_act(l, L, threadIdx.x) == l) stab[atomicAdd(&nstab, 1)] = threadIdx.x;
  __syncthreads();
  const int ns = nstab;
  for (uint32_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    const uint32_t src = transposed ? swp[r] : r;
    const double v = tv[src] * x[src];
    const uint32_t rt = idx[r] & lm;
    for (int q = 0; q < ns; ++q) tmp[spad((int)layer_act(rt, L, stab[q]))] = v;
  }
  __syncthreads();
  tile_rounds<double, KB, Kron<double>>(tmp, L, 0, 0, c);
  for (uint32_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    const uint32_t dst = transposed ? r : swp[r];
    y[dst] = tv[dst] * (double)dup[dst] * (tmp[spad((int)(idx[r] & lm))] * post);
  }
}

int grid_n(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 16));
}

}  // namespace

void build_two_layer(Op& op) {
  const int L = op.L;
  if (L > 14) fail(TM_ERR_LIMIT, "two-layer operators support L <= 14 (4^L states)");
  const double bj = op.mp.betaJ, k = op.mp.kappa, k2 = op.mp.kappa2, h = op.mp.h;
  op.nstate = 1ll << (2 * L);
  cudaStream_t s = op.stream;
  // output factor of the r-form butterflies (K_YAT, K_YAM)
  op.kron.out64 = kron_out_factor(bj * k, L, std::exp(-2.0 * std::fabs(bj * k))) *
                  (op.kind == K_YAT ? op.normfactor : 1.0);
  if (op.kind == K_YAT || op.kind == K_Y2AT) {
    op.n = op.nstate;
    op.tvec.alloc((size_t)op.n * 8);
    op.ws_a.alloc((size_t)op.n * 8);
    if (op.kind == K_YAT)
      yat_tvec_kernel<<<grid_n(op.n), 256, 0, s>>>(op.tvec.as<double>(), L, bj, h, op.kron.out64);
    else
      y2at_tvec_kernel<<<grid_n(op.n), 256, 0, s>>>(op.tvec.as<double>(), L, bj, h);
    TM_CKK("two_layer_tvec");
    TM_CK(cudaStreamSynchronize(s));
    return;
  }
  // reduced: orbits of the two-layer group
  op.grp.kind = G_Y2D;
  op.grp.L = L;
  op.grp.nbits = 2 * L;
  op.grp.periodic = 1;
  op.grp.flip = op.censym;
  build_orbit_table(op);
  const int64_t R = op.n;
  GroupDev g = to_dev(op.grp);
  op.swp.alloc((size_t)R * 4);
  yswap_kernel<<<grid_n(R), 256, 0, s>>>(g, op.idx.as<uint32_t>(), R, op.ws_a.as<uint32_t>(),
                                         op.ws_b.as<uint32_t>(), op.swp.as<uint32_t>());
  TM_CKK("two_layer_swap");
  op.tvec.alloc((size_t)R * 8);
  yam_tvec_kernel<<<grid_n(R), 256, 0, s>>>(op.idx.as<uint32_t>(), op.dup.as<uint16_t>(), op.tvec.as<double>(), R,
                                            L, op.ltype, bj, k, k2, h, op.nfexp);
  TM_CKK("two_layer_tvec");
  // blocks of representatives sharing the left (high) layer
  std::vector<uint32_t> idx((size_t)R), starts;
  TM_CK(cudaMemcpyAsync(idx.data(), op.idx.p, (size_t)R * 4, cudaMemcpyDeviceToHost, s));
  TM_CK(cudaStreamSynchronize(s));
  for (int64_t r = 0; r < R; ++r)
    if (r == 0 || (idx[r] >> L) != (idx[r - 1] >> L)) starts.push_back((uint32_t)r);
  starts.push_back((uint32_t)R);
  op.nblocks = (int)starts.size() - 1;
  op.bstart.alloc(starts.size() * 4);
  TM_CK(cudaMemcpyAsync(op.bstart.p, starts.data(), starts.size() * 4, cudaMemcpyHostToDevice, s));
  TM_CK(cudaStreamSynchronize(s));
  op.ws_a.release();
  op.ws_b.release();
}

void matvec_two_layer(const Op& op, const double* x, double* y, cudaStream_t s) {
  const Op& b = op.parent ? *op.parent : op;
  const bool tr = op.transposed;
  const int L = b.L;
  const double bj = b.mp.betaJ, k = b.mp.kappa;
  if (b.kind == K_YAT) {
    kron_swap_product(b, x, y, b.ws_a.as<double>(), tr, s);
  } else if (b.kind == K_Y2AT) {
    // bzwj1 = e^{+-K}, bzwj2 = e^{-+2K kappa} (TMat/tmat.cpp:247-253)
    // ln e2[0], ln rho_0, ln rho_1
    const double le2 = -2.0 * bj * k, lr[2] = {-2.0 * bj - le2, 2.0 * bj - le2};
    PairCoef c;
    const double growth = L * (std::log1p(std::exp(le2)) + std::log1p(std::exp(std::max(lr[0], lr[1]))));
    const int turn = growth < 300.0 ? 0 : (le2 > 0.0 ? 1 : 0) | (lr[0] > 0.0 ? 2 : 0) | (lr[1] > 0.0 ? 4 : 0);
    double lt[3] = {le2, lr[0], lr[1]};  // ln of what was turned round
    for (int i = 0; i < 3; ++i)
      if (!((turn >> i) & 1)) lt[i] = 0.0;
    c.e2 = std::exp(turn & 1 ? -le2 : le2);
    for (int j = 0; j < 2; ++j) c.rho[j] = std::exp(((turn >> (j + 1)) & 1) ? -lr[j] : lr[j]);
    decltype(&pair_kernel<0>) const kernels[8] = {pair_kernel<0>, pair_kernel<1>, pair_kernel<2>, pair_kernel<3>,
                                                  pair_kernel<4>, pair_kernel<5>, pair_kernel<6>, pair_kernel<7>};
    PairTab tab{};
    for (int q = 0; q <= L; ++q) {
      const double ln = bj * (L - 2.0 * q) + L * lt[0] + (L - q) * lt[1] + q * lt[2];
      // (the factor alone may overflow where a tiny normfactor brings it back)
      tab.d[q] = ln < 700.0 ? b.normfactor * std::exp(ln)
                            : (b.normfactor > 0.0 ? std::exp(ln + std::log(b.normfactor)) : 0.0);
    }
    const double* tv = b.tvec.as<double>();
    int lo = 0;
    const double* src = x;
    while (lo < L) {
      const int cb = (lo == 0) ? 0 : std::min(3, lo);
      const int np = std::min(L - lo, (kMaxTileBits - cb) / 2);
      const int tile = 1 << (cb + 2 * np);
      const size_t shm = (size_t)(tile + tile / 32 + 1) * sizeof(double);
      const bool last = (lo + np >= L);
      kernels[turn]<<<(unsigned)(1u << (2 * L - cb - 2 * np)), std::min(512, std::max(32, tile / 4)), shm, s>>>(
          src, y, L, lo, np, cb, c, lo == 0 ? tv : nullptr, last ? tv : nullptr, tab);
      TM_CKK("two_layer_pairs");
      src = y;
      lo += np;
    }
  } else if (b.kind == K_YAM) {
    const size_t shm = (size_t)((1 << L) + (1 << L) / 32 + 1) * sizeof(double);
    const int ng = 2 * L * (b.censym ? 2 : 1);
    const Kron<double> c{std::exp(-2.0 * std::fabs(bj * k)), bj * k > 0 ? 1 : 0};
    auto go = [&](auto kb) {
      constexpr int KB = decltype(kb)::value;
      raise_smem_limit((const void*)yam_block_kernel<KB>, shm);
      const int threads = std::min(512, std::max(128, (1 << L) >> KB));
      yam_block_kernel<KB><<<(unsigned)b.nblocks, threads, shm, s>>>(
          x, y, b.idx.as<uint32_t>(), b.dup.as<uint16_t>(), b.tvec.as<double>(), b.swp.as<uint32_t>(),
          b.bstart.as<uint32_t>(), L, ng, tr ? 1 : 0, c, b.kron.out64);
    };
    if (L >= 12)
      go(std::integral_constant<int, 4>());
    else if (L >= 9)
      go(std::integral_constant<int, 2>());
    else
      go(std::integral_constant<int, 1>());
    TM_CKK("two_layer_block");
  } else {
    fail(TM_ERR_ARG, "not a two-layer operator");
  }
}

}  // namespace ltm
