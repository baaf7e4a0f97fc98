// Adjoint of the leading eigenvalues: d ln(lambda)/d(betaJ, kappa, kappa2, h).
//
// No reference counterpart (the reference only reports eigenvalues and the
// magnetisation / domain-wall moments of TMat/tmatphys.cpp).  For an
// eigenpair (lambda, r) with left vector l (l = r for symmetric operators):
//   d lambda = l^T (dT) r / (l^T r).
// Every operator here is T = p * Tv' * Th * Tv' (Tv' = the operator's Tvec:
// the square-root intra-layer Boltzmann weight, times nf^(1/2) / sqrt(dup) in
// the reduced forms).  Tv' is diagonal, so with g(s) = d ln Tv'(s)/d theta:
//   d ln lambda = 2 <g>_{l r} + l^T (p Tv' dTh Tv') r / (lambda l^T r),
// where <g>_{l r} = sum l_i r_i g(s_i) / sum l_i r_i.  The first term is a
// fused weighted reduction over the basis.  The second is nonzero only for
// theta = betaJ (Th depends on K = betaJ alone for the Kronecker-core
// operators, which are symmetric: l = r).  It is a weighted sum of squared
// Hadamard coefficients of Tv' r (kron_power, tm_core.cu).  The normfactor terms cancel: the
// result is the derivative of the reported eigenvalue lambda/normfactor.
#include <cmath>
#include <functional>
#include <vector>

#include "tm_chain.h"
#include "tm_group.cuh"
#include "tm_internal.h"

namespace ltm {

namespace {

struct GradParams {
  int kind, L, s1, s2, boundary;
  double bj, k, k2, h;
};

// d(exponent of Tv')/d theta without the normfactor terms, theta = (bJ, k, k2, h)
__device__ void gvec(const GradParams& p, uint64_t s, double g[4]) {
  const int L = p.L;
  const uint64_t mask = (1ull << L) - 1;
  int n0 = popc64(s);
  g[0] = g[1] = g[2] = g[3] = 0.0;
  if (p.kind == K_XAT) {
    int n1, n2, ns1 = L, ns2 = L;
    uint64_t a, b;
    switch (p.boundary) {
      case 0:
        n1 = popc64(s ^ rotr(s, L, 1));
        n2 = popc64(s ^ rotr(s, L, 2));
        break;
      case 1:
        n1 = popc64((s & (mask >> 1)) ^ (s >> 1));
        n2 = popc64((s & (mask >> 2)) ^ (s >> 2));
        ns1 = L - 1;
        ns2 = L - 2;
        break;
      case 5:
      case 9:
        a = (s << 1) | (p.boundary == 9 ? 1ull : 0ull);
        b = s >> 1;
        n1 = popc64(s ^ a);
        n2 = popc64((a & mask) ^ b);
        ns1 = L + 1;
        break;
      default:
        a = (s << 1) | (p.boundary == 17 ? 1ull : 0ull);
        b = (s << 2) | (p.boundary == 17 ? 3ull : 0ull);
        n1 = popc64(s ^ a);
        n2 = popc64(s ^ b);
        ns1 = L + 1;
        ns2 = L + 2;
        break;
    }
    g[0] = -0.5 * (2.0 * n1 - ns1) + 0.5 * p.k * (2.0 * n2 - ns2) - 0.5 * p.h * (2.0 * n0 - L);
    g[1] = 0.5 * p.bj * (2.0 * n2 - ns2);
    g[3] = -0.5 * p.bj * (2.0 * n0 - L);
  } else if (p.kind == K_XAM) {
    int n1, n2;
    if (!p.boundary) {
      n1 = popc64(s ^ rotr(s, L, 1));
      n2 = popc64(s ^ rotr(s, L, 2));
    } else {
      n1 = popc64((s & (mask >> 1)) ^ (s >> 1));
      n2 = popc64((s & (mask >> 2)) ^ (s >> 2));
    }
    g[0] = -0.5 * (2 * n1 - L) + 0.5 * p.k * (2 * n2 - L) - 0.5 * p.h * (2 * n0 - L);
    g[1] = 0.5 * p.bj * (2 * n2 - L);
    g[3] = -0.5 * p.bj * (2 * n0 - L);
  } else if (p.kind == K_ZBT || p.kind == K_ZBM || p.kind == K_XDT || p.kind == K_XDM) {
    aux_tvec_grad(p.kind, L, p.boundary, p.bj, p.k2, p.h, s, g);
  } else if (p.kind == K_XAM3) {
    int n1a = popc64(s ^ rshift3d(s, p.s1, p.s2, 1));
    int n1b = popc64(s ^ dshift3d(s, p.s1, p.s2, 1));
    int n2 = popc64(s ^ rshift3d(s, p.s1, p.s2, 2));
    g[0] = -(n1a + n1b - L) + 0.5 * p.k * (2 * n2 - L) - 0.5 * p.h * (2 * n0 - L);
    g[1] = 0.5 * p.bj * (2 * n2 - L);
    g[3] = -0.5 * p.bj * (2 * n0 - L);
  }
}

__global__ void diag_grad_kernel(GradParams p, const double* __restrict__ qr, const double* __restrict__ ql,
                                 const uint32_t* __restrict__ idx, int64_t n, double* __restrict__ part) {
  double acc[5] = {0, 0, 0, 0, 0};
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) {
    uint64_t s = idx ? (uint64_t)idx[i] : (uint64_t)i;
    double w = qr[i] * (ql ? ql[i] : qr[i]);
    double g[4];
    gvec(p, s, g);
    for (int k = 0; k < 4; ++k) acc[k] += w * g[k];
    acc[4] += w;
  }
  __shared__ double sh[5][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int k = 0; k < 5; ++k) {
    double v = acc[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sh[k][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    double t = 0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sh[threadIdx.x][q];
    part[(int64_t)blockIdx.x * 5 + threadIdx.x] = t;
  }
}

// sum_i l_i y_i, block sums
__global__ void __launch_bounds__(256) dot_kernel(const double* __restrict__ l, const double* __restrict__ y,
                                                  int64_t n, double* __restrict__ part) {
  double acc = 0.0;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) acc = fma(l[i], y[i], acc);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  __shared__ double sh[8];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sh[q];
    part[blockIdx.x] = t;
  }
}

int nblocks(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 4));
}

}  // namespace

void ensure_state_map(Op& op);

// the chain's tangent products by betaJ, kappa and (BNNNI) kappa2, each handed
// to `take` before the next overwrites y (tm_aux.cu)
void matvec_aux_tangents(const Op& op, const double* x, double* y, cudaStream_t s,
                         const std::function<void(int)>& take);
// v^T (dTh / dK) v of the Kronecker factor, block sums (tm_core.cu)
int64_t kron_power(const Op& op, const double* x, DBuf& part, cudaStream_t s);

// Aux-bit operators (DNNI, diagonal BNNNI): T = D_out C D_in with the
// diagonal Boltzmann weights D (Tvec, times dup in the reduced output) and
// the chain C of local step gates built from b1 = e^{+-bJ}, b2 = e^{-+bJ k},
// b3 = e^{-+bJ k2}.  d ln(lambda) = 2 <g>_{lr} + <l, D_out (dC) D_in r> /
// (lambda <l, r>); the second term is a tangent product of the chain
// (matvec_aux_tangents) per parameter the gates depend on.
// (the partial sums of every term come back in one copy)
void adjoint_grad(const Op& op, const double* qr_h, const double* ql_h, double lam, double grad[4]) {
  const bool aux = (op.kind == K_ZBT || op.kind == K_ZBM || op.kind == K_XDT || op.kind == K_XDM);
  if (op.kind != K_XAT && op.kind != K_XAM && op.kind != K_XAM3 && !aux)
    fail(TM_ERR_UNSUPPORTED, "adjoint provided for the x-ANNNI, DNNI and diagonal BNNNI operators");
  cudaStream_t s = op.stream;
  const int64_t n = op.n;
  const bool reduced = (op.kind == K_XAM || op.kind == K_XAM3 || op.kind == K_ZBM || op.kind == K_XDM);
  DBuf dqr, dql, part;
  dqr.alloc((size_t)n * 8);
  TM_CK(cudaMemcpyAsync(dqr.p, qr_h, (size_t)n * 8, cudaMemcpyHostToDevice, s));
  const double* qlp = nullptr;
  if (ql_h) {
    dql.alloc((size_t)n * 8);
    TM_CK(cudaMemcpyAsync(dql.p, ql_h, (size_t)n * 8, cudaMemcpyHostToDevice, s));
    qlp = dql.as<double>();
  }
  GradParams gp{op.kind, op.L, op.size1, op.size2, op.boundary, op.mp.betaJ, op.mp.kappa, op.mp.kappa2, op.mp.h};
  const int nb = nblocks(n);
  part.alloc((size_t)nb * 8 * 8);  // 5 sums per block, then up to 3 quadratic forms
  diag_grad_kernel<<<nb, 256, 0, s>>>(gp, dqr.as<double>(), qlp, reduced ? op.idx.as<uint32_t>() : nullptr, n,
                                      part.as<double>());
  TM_CKK("diag_grad");
  const int nquad = !aux ? 1 : (op.kind == K_ZBT || op.kind == K_ZBM) ? 3 : 2;  // DNNI gates: no kappa2
  std::vector<double> hp((size_t)nb * 5), hq;
  DBuf quad;
  int64_t per = nb;  // partial sums per quadratic form
  if (aux) {
    DBuf y;
    y.alloc((size_t)n * 8);
    matvec_aux_tangents(op, dqr.as<double>(), y.as<double>(), s, [&](int t) {
      dot_kernel<<<nb, 256, 0, s>>>(qlp ? qlp : dqr.as<double>(), y.as<double>(), n,
                                    part.as<double>() + (size_t)nb * (5 + t));
      TM_CKK("grad_dot");
    });
    hp.resize((size_t)nb * (5 + nquad));
  } else {
    if (reduced) ensure_state_map(const_cast<Op&>(op));
    per = kron_power(op, dqr.as<double>(), quad, s);
    hq.resize((size_t)per);
    TM_CK(cudaMemcpyAsync(hq.data(), quad.p, hq.size() * 8, cudaMemcpyDeviceToHost, s));
  }
  TM_CK(cudaMemcpyAsync(hp.data(), part.p, hp.size() * 8, cudaMemcpyDeviceToHost, s));
  TM_CK(cudaStreamSynchronize(s));
  double sums[5] = {0, 0, 0, 0, 0};
  for (int b = 0; b < nb; ++b)
    for (int k = 0; k < 5; ++k) sums[k] += hp[(size_t)b * 5 + k];
  const double wsum = sums[4];
  for (int k = 0; k < 4; ++k) grad[k] = 2.0 * sums[k] / wsum;
  const double pc = (op.kind == K_XAT) ? op.normfactor : 1.0;
  for (int t = 0; t < nquad; ++t) {
    const double* h = aux ? hp.data() + (size_t)nb * (5 + t) : hq.data();
    double q = 0.0;
    for (int64_t b = 0; b < per; ++b) q += h[b];
    grad[t] += pc * q / (lam * wsum);
  }
}

}  // namespace ltm
