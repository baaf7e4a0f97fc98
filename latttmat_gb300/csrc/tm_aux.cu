// Aux-bit transfer-matrix cores: DNNI (one carried bit) and diagonal
// BNNNI+3NN (two carried bits), full operators and their reduced forms.
//
// DNNI (XDTMatVecProd2D, TMat/tmat.cpp:322-476): the inter-layer factor couples
// each new spin to three old ones (same site and both diagonals), so it is
// swept site by site with the previous old spin carried in an auxiliary bit.
// The diagonal BNNNI TM (ZBTMatVecProd2D, TMat/tmat.cpp:480-662) sweeps two
// sites per step with two carried bits; its transpose swaps the roles of the
// coupling factors (optdirection = 1).
//
// Undoing the reference's rotation of the state after every step leaves local
// gates in a fixed frame: step t rewrites the carried letter and the letter
// (one or two sites) at its position, with weights that depend on the next old
// letter (at the end of the ring, on the first one: everything runs once per
// value of it, the "lastbit").  Here the ring is walked from the top of the state
// down, so that
//   - a prefix of the new state is known after every step, and a reduced
//     operator keeps only the prefixes that lead to an orbit's smallest state
//     (tm_tree.cu): at L = 24 (BNNNI) a third of the elements are left after
//     four of the twelve steps and a sixth after seven;
//   - the remaining old bits stay contiguous, whatever the prefixes are.
// A pass keeps a tile of 2^10..2^14 elements (some letters, a contiguous chunk
// of the bits below them, the carried letter) in shared memory for several
// steps; the first pass builds its tiles from x with the first step already
// applied (the carried letter has one value per state there), the last holds
// all lastbit values of a node, sums them and the carried letters and writes
// y.  A step takes two
// multiply-adds and one multiply per output (BNNNI; one and one for DNNI)
// through factored tables (ChainTab).  FP32 and double-float steps are scaled
// by the inverse of their largest row sum; the product of the scales is
// applied at the output.
#include <algorithm>
#include <cmath>
#include <functional>
#include <type_traits>
#include <vector>

#include "tm_chain.h"
#include "tm_df.cuh"
#include "tm_internal.h"

namespace ltm {

namespace {

int grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)num_sms() * 32));
}

// x + rho y in the chain's arithmetic (double-float: renormalised by the
// multiply that follows)
__device__ __forceinline__ float xpry(float rho, float y, float x) { return fmaf(rho, y, x); }
__device__ __forceinline__ double xpry(double rho, double y, double x) { return fma(rho, y, x); }
__device__ __forceinline__ dfloat xpry(dfloat rho, dfloat y, dfloat x) { return df_fma_unnorm(rho, y, x); }
__device__ __forceinline__ tangent xpry(tangent rho, tangent y, tangent x) { return x + rho * y; }

// element type of the pre-scaled input vector u (tangent: its value)
template <class T>
struct ChainIn {
  using U = T;
};
template <>
struct ChainIn<tangent> {
  using U = dfloat;
};
__device__ __forceinline__ void to_elem(float u, float& v) { v = u; }
__device__ __forceinline__ void to_elem(double u, double& v) { v = u; }
__device__ __forceinline__ void to_elem(dfloat u, dfloat& v) { v = u; }
__device__ __forceinline__ void to_elem(dfloat u, tangent& v) { v = tangent(u, dfloat(0.f, 0.f)); }

// x times its FP64 weight in the chain's arithmetic
__device__ __forceinline__ void weigh_in(float x, double t, float& v) { v = scale_round(x, t); }
__device__ __forceinline__ void weigh_in(double x, double t, float& v) { v = (float)(x * t); }
__device__ __forceinline__ void weigh_in(double x, double t, double& v) { v = x * t; }
__device__ __forceinline__ void weigh_in(double x, double t, dfloat& v) { v = dfloat(x * t); }
__device__ __forceinline__ void weigh_in(double x, double t, tangent& v) { v = tangent(x * t); }

// fold: sums of the carried letters and lastbit passes, without the FP64 pipe
// except in FP64 (double-float keeps 48 bits; FP32 values sum exactly enough)
template <class T>
struct FoldAcc {
  using A = dfloat;
};
template <>
struct FoldAcc<double> {
  using A = double;
};
__device__ __forceinline__ dfloat fold_add(dfloat a, float x) { return a + dfloat(x, 0.f); }
__device__ __forceinline__ double fold_add(double a, double x) { return a + x; }
__device__ __forceinline__ dfloat fold_add(dfloat a, dfloat x) { return a + x; }
__device__ __forceinline__ dfloat fold_add(dfloat a, tangent x) { return a + x.d; }

// ------------------------------------------------------------------ tile slots
// A slot holds the S values of the carried letter.  It is kept as 16-byte (8
// for DNNI in FP32) vectors, each in a plane of its own: neighbouring slots
// are then neighbouring vectors, where whole 32-byte slots would use half the
// banks per access.  Vector i of a plane sits at i + i / 8 (8-byte
// vectors: i + i / 16), one pad per 128 bytes, so that strided letters spread
// over the banks, and planes are 64 bytes apart modulo 128.  Double-float
// slots are planar (hi words, then lo words), the order the packed FP32 lanes
// take them in.
template <class T, int S>
struct SlotT {
  static constexpr int kBytes = S * (int)sizeof(T);
  using V = typename std::conditional<kBytes == 8, uint2, uint4>::type;
  static constexpr int kVecs = kBytes / (int)sizeof(V);
  static constexpr int kShift = (kBytes == 8) ? 4 : 3;
};

__host__ __device__ __forceinline__ int slot_plane(int slots, int slot_bytes) {
  const int n = slots + (slots >> (slot_bytes == 8 ? 4 : 3));
  return slot_bytes <= 16 ? n : ((n + 7) & ~7) + 4;
}

// vector k of slot i
template <class T, int S>
__device__ __forceinline__ typename SlotT<T, S>::V* slot_vec(unsigned char* sm, int plane, int i, int k) {
  return reinterpret_cast<typename SlotT<T, S>::V*>(sm) + k * plane + i + (i >> SlotT<T, S>::kShift);
}

// a slot in a pass buffer (its vectors are consecutive there)
template <class T, int S>
__device__ __forceinline__ void vec_to_slot(const typename SlotT<T, S>::V (&raw)[SlotT<T, S>::kVecs], T (&v)[S]) {
  if constexpr (std::is_same<T, dfloat>::value) {
    const float* f = reinterpret_cast<const float*>(raw);
#pragma unroll
    for (int q = 0; q < S; ++q) v[q] = dfloat(f[q], f[S + q]);
  } else {
    const T* e = reinterpret_cast<const T*>(raw);
#pragma unroll
    for (int q = 0; q < S; ++q) v[q] = e[q];
  }
}
template <class T, int S>
__device__ __forceinline__ void slot_to_vec(const T (&v)[S], typename SlotT<T, S>::V (&raw)[SlotT<T, S>::kVecs]) {
  if constexpr (std::is_same<T, dfloat>::value) {
    float* f = reinterpret_cast<float*>(raw);
#pragma unroll
    for (int q = 0; q < S; ++q) {
      f[q] = v[q].hi;
      f[S + q] = v[q].lo;
    }
  } else {
    T* e = reinterpret_cast<T*>(raw);
#pragma unroll
    for (int q = 0; q < S; ++q) e[q] = v[q];
  }
}

template <class T, int S>
__device__ __forceinline__ void slot_ld(unsigned char* sm, int plane, int i, T (&v)[S]) {
  typename SlotT<T, S>::V raw[SlotT<T, S>::kVecs];
#pragma unroll
  for (int k = 0; k < SlotT<T, S>::kVecs; ++k) raw[k] = *slot_vec<T, S>(sm, plane, i, k);
  vec_to_slot<T, S>(raw, v);
}

template <class T, int S>
__device__ __forceinline__ void slot_st(unsigned char* sm, int plane, int i, const T (&v)[S]) {
  typename SlotT<T, S>::V raw[SlotT<T, S>::kVecs];
  slot_to_vec<T, S>(v, raw);
#pragma unroll
  for (int k = 0; k < SlotT<T, S>::kVecs; ++k) *slot_vec<T, S>(sm, plane, i, k) = raw[k];
}

// ------------------------------------------------------------------ steps
// DNNI: RL consecutive letters (top first) of a thread's 2^RL slots.  The
// letter after each is the next one of the group, or `ctl` after the last.
template <class T, int RL>
__device__ __forceinline__ void dnni_steps(T (&v)[1 << RL][2], const ChainTab<T>& tab, int ctl) {
  const T rho = tab.rho1;
#pragma unroll
  for (int j = 0; j < RL; ++j) {
    const int bit = 1 << (RL - 1 - j);
#pragma unroll
    for (int w = 0; w < (1 << RL); ++w) {
      if (w & bit) continue;
      const int c = (j < RL - 1) ? ((w >> (RL - 2 - j)) & 1) : ctl;
      const T* z = tab.zu + c * 4;
      T in[2][2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        in[0][q] = v[w][q];
        in[1][q] = v[w | bit][q];
      }
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        v[w][a] = z[a] * xpry(rho, in[a][1], in[a][0]);
        v[w | bit][a] = z[2 + a] * xpry(rho, in[a][0], in[a][1]);
      }
    }
  }
}

// BNNNI: one letter; v[a'][q] in, v[s'][a'] out
template <class T>
__device__ __forceinline__ void bnnni_step(T (&v)[4][4], const ChainTab<T>& tab, int ctl) {
  T out[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const T* z = tab.zu + ctl * 16 + a * 4;
    T t[2][2];
#pragma unroll
    for (int qr = 0; qr < 2; ++qr) {
      t[0][qr] = xpry(tab.rho1, v[a][2 + qr], v[a][qr]);
      t[1][qr] = xpry(tab.rho1, v[a][qr], v[a][2 + qr]);
    }
#pragma unroll
    for (int sv = 0; sv < 4; ++sv) out[sv][a] = z[sv] * xpry(tab.rho2[sv], t[sv >> 1][1], t[sv >> 1][0]);
  }
#pragma unroll
  for (int sv = 0; sv < 4; ++sv)
#pragma unroll
    for (int a = 0; a < 4; ++a) v[sv][a] = out[sv][a];
}

// Shared-memory step tables of a block: the ChainTab, and for double-float
// BNNNI also its planar form for the packed lanes.
template <class T>
struct ChainSh {
  ChainTab<T> tab;
  T two[64];  // first pass: zu[c][s', a'] w2[s'][lb] of the second step, [c][s'][a']
};
struct ChainShDF {
  ChainTab<dfloat> tab;
  dfloat two[64];
  float2 zh[32], zl[32];  // [c][a'][s' pair]
  float2 r2h[2], r2l[2];  // [sl]: (sr = 0, 1)
};

// bnnni_step on the packed FP32 lanes: the two-term sums over ql pair the
// values of qr, those over qr pair the results of sr.  31 packed operations
// per output pair, as the scalar sequence would take per output.
__device__ __forceinline__ void bnnni_step_df(float4 (&h)[4], float4 (&l)[4], const ChainShDF& sh, int ctl) {
  const dfloat r1 = sh.tab.rho1;
  const float2 rh = make_float2(r1.hi, r1.hi), rl = make_float2(r1.lo, r1.lo), rn = make_float2(-r1.hi, -r1.hi);
  float oh[4][4], ol[4][4];  // [s'][a']
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const float2 h0 = make_float2(h[a].x, h[a].y), h1 = make_float2(h[a].z, h[a].w);
    const float2 l0 = make_float2(l[a].x, l[a].y), l1 = make_float2(l[a].z, l[a].w);
    float2 th[2], tl[2];
    df2_fma_unnorm(rh, rl, rn, h1, l1, h0, l0, th[0], tl[0]);
    df2_fma_unnorm(rh, rl, rn, h0, l0, h1, l1, th[1], tl[1]);
#pragma unroll
    for (int sl = 0; sl < 2; ++sl) {
      const float2 qh = sh.r2h[sl], ql = sh.r2l[sl];
      float2 dh, dl;
      df2_fma_unnorm(qh, ql, make_float2(-qh.x, -qh.y), make_float2(th[sl].y, th[sl].y),
                     make_float2(tl[sl].y, tl[sl].y), make_float2(th[sl].x, th[sl].x),
                     make_float2(tl[sl].x, tl[sl].x), dh, dl);
      const int k = ctl * 8 + a * 2 + sl;
      float2 ph, pl;
      df2_mul(dh, dl, sh.zh[k], sh.zl[k], ph, pl);
      oh[2 * sl][a] = ph.x;
      oh[2 * sl + 1][a] = ph.y;
      ol[2 * sl][a] = pl.x;
      ol[2 * sl + 1][a] = pl.y;
    }
  }
#pragma unroll
  for (int sv = 0; sv < 4; ++sv) {
    h[sv] = make_float4(oh[sv][0], oh[sv][1], oh[sv][2], oh[sv][3]);
    l[sv] = make_float4(ol[sv][0], ol[sv][1], ol[sv][2], ol[sv][3]);
  }
}

template <class T, int KS>
using ChainShared = typename std::conditional<std::is_same<T, dfloat>::value && KS == 2, ChainShDF, ChainSh<T>>::type;

// the block's step tables from global (or parameter) memory
template <class T, int KS>
__device__ __forceinline__ void chain_tables(ChainShared<T, KS>& sh, const ChainTab<T>& tab) {
  constexpr int n = (int)(sizeof(ChainTab<T>) / 4);
  for (int k = threadIdx.x; k < n; k += blockDim.x)
    reinterpret_cast<uint32_t*>(&sh.tab)[k] = reinterpret_cast<const uint32_t*>(&tab)[k];
  if constexpr (std::is_same<T, dfloat>::value && KS == 2) {
    for (int k = threadIdx.x; k < 32; k += blockDim.x) {
      const dfloat a = tab.zu[2 * k], b = tab.zu[2 * k + 1];
      sh.zh[k] = make_float2(a.hi, b.hi);
      sh.zl[k] = make_float2(a.lo, b.lo);
    }
    for (int k = threadIdx.x; k < 2; k += blockDim.x) {
      const dfloat a = tab.rho2[2 * k], b = tab.rho2[2 * k + 1];
      sh.r2h[k] = make_float2(a.hi, b.hi);
      sh.r2l[k] = make_float2(a.lo, b.lo);
    }
  }
}

// Buffers of one product.
template <class T, class IO>
struct ChainIO {
  const T* src;        // previous pass's output
  T* dst;              // this pass's output
  const typename ChainIn<T>::U* u;  // first pass: input times Tvec, or null:
  const IO* x;         //   x * pre
  const double* pre;
  const uint32_t* smap;  // reduced: state -> row
  IO* y;               // last pass
  const double* tv;    //   y = sum * tv [* dup] * post
  const uint16_t* dup;
  ScaleF post;
};

// letters per round held in registers
template <class T, int KS>
struct RoundLetters {
  static constexpr int value = (KS == 2) ? 1 : (sizeof(T) == 4 ? 3 : (sizeof(T) == 8 ? 2 : 1));
};

// What a round needs beside the tile.
template <class T, class IO>
struct RoundArgs {
  const ChainIO<T, IO>* io;
  uint64_t src0, dst0;   // slots: (lb, node) base of the source (lb: last passes add it) and destination
  uint64_t src_lb;       // slots per lastbit value in the source (last passes)
  uint64_t out0;         // first child node of the tile (full operators)
  uint64_t low0;         // the block's outer old bits
  int end_ctl;           // letter after the product's last one (-1: the lastbit value)
  const uint2* nodes;    // tree: the round's nodes (children known), or null
};

enum { kRoundIn = 1, kRoundOut = 2 };

// One round on RL letters from depth d of the pass; the words of depth d are
// nodes [0, cnt) from `words` (full operators: 0 .. cnt - 1).  IN: the slots
// come straight from the previous pass's buffer; OUT: they go straight to this
// pass's buffer; otherwise both stay in the shared-memory tile.  A pass's
// first and last rounds skip it that way: one write and one read of the
// traffic through shared memory, which with the instructions that move it
// bounds the FP32 passes, are saved at each end (the second DNNI pass at
// L = 26 took 0.61 ms with the tile at both ends, 0.53 ms so).  The last pass
// keeps the tile for its sums: summed in registers and over lanes, with
// strided outputs, it took 1.03 ms against 0.86 ms.
template <class T, int KS, int RL, int IOF, class IO>
__device__ __forceinline__ void chain_round(unsigned char* sm, int plane, const ChainShared<T, KS>& sh,
                                            const ChainPass& cp, int d, const uint16_t* __restrict__ words, int cnt,
                                            const RoundArgs<T, IO>& A) {
  constexpr int S = 1 << KS, W = 1 << (KS * RL);
  using V = typename SlotT<T, S>::V;
  constexpr int kVecs = SlotT<T, S>::kVecs;
  constexpr bool kPacked = std::is_same<T, dfloat>::value && KS == 2;
  const int bl = KS * (cp.T - d - RL) + cp.tb;  // tile bits below the round's letters
  const int wmask = (1 << (KS * d)) - 1, tmask = (1 << cp.tb) - 1;
  const bool inside = d + RL < cp.T;
  const int total = cnt << bl;
  // (whole lastbit groups stay together: total is a multiple of 2^tb)
  for (int gi = threadIdx.x; gi < total; gi += blockDim.x) {
    const int pi = gi >> bl, lo = gi & ((1 << bl) - 1);
    const int p = words ? ((int)__ldg(words + pi) & wmask) : pi;
    const int base = (p << (KS * RL + bl)) | lo;
    int ctl;
    if (inside)
      ctl = (lo >> (bl - KS)) & (S - 1);
    else if (cp.last)
      ctl = A.end_ctl < 0 ? lo & (S - 1) : A.end_ctl;
    else
      ctl = (int)((A.low0 | (uint64_t)(lo & tmask)) >> (cp.rest - KS)) & (S - 1);
    T v[W][S];
    float4 h[4], l[4];
    if constexpr ((IOF & kRoundIn) != 0) {
      const uint64_t at = A.src0 + ((uint64_t)(lo >> cp.tb) << cp.rest) +
                          (cp.last ? (uint64_t)(lo & tmask) * A.src_lb : (uint64_t)(lo & tmask));
      const V* src = reinterpret_cast<const V*>(A.io->src) + at * kVecs;
      const int sh_w = KS * (cp.T - RL) + cp.rest;  // (d = 0)
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const V* q = src + (((uint64_t)w << sh_w) * kVecs);
        if constexpr (kPacked) {
          h[w] = *reinterpret_cast<const float4*>(q);
          l[w] = *reinterpret_cast<const float4*>(q + 1);
        } else {
          V raw[kVecs];
#pragma unroll
          for (int k = 0; k < kVecs; ++k) raw[k] = q[k];
          vec_to_slot<T, S>(raw, v[w]);
        }
      }
    } else {
#pragma unroll
      for (int w = 0; w < W; ++w) {
        if constexpr (kPacked) {
          h[w] = *reinterpret_cast<const float4*>(slot_vec<T, 4>(sm, plane, base | (w << bl), 0));
          l[w] = *reinterpret_cast<const float4*>(slot_vec<T, 4>(sm, plane, base | (w << bl), 1));
        } else {
          slot_ld<T, S>(sm, plane, base | (w << bl), v[w]);
        }
      }
    }
    if constexpr (kPacked)
      bnnni_step_df(h, l, sh, ctl);
    else if constexpr (KS == 1)
      dnni_steps<T, RL>(v, sh.tab, ctl);
    else
      bnnni_step<T>(v, sh.tab, ctl);
    if constexpr ((IOF & kRoundOut) != 0) {
      // bl = tb here; the children of word p: consecutive in a full operator,
      // those of its mask in a tree (one letter per round)
      uint2 nd = make_uint2(0u, ~0u);
      if (A.nodes) nd = __ldg(A.nodes + pi);
      const uint64_t first = A.nodes ? (uint64_t)nd.x : A.out0 + ((uint64_t)p << (KS * RL));
#pragma unroll
      for (int w = 0; w < W; ++w) {
        if (!((nd.y >> w) & 1u)) continue;
        const uint64_t child = first + (A.nodes ? (uint64_t)__popc(nd.y & ((1u << w) - 1u)) : (uint64_t)w);
        V* q = reinterpret_cast<V*>(A.io->dst) + (A.dst0 + (child << cp.rest) + (uint64_t)(lo & tmask)) * kVecs;
        if constexpr (kPacked) {
          *reinterpret_cast<float4*>(q) = h[w];
          *reinterpret_cast<float4*>(q + 1) = l[w];
        } else {
          V raw[kVecs];
          slot_to_vec<T, S>(v[w], raw);
#pragma unroll
          for (int k = 0; k < kVecs; ++k) q[k] = raw[k];
        }
      }
    } else {
#pragma unroll
      for (int w = 0; w < W; ++w) {
        if constexpr (kPacked) {
          *reinterpret_cast<float4*>(slot_vec<T, 4>(sm, plane, base | (w << bl), 0)) = h[w];
          *reinterpret_cast<float4*>(slot_vec<T, 4>(sm, plane, base | (w << bl), 1)) = l[w];
        } else {
          slot_st<T, S>(sm, plane, base | (w << bl), v[w]);
        }
      }
    }
  }
  if constexpr ((IOF & kRoundOut) == 0) __syncthreads();
}

// a round of RL letters or the fewer that are left, by where its slots are
template <class T, int KS, int RL, class IO>
__device__ __forceinline__ void chain_round_n(int n, int iof, unsigned char* sm, int plane,
                                              const ChainShared<T, KS>& sh, const ChainPass& cp, int d,
                                              const uint16_t* words, int cnt, const RoundArgs<T, IO>& A) {
  if constexpr (RL > 1) {
    if (n < RL) {
      chain_round_n<T, KS, RL - 1, IO>(n, iof, sm, plane, sh, cp, d, words, cnt, A);
      return;
    }
  }
  switch (iof) {
    case 0: chain_round<T, KS, RL, 0, IO>(sm, plane, sh, cp, d, words, cnt, A); break;
    case 1: chain_round<T, KS, RL, 1, IO>(sm, plane, sh, cp, d, words, cnt, A); break;
    case 2: chain_round<T, KS, RL, 2, IO>(sm, plane, sh, cp, d, words, cnt, A); break;
    default: chain_round<T, KS, RL, 3, IO>(sm, plane, sh, cp, d, words, cnt, A); break;
  }
}

constexpr int kChainMaxT = 16;  // letters of a pass

// The first two steps of a closed ring applied to x.  After the first one the
// carried letter of a state is its top letter (the lastbit value lb), so the
// second step's sum has one term too:
//   out(s'_0, s'_1; a' = a) = zu[c][s'_1, a] w1[s'_1][lb]
//                             zu[a][s'_0, lb] w1[s'_0][q] x(lb, a, below)
// with q the bottom letter and c the third.  A thread forms all words s'_0
// s'_1 (those of the mask) of one `below` from its S states.  Against a first
// step at the load and a full second step this took 0.31 of 1.01 ms off the
// first BNNNI pass at L = 24 in double-float.
template <class T, int KS, class IO>
__device__ __forceinline__ void chain_first_two(unsigned char* sm, int plane, const ChainIO<T, IO>& io,
                                                const ChainShared<T, KS>& sh, const ChainPass& cp, int L, int lb0,
                                                uint64_t low0, uint32_t allowed) {
  constexpr int S = 1 << KS;
  const int fb = KS * (cp.T - 2) + cp.tb;
  const int tmask = (1 << cp.tb) - 1;
  // (small tiles: a thread per s'_0, so that all threads have work)
  const bool split = (1 << fb) < (int)blockDim.x;
  for (int item = threadIdx.x; item < (split ? S << fb : 1 << fb); item += blockDim.x) {
    const int e = item & ((1 << fb) - 1);
    const int lb = cp.last ? e & tmask : lb0;
    const uint64_t below = ((uint64_t)(e >> cp.tb) << cp.rest) | (cp.last ? 0ull : low0 | (uint64_t)(e & tmask));
    T x[S];
    if (io.u) {
      uint64_t at[S];
#pragma unroll
      for (int a = 0; a < S; ++a) {
        const uint64_t r = ((uint64_t)lb << (L - KS)) | ((uint64_t)a << (L - 2 * KS)) | below;
        at[a] = io.smap ? io.smap[r] : r;
      }
#pragma unroll
      for (int a = 0; a < S; ++a) to_elem(io.u[at[a]], x[a]);
    } else if (io.smap) {
      uint32_t at[S];
#pragma unroll
      for (int a = 0; a < S; ++a)
        at[a] = io.smap[((uint64_t)lb << (L - KS)) | ((uint64_t)a << (L - 2 * KS)) | below];
#pragma unroll
      for (int a = 0; a < S; ++a) weigh_in(io.x[at[a]], io.pre[at[a]], x[a]);
    } else {
#pragma unroll
      for (int a = 0; a < S; ++a) {
        const uint64_t r = ((uint64_t)lb << (L - KS)) | ((uint64_t)a << (L - 2 * KS)) | below;
        weigh_in(io.x[r], io.pre[r], x[a]);
      }
    }
    const int c = (int)(below >> (L - 3 * KS)) & (S - 1);  // (three letters at least: the caller)
    for (int s0 = split ? item >> fb : 0; s0 < (split ? (item >> fb) + 1 : S); ++s0) {
      if (!((allowed >> (s0 * S)) & ((1u << S) - 1u))) continue;
      T xa[S];
#pragma unroll
      for (int a = 0; a < S; ++a) {
        const int q = (int)below & (S - 1);
        xa[a] = sh.tab.zu[a * S * S + (KS == 1 ? s0 * S + lb : lb * S + s0)] * (sh.tab.w1[s0 * S + q] * x[a]);
      }
#pragma unroll
      for (int s1 = 0; s1 < S; ++s1) {
        if (!((allowed >> (s0 * S + s1)) & 1u)) continue;
        T o[S];
#pragma unroll
        for (int a = 0; a < S; ++a) {
          if (cp.last)
            o[a] = sh.tab.zu[c * S * S + (KS == 1 ? s1 * S + a : a * S + s1)] * (sh.tab.w2[s1 * S + lb] * xa[a]);
          else
            o[a] = sh.two[c * S * S + s1 * S + a] * xa[a];
        }
        slot_st<T, S>(sm, plane, ((s0 * S + s1) << fb) | e, o);
      }
    }
  }
}

// The fold of word w in FP64, for sums that leave the FP32 exponent range (two
// FP32 words make a NaN of an infinite sum).  Not inlined: see scale_round_f64.
__device__ __forceinline__ double part64(float x) { return x; }
__device__ __forceinline__ double part64(double x) { return x; }
__device__ __forceinline__ double part64(dfloat x) { return (double)x; }
__device__ __forceinline__ double part64(tangent x) { return (double)x.d; }
template <class T, int S>
static __device__ __noinline__ double fold_f64(unsigned char* sm, int plane, int slot0, int nlb) {
  double a = 0.0;
  for (int t = 0; t < nlb; ++t) {
    T v[S];
    slot_ld<T, S>(sm, plane, slot0 | t, v);
    for (int q = 0; q < S; ++q) a += part64(v[q]);
  }
  return a;
}
__device__ __forceinline__ bool fold_ok(dfloat a) { return fabsf(a.hi) < 3e38f; }
__device__ __forceinline__ bool fold_ok(double) { return true; }

// One block of a pass (the tables in sh are loaded and synchronised).
//   KS = 1: DNNI (permute_mult_T1 / _last, TMat/tmat.cpp:344-376); KS = 2:
//   diagonal BNNNI (TMat/tmat.cpp:521-588).
// bc: 0 closed ring; 5, 9: DNNI open boundaries (TMat/tmat.cpp:392-457), the
// sites beyond the ends fixed to 0 (9: to 1 below site 0).
template <class T, int KS, class IO>
__device__ __forceinline__ void chain_block(const ChainIO<T, IO>& io, ChainShared<T, KS>& sh, const ChainPass& cp,
                                            const TreeDev& tr, int L, int bc, uint64_t blk) {
  constexpr int S = 1 << KS, RL = RoundLetters<T, KS>::value;
  using Acc = typename FoldAcc<T>::A;
  using V = typename SlotT<T, S>::V;
  constexpr int kVecs = SlotT<T, S>::kVecs;
  extern __shared__ __align__(16) unsigned char sm[];
  const int wbits = KS * cp.T;
  const int plane = slot_plane(1 << (wbits + cp.tb), SlotT<T, S>::kBytes);
  __shared__ uint32_t rg0[kChainMaxT + 1], rgn[kChainMaxT + 1];
  // block -> (lb, node, outer old bits)
  const int ob = cp.rest - cp.cb;
  const uint64_t low0 = (blk & ((1ull << ob) - 1)) << cp.cb;
  const uint64_t nl = blk >> ob;
  const int lb_outer = cp.last ? 0 : (int)(nl / (uint64_t)cp.nin);
  const uint64_t node = nl - (uint64_t)lb_outer * (uint64_t)cp.nin;
  const bool tree = tr.nodes != nullptr;
  if (threadIdx.x == 0) {
    // (one range per turn, written at the turn's end: with the first range
    // written inside the loop and a break at its end, nvcc 13.0 stored the
    // ranges of one instantiation one place too far)
    uint32_t r0 = (uint32_t)node, r1 = r0 + 1;
    rg0[0] = r0;
    rgn[0] = 1;
#pragma unroll 1
    for (int j = 1; j <= cp.T; ++j) {
      if (tree) {
        const uint2* nd = tr.nodes + tr.off[cp.t0 + j - 1];
        const uint2 a = nd[r0], b = nd[r1 - 1];
        r0 = a.x;
        r1 = b.x + __popc(b.y);
      } else {
        r0 = 0;
        r1 = 1u << (KS * j);
      }
      rg0[j] = r0;
      rgn[j] = r1 - r0;
    }
  }
  const int tmask = (1 << cp.tb) - 1;
  const bool two = cp.first && bc == 0 && cp.T >= (cp.last ? 3 : 2);
  if (two) {
    __shared__ uint32_t allowed;  // words of the first two letters
    if (threadIdx.x == 0) {
      uint32_t m = 0;
      if (tree) {
        const uint2 root = tr.nodes[tr.off[0]];
        for (int s0 = 0, k = 0; s0 < S; ++s0)
          if ((root.y >> s0) & 1u) m |= tr.nodes[tr.off[1] + root.x + k++].y << (s0 * S);
      } else {
        m = S == 4 ? 0xffffu : 0xfu;
      }
      allowed = m;
    }
    if (!cp.last)
      for (int k = threadIdx.x; k < S * S * S; k += blockDim.x) {
        const int c = k / (S * S), s1 = (k / S) % S, a = k % S;
        sh.two[k] = sh.tab.zu[c * S * S + (KS == 1 ? s1 * S + a : a * S + s1)] * sh.tab.w2[s1 * S + lb_outer];
      }
    __syncthreads();
    chain_first_two<T, KS, IO>(sm, plane, io, sh, cp, L, lb_outer, low0, allowed);
  } else if (cp.first) {
    // The first step applied to x: the carried letter of state r is its
    // bottom letter, the ring's first old letter is its top one (closed: the
    // lastbit value), which becomes the carried letter.  Two states per
    // thread and turn, so that their gathers are in flight together.
    const int fb = KS * (cp.T - 1) + cp.tb;  // tile bits below the first letter
    constexpr int A0 = S;
    for (int e0 = threadIdx.x; e0 < (1 << fb); e0 += 2 * blockDim.x) {
      uint64_t below[2];
      T v[2][A0];
      const int na = bc == 0 ? 1 : S;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = e0 + h * (int)blockDim.x;
        const int k = e & tmask;
        below[h] = ((uint64_t)(e >> cp.tb) << cp.rest) | (cp.last ? 0ull : low0 | (uint64_t)k);
      }
      if (io.u) {
        uint64_t at[2][A0];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int a = 0; a < A0; ++a) {
            const int e = e0 + h * (int)blockDim.x;
            if (e < (1 << fb) && a < na) {
              const int top = bc ? a : (cp.last ? e & tmask : lb_outer);
              const uint64_t r = ((uint64_t)top << (L - KS)) | below[h];
              at[h][a] = io.smap ? io.smap[r] : r;
            }
          }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int a = 0; a < A0; ++a)
            if (e0 + h * (int)blockDim.x < (1 << fb) && a < na) to_elem(io.u[at[h][a]], v[h][a]);
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int a = 0; a < A0; ++a) {
            const int e = e0 + h * (int)blockDim.x;
            if (e < (1 << fb) && a < na) {
              const int top = bc ? a : (cp.last ? e & tmask : lb_outer);
              const uint64_t r = ((uint64_t)top << (L - KS)) | below[h];
              const uint64_t at = io.smap ? io.smap[r] : r;
              weigh_in(io.x[at], io.pre[at], v[h][a]);
            }
          }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = e0 + h * (int)blockDim.x;
        if (e >= (1 << fb)) break;
        const int c = (int)(below[h] >> (L - 2 * KS)) & (S - 1);
        const int lb = cp.last ? e & tmask : lb_outer;
        int q = (int)(below[h] & (S - 1));
        if (bc) {
#pragma unroll
          for (int a = 0; a < A0; ++a)
            v[h][a] = v[h][a] * (sh.tab.b2[(int)(below[h] & 1) ^ (bc == 9)] * sh.tab.b2[a & 1]);
          q = 0;
        }
#pragma unroll
        for (int sv = 0; sv < S; ++sv) {
          T o[S];
          if (bc == 0) {
            // (one product, then selects: all S carried letters' products
            // would run, predicated or not)
            const T z = sh.tab.zu[c * S * S + (KS == 1 ? sv * S + lb : lb * S + sv)] * (sh.tab.w1[sv * S + q] * v[h][0]);
#pragma unroll
            for (int a = 0; a < S; ++a) o[a] = (a == lb) ? z : T(0);
          } else {
#pragma unroll
            for (int a = 0; a < S; ++a)
              o[a] = sh.tab.zu[c * S * S + (KS == 1 ? sv * S + a : a * S + sv)] * (sh.tab.w1[sv * S + q] * v[h][a]);
          }
          slot_st<T, S>(sm, plane, (sv << fb) | e, o);
        }
      }
    }
  }
  __syncthreads();
  RoundArgs<T, IO> A;
  A.io = &io;
  A.src0 = (((uint64_t)lb_outer * cp.nin + node) << (cp.rest + wbits)) + low0;
  A.src_lb = (uint64_t)cp.nin << (cp.rest + wbits);
  A.dst0 = (((uint64_t)lb_outer * cp.nout) << cp.rest) + low0;
  A.out0 = tree ? 0 : node << wbits;
  A.low0 = low0;
  A.end_ctl = bc == 0 ? -1 : (bc == 9 ? 1 : 0);
  // a tree's children are looked up one letter at a time: its last round has
  // one letter
  const int d0 = two ? 2 : (cp.first ? 1 : 0);
  for (int d = d0; d < cp.T;) {
    const int left = cp.T - d;
    int n = left < RL ? left : RL;
    if (tree && !cp.last && n == left && n > 1) --n;
    const bool out = !cp.last && d + n == cp.T;
    const uint16_t* words = tree ? tr.words + tr.off[cp.t0 + d] + rg0[d] : nullptr;
    A.nodes = (tree && out) ? tr.nodes + tr.off[cp.t0 + d] + rg0[d] : nullptr;
    chain_round_n<T, KS, RL, IO>(n, (d == 0 ? kRoundIn : 0) | (out ? kRoundOut : 0), sm, plane, sh, cp, d, words,
                                 (int)rgn[d], A);
    d += n;
  }
  if (cp.last) {
    const uint16_t* words = tree ? tr.words + tr.off[cp.t0 + cp.T] + rg0[cp.T] : nullptr;
    const uint64_t out0 = tree ? rg0[cp.T] : node << wbits;
    for (int i = threadIdx.x; i < (int)rgn[cp.T]; i += blockDim.x) {
      const int w = words ? ((int)__ldg(words + i) & ((1 << wbits) - 1)) : i;
      Acc acc = Acc(0);
#pragma unroll
      for (int t = 0; t < S; ++t) {
        if (t > tmask) break;
        T v[S];
        slot_ld<T, S>(sm, plane, (w << cp.tb) | t, v);
#pragma unroll
        for (int q = 0; q < S; ++q) acc = fold_add(acc, v[q]);
      }
      const uint64_t r = out0 + i;
      double t = io.tv[r];
      if (io.dup) t *= (double)io.dup[r];
      if (!fold_ok(acc))
        io.y[r] = (IO)(fold_f64<T, S>(sm, plane, w << cp.tb, tmask + 1) * t * io.post.f64);
      else if constexpr (sizeof(IO) == 4)
        io.y[r] = scale_round(acc, t, io.post);
      else
        io.y[r] = (double)acc * t * io.post.f64;
    }
  } else if (d0 == cp.T) {
    // (a pass of the first letters alone: the tile goes out as it is)
    const uint16_t* words = tree ? tr.words + tr.off[cp.t0 + cp.T] + rg0[cp.T] : nullptr;
    const uint64_t out0 = tree ? rg0[cp.T] : node << wbits;
    V* dst = reinterpret_cast<V*>(io.dst) + (A.dst0 + (out0 << cp.rest)) * kVecs;
    for (int e = threadIdx.x; e < ((int)rgn[cp.T] << cp.cb) * kVecs; e += blockDim.x) {
      const int i = e / kVecs, k = e % kVecs;
      const int n = i >> cp.cb;
      const int w = words ? ((int)__ldg(words + n) & ((1 << wbits) - 1)) : n;
      const V raw = *slot_vec<T, S>(sm, plane, (w << cp.cb) | (i & tmask), k);
      dst[(((uint64_t)n << cp.rest) | (uint64_t)(i & tmask)) * kVecs + k] = raw;
    }
  }
}

// Measured at the sizes of the sweep and the full operators, against in-place
// passes of all 2^L states with four multiply-adds and one multiply per
// output: BNNNI (reduced) at L = 24 in double-float 10.1 -> 1.47 ms, DNNI
// (full) at L = 26 in FP32 5.18 -> 2.04 ms.  No unit is at its peak: the three
// double-float passes issue in 48, 47 and 42% of all cycles (FP32 pipe 36, 52
// and 47%, shared memory 52, 47 and 53%, 24% of the warps resident at 124
// registers), the FP32 ones in 68, 72 and 71% (shared memory 38, 47 and 61%,
// memory 33, 50 and 28%).
template <class T>
constexpr int chain_min_blocks() {
  return sizeof(T) == 4 ? 4 : 2;
}

template <class T, int KS, class IO>
__global__ void __launch_bounds__(256, chain_min_blocks<T>())
    chain_kernel(const __grid_constant__ ChainIO<T, IO> io, const __grid_constant__ ChainTab<T> tab,
                 const __grid_constant__ ChainPass cp, const __grid_constant__ TreeDev tr, int L, int bc) {
  __shared__ __align__(16) ChainShared<T, KS> sh;
  chain_tables<T, KS>(sh, tab);
  __syncthreads();
  chain_block<T, KS, IO>(io, sh, cp, tr, L, bc, blockIdx.x);
}

// u = x tvec in the product's arithmetic, for reduced operators above
// kChainFold bits.  Below, the first pass gathers x and the weight of every
// state itself: the 2^L gathers more cost less than a launch there (with a
// scaling launch / without, us: DNNI L = 15 FP32 20.5 / 16.4, L = 17 FP64 43.0 /
// 39.0, BNNNI L = 16 double-float 26.7 / 24.6, L = 18 49.2 / 53.3).
constexpr int kChainFold = 17;
template <class U, class IO>
__global__ void chain_scale_in(const IO* __restrict__ x, const double* __restrict__ tv, U* __restrict__ u, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) {
    U v;
    weigh_in(x[i], tv[i], v);
    u[i] = v;
  }
}

// ------------------------------------------------------------------ batched product
// u of every member in `MODE` (kSweepRows rows per block)
template <class U, int MODE>
__global__ void __launch_bounds__(256) chain_batch_scale_in(const ChainInst* __restrict__ inst,
                                                            const int2* __restrict__ km,
                                                            const int64_t* __restrict__ rstart,
                                                            const int* __restrict__ rmem) {
  const int s_i = rmem[blockIdx.x];  // the member of this row block
  const ChainInst& I = inst[s_i];
  const int2 kmi = km[s_i];
  if (kmi.y != MODE) return;
  const int64_t r0 = ((int64_t)blockIdx.x - rstart[s_i]) * kSweepRows;
  const int64_t r1 = min(r0 + (int64_t)kSweepRows, I.n);
  const double* x = I.V + (int64_t)kmi.x * I.ldv;
  U* u = reinterpret_cast<U*>(I.u);
  for (int64_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    U v;
    weigh_in(x[r], I.tvec[r], v);
    u[r] = v;
  }
}

template <class T, int MODE>
__device__ __forceinline__ const ChainTab<T>* inst_tab(const ChainInst& I, int theta) {
  if constexpr (MODE == kModeF32)
    return &I.c32;
  else if constexpr (MODE == kModeDF)
    return &I.cdf;
  else if constexpr (MODE == kModeTangent)
    return &I.ctan[theta];
  else
    return &I.c64;
}

// One pass over every batch member's tiles: a block takes its member from the
// per-block member map, then runs the same tile body as chain_kernel on
// kBatchTiles consecutive tiles of that member's geometry (copied to shared
// memory).  km[i] = (Krylov column the member extends, product mode).
template <class T, int KS, int MODE>
__global__ void __launch_bounds__(256, chain_min_blocks<T>())
    chain_batch_kernel(const ChainInst* __restrict__ inst, const int2* __restrict__ km, const int64_t* __restrict__ start,
                       const int* __restrict__ bmem, int pass, int theta) {
  __shared__ ChainPass cps;
  __shared__ TreeDev trs;
  __shared__ __align__(16) ChainShared<T, KS> sh;
  const int s_i = bmem[blockIdx.x];  // the member of this block
  const ChainInst& I = inst[s_i];
  const int64_t blk = (int64_t)blockIdx.x - start[s_i];
  const int np = (sizeof(T) == 4) ? I.np4 : (sizeof(T) == 8 ? I.np8 : I.np16);
  const int2 kmi = km[s_i];
  if (kmi.y != MODE || pass >= np) return;  // uniform over the block
  auto copy = [](void* dst, const void* src, int bytes) {
    for (int q = threadIdx.x; q < bytes / 4; q += blockDim.x)
      reinterpret_cast<uint32_t*>(dst)[q] = reinterpret_cast<const uint32_t*>(src)[q];
  };
  copy(&cps, (sizeof(T) == 4) ? &I.p4[pass] : (sizeof(T) == 8 ? &I.p8[pass] : &I.p16[pass]), (int)sizeof(ChainPass));
  copy(&trs, &I.tree, (int)sizeof(TreeDev));
  chain_tables<T, KS>(sh, *inst_tab<T, MODE>(I, theta));
  __syncthreads();
  const int64_t ntiles = ((int64_t)(cps.last ? 1 : cps.nlb) * cps.nin) << (cps.rest - cps.cb);
  ChainIO<T, double> io;
  T* const buf[2] = {reinterpret_cast<T*>(I.P), reinterpret_cast<T*>(trs.nodes ? I.Q : I.P)};
  io.src = buf[(pass + 1) & 1];
  io.dst = buf[pass & 1];
  io.u = reinterpret_cast<const typename ChainIn<T>::U*>(I.u);
  io.x = nullptr;
  io.pre = nullptr;
  io.smap = I.smap;
  io.y = I.w;
  io.tv = I.tvec;
  io.dup = I.dup;
  const double gs = (MODE == kModeF32) ? I.gs32 : (MODE == kModeF64 ? I.gs64 : I.gsdf);  // tangent steps as DF
  io.post.f64 = gs * I.nf;
  for (int q = 0; q < kBatchTiles; ++q) {
    const int64_t tile = blk * kBatchTiles + q;
    if (tile >= ntiles) break;  // uniform over the block
    if (q) __syncthreads();     // the previous tile's last reads of shared memory
    chain_block<T, KS, double>(io, sh, cps, trs, I.L, I.bc, (uint64_t)tile);
  }
}

}  // namespace

AuxCoef coef_of(const Op& op) {
  AuxCoef c;
  const double bj = op.mp.betaJ;
  c.b1[0] = std::exp(bj);
  c.b1[1] = 1.0 / c.b1[0];
  c.b2[0] = std::exp(-bj * op.mp.kappa);
  c.b2[1] = 1.0 / c.b2[0];
  c.b3[0] = std::exp(-bj * op.mp.kappa2);
  c.b3[1] = 1.0 / c.b3[0];
  return c;
}

namespace {

// value and derivative by one parameter (host)
struct Dual {
  double v = 0.0, d = 0.0;
  Dual() {}
  Dual(double v_, double d_ = 0.0) : v(v_), d(d_) {}
};
Dual operator*(Dual a, Dual b) { return Dual(a.v * b.v, a.d * b.v + a.v * b.d); }
Dual operator/(Dual a, Dual b) { return Dual(a.v / b.v, (a.d - a.v / b.v * b.d) / b.v); }

double value(double x) { return x; }
double value(Dual x) { return x.v; }
template <class T>
T tab_elem(double x) {
  return (T)x;
}
template <class T>
T tab_elem(Dual x) {
  return tangent(x.v, x.d);
}

// A bound on ln of the operator's Tvec entries (aux_tvec_grad's terms, with the
// normfactor that the BNNNI and reduced forms hold) and of the factors that an
// open boundary adds at both ends.
double weight_bound(const Op& op) {
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  const double aK = std::fabs(op.mp.betaJ);
  double b = 0.5 * aK * (op.L + 1) * (1.0 + std::fabs(op.mp.h) + (zb ? std::fabs(op.mp.kappa2) : 0.0));
  if (op.kind != K_XDT) b += 0.5 * op.mp.betaJ * op.nfexp;
  if (!zb && op.boundary) b += 2.0 * aK * std::fabs(op.mp.kappa);
  return b;
}

// The step tables (see ChainTab) from the factors b1 = e^{+-K}, b2 =
// e^{-+K kappa}, b3 = e^{-+K kappa2} (TMat/tmat.cpp:344-376, 521-588) and
// their derivatives; returns the largest row sum of a step, whose inverse
// normalises the FP32 and double-float steps.  lnmax: ln of the largest input
// weight (up: 1 / the power of two in w1, see ChainTab).  The ring is walked from the
// top, so the carried letter q is the neighbour above and the control c the
// one below: the reference's factors of the lower neighbour (dir 0: b1[sr^al]
// b2[sr^ar] b2[sl^al]; dir 1: b2[sr^ar] b2[sl^al]) belong to c, those of the
// upper one (dir 0: b2[sr^fr] b2[sl^fl]; dir 1: b1[sl^fr] b2[sr^fr]
// b2[sl^fl]) to q.
template <class T>
double chain_tab(bool zb, int dir, const AuxCoef& c, const AuxCoef* dc, bool norm, ChainTab<T>& tab, double lnmax,
                 double* up, double* bias = nullptr) {
  // (formed for every product: plain values but for tangent pairs)
  using D = typename std::conditional<std::is_same<T, tangent>::value, Dual, double>::type;
  D b1[2], b2[2], b3[2];
  for (int k = 0; k < 2; ++k) {
    b1[k] = D(c.b1[k]);
    b2[k] = D(c.b2[k]);
    b3[k] = D(c.b3[k]);
    if constexpr (std::is_same<T, tangent>::value) {
      b1[k].d = dc->b1[k];
      b2[k].d = dc->b2[k];
      b3[k].d = dc->b3[k];
    }
  }
  const int S = zb ? 4 : 2;
  D rho1 = b2[1] / b2[0], rho2[4] = {}, w1[16], zu[64];
  if (!zb) {
    for (int s = 0; s < 2; ++s)
      for (int q = 0; q < 2; ++q) {
        w1[s * 2 + q] = (s == q) ? D(1.0) : rho1;
        for (int k = 0; k < 2; ++k) zu[k * 4 + s * 2 + q] = b2[k ^ s] * b1[s ^ q] * b2[0];  // q is a' here
      }
  } else {
    for (int s = 0; s < 4; ++s) {
      const int sl = s >> 1, sr = s & 1;
      D f = b2[0] * b2[sr];
      rho2[s] = b2[sr ^ 1] / b2[sr];
      if (dir) {
        f = f * b1[sl];
        rho2[s] = rho2[s] * b1[sl ^ 1] / b1[sl];
      }
      for (int q = 0; q < 4; ++q) {
        const int ql = q >> 1, qr = q & 1;
        w1[s * 4 + q] = (sl == ql ? D(1.0) : rho1) * (qr ? rho2[s] : D(1.0));
        // q as a' = (pl, pr)
        const D u = (dir ? b1[sl ^ qr] : b1[sr ^ ql]) * b3[sr ^ qr] * b3[sl ^ ql];
        for (int k = 0; k < 4; ++k) {
          const int cl = k >> 1, cr = k & 1;
          const D z = dir ? b2[sr ^ cr] * b2[sl ^ cl] : b1[sr ^ cl] * b2[sr ^ cr] * b2[sl ^ cl];
          zu[k * 16 + q * 4 + s] = z * u * f;
        }
      }
    }
  }
  double gb = 0.0;
  for (int k = 0; k < S; ++k)
    for (int s = 0; s < S; ++s) {
      double sum = 0.0;
      for (int q = 0; q < S; ++q) sum += value(w1[s * S + q]);
      for (int a = 0; a < S; ++a) gb = std::max(gb, value(zu[k * S * S + (zb ? a * S + s : s * S + a)]) * sum);
    }
  // What rounding the tables adds to a step, as the ratio of its exact to its
  // rounded sum over all inputs and outputs: every step shares it, so the
  // product's output factor takes it out (FP32: 3e-8 per entry, L of them).
  const D g(norm ? 1.0 / gb : 1.0);
  if (std::is_same<T, float>::value && bias) {
    const float r1 = (float)value(rho1);
    double exact = 0.0, rounded = 0.0;
    for (int k = 0; k < S; ++k)
      for (int s = 0; s < S; ++s) {
        double se = 0.0, sr = 0.0;
        for (int q = 0; q < S; ++q) {
          se += value(w1[s * S + q]);
          sr += !zb ? (s == q ? 1.0 : (double)r1)
                    : ((s >> 1) == (q >> 1) ? 1.0 : (double)r1) * ((q & 1) ? (double)(float)value(rho2[s]) : 1.0);
        }
        for (int a = 0; a < S; ++a) {
          const double z = value(zu[k * S * S + (zb ? a * S + s : s * S + a)]) * value(g);
          exact += z * se;
          rounded += (double)(float)z * sr;
        }
      }
    *bias = exact / rounded;
  }
  // (e^80 of e^88.7: vectors of unit norm leave room)
  double top = 0.0;
  for (int s = 0; zb && s < 4; ++s) top = std::max(top, value(rho2[s]));
  const double sums = (1.0 + value(rho1)) * (1.0 + top);
  int k = 0;
  if (norm && !(sums < 1e4 && lnmax < 70.0)) {
    const double grow = std::log(sums), over = std::min(grow, lnmax + grow - 80.0);
    if (over > 0.0) k = (int)std::ceil(std::min(over, 80.0) / std::log(2.0));
  }
  *up = std::ldexp(1.0, k);
  tab.rho1 = tab_elem<T>(rho1);
  for (int k = 0; k < 4; ++k) tab.rho2[k] = tab_elem<T>(rho2[k]);
  for (int k = 0; k < 2; ++k) tab.b2[k] = tab_elem<T>(b2[k]);
  for (int k = 0; k < S * S; ++k) {
    tab.w1[k] = tab_elem<T>(w1[k] * D(1.0 / *up));
    tab.w2[k] = tab_elem<T>(w1[k]);
  }
  for (int k = 0; k < S * S * S; ++k) tab.zu[k] = tab_elem<T>(zu[k] * g);
  return gb;
}

}  // namespace

// Batch members keep no product buffers of their own: the batch owns them.
static thread_local bool g_batch_member = false;
BatchMemberScope::BatchMemberScope() : prev(g_batch_member) { g_batch_member = true; }
BatchMemberScope::~BatchMemberScope() { g_batch_member = prev; }

void build_aux(Op& op) {
  const int L = op.L;
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  const bool reduced = (op.kind == K_XDM || op.kind == K_ZBM);
  if (zb && L % 2) fail(TM_ERR_ARG, "diagonal BNNNI operators need an even width");
  if (reduced) build_prefix_tree(op, L, std::vector<int>(zb ? L / 2 : L, zb ? 2 : 1), true, op.tree);
  if (g_batch_member) return;
  if (!reduced) {  // one buffer, written in place
    const int nlb = zb ? 4 : (op.boundary == 0 ? 2 : 1);
    op.ws_a.alloc((size_t)8 * nlb << (L + (zb ? 2 : 1)));
    return;
  }
  // the two pass buffers of any plan the tuning table can choose
  int64_t most[2] = {1, 1};
  for (size_t elem : {(size_t)4, (size_t)8})
    for (int tb = 10; tb <= (elem == 8 ? 13 : 14); ++tb) {
      int64_t need[2];
      chain_buffer_elems(op, chain_plan(op, elem, tb), need);
      for (int k = 0; k < 2; ++k) most[k] = std::max(most[k], need[k] * (int64_t)elem);
    }
  op.ws_a.alloc((size_t)most[0]);
  op.ws_b.alloc((size_t)most[1]);
  op.ws_c.alloc((size_t)op.n * 8);
}

// ------------------------------------------------------------------ autotuner inputs
namespace {
__global__ void tune_fill_kernel(double* v, int64_t n, uint64_t seed) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) {
    uint64_t z = seed + 0x9e3779b97f4a7c15ull * (uint64_t)(i + 1);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    v[i] = (double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5;
  }
}
__global__ void tune_f32_kernel(const double* __restrict__ x, float* __restrict__ y, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += st) y[i] = (float)x[i];
}
}  // namespace

void fill_uniform_dev(double* v, int64_t n, uint64_t seed, cudaStream_t s) {
  tune_fill_kernel<<<grid_for(n), 256, 0, s>>>(v, n, seed);
  TM_CKK("tune_fill");
}
void to_f32_dev(const double* x, float* y, int64_t n, cudaStream_t s) {
  tune_f32_kernel<<<grid_for(n), 256, 0, s>>>(x, y, n);
  TM_CKK("tune_f32");
}

// ------------------------------------------------------------------ pass plans
// The passes of one product.  A tile of 2^tile_bits elements holds the carried
// letter, a chunk of the old bits below the pass's letters (at
// least 128 bytes' worth of slots, for coalescing) and the pass's letters; the
// last pass has no bits below, holds the lastbit values instead and takes as
// many letters as fit; the others share the rest evenly, the first one (whose
// gathers want long chunks) the fewest.
//   Small operators would leave most SMs without a block that way (DNNI, full,
// open, L = 12 in FP64: two blocks of 2^11 slots in the last pass): the last
// pass then hands letters to the others, down to an even split, and the chunks
// shrink to two slots, until a pass has `blocks` blocks.  The buffers of such
// operators stay in L2, where short runs cost little.  With the greedy split /
// 128 / 256 / 512 blocks, us: full DNNI L = 12 FP64 43.0 / 17.4 / 17.4 / 17.4,
// L = 17 FP64 - / 57.4 / 51.2 / 50.7, L = 18 FP32 - / 22.5 / 18.5 / 18.5, reduced
// BNNNI L = 18 FP32 - / 29.7 / 29.9 / 36.9.
ChainPlan chain_plan(const Op& op, size_t elem, int tile_bits, int blocks) {
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  const int KS = zb ? 2 : 1, m = op.L / KS;
  const int bc = zb ? 0 : op.boundary;
  const int slot = (1 << KS) * (int)elem;
  const int cbn = (slot == 8) ? 4 : (slot == 16) ? 3 : (slot == 32) ? 2 : 1;
  const int lbb = (bc == 0) ? KS : 0;
  const int capl = std::min(kChainMaxT, std::max(1, (tile_bits - KS - lbb) / KS));
  const int cap = std::min(kChainMaxT, std::max(1, (tile_bits - KS - cbn) / KS));
  int lead = std::max(0, m - capl);  // letters before the last pass
  const int npass = 1 + (lead + cap - 1) / cap;
  if (npass > kChainMaxPass) fail(TM_ERR_LIMIT, "too many chain passes");
  auto nodes = [&](int t) { return op.tree.nlev ? op.tree.n[t] : (int64_t)1 << (KS * t); };
  const int even = std::min(cap * (npass - 1), m * (npass - 1) / npass);
  while (lead < even && nodes(lead) < blocks) ++lead;
  ChainPlan out;
  int t0 = 0;
  for (int p = 0; p < npass; ++p) {
    ChainPass cp{};
    cp.t0 = t0;
    cp.T = (p == npass - 1) ? m - t0 : (lead - t0) / (npass - 1 - p);
    cp.rest = op.L - KS * (t0 + cp.T);
    cp.cb = std::min(std::max(cbn, tile_bits - KS - KS * cp.T), cp.rest);
    cp.first = (p == 0);
    cp.last = (p == npass - 1);
    cp.nlb = (bc == 0) ? 1 << KS : 1;
    cp.nin = nodes(t0);
    cp.nout = nodes(t0 + cp.T);
    while (cp.cb > 1 && chain_pass_blocks(cp) < blocks) --cp.cb;
    cp.tb = cp.last ? lbb : cp.cb;
    out.p[out.n++] = cp;
    t0 += cp.T;
  }
  return out;
}

// blocks of one pass and its dynamic shared memory
int64_t chain_pass_blocks(const ChainPass& cp) {
  return ((int64_t)(cp.last ? 1 : cp.nlb) * cp.nin) << (cp.rest - cp.cb);
}
size_t chain_pass_smem(const ChainPass& cp, bool zb, size_t elem) {
  const int KS = zb ? 2 : 1, bytes = (1 << KS) * (int)elem;
  const int vec = std::min(bytes, 16);
  return (size_t)slot_plane(1 << (KS * cp.T + cp.tb), bytes) * (bytes / vec) * vec;
}
// (a full operator's passes write every element where they read it: one
// buffer, in place)
void chain_buffer_elems(const Op& op, const ChainPlan& plan, int64_t need[2]) {
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  need[0] = need[1] = 0;
  for (int p = 0; p + 1 < plan.n; ++p)
    need[op.tree.nlev ? p & 1 : 0] = std::max(need[op.tree.nlev ? p & 1 : 0], ((int64_t)plan[p].nlb * plan[p].nout) << (plan[p].rest + (zb ? 2 : 1)));
}

namespace {
TreeDev tree_dev(const Op& op) {
  TreeDev t{};
  if (!op.tree.nlev) return t;
  t.nodes = op.tree.nodes.as<uint2>();
  t.words = op.tree.words.as<uint16_t>();
  for (int i = 0; i <= op.tree.nlev; ++i) t.off[i] = (uint32_t)op.tree.off[i];
  return t;
}
}  // namespace

// y = T x (or T^T x for transposed views); scaled: FP32 result divided by the
// returned factor, the step normalisation or, where the rest of the output
// factor would take FP32 results out of their range (scale_fits), all of it.
// T: arithmetic and pass-buffer type (float, double, or dfloat: FP64-accurate
// products on the FP32 pipes); IO: element type of x and y.
template <class T, class IO = T>
double matvec_aux_dir(const Op& op, const IO* x, IO* y, bool scaled, int dir, cudaStream_t s,
                      const AuxCoef* dcoef = nullptr, void* buf0 = nullptr, void* buf1 = nullptr) {
  using U = typename ChainIn<T>::U;
  const int L = op.L;
  const bool reduced = (op.kind == K_XDM || op.kind == K_ZBM);
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  // FP32 and double-float steps (tangent pairs included) are normalised
  // (FP32 exponent range)
  const bool norm = !std::is_same<T, double>::value;
  ChainTab<T> tab;  // (DNNI leaves the end of its arrays as it is)
  double bias = 1.0, up = 1.0;
  const double gb = chain_tab<T>(zb, dir, coef_of(op), dcoef, norm, tab, weight_bound(op), &up, &bias);
  const int nsteps = zb ? L / 2 : L;
  const double gscale = norm ? std::pow(gb, (double)nsteps) * up : 1.0;
  const double sf = (scaled ? 1.0 : gscale) * std::pow(bias, (double)nsteps);
  const int bc = zb ? 0 : op.boundary;
  int tile_bits = 0, threads = 0;
  chain_tuning(L, sizeof(T), zb, tile_bits, threads);
  T* buf[2] = {buf0 ? static_cast<T*>(buf0) : op.ws_a.as<T>(), buf1 ? static_cast<T*>(buf1) : op.ws_b.as<T>()};
  if (!op.tree.nlev) buf[1] = buf[0];
  ChainIO<T, IO> io{};
  io.tv = op.tvec.as<double>();
  io.y = y;
  const double f = ((zb || reduced) ? 1.0 : op.normfactor) * sf;
  const bool whole = scaled && !scale_fits(f);
  io.post = scale_factor(whole ? 1.0 : f);
  io.x = x;
  io.pre = op.tvec.as<double>();
  if (reduced) {
    io.smap = op.smap.as<uint32_t>();
    io.dup = op.dup.as<uint16_t>();
    if (L > kChainFold) {
      U* u = op.ws_c.as<U>();
      chain_scale_in<U, IO><<<grid_for(op.n), 256, 0, s>>>(x, op.tvec.as<double>(), u, op.n);
      TM_CKK("chain_scale_in");
      io.u = u;
    }
  }
  const TreeDev tr = tree_dev(op);
  int p = 0;
  for (const ChainPass& cp : chain_plan(op, sizeof(T), tile_bits)) {
    const int64_t nblocks = chain_pass_blocks(cp);
    const size_t shm = chain_pass_smem(cp, zb, sizeof(T));
    io.src = buf[(p + 1) & 1];
    io.dst = buf[p & 1];
    if (zb) {
      raise_smem_limit((const void*)chain_kernel<T, 2, IO>, shm);
      chain_kernel<T, 2, IO><<<(unsigned)nblocks, threads, shm, s>>>(io, tab, cp, tr, L, bc);
    } else {
      raise_smem_limit((const void*)chain_kernel<T, 1, IO>, shm);
      chain_kernel<T, 1, IO><<<(unsigned)nblocks, threads, shm, s>>>(io, tab, cp, tr, L, bc);
    }
    TM_CKK("aux_chain");
    ++p;
  }
  return scaled ? (whole ? gscale * f : gscale) : 1.0;
}

// ------------------------------------------------------------------ batch members
void chain_inst_fill(const Op& op, int dir, ChainInst& rec, int tb4, int tb8) {
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  const bool reduced = (op.kind == K_XDM || op.kind == K_ZBM);
  const int L = op.L;
  rec.L = L;
  rec.zb = zb;
  rec.bc = zb ? 0 : op.boundary;
  rec.dir = dir;
  rec.nlb = (rec.bc == 0) ? (zb ? 4 : 2) : 1;
  rec.n = op.n;
  // full DNNI applies the normfactor at the output; the BNNNI Tvec holds it
  rec.nf = (reduced || zb) ? 1.0 : op.normfactor;
  const AuxCoef c = coef_of(op);
  double bias = 1.0, up = 1.0, none = 1.0;
  const double lnmax = weight_bound(op);
  const double gb = chain_tab<float>(zb, dir, c, nullptr, true, rec.c32, lnmax, &up, &bias);
  chain_tab<dfloat>(zb, dir, c, nullptr, true, rec.cdf, lnmax, &up);
  chain_tab<double>(zb, dir, c, nullptr, false, rec.c64, lnmax, &none);
  const int nsteps = zb ? L / 2 : L;
  rec.gsdf = std::pow(gb, (double)nsteps) * up;
  rec.gs32 = rec.gsdf * std::pow(bias, (double)nsteps);
  rec.gs64 = 1.0;
  int th = 0;
  if (tb4 <= 0) chain_tuning(L, 4, zb, tb4, th);
  if (tb8 <= 0) chain_tuning(L, 8, zb, tb8, th);
  int tb16 = 0;
  chain_tuning(L, 16, zb, tb16, th);
  const ChainPlan p16 = chain_plan(op, 16, tb16, 0);
  rec.np16 = p16.n;
  std::copy(p16.begin(), p16.end(), rec.p16);
  for (int t = 0; t < 3; ++t) {
    const AuxCoef db = aux_coef_derivative(op.mp.betaJ, op.mp.kappa, op.mp.kappa2, t);
    chain_tab<tangent>(zb, dir, c, &db, true, rec.ctan[t], lnmax, &up);  // the normalisation is a constant: no derivative
  }
  rec.tree = tree_dev(op);
  rec.kind = op.kind;
  rec.bj = op.mp.betaJ;
  rec.kap = op.mp.kappa;
  rec.kap2 = op.mp.kappa2;
  rec.h = op.mp.h;
  const ChainPlan p4 = chain_plan(op, 4, tb4, 0), p8 = chain_plan(op, 8, tb8, 0);
  rec.np4 = p4.n;
  rec.np8 = p8.n;
  std::copy(p4.begin(), p4.end(), rec.p4);
  std::copy(p8.begin(), p8.end(), rec.p8);
  rec.smap = reduced ? op.smap.as<uint32_t>() : nullptr;
  rec.tvec = op.tvec.as<double>();
  rec.idx = reduced ? op.idx.as<uint32_t>() : nullptr;
  rec.dup = reduced ? op.dup.as<uint16_t>() : nullptr;
}

namespace {
template <class T, int KS, int MODE>
int batch_passes(const ChainBatch& B, const int2* km, const ChainBatch::Plan& P, cudaStream_t s, int theta) {
  int launches = 1;
  chain_batch_scale_in<typename ChainIn<T>::U, MODE><<<(unsigned)B.nrblk, 256, 0, s>>>(B.inst, km, B.rstart, B.rmem);
  TM_CKK("chain_batch_scale_in");
  for (int p = 0; p < P.np; ++p) {
    if (P.nblk[p] == 0) continue;
    raise_smem_limit((const void*)chain_batch_kernel<T, KS, MODE>, P.smem);
    chain_batch_kernel<T, KS, MODE><<<(unsigned)P.nblk[p], P.threads, P.smem, s>>>(
        B.inst, km, P.start + (size_t)p * (B.count + 1), P.bmem + P.boff[p], p, theta);
    TM_CKK("chain_batch");
    ++launches;
  }
  return launches;
}

template <int KS>
int batch_product(const ChainBatch& B, const int2* km, int mode, cudaStream_t s, int theta) {
  if (mode == kModeF32) return batch_passes<float, KS, kModeF32>(B, km, B.p4, s, theta);
  if (mode == kModeDF) return batch_passes<dfloat, KS, kModeDF>(B, km, B.p8, s, theta);
  if (mode == kModeTangent) return batch_passes<tangent, KS, kModeTangent>(B, km, B.p16, s, theta);
  return batch_passes<double, KS, kModeF64>(B, km, B.p8, s, theta);
}
}  // namespace

int chain_batch_product(const ChainBatch& B, const int2* km, int mode, cudaStream_t s, int theta) {
  return B.zb ? batch_product<2>(B, km, mode, s, theta) : batch_product<1>(B, km, mode, s, theta);
}

// ------------------------------------------------------------------ autotuner
// Time the operator's product (FP32, or the 8-byte double-float engine) over
// the tile sizes and block sizes the chain kernels take, CUDA events on the
// operator's stream, and keep the fastest for this (element size, carried
// bits, width) in the tuning table.  Results do not depend on the choice
// (same arithmetic per element, in the same order).
void chain_autotune(const Op& op0, tm_dtype dt, int& best_tb, int& best_th, double& best_ms) {
  const Op& op = op0.parent ? *op0.parent : op0;
  if (op.kind != K_ZBT && op.kind != K_ZBM && op.kind != K_XDT && op.kind != K_XDM)
    fail(TM_ERR_UNSUPPORTED, "the autotuner covers the aux-bit operators (models B and D)");
  if (!op.ws_a.p) fail(TM_ERR_ARG, "operator has no product buffers (a sweep member)");
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  const size_t elem = (dt == TM_F32) ? 4 : 8;
  cudaStream_t s = op.stream;
  AllocStream guard(s);
  DBuf x, y, x32, y32;
  x.alloc((size_t)op.n * 8);
  y.alloc((size_t)op.n * 8);
  x32.alloc((size_t)op.n * 4);
  y32.alloc((size_t)op.n * 4);
  fill_uniform_dev(x.as<double>(), op.n, 7, s);
  to_f32_dev(x.as<double>(), x32.as<float>(), op.n, s);
  chain_tuning(op.L, elem, zb, best_tb, best_th);
  const int tbs[4] = {11, 12, 13, 14};
  const int ths[2] = {128, 256};
  ChainTuneKeep tried(op.L, elem, zb);  // the entry as it was, should a step throw
  struct Events {
    cudaEvent_t e[2] = {nullptr, nullptr};
    ~Events() {
      for (cudaEvent_t v : e)
        if (v) cudaEventDestroy(v);
    }
  } ev;
  for (cudaEvent_t& v : ev.e) TM_CK(cudaEventCreate(&v));
  best_ms = 1e30;
  for (int tb : tbs) {
    if (tb > (elem == 8 ? 13 : 14)) continue;
    for (int th : ths) {
      chain_set_tuning(op.L, elem, zb, tb, th);
      auto run = [&]() {
        if (elem == 4)
          matvec_aux_dir<float>(op, x32.as<float>(), y32.as<float>(), true, 0, s);
        else
          matvec_aux_dir<dfloat, double>(op, x.as<double>(), y.as<double>(), false, 0, s);
      };
      run();
      TM_CK(cudaEventRecord(ev.e[0], s));
      for (int r = 0; r < 3; ++r) run();
      TM_CK(cudaEventRecord(ev.e[1], s));
      TM_CK(cudaEventSynchronize(ev.e[1]));
      float ms = 0.f;
      TM_CK(cudaEventElapsedTime(&ms, ev.e[0], ev.e[1]));
      if (ms / 3.0 < best_ms) {
        best_ms = ms / 3.0;
        best_tb = tb;
        best_th = th;
      }
    }
  }
  tried.set(best_tb, best_th);
}

template <class T>
double matvec_aux(const Op& op, const T* x, T* y, bool scaled, cudaStream_t s) {
  const Op& base = op.parent ? *op.parent : op;
  return matvec_aux_dir<T>(base, x, y, scaled, op.transposed ? 1 : 0, s);
}

template double matvec_aux<float>(const Op&, const float*, float*, bool, cudaStream_t);
template double matvec_aux<double>(const Op&, const double*, double*, bool, cudaStream_t);

// Tangent products of the adjoint: y = D_out (dC/dtheta) D_in x, the chain
// steps differentiated with respect to betaJ, kappa and (BNNNI) kappa2 in turn
// (the Boltzmann weights Tvec held fixed); take(t) uses y before the next.
void matvec_aux_tangents(const Op& op, const double* x, double* y, cudaStream_t s,
                         const std::function<void(int)>& take) {
  // pass buffers at 16 bytes per element (the operator's hold 8)
  const bool zb = (op.kind == K_ZBT || op.kind == K_ZBM);
  int tb = 0, th = 0;
  chain_tuning(op.L, 16, zb, tb, th);
  int64_t need[2];
  chain_buffer_elems(op, chain_plan(op, 16, tb), need);
  AllocStream guard(s);
  DBuf P;
  P.alloc((size_t)(need[0] + need[1]) * 16 + 16);
  tangent* buf = P.as<tangent>();
  for (int t = 0; t < (zb ? 3 : 2); ++t) {
    const AuxCoef db = aux_coef_derivative(op.mp.betaJ, op.mp.kappa, op.mp.kappa2, t);
    matvec_aux_dir<tangent, double>(op, x, y, false, 0, s, &db, buf, buf + need[0]);
    take(t);
  }
}

// FP64-accurate product in double-float arithmetic (the solver's refinement
// products for the aux-bit operators)
void matvec_aux_df(const Op& op, const double* x, double* y, cudaStream_t s) {
  const Op& base = op.parent ? *op.parent : op;
  matvec_aux_dir<dfloat, double>(base, x, y, false, op.transposed ? 1 : 0, s);
}

}  // namespace ltm
