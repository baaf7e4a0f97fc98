// Prefix trees of orbit representatives.
//
// A representative is the smallest state of its orbit, so its top k bits are
// one of a few k-bit prefixes: for the translation groups about 2/k of all of
// them (a prefix that some rotation of the state could undercut starts no
// representative).  A product that builds its output bits from the top down
// therefore keeps, after k bits, only the elements whose new bits are such a
// prefix, and its work shrinks as it goes instead of staying at 2^L per bit.
//
// The tree has one level per step of the product: level i holds the distinct
// b_i-bit prefixes of the representatives in ascending order (level 0 the
// empty one, the last level the representatives themselves).  A node is
// {index of its first child in the next level, mask of its children's step
// bits}; children are consecutive and ascending, so child j of a node sits at
// first + popc(mask below bit j).  Everything follows from the sorted list:
// representative r opens a new node at every level deeper than the prefix it
// shares with r - 1.
#include <vector>

#include "tm_internal.h"

namespace ltm {

namespace {

constexpr int kTreeBlock = 1024;

struct TreeLevels {
  int nlev;              // levels 0 .. nlev
  int nbits;             // bits of a representative
  int b[kTreeMaxLevels + 1];
  uint2* nodes[kTreeMaxLevels + 1];  // levels 0 .. nlev - 1
  uint16_t* words[kTreeMaxLevels + 1];
};

// length of the prefix that representative r shares with r - 1 (-1: r = 0)
__device__ __forceinline__ int shared_prefix(const uint32_t* __restrict__ idx, int64_t r, int nbits) {
  if (r == 0) return -1;
  return nbits - (32 - __clz(idx[r] ^ idx[r - 1]));
}

// new nodes per level among this block's representatives: cnt[level][block]
__global__ void __launch_bounds__(kTreeBlock) tree_count_kernel(const uint32_t* __restrict__ idx, int64_t n,
                                                                TreeLevels T, uint32_t* __restrict__ cnt) {
  const int64_t r = (int64_t)blockIdx.x * kTreeBlock + threadIdx.x;
  const int c = (r < n) ? shared_prefix(idx, r, T.nbits) : T.nbits;
  for (int i = 0; i <= T.nlev; ++i) {
    const int k = __syncthreads_count(c < T.b[i]);
    if (threadIdx.x == 0) cnt[(int64_t)i * gridDim.x + blockIdx.x] = (uint32_t)k;
  }
}

// exclusive scan of one level's block counts (a block per level), totals out
__global__ void __launch_bounds__(kTreeBlock) tree_scan_kernel(uint32_t* __restrict__ cnt, int64_t nblk,
                                                               uint32_t* __restrict__ total) {
  __shared__ uint32_t ws[32];
  __shared__ uint32_t carry;
  uint32_t* a = cnt + (int64_t)blockIdx.x * nblk;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t i0 = 0; i0 < nblk; i0 += kTreeBlock) {
    const int64_t i = i0 + threadIdx.x;
    const uint32_t v = (i < nblk) ? a[i] : 0u;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws[wid] = x;
    __syncthreads();
    if (wid == 0) {
      uint32_t w = ws[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      ws[lane] = w;
    }
    __syncthreads();
    const uint32_t base = carry + (wid ? ws[wid - 1] : 0u);
    if (i < nblk) a[i] = base + x - v;
    __syncthreads();
    if (threadIdx.x == 0) carry += ws[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// children of every node: representative r, new from level f on, adds its
// level-i node to the mask of its level-(i-1) node, and is that node's first
// child where the latter is new with it
__global__ void __launch_bounds__(kTreeBlock) tree_fill_kernel(const uint32_t* __restrict__ idx, int64_t n,
                                                               TreeLevels T, const uint32_t* __restrict__ cnt) {
  __shared__ uint32_t ws[32];
  const int64_t r = (int64_t)blockIdx.x * kTreeBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c = (r < n) ? shared_prefix(idx, r, T.nbits) : T.nbits;
  const uint32_t s = (r < n) ? idx[r] : 0u;
  uint32_t parent = 0;
  for (int i = 0; i <= T.nlev; ++i) {
    const bool fresh = c < T.b[i];
    const uint32_t bal = __ballot_sync(0xffffffffu, fresh);
    if (lane == 0) ws[wid] = __popc(bal);
    __syncthreads();
    uint32_t before = cnt[(int64_t)i * gridDim.x + blockIdx.x];
    for (int w = 0; w < wid; ++w) before += ws[w];
    // the node of r at this level: the last new one up to r
    const uint32_t node = before + __popc(bal & (0xffffffffu >> (31 - lane))) - 1u;
    if (i > 0 && fresh) {
      const int step = T.b[i] - T.b[i - 1];
      const uint32_t word = (s >> (T.nbits - T.b[i])) & ((1u << step) - 1u);
      uint2* nd = T.nodes[i - 1] + parent;
      atomicOr(&nd->y, 1u << word);
      if (c < T.b[i - 1]) nd->x = node;
      if (T.words[i]) T.words[i][node] = (uint16_t)(s >> (T.nbits - T.b[i]));
    }
    parent = node;
    __syncthreads();
  }
}

}  // namespace

// Levels after steps[0], steps[0] + steps[1], ... bits (each step at most 5
// bits, together nbits) of the representatives in op.idx; words: with the
// last 16 bits of every node's prefix.
void build_prefix_tree(const Op& op, int nbits, const std::vector<int>& steps, bool words, PrefixTree& out) {
  const int64_t n = op.n;
  cudaStream_t s = op.stream;
  const int nlev = (int)steps.size();
  if (nlev < 1 || nlev > kTreeMaxLevels || nbits > 32) fail(TM_ERR_LIMIT, "prefix tree: too many levels");
  TreeLevels T{};
  T.nlev = nlev;
  T.nbits = nbits;
  for (int i = 0; i < nlev; ++i) T.b[i + 1] = T.b[i] + steps[i];
  if (T.b[nlev] != nbits) fail(TM_ERR_ARG, "prefix tree: steps do not cover the state");
  const int64_t nblk = (n + kTreeBlock - 1) / kTreeBlock;
  DBuf cnt;  // counts per level and block, then the totals per level
  {
    AllocStream pool(s);  // (freed in stream order: a cudaFree would wait for the device)
    cnt.alloc((size_t)(nlev + 1) * (nblk + 1) * 4);
  }
  uint32_t* tot = cnt.as<uint32_t>() + (size_t)(nlev + 1) * nblk;
  tree_count_kernel<<<(unsigned)nblk, kTreeBlock, 0, s>>>(op.idx.as<uint32_t>(), n, T, cnt.as<uint32_t>());
  TM_CKK("tree_count");
  tree_scan_kernel<<<nlev + 1, kTreeBlock, 0, s>>>(cnt.as<uint32_t>(), nblk, tot);
  TM_CKK("tree_scan");
  uint32_t h[kTreeMaxLevels + 1] = {0};
  TM_CK(cudaMemcpyAsync(h, tot, (size_t)(nlev + 1) * 4, cudaMemcpyDeviceToHost, s));
  TM_CK(cudaStreamSynchronize(s));
  int64_t sum = 0;
  for (int i = 0; i <= nlev; ++i) {
    out.b[i] = T.b[i];
    out.n[i] = (i == 0) ? 1 : h[i];
    out.off[i] = sum;
    sum += out.n[i];
  }
  out.nodes.alloc((size_t)out.off[nlev] * sizeof(uint2));
  TM_CK(cudaMemsetAsync(out.nodes.p, 0, (size_t)out.off[nlev] * sizeof(uint2), s));
  if (words) out.words.alloc((size_t)sum * 2);
  for (int i = 0; i < nlev; ++i) T.nodes[i] = out.level(i);
  for (int i = 0; words && i <= nlev; ++i) T.words[i] = out.words.as<uint16_t>() + out.off[i];
  tree_fill_kernel<<<(unsigned)nblk, kTreeBlock, 0, s>>>(op.idx.as<uint32_t>(), n, T, cnt.as<uint32_t>());
  TM_CKK("tree_fill");
  out.nlev = nlev;  // (last: a tree whose tables could not be built is no tree)
}

}  // namespace ltm
