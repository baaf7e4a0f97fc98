// Tuning table of the chain passes: tile bits and threads per block by
// (element size, carried bits, width).
#include <mutex>

#include "tm_chain.h"

namespace ltm {

// Defaults: 2^13-element tiles and 256 threads for 4-byte elements, 2^12 and
// 128 for 8-byte ones (32 KB either way; 64 or more groups per warp-round at
// either size).  Over BNNNI widths 16-24 and DNNI widths
// 20-26 these are within 10% of the fastest of all tile and block sizes;
// tm_chain_autotune and tm_chain_set_tuning override entries at run time.
namespace {
std::mutex g_tune_mu;
ChainTune g_tune[2][2][33];  // [elem 4/8][zb][L]
}  // namespace

void chain_tuning(int L, size_t elem, bool zb, int& tile_bits, int& threads) {
  if (elem >= 16) {  // tangent pairs (adjoint): 32 KB tiles, fewer threads
    tile_bits = 11;
    threads = 128;
    return;
  }
  tile_bits = (elem == 8) ? 12 : 13;
  threads = (elem == 8) ? 128 : 256;
  if (L < 0 || L > 32) return;
  std::lock_guard<std::mutex> lock(g_tune_mu);
  const ChainTune& t = g_tune[elem == 8][zb ? 1 : 0][L];
  if (t.tile_bits) tile_bits = t.tile_bits;
  if (t.threads) threads = t.threads;
}

void chain_set_tuning(int L, size_t elem, bool zb, int tile_bits, int threads) {
  if (L < 0 || L > 32) fail(TM_ERR_ARG, "width out of range");
  if (tile_bits && (tile_bits < 10 || tile_bits > (elem == 8 ? 13 : 14))) fail(TM_ERR_ARG, "tile bits out of range");
  if (threads && threads != 64 && threads != 128 && threads != 256) fail(TM_ERR_ARG, "threads must be 64, 128 or 256");
  std::lock_guard<std::mutex> lock(g_tune_mu);
  g_tune[elem == 8][zb ? 1 : 0][L] = ChainTune{tile_bits, threads};
}

ChainTuneKeep::ChainTuneKeep(int L_, size_t elem_, bool zb_) : L(L_), elem(elem_), zb(zb_) {
  if (L < 0 || L > 32) fail(TM_ERR_ARG, "width out of range");
  std::lock_guard<std::mutex> lock(g_tune_mu);
  entry = g_tune[elem == 8][zb ? 1 : 0][L];
}
ChainTuneKeep::~ChainTuneKeep() {
  std::lock_guard<std::mutex> lock(g_tune_mu);
  g_tune[elem == 8][zb ? 1 : 0][L] = entry;
}

}  // namespace ltm
