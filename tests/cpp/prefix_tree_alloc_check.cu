// build_prefix_tree with every device call failing and the k-th allocation
// throwing: a tree that could not be completed has to stay "no tree", and a
// later build has to start again.  Runs without a GPU (no device is visible to
// it: the launches do nothing).
#include "tm_tree.cu"

#include <cstdio>
#include <cstdlib>

namespace ltm {
static int g_left = 0;
void fail(tm_status code, const std::string& msg) { throw Failure{code, msg}; }
void check_cuda(cudaError_t, const char*, const char*, int) {}
void note_launch() {}
AllocStream::AllocStream(cudaStream_t) : prev(nullptr) {}
AllocStream::~AllocStream() {}
void DBuf::alloc(size_t b) {
  release();
  if (g_left-- <= 0) fail(TM_ERR_NOMEM, "out of device memory");
  p = std::malloc(b < 65536 ? 65536 : b);
}
void DBuf::release() {
  std::free(p);
  p = nullptr;
}
}  // namespace ltm

int main() {
  for (int words = 0; words < 2; ++words) {
    ltm::Op op;
    op.n = 100;
    ltm::PrefixTree tree;
    for (int ok = 0; ok < 3; ++ok) {  // counts, nodes, words
      ltm::g_left = ok;
      bool threw = false;
      try {
        ltm::build_prefix_tree(op, 12, {4, 4, 4}, words != 0, tree);
      } catch (const ltm::Failure&) {
        threw = true;
      }
      if (threw != (ok < 2 + words)) return std::printf("allocation %d: threw %d\n", ok, threw), 1;
      if (threw && tree.nlev) return std::printf("allocation %d failed, nlev = %d\n", ok, tree.nlev), 1;
    }
    ltm::g_left = 3;
    ltm::build_prefix_tree(op, 12, {4, 4, 4}, words != 0, tree);
    if (tree.nlev != 3) return std::printf("complete build, nlev = %d\n", tree.nlev), 1;
  }
  std::printf("ok\n");
  return 0;
}
