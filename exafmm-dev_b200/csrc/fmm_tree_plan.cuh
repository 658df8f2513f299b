// Sizes of the adaptive tree's build (fmm_tree.cu) that the host works out: no CUDA in them, so
// that they can be checked without a device.
#pragma once
#include <algorithm>
#include <cstddef>

namespace fmmb200 {

// Blocks of the tree kernel that are resident together on `sms` SMs that hold `per` of them each,
// `want` of which each is to take at most (more make dearer barriers).
inline int tree_most(int sms, int per, int want) { return std::max(1, sms * std::min(per, want)); }

// Blocks of the tree kernel, at most `most`: a warp for every few nodes of the widest level
// (fewer blocks make cheaper barriers).  Any ncrit that an int holds.
inline int tree_blocks(int n, int ncrit, int most) {
  const long long per = 4LL * ncrit, want = (n + per - 1) / per;
  return (int)std::max(1LL, std::min<long long>(want, most));
}

// Most nodes of a tree: the interaction lists hold 27-bit cells.
constexpr size_t kTreeMaxNodes = (size_t{1} << 27) - 1;

// Nodes to make room for at first; 0: more roots than a tree may have nodes.
inline size_t tree_first_nodes(int n, int ncrit, int nroots, size_t most = kTreeMaxNodes) {
  if ((size_t)nroots > most) return 0;
  return std::min(most, std::max<size_t>(1024, 4 * (size_t)(n / ncrit) + 64 + nroots));
}
// and after a build that needed more than the `had` nodes there was room for; 0: it cannot be built
inline size_t tree_more_nodes(size_t had, size_t most = kTreeMaxNodes) {
  return had < most ? std::min(most, 2 * had) : 0;
}

}  // namespace fmmb200
