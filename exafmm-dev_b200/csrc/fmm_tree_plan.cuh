// Sizes of the adaptive tree's build (fmm_tree.cu) that the host works out: no CUDA in them, so
// that they can be checked without a device.
#pragma once
#include <algorithm>

namespace fmmb200 {

// Blocks of the tree kernel, at most `most`: a warp for every few nodes of the widest level
// (fewer blocks make cheaper barriers).  Any ncrit that an int holds.
inline int tree_blocks(int n, int ncrit, int most) {
  const long long per = 4LL * ncrit, want = (n + per - 1) / per;
  return (int)std::max(1LL, std::min<long long>(want, most));
}

}  // namespace fmmb200
