// Host build of the tree build's sizes (exafmm-dev_b200/csrc/fmm_tree_plan.cuh) for
// tests/test_tree_plan.py.
#include "fmm_tree_plan.cuh"

extern "C" {
int tree_blocks(int n, int ncrit, int most) { return fmmb200::tree_blocks(n, ncrit, most); }
}
