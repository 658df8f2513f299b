// Host build of the tree build's sizes (exafmm-dev_b200/csrc/fmm_tree_plan.cuh) for
// tests/test_tree_plan.py.
#include "fmm_tree_plan.cuh"

extern "C" {
int tree_most(int sms, int per, int want) { return fmmb200::tree_most(sms, per, want); }
int tree_blocks(int n, int ncrit, int most) { return fmmb200::tree_blocks(n, ncrit, most); }
unsigned long long tree_first_nodes(int n, int ncrit, int nroots, unsigned long long most) {
  return most ? fmmb200::tree_first_nodes(n, ncrit, nroots, most)
              : fmmb200::tree_first_nodes(n, ncrit, nroots);
}
unsigned long long tree_more_nodes(unsigned long long had, unsigned long long most) {
  return most ? fmmb200::tree_more_nodes(had, most) : fmmb200::tree_more_nodes(had);
}
}
