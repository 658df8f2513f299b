// Adaptive octree build on the device, bit-exact with BuildTree (include/build_tree_tbb.h).
//
// The reference splits a node while it holds more than ncrit bodies (:172), scattering its
// bodies stably by octant (x > Xc) + 2 (y > Yc) + 4 (z > Zc) (:59, :101) around a centre
// that each level moves by +-R0 / 2^(level+1) (:199-203).  Here every body walks that same
// chain of centres once (k_keys), recording its octant at each of kMaxLevel levels as a
// 63-bit path key; a stable radix sort by key then lays the bodies out in octant order, and
// nodes are carved out of the sorted keys level by level (k_tree), each node's
// octant sub-ranges found by binary search.  Bodies inside a leaf keep their input order, as
// the stable partitions leave them: ranked by the leaf's warp (k_tree), or, with leaves above
// kRankBodies, by a second stable sort by leaf-truncated key.
// Cells take the reference's layout (Nodes2cells :250-294): root first, the children of a
// cell contiguous, each child's subtree after the previous child's.
#include <algorithm>
#include <cfloat>

#include <climits>

#include "fmm_grid.cuh"
#include "fmm_solver.cuh"
#include "fmm_tree_plan.cuh"

namespace fmmb200 {

template <typename T> __device__ __forceinline__ T tmax();
template <> __device__ __forceinline__ float tmax<float>() { return FLT_MAX; }
template <> __device__ __forceinline__ double tmax<double>() { return DBL_MAX; }

// ---------------------------------------------------------------- bounds
// BoundBox::getBounds (include/bound_box.h:76-88): elementwise min / max of positions, per
// chunk of one root's bodies (one block per chunk), then per root (one block per root).
// Min and max are exact whatever the order in which values meet.

// the block's min / max of mn, mx (per thread) into thread 0's mn, mx
template <typename T> __device__ __forceinline__ void block_minmax(T* mn, T* mx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      T a = __shfl_xor_sync(0xffffffffu, mn[d], o);
      T c = __shfl_xor_sync(0xffffffffu, mx[d], o);
      mn[d] = a < mn[d] ? a : mn[d];
      mx[d] = c > mx[d] ? c : mx[d];
    }
  __shared__ T sh[32][6];
  int w = threadIdx.x >> 5;
  if (lane_id() == 0)
    for (int d = 0; d < 3; d++) sh[w][d] = mn[d], sh[w][3 + d] = mx[d];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 1; k < (int)(blockDim.x >> 5); k++)
      for (int d = 0; d < 3; d++) {
        mn[d] = sh[k][d] < mn[d] ? sh[k][d] : mn[d];
        mx[d] = sh[k][3 + d] > mx[d] ? sh[k][3 + d] : mx[d];
      }
}

template <typename T>
__global__ void k_minmax_chunks(const vec4<T>* __restrict__ b, const int* __restrict__ cb,
                                const int* __restrict__ ce, T* __restrict__ part) {
  T mn[3] = {tmax<T>(), tmax<T>(), tmax<T>()};
  T mx[3] = {-tmax<T>(), -tmax<T>(), -tmax<T>()};
  const int e = ce[blockIdx.x];
  for (int i = cb[blockIdx.x] + threadIdx.x; i < e; i += blockDim.x) {
    vec4<T> p = b[i];
    mn[0] = p.x < mn[0] ? p.x : mn[0];
    mn[1] = p.y < mn[1] ? p.y : mn[1];
    mn[2] = p.z < mn[2] ? p.z : mn[2];
    mx[0] = p.x > mx[0] ? p.x : mx[0];
    mx[1] = p.y > mx[1] ? p.y : mx[1];
    mx[2] = p.z > mx[2] ? p.z : mx[2];
  }
  block_minmax(mn, mx);
  if (threadIdx.x == 0)
    for (int d = 0; d < 3; d++) part[6 * blockIdx.x + d] = mn[d], part[6 * blockIdx.x + 3 + d] = mx[d];
}

// BuildTree::bounds2box (include/build_tree_tbb.h:298-310), one block per root over the
// root's chunk bounds; box[16 r ..] = X0[3], R0, Xmin[3], Xmax[3]
template <typename T>
__global__ void k_box(int nroots, const int* __restrict__ chunk_lo, const T* __restrict__ part,
                      int shared, T* __restrict__ box) {
  const int r = blockIdx.x;
  if (r >= nroots) return;
  // shared: every root takes the box of the bounds of all bodies (BoundBox::getBounds of
  // the targets, then of the sources with those bounds, include/bound_box.h:91-97)
  const int c0 = shared ? chunk_lo[0] : chunk_lo[r], c1 = shared ? chunk_lo[nroots] : chunk_lo[r + 1];
  T mn[3] = {tmax<T>(), tmax<T>(), tmax<T>()};
  T mx[3] = {-tmax<T>(), -tmax<T>(), -tmax<T>()};
  for (int k = c0 + threadIdx.x; k < c1; k += blockDim.x)
    for (int d = 0; d < 3; d++) {
      T a = part[6 * k + d], c = part[6 * k + 3 + d];
      mn[d] = a < mn[d] ? a : mn[d];
      mx[d] = c > mx[d] ? c : mx[d];
    }
  block_minmax(mn, mx);
  if (threadIdx.x != 0) return;
  T X[3], R = 0;
  for (int d = 0; d < 3; d++) X[d] = div_rn(add_rn(mx[d], mn[d]), (T)2);
  for (int d = 0; d < 3; d++) {
    T a = sub_rn(X[d], mn[d]);
    R = R < a ? a : R;
    T c = sub_rn(mx[d], X[d]);
    R = R < c ? c : R;
  }
  T* bx = box + 16 * r;
  for (int d = 0; d < 3; d++) bx[d] = X[d], bx[4 + d] = mn[d], bx[7 + d] = mx[d];
  bx[3] = (T)__dmul_rn((double)R, 1.00001);
}

// ---------------------------------------------------------------- path keys
template <typename T>
__global__ void k_keys(const vec4<T>* __restrict__ b, int n, const T* __restrict__ box,
                       const int* __restrict__ root_first, int nroots,
                       unsigned long long* __restrict__ keys, int* __restrict__ idx) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // root of body i: last r with root_first[r] <= i
  int lo = 0, hi = nroots - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (root_first[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  const T* bx = box + 16 * lo;
  vec4<T> p = b[i];
  T c0 = bx[0], c1 = bx[1], c2 = bx[2], R0 = bx[3];
  unsigned long long key = 0;
  T sc = T(0.5);  // 2^-(l+1), exact
  for (int l = 0; l < kMaxLevel; l++) {
    // R0 / 2^(l+1) as the product with 2^-(l+1): the same real number, so the same
    // rounding as the reference's division
    T r = mul_rn(R0, sc);
    sc = mul_rn(sc, T(0.5));
    int o = (p.x > c0) | ((p.y > c1) << 1) | ((p.z > c2) << 2);
    key = (key << 3) | (unsigned)o;
    c0 = add_rn(c0, (o & 1) ? r : -r);
    c1 = add_rn(c1, (o & 2) ? r : -r);
    c2 = add_rn(c2, (o & 4) ? r : -r);
  }
  keys[i] = key;
  idx[i] = i;
}

// forest sort helpers: root of each key-sorted body (binary search of its input index in
// the roots' first bodies), then a gather through the root-sorted permutation
__global__ void k_root_of(int n, const int* __restrict__ body, const int* __restrict__ root_first,
                          int nroots, unsigned* __restrict__ root, int* __restrict__ pos) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int b = body[i];
  int lo = 0, hi = nroots - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (root_first[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  root[i] = (unsigned)lo;
  pos[i] = i;
}

__global__ void k_gather_kv(int n, const int* __restrict__ perm,
                            const unsigned long long* __restrict__ kin,
                            const int* __restrict__ vin, unsigned long long* __restrict__ kout,
                            int* __restrict__ vout) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int j = perm[i];
  kout[i] = kin[j];
  vout[i] = vin[j];
}

__device__ __forceinline__ int digit_at(unsigned long long key, int level) {
  return (int)((key >> (3 * (kMaxLevel - 1 - level))) & 7ULL);
}

// ---------------------------------------------------------------- the tree, in one kernel
// Everything between the key sort and the cells is a few dozen small steps, each over one
// level of nodes and each needing the one before: as launches of their own (a split, a scan
// and an emission per level, the subtree sizes up and the cell slots down) they were 45 to 75
// launches of 2-4 us.  k_tree runs them as one cooperative launch with a barrier of its blocks
// between steps (about 1.5 us).  Bound by latency throughout: a warp's split is two to three
// dependent rounds of key reads.
//
// control block of k_tree (ints, zero before the launch except where said)
enum {
  TC_ARRIVED, TC_FAULT, TC_BIG,  // TC_BIG: a leaf of more than kRankBodies bodies
  TC_LEAVES,
  TC_COUNT = 8,       // [l]: nodes of level l (l > 0)
  TC_FULL = 40,       // [l]: the children of level l did not fit the node arrays
  TC_DEEP = 72,       // [l]: level l splits on a digit the keys were not sorted by
  TC_INTS = 104
};

// largest leaf whose bodies k_tree puts in input order itself
constexpr int kRankBodies = 128;

template <typename T> struct TreeArgs {
  const unsigned long long* keys;  // sorted within each root on their first `levels` digits
  const int* sidx;                 // input index of each sorted key
  const vec4<T>* bodies_in;
  const T* box;
  const int* root_first;
  int nroots, ncrit, levels, ncap;
  int rank;   // put the bodies of each leaf in input order (order, bodies)
  int cluster;  // the launch is one cluster
  int radii;  // and set the cells' final radii and monopoles (before the error-optimised ones)
  int use_rmax;
  T theta;
  int* ctl;
  int *nbegin, *ncount, *nparent, *nchildn, *nfirst, *nnode, *npos, *ncb, *nlevel, *nsid;
  T *nX, *nM0;
  int* cbase;
  int *order, *iparent, *ichild, *nchild, *ibody, *nbody, *clevel, *croot, *leaves;
  vec4<T>* bodies;
  unsigned long long* icell;
  int4* info;
  vec4<T>* cX;
  T* m0;
};

// A warp finds the 7 octant boundaries of a node's sorted key range [b, b + c) together by
// 32-ary searches (32 samples per boundary and round, all loads of a round independent), so
// a node needs log32(c) dependent rounds instead of the 7 log2(c) of a binary search per
// boundary.  slo[o]: the first index whose octant digit is >= o.
__device__ __forceinline__ void octant_starts(int lane, int b, int c, int level,
                                              const unsigned long long* __restrict__ keys,
                                              int* slo) {
  int shi[8];
#pragma unroll
  for (int o = 1; o < 8; o++) {
    slo[o] = b;
    shi[o] = b + c;
  }
  // invariant: the first index whose octant digit is >= o lies in [slo[o], shi[o]]
  for (;;) {
    bool open = false;
#pragma unroll
    for (int o = 1; o < 8; o++) open |= slo[o] < shi[o];
    if (!open) break;
    unsigned ball[8];
    int step[8];
#pragma unroll
    for (int o = 1; o < 8; o++) {
      const int len = shi[o] - slo[o];
      step[o] = len <= 32 ? 1 : (len + 31) / 32;
      const long long idx = slo[o] + (long long)lane * step[o];
      const bool pred = len > 0 && idx < shi[o] && digit_at(keys[idx], level) < o;
      ball[o] = __ballot_sync(0xffffffffu, pred);
    }
#pragma unroll
    for (int o = 1; o < 8; o++) {
      if (slo[o] >= shi[o]) continue;
      const int t = __popc(ball[o]);
      if (step[o] == 1) {
        slo[o] = shi[o] = slo[o] + t;
      } else if (t == 0) {
        shi[o] = slo[o];
      } else {
        const long long nlo = slo[o] + (long long)(t - 1) * step[o] + 1;
        const long long nhi = slo[o] + (long long)t * step[o];
        shi[o] = (int)(nhi < shi[o] ? nhi : shi[o]);
        slo[o] = (int)nlo;
      }
    }
  }
}

// The bodies of a leaf of at most 32 K bodies (a warp): their input indices, in key order,
// ranked and written back ascending (the stable partitions of the reference keep input
// order), the bodies with them; with radii, the leaf's radius (setRmax, R /= theta) and the
// sum of its charges in body order, as the P2M kernels form them.
template <typename T, int K>
__device__ __forceinline__ void rank_leaf(const TreeArgs<T>& a, int lane, int v, int b0, int n,
                                          T X0, T X1, T X2, T R) {
  int id[K], r[K];
  T rmax = 0;
#pragma unroll
  for (int k = 0; k < K; k++) {
    id[k] = lane + 32 * k < n ? a.sidx[b0 + lane + 32 * k] : INT_MAX;
    r[k] = 0;
  }
#pragma unroll
  for (int q = 0; q < K; q++)
    for (int i = 0; i < min(32, n - 32 * q); i++) {
      const int u = __shfl_sync(0xffffffffu, id[q], i);
#pragma unroll
      for (int k = 0; k < K; k++) r[k] += u < id[k];
    }
#pragma unroll
  for (int k = 0; k < K; k++)
    if (lane + 32 * k < n) {
      const vec4<T> b = a.bodies_in[id[k]];
      a.order[b0 + r[k]] = id[k];
      a.bodies[b0 + r[k]] = b;
      const T d = sqrt_rn(norm_rn(sub_rn(X0, b.x), sub_rn(X1, b.y), sub_rn(X2, b.z)));
      rmax = d > rmax ? d : rmax;
    }
  if (!a.radii) return;
  __syncwarp();
  T q = 0;
  for (int base = 0; base < n; base += 32) {
    const int cnt = min(32, n - base);
    const T w = lane < cnt ? a.bodies[b0 + base + lane].w : T(0);
    for (int i = 0; i < cnt; i++) q = add_rn(q, __shfl_sync(0xffffffffu, w, i));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const T u = __shfl_xor_sync(0xffffffffu, rmax, o);
    rmax = u > rmax ? u : rmax;
  }
  if (lane == 0) {
    if (a.use_rmax) R = rmax < R ? rmax : R;
    a.nX[4 * v + 3] = div_rn(R, a.theta);
    a.nM0[v] = q;
  }
}

// One node of BuildNodes (include/build_tree_tbb.h:165-218), a warp: a node with more than
// ncrit bodies gets one child per non-empty octant, from node `next` on; any other is a leaf.
template <typename T>
__device__ __forceinline__ void tree_node(const TreeArgs<T>& a, int lane, int v, int level,
                                          int next) {
  const int b = a.nbegin[v], c = a.ncount[v], root = a.nsid[v];
  const T R0 = a.box[16 * root + 3];
  const T X0 = a.nX[4 * v], X1 = a.nX[4 * v + 1], X2 = a.nX[4 * v + 2];
  if (c > a.ncrit && level < kMaxLevel) {
    if (level >= a.levels) {
      if (lane == 0) atomicExch(&a.ctl[TC_DEEP + level], 1);
      return;
    }
    int slo[8];
    octant_starts(lane, b, c, level, a.keys, slo);
    int s = b, e = b + c;  // the range of octant `lane`
#pragma unroll
    for (int o = 1; o < 8; o++) {
      if (lane == o) s = slo[o];
      if (lane == o - 1) e = slo[o];
    }
    const unsigned m = __ballot_sync(0xffffffffu, lane < 8 && e > s);
    const int nch = __popc(m);
    int first = 0;
    if (lane == 0) first = next + atomicAdd(&a.ctl[TC_COUNT + level + 1], nch);
    first = __shfl_sync(0xffffffffu, first, 0);
    if (first + nch > a.ncap) {
      if (lane == 0) atomicExch(&a.ctl[TC_FULL + level], 1);
      return;
    }
    if (m >> lane & 1) {
      const int u = first + __popc(m & ((1u << lane) - 1));
      const T r = div_rn(R0, (T)(1 << (level + 1)));
      a.nbegin[u] = s;
      a.ncount[u] = e - s;
      a.nparent[u] = v;
      a.nlevel[u] = level + 1;
      a.nsid[u] = root;
      a.nX[4 * u] = add_rn(X0, (lane & 1) ? r : -r);
      a.nX[4 * u + 1] = add_rn(X1, (lane & 2) ? r : -r);
      a.nX[4 * u + 2] = add_rn(X2, (lane & 4) ? r : -r);
    }
    if (lane == 0) {
      a.nchildn[v] = nch;
      a.nfirst[v] = first;
    }
    return;
  }
  if (lane == 0) {
    a.nchildn[v] = 0;
    a.nfirst[v] = -1;
    a.nnode[v] = 1;
  }
  if (!a.rank) return;
  const T R = div_rn(R0, (T)(1 << level));
  if (c <= 64) rank_leaf<T, 2>(a, lane, v, b, c, X0, X1, X2, R);
  else if (c <= kRankBodies) rank_leaf<T, kRankBodies / 32>(a, lane, v, b, c, X0, X1, X2, R);
  else if (lane == 0) {
    atomicExch(&a.ctl[TC_BIG], 1);
    if (a.radii) {  // (defined values for the cells above; the structure pass sets them anew)
      a.nX[4 * v + 3] = R;
      a.nM0[v] = 0;
    }
  }
}

// The subtree size (NNODE, include/build_tree_tbb.h:215-217) of a split node, and with radii
// its radius and monopole from its children's (include/up_down_pass.h:60-84).
template <typename T> __device__ __forceinline__ void tree_up(const TreeArgs<T>& a, int v, int level) {
  const int nch = a.nchildn[v];
  if (nch == 0) return;
  const int u0 = a.nfirst[v];
  int size = 1;
  T rr = 0, q = 0;
  const T X0 = a.nX[4 * v], X1 = a.nX[4 * v + 1], X2 = a.nX[4 * v + 2];
  for (int u = u0; u < u0 + nch; u++) {
    size += a.nnode[u];
    if (!a.radii) continue;
    const T d = add_rn(sqrt_rn(norm_rn(sub_rn(X0, a.nX[4 * u]), sub_rn(X1, a.nX[4 * u + 1]),
                                       sub_rn(X2, a.nX[4 * u + 2]))),
                       a.nX[4 * u + 3]);
    rr = d > rr ? d : rr;
    q = add_rn(q, a.nM0[u]);
  }
  a.nnode[v] = size;
  if (a.radii) {
    T R = div_rn(a.box[16 * a.nsid[v] + 3], (T)(1 << level));
    if (a.use_rmax) R = rr < R ? rr : R;
    a.nX[4 * v + 3] = div_rn(R, a.theta);
    a.nM0[v] = q;
  }
}

// The cell of node v, and its children's slots: Nodes2cells (include/build_tree_tbb.h:250-294:
// children at CN, the next free slot after the child block, each child's subtree after the
// previous child's) with the Morton index of getKey (:240-249) in 64-bit arithmetic.
template <typename T>
__device__ __forceinline__ void tree_cell(const TreeArgs<T>& a, int v, int level) {
  const int root = a.nsid[v];
  const int rc = a.nroots == 1 ? 0 : a.cbase[root];
  const int c = level == 0 ? rc : a.npos[v], cb = level == 0 ? rc + 1 : a.ncb[v];
  const int nch = a.nchildn[v], u0 = a.nfirst[v], par = a.nparent[v];
  if (level == 0) a.npos[v] = c;
  int acc = cb + nch;
  for (int k = 0; k < nch; k++) {
    a.npos[u0 + k] = cb + k;
    a.ncb[u0 + k] = acc;
    acc += a.nnode[u0 + k] - 1;
  }
  const T* box = a.box + 16 * root;
  const T R0 = box[3], R = div_rn(R0, (T)(1 << level));
  const T X[3] = {a.nX[4 * v], a.nX[4 * v + 1], a.nX[4 * v + 2]};
  const int b = a.nbegin[v], nb = a.ncount[v], ch = nch ? cb : 0;
  a.croot[c] = rc;
  a.iparent[c] = level == 0 ? c : a.npos[par];
  a.nchild[c] = nch;
  a.ichild[c] = ch;
  a.ibody[c] = b;
  a.nbody[c] = nb;
  a.clevel[c] = level;
  a.info[c] = make_int4(nch, ch, nb, b);
  const T diam = mul_rn((T)2, R);
  int iX[3];
  for (int d = 0; d < 3; d++) iX[d] = (int)div_rn(sub_rn(X[d], sub_rn(box[d], R0)), diam);
  unsigned long long index = ((1ULL << (3 * level)) - 1) / 7;
  for (int l = 0; l < level; l++)
    for (int d = 0; d < 3; d++) {
      index += (unsigned long long)(iX[d] & 1) << (3 * l + d);
      iX[d] >>= 1;
    }
  a.icell[c] = index;
  a.cX[c] = make_v4<T>(X[0], X[1], X[2], a.radii ? a.nX[4 * v + 3] : R);
  if (a.radii) a.m0[c] = a.nM0[v];
}

constexpr int kTreeThreads = 256, kTreeBlocks = 3;  // threads of a block, blocks per SM
constexpr int kTreeCluster = 8;  // blocks of a launch of one cluster

template <typename T>
__global__ void __launch_bounds__(kTreeThreads, kTreeBlocks) k_tree(TreeArgs<T> a) {
  GridBarrier bar{(unsigned*)&a.ctl[TC_ARRIVED], &a.ctl[TC_FAULT], 0, a.cluster != 0};
  __shared__ int lv[kMaxLevel + 3];
  const int lane = lane_id();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  // one root node per non-empty solve, in solve order
  for (int r = tid; r < a.nroots; r += nt) {
    a.nbegin[r] = a.root_first[r];
    a.ncount[r] = a.root_first[r + 1] - a.root_first[r];
    a.nparent[r] = -1;
    a.nlevel[r] = 0;
    a.nsid[r] = r;
    for (int d = 0; d < 3; d++) a.nX[4 * r + d] = a.box[16 * r + d];
  }
  if (!bar.sync()) return;
  int lo = 0, hi = a.nroots, level = 0;
  for (;; level++) {
    if (threadIdx.x == 0) lv[level] = lo;
    for (int v = lo + (tid >> 5); v < hi; v += nt >> 5) tree_node(a, lane, v, level, hi);
    if (!bar.sync()) return;
    // (flags and counts of this level: no block writes them any more)
    if (*(volatile int*)&a.ctl[TC_FULL + level] || *(volatile int*)&a.ctl[TC_DEEP + level]) return;
    const int cnt = *(volatile int*)&a.ctl[TC_COUNT + level + 1];
    if (cnt == 0) break;
    lo = hi;
    hi += cnt;
  }
  if (threadIdx.x == 0) lv[level + 1] = hi;
  __syncthreads();
  for (int l = level - 1; l >= 0; l--) {
    for (int v = lv[l] + tid; v < lv[l + 1]; v += nt) tree_up(a, v, l);
    if (!bar.sync()) return;
  }
  if (a.nroots > 1) {  // first cell of each root: exclusive scan of the roots' subtree sizes
    if (blockIdx.x == 0 && threadIdx.x < 32) {
      int run = 0;
      for (int r0 = 0; r0 < a.nroots; r0 += 32) {
        const int n = r0 + lane < a.nroots ? a.nnode[r0 + lane] : 0;
        int incl = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, incl, d);
          if (lane >= d) incl += u;
        }
        if (r0 + lane < a.nroots) a.cbase[r0 + lane] = run + incl - n;
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    if (!bar.sync()) return;
  } else if (tid == 0) {
    a.cbase[0] = 0;
  }
  for (int l = 0; l <= level; l++) {
    // (a warp's leaves take one atomic; their order does not matter to any result)
    for (int v0 = lv[l] + tid - lane; v0 < lv[l + 1]; v0 += nt) {
      const int v = v0 + lane;
      const bool in = v < lv[l + 1];
      if (in) tree_cell(a, v, l);
      const unsigned m = __ballot_sync(0xffffffffu, in && a.nchildn[in ? v : 0] == 0);
      int at = 0;
      if (lane == 0 && m) at = atomicAdd(&a.ctl[TC_LEAVES], __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (m >> lane & 1) a.leaves[at + __popc(m & ((1u << lane) - 1))] = a.npos[v];
    }
    if (l < level && !bar.sync()) return;
  }
}

// Blocks of k_tree that this device (or this process's share of it) holds at a time: its launch
// is refused with more.
template <typename T> static int tree_resident(SolverBase& s) {
  if (s.tree_most == 0) {
    int sms = 0, per = 0;
    FMM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.cfg.device));
    FMM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_tree<T>, kTreeThreads, 0));
    s.tree_most = tree_most(sms, per, kTreeBlocks);
  }
  return s.tree_most;
}

// (NCHILD, ICHILD, NBODY, IBODY) of every cell in one 16-byte record, for the traversal
__global__ void k_cell_info(int ncells, const int* __restrict__ nchild,
                            const int* __restrict__ ichild, const int* __restrict__ nbody,
                            const int* __restrict__ ibody, int4* __restrict__ info) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < ncells) info[c] = make_int4(nchild[c], ichild[c], nbody[c], ibody[c]);
}

void fill_cell_info(SolverBase& s) {
  s.c_info.ensure(s.ncells);
  k_cell_info<<<ceil_div(s.ncells, 256), 256, 0, s.stream>>>(
      s.ncells, s.c_nchild.p, s.c_ichild.p, s.c_nbody.p, s.c_ibody.p, s.c_info.p);
  FMM_LAUNCH_CHECK();
}

// leaf level of every sorted body (leaves only; ranges partition the bodies)
__global__ void k_leaf_levels(int nnodes, const int* __restrict__ nchildn,
                              const int* __restrict__ nbegin, const int* __restrict__ ncount,
                              const int* __restrict__ nlevel, int* __restrict__ blev) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nnodes || nchildn[v] != 0) return;
  int lev = nlevel[v];
  for (int b = nbegin[v]; b < nbegin[v] + ncount[v]; b++) blev[b] = lev;
}

// every cell's radius as before any solve sets it: the half side of its box (a tree kernel that
// sets final radii leaves those of a tree with a leaf it could not rank unfinished)
template <typename T>
__global__ void k_box_radii(int nnodes, const int* __restrict__ nlevel,
                            const int* __restrict__ nsid, const int* __restrict__ npos,
                            const T* __restrict__ box, vec4<T>* __restrict__ cX) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < nnodes) cX[npos[v]].w = div_rn(box[16 * nsid[v] + 3], (T)(1 << nlevel[v]));
}

// key truncated to the body's leaf, scattered back to input order
__global__ void k_tkey(int n, const unsigned long long* __restrict__ skeys,
                       const int* __restrict__ sidx, const int* __restrict__ blev,
                       unsigned long long* __restrict__ tkey, int* __restrict__ iota) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n) return;
  int lev = blev[b];
  unsigned long long mask = lev == 0 ? 0ULL : (~0ULL << (3 * (kMaxLevel - lev)));
  tkey[sidx[b]] = skeys[b] & mask;
  iota[b] = b;
}

template <typename T>
__global__ void k_permute(int n, const vec4<T>* __restrict__ in, const int* __restrict__ order,
                          vec4<T>* __restrict__ out) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < n) out[b] = in[order[b]];
}

// Sort (key, body) pairs by (root, key), stable: one radix sort on the key over all roots,
// then a stable radix sort on the root id (least significant digit first), so the result is
// each root's range sorted on its own, as when the root is solved alone.  (CUB's segmented
// sort gives each segment one thread block, which is slow for a few large segments.)
template <typename T>
static void forest_sort(Solver<T>& s, const unsigned long long* kin, unsigned long long* kout,
                        const int* vin, int* vout, int n, int nroots, int end_bit,
                        int begin_bit = 0) {
  if (nroots == 1) {
    sort_pairs_u64(s, kin, kout, vin, vout, n, end_bit, begin_bit);
    return;
  }
  const int TB = 256;
  s.fs_keys.ensure(n);
  s.fs_idx.ensure(n);
  s.fs_root.ensure(n);
  s.fs_root2.ensure(n);
  s.fs_pos.ensure(n);
  s.fs_pos2.ensure(n);
  sort_pairs_u64(s, kin, s.fs_keys.p, vin, s.fs_idx.p, n, end_bit, begin_bit);
  k_root_of<<<ceil_div(n, TB), TB, 0, s.stream>>>(n, s.fs_idx.p, s.root_first, nroots,
                                                  s.fs_root.p, s.fs_pos.p);
  FMM_LAUNCH_CHECK();
  int bits = 1;
  while ((1LL << bits) < (long long)nroots) bits++;
  sort_pairs_u32(s, s.fs_root.p, s.fs_root2.p, s.fs_pos.p, s.fs_pos2.p, n, bits);
  k_gather_kv<<<ceil_div(n, TB), TB, 0, s.stream>>>(n, s.fs_pos2.p, s.fs_keys.p, s.fs_idx.p,
                                                    kout, vout);
  FMM_LAUNCH_CHECK();
}

// ---------------------------------------------------------------- uniform Morton tree
// BuildTree of include/build_tree_omp.h:214-262 (the builder of an OpenMP build without TBB,
// include/build_tree.h:12-13): every leaf at the depth `level` the host computes as the
// reference does (:218), bodies keyed by the interleaved bits of their grid cell at the
// leaf size d (getKey :36-57), stably sorted by key (radixSort :59-121), one leaf per run of
// equal keys (bodies2leafs :130-158), the parents of each level one per run of equal
// key / 8^l (leafs2cells :160-198), then the cell array reversed (reverseOrder :200-211):
// root first, each level in descending key order, children contiguous.  The cells are
// formed in the reference's construction order (leaves ascending, then each level above)
// and written at index ncells - 1 - c, with the reference's values throughout, including
// its root IPARENT (ncells - 1) and leaf ICHILD (ncells).
constexpr int kUniformMaxLevel = 10;  // the reference's `int id` holds 3 level bits (:45)

// the cell size of a level as getKey declares it: `float d = 2 * box.R / (1 << level)`
// evaluated in the working precision, then made a float (:38); a level above doubles it
// in float (:166)
template <typename T>
__device__ __forceinline__ float uniform_d(const T* __restrict__ box, int level) {
  return (float)div_rn(mul_rn(T(2), box[3]), (T)(1 << level));
}
// grid index along one axis: (X - Xmin) / d in the working precision (d promoted), truncated
template <typename T> __device__ __forceinline__ int uniform_ix(T x, T xmin, float d) {
  return (int)div_rn(sub_rn(x, xmin), (T)d);
}

template <typename T>
__global__ void k_ukeys(const vec4<T>* __restrict__ b, int n, const T* __restrict__ box,
                        int level, unsigned long long* __restrict__ key, int* __restrict__ idx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float d = uniform_d(box, level);
  const vec4<T> x = b[i];
  int ix = uniform_ix(x.x, box[4], d), iy = uniform_ix(x.y, box[5], d),
      iz = uniform_ix(x.z, box[6], d);
  int id = 0;
  for (int l = 0; l < level; l++) {
    id += (ix & 1) << (3 * l);
    id += (iy & 1) << (3 * l + 1);
    id += (iz & 1) << (3 * l + 2);
    ix >>= 1;
    iy >>= 1;
    iz >>= 1;
  }
  key[i] = (unsigned long long)id;
  idx[i] = i;
}

// run heads one level up: child c (construction index cb + c; its first body fb[cb + c], or
// the body c itself when fb is null) starts a new cell when its key shifted right by
// `shift` differs from its predecessor's; flags[m] = 0 closes the scan
__global__ void k_uheads(int m, int cb, const int* __restrict__ fb,
                         const unsigned long long* __restrict__ key, int shift,
                         int* __restrict__ flags) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > m) return;
  if (c == m) {
    flags[m] = 0;
    return;
  }
  const int b = fb ? fb[cb + c] : c;
  const int bp = c == 0 ? 0 : (fb ? fb[cb + c - 1] : c - 1);
  flags[c] = c == 0 || (key[b] >> shift) != (key[bp] >> shift);
}

// the cells of one level from the run heads of the level below (construction order: the new
// cells from ce on); body runs for the leaves (fb == null), cell runs above (ch0, par)
__global__ void k_uemit(int m, int cb, int ce, const int* __restrict__ flags,
                        const int* __restrict__ pos, int* __restrict__ fb,
                        int* __restrict__ ch0, int* __restrict__ par, bool leaves) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m) return;
  const int r = pos[c] + flags[c] - 1;  // the new cell this child (or body) belongs to
  if (flags[c]) {
    fb[ce + r] = leaves ? c : fb[cb + c];
    ch0[ce + r] = leaves ? 0 : cb + c;
  }
  if (!leaves) par[cb + c] = ce + r;
}

struct UniformLevels {
  int begin[kUniformMaxLevel + 2];  // construction range of level l: [begin[l], end[l])
  int end[kUniformMaxLevel + 2];
};

// cell records at index ncells - 1 - c for construction index c (reverseOrder)
template <typename T>
__global__ void k_ucells(int nc, int n, int level, UniformLevels lv, const T* __restrict__ box,
                         const int* __restrict__ fb, const int* __restrict__ ch0,
                         const int* __restrict__ par, const unsigned long long* __restrict__ key,
                         const vec4<T>* __restrict__ bodies, int* __restrict__ iparent,
                         int* __restrict__ ichild, int* __restrict__ nchild,
                         int* __restrict__ ibody, int* __restrict__ nbody,
                         int* __restrict__ clevel, unsigned long long* __restrict__ icell,
                         vec4<T>* __restrict__ cX, int* __restrict__ croot) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  int L = level;
  while (c >= lv.end[L]) L--;  // levels are laid out leaves first
  const int f = nc - 1 - c;
  const int b = fb[c];
  const int nb = (c + 1 < lv.end[L] ? fb[c + 1] : n) - b;
  int nch = 0;
  if (L < level) nch = (c + 1 < lv.end[L] ? ch0[c + 1] : lv.end[L + 1]) - ch0[c];
  // reverseOrder: ICHILD = perm[ICHILD] - NCHILD + 1 (a leaf's ICHILD 0 goes to nc),
  // IPARENT = perm[IPARENT] (the root's IPARENT 0 goes to nc - 1)
  ichild[f] = (nc - 1 - (L < level ? ch0[c] : 0)) - nch + 1;
  iparent[f] = nc - 1 - (L > 0 ? par[c] : 0);
  nchild[f] = nch;
  ibody[f] = b;
  nbody[f] = nb;
  clevel[f] = L;
  icell[f] = key[b] >> (3 * (level - L));
  // centre and radius from the cell's first body at the level's cell size (:148-151,
  // :182-185): d (ix + .5) + Xmin in double, stored in the working precision
  float dl = uniform_d(box, level);
  for (int k = L; k < level; k++) dl *= 2.f;
  const vec4<T> x = bodies[b];
  const T xs[3] = {x.x, x.y, x.z};
  T X[3];
  for (int k = 0; k < 3; k++) {
    const int ik = uniform_ix(xs[k], box[4 + k], dl);
    X[k] = (T)__dadd_rn(__dmul_rn((double)dl, (double)ik + 0.5), (double)box[4 + k]);
  }
  cX[f] = make_v4<T>(X[0], X[1], X[2], (T)__dmul_rn((double)dl, 0.5));
  croot[f] = 0;
}

__global__ void k_iota(int n, int first, int* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = first + i;
}

// depth of the uniform tree for n bodies (include/build_tree_omp.h:218): host arithmetic,
// the reference's own expression (integer n / ncrit, libm log)
int uniform_level(int n, int ncrit) {
  return n >= ncrit ? 1 + int(log((double)(n / ncrit)) / M_LN2 / 3) : 0;
}

template <typename T> static void build_uniform(Solver<T>& s) {
  const int n = s.n, TB = 256;
  const int level = uniform_level(n, s.cfg.ncrit);
  if (level > kUniformMaxLevel)
    throw FmmError(FMM_ERR_NOT_SUPPORTED,
                   "uniform tree deeper than 10 levels (the reference's 32-bit Morton keys "
                   "overflow there)");
  // getKey, radixSort (stable, on the key's 3 level bits), permute
  s.keys.ensure(n);
  s.keys2.ensure(n);
  s.idx.ensure(n);
  s.idx2.ensure(n);
  k_ukeys<T><<<ceil_div(n, TB), TB, 0, s.stream>>>(s.bodies_in.p, n, s.box.p, level, s.keys.p,
                                                   s.idx.p);
  FMM_LAUNCH_CHECK();
  sort_pairs_u64(s, s.keys.p, s.keys2.p, s.idx.p, s.idx2.p, n, std::max(3 * level, 1));
  s.order.ensure(n);
  FMM_CUDA(cudaMemcpyAsync(s.order.p, s.idx2.p, sizeof(int) * n, cudaMemcpyDeviceToDevice,
                           s.stream));
  s.bodies.ensure(n);
  k_permute<T><<<ceil_div(n, TB), TB, 0, s.stream>>>(n, s.bodies_in.p, s.order.p, s.bodies.p);
  FMM_LAUNCH_CHECK();
  // cells in construction order, level by level from the leaves: first body (nbegin),
  // first child (nfirst), parent (nparent); run heads and their scan in nsplit / coff.
  // Level l holds at most min(n, 8^l) cells.
  size_t cap = 16;
  for (int L = 0; L <= level; L++) cap += std::min<size_t>((size_t)n, (size_t)1 << (3 * L));
  s.nbegin.ensure(cap);
  s.nfirst.ensure(cap);
  s.nparent.ensure(cap);
  s.nsplit.ensure((size_t)n + 1);
  s.coff.ensure((size_t)n + 1);
  UniformLevels lv{};
  int cb = 0, m = n, ce = 0;  // the level below: construction range [cb, cb + m)
  for (int L = level; L >= 0; L--) {
    const bool leaves = L == level;
    const int shift = 3 * (level - L);
    k_uheads<<<ceil_div(m + 1, TB), TB, 0, s.stream>>>(m, cb, leaves ? nullptr : s.nbegin.p,
                                                       s.keys2.p, shift, s.nsplit.p);
    FMM_LAUNCH_CHECK();
    exclusive_sum_int(s, s.nsplit.p, s.coff.p, m + 1);
    FMM_CUDA(cudaMemcpyAsync(s.scal_host, s.coff.p + m, sizeof(int), cudaMemcpyDeviceToHost,
                             s.stream));
    k_uemit<<<ceil_div(m, TB), TB, 0, s.stream>>>(m, cb, ce, s.nsplit.p, s.coff.p, s.nbegin.p,
                                                  s.nfirst.p, s.nparent.p, leaves);
    FMM_LAUNCH_CHECK();
    FMM_CUDA(cudaStreamSynchronize(s.stream));
    const int cnt = s.scal_host[0];
    lv.begin[L] = ce;
    lv.end[L] = ce + cnt;
    cb = ce;
    m = cnt;
    ce += cnt;
  }
  const int nc = ce;
  // reverseOrder into the reference's cell layout
  s.c_iparent.ensure(nc); s.c_ichild.ensure(nc); s.c_nchild.ensure(nc);
  s.c_ibody.ensure(nc); s.c_nbody.ensure(nc); s.c_level.ensure(nc);
  s.c_icell.ensure(nc);
  s.cX.ensure(nc);
  s.c_root.ensure(nc);
  k_ucells<T><<<ceil_div(nc, TB), TB, 0, s.stream>>>(
      nc, n, level, lv, s.box.p, s.nbegin.p, s.nfirst.p, s.nparent.p, s.keys2.p, s.bodies.p,
      s.c_iparent.p, s.c_ichild.p, s.c_nchild.p, s.c_ibody.p, s.c_nbody.p, s.c_level.p,
      s.c_icell.p, s.cX.p, s.c_root.p);
  FMM_LAUNCH_CHECK();
  s.c_info.ensure(nc);
  k_cell_info<<<ceil_div(nc, TB), TB, 0, s.stream>>>(nc, s.c_nchild.p, s.c_ichild.p,
                                                     s.c_nbody.p, s.c_ibody.p, s.c_info.p);
  FMM_LAUNCH_CHECK();
  // the level passes walk cells level by level: node v is cell v (npos the identity), the
  // cells of level l at [nc - end[l], nc - begin[l]); every leaf is on the deepest level
  s.npos.ensure(nc);
  k_iota<<<ceil_div(nc, TB), TB, 0, s.stream>>>(nc, 0, s.npos.p);
  FMM_LAUNCH_CHECK();
  const int nleaves = lv.end[level] - lv.begin[level];
  s.leaves.ensure(nleaves);
  k_iota<<<ceil_div(nleaves, TB), TB, 0, s.stream>>>(nleaves, nc - nleaves, s.leaves.p);
  FMM_LAUNCH_CHECK();
  s.level_lo.clear();
  for (int L = 0; L <= level; L++) s.level_lo.push_back(nc - lv.end[L]);
  s.level_lo.push_back(nc);
  s.cbase.ensure(2);
  FMM_CUDA(cudaMemsetAsync(s.cbase.p, 0, sizeof(int), s.stream));
  s.root_cell.assign(1, 0);
  s.maxlevel = level;
  s.ncells = nc;
  s.nleaves = nleaves;
  s.tree_plan = 0;
}

template <typename T> void build_tree(Solver<T>& s, bool radii) {
  const int n = s.n;
  const int TB = 256;
  s.kc_valid = false;  // the host copies of the cells' index fields are stale
  s.radii_set = false;
  s.level_lo.clear();
  s.ncells = s.maxlevel = s.nleaves = 0;
  // roots: non-empty solves in order
  const int nsolves = (int)s.seg.size() - 1;
  s.root_solve.clear();
  std::vector<int> rfirst;
  for (int q = 0; q < nsolves; q++)
    if (s.seg[q + 1] > s.seg[q]) {
      s.root_solve.push_back(q);
      rfirst.push_back(s.seg[q]);
    }
  rfirst.push_back(n);
  const int nroots = (int)s.root_solve.size();
  if (s.cfg.tree == FMM_TREE_UNIFORM && (nroots > 1 || s.ij))
    throw FmmError(FMM_ERR_NOT_SUPPORTED,
                   "the uniform tree builds one tree per call (no batches, no separate target "
                   "and source trees)");
  s.nroots = nroots;
  s.box.ensure(16 * (size_t)std::max(nroots, 1));
  if (nroots == 0) {
    FMM_CUDA(cudaMemsetAsync(s.box.p, 0, 16 * sizeof(T), s.stream));
    s.root_cell.clear();
    return;
  }
  // bounds per root over chunks of at most 4096 bodies (256 blocks at 2^20 bodies); the
  // roots' first bodies, the chunks' ranges and the roots' first chunks in one upload from
  // pinned memory (the last solve's was waited for when its tree was read back, a failed one's
  // when it returned)
  const int CH = 4096;
  int nch = 0;
  for (int r = 0; r < nroots; r++) nch += ceil_div(rfirst[r + 1] - rfirst[r], CH);
  const size_t up = 2 * (size_t)(nroots + 1) + 2 * (size_t)nch;
  s.d_seg.ensure(up);
  if (up > s.seg_host_cap) {
    if (s.seg_host) s.roots_retired.push_back((int2*)s.seg_host);
    s.seg_host = nullptr;
    s.seg_host_cap = 0;
    FMM_CUDA(cudaMallocHost((void**)&s.seg_host, 2 * up * sizeof(int)));
    s.seg_host_cap = 2 * up;
  }
  {
    int *hr = s.seg_host, *hlo = hr + nroots + 1, *hb = hlo + nroots + 1, *he = hb + nch;
    std::copy(rfirst.begin(), rfirst.end(), hr);
    int k = 0;
    for (int r = 0; r < nroots; r++) {
      hlo[r] = k;
      for (int b0 = rfirst[r]; b0 < rfirst[r + 1]; b0 += CH, k++) {
        hb[k] = b0;
        he[k] = std::min(b0 + CH, rfirst[r + 1]);
      }
    }
    hlo[nroots] = k;
  }
  FMM_CUDA(cudaMemcpyAsync(s.d_seg.p, s.seg_host, up * sizeof(int), cudaMemcpyHostToDevice,
                           s.stream));
  s.root_first = s.d_seg.p;
  const int *dlo = s.root_first + nroots + 1, *dcb = dlo + nroots + 1, *dce = dcb + nch;
  s.minmax_part.ensure(6 * (size_t)nch);
  k_minmax_chunks<T><<<nch, TB, 0, s.stream>>>(s.bodies_in.p, dcb, dce, s.minmax_part.p);
  FMM_LAUNCH_CHECK();
  k_box<T><<<nroots, TB, 0, s.stream>>>(nroots, dlo, s.minmax_part.p,
                                        s.ij && s.ij_common_box ? 1 : 0, s.box.p);
  FMM_LAUNCH_CHECK();
  phase_end(s, FMM_PHASE_BOUNDS);
  phase_begin(s, FMM_PHASE_TREE);
  if (s.cfg.tree == FMM_TREE_UNIFORM) {
    build_uniform(s);
    return;
  }
  s.keys.ensure(n);
  s.keys2.ensure(n);
  s.idx.ensure(n);
  s.idx2.ensure(n);
  s.order.ensure(n);
  s.bodies.ensure(n);
  s.cbase.ensure(nroots + 1);
  s.tree_ctl.ensure(TC_INTS);
  const bool rank = s.cfg.ncrit <= kRankBodies;
  // With a plan of L levels to split, the keys are sorted on their top L digits only: the
  // splits read no deeper digit, and the bodies of a leaf are put in input order afterwards
  // whatever the order of their deeper digits.  A tree that turns out deeper is built again
  // with the keys sorted on every digit.
  int levels = s.tree_plan > 0 && rank ? std::min(s.tree_plan + 1, kMaxLevel) : kMaxLevel;
  size_t cap = tree_first_nodes(n, s.cfg.ncrit, nroots);
  int* hc = s.scal_host + kTreeHost;
  bool sorted = false;
  for (;;) {
    if (cap == 0)
      throw FmmError(FMM_ERR_NOT_SUPPORTED, "more than 2^27 - 1 cells (list pairs hold 27-bit cells)");
    if (!sorted) {
      k_keys<T><<<ceil_div(n, TB), TB, 0, s.stream>>>(s.bodies_in.p, n, s.box.p, s.root_first,
                                                      nroots, s.keys.p, s.idx.p);
      FMM_LAUNCH_CHECK();
      forest_sort(s, s.keys.p, s.keys2.p, s.idx.p, s.idx2.p, n, nroots, 3 * kMaxLevel,
                  3 * (kMaxLevel - levels));
      sorted = true;
    }
    DevArr<int>* narr[] = {&s.nbegin, &s.ncount, &s.nparent, &s.nchildn, &s.nfirst, &s.nnode,
                           &s.npos, &s.ncb, &s.nlevel, &s.nsid, &s.c_iparent, &s.c_ichild,
                           &s.c_nchild, &s.c_ibody, &s.c_nbody, &s.c_level, &s.c_root, &s.leaves};
    size_t ncap = kTreeMaxNodes;
    for (auto* q : narr) {
      q->ensure(cap);
      ncap = std::min(ncap, q->cap);
    }
    s.nX.ensure(4 * cap);
    s.nM0.ensure(cap);
    s.m0.ensure(cap);
    s.c_icell.ensure(cap);
    s.c_info.ensure(cap);
    s.cX.ensure(cap);
    ncap = std::min({ncap, s.nX.cap / 4, s.nM0.cap, s.m0.cap, s.c_icell.cap, s.c_info.cap, s.cX.cap});
    TreeArgs<T> t{};
    t.keys = s.keys2.p;
    t.sidx = s.idx2.p;
    t.bodies_in = s.bodies_in.p;
    t.box = s.box.p;
    t.root_first = s.root_first;
    t.nroots = nroots;
    t.ncrit = s.cfg.ncrit;
    t.levels = levels;
    t.ncap = (int)ncap;
    t.rank = rank;
    t.radii = rank && radii;
    t.use_rmax = s.cfg.use_rmax;
    t.theta = (T)s.cfg.theta;
    t.ctl = s.tree_ctl.p;
    t.nbegin = s.nbegin.p, t.ncount = s.ncount.p, t.nparent = s.nparent.p;
    t.nchildn = s.nchildn.p, t.nfirst = s.nfirst.p, t.nnode = s.nnode.p, t.npos = s.npos.p;
    t.ncb = s.ncb.p, t.nlevel = s.nlevel.p, t.nsid = s.nsid.p, t.nX = s.nX.p, t.nM0 = s.nM0.p;
    t.cbase = s.cbase.p, t.order = s.order.p, t.iparent = s.c_iparent.p, t.ichild = s.c_ichild.p;
    t.nchild = s.c_nchild.p, t.ibody = s.c_ibody.p, t.nbody = s.c_nbody.p;
    t.clevel = s.c_level.p, t.croot = s.c_root.p, t.leaves = s.leaves.p, t.bodies = s.bodies.p;
    t.icell = s.c_icell.p, t.info = s.c_info.p, t.cX = s.cX.p, t.m0 = s.m0.p;
    int blocks = tree_blocks(n, s.cfg.ncrit, tree_resident<T>(s));
    FMM_CUDA(cudaMemsetAsync(s.tree_ctl.p, 0, TC_INTS * sizeof(int), s.stream));
    void* args[] = {&t};
    if (blocks <= 2 * kTreeCluster) {
      // a few blocks: one cluster, whose barrier costs a fifth (1,000 bodies:
      // tree 0.115 -> 0.094 ms, a solve 0.465 -> 0.443)
      blocks = std::min(blocks, kTreeCluster);
      t.cluster = 1;
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = blocks;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(blocks);
      cfg.blockDim = dim3(kTreeThreads);
      cfg.stream = s.stream;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      FMM_CUDA(cudaLaunchKernelExC(&cfg, (const void*)k_tree<T>, args));
    } else {
      FMM_CUDA(cudaLaunchCooperativeKernel((const void*)k_tree<T>, dim3(blocks),
                                           dim3(kTreeThreads), args, 0, s.stream));
    }
    FMM_LAUNCH_CHECK();
    FMM_CUDA(cudaMemcpyAsync(hc, s.tree_ctl.p, TC_INTS * sizeof(int), cudaMemcpyDeviceToHost,
                             s.stream));
    s.root_cell.assign(nroots, 0);
    if (nroots > 1)
      FMM_CUDA(cudaMemcpyAsync(s.root_cell.data(), s.cbase.p, sizeof(int) * nroots,
                               cudaMemcpyDeviceToHost, s.stream));
    FMM_CUDA(cudaStreamSynchronize(s.stream));
    if (hc[TC_FAULT]) throw FmmError(FMM_ERR_DEVICE, "the tree build's blocks lost one another");
    bool full = false, deep = false;
    for (int l = 0; l < kMaxLevel; l++) {
      full |= hc[TC_FULL + l] != 0;
      deep |= hc[TC_DEEP + l] != 0;
    }
    if (deep) {
      levels = kMaxLevel;
      sorted = false;
    }
    if (full) cap = tree_more_nodes(ncap);
    if (!deep && !full) break;
  }
  s.level_lo.assign({0, nroots});
  for (int l = 1; hc[TC_COUNT + l]; l++) s.level_lo.push_back(s.level_lo.back() + hc[TC_COUNT + l]);
  const int nlev = (int)s.level_lo.size() - 1, nnodes = s.level_lo.back();
  s.tree_plan = nlev;
  s.maxlevel = nlev - 1;
  s.ncells = nnodes;
  s.nleaves = hc[TC_LEAVES];
  if (rank && !hc[TC_BIG]) {
    s.radii_set = radii;
    return;
  }
  if (rank && radii) {  // (the structure pass then forms the radii from the boxes')
    k_box_radii<T><<<ceil_div(nnodes, TB), TB, 0, s.stream>>>(nnodes, s.nlevel.p, s.nsid.p,
                                                              s.npos.p, s.box.p, s.cX.p);
    FMM_LAUNCH_CHECK();
  }
  // leaves of more bodies than a warp ranks: stable sort by leaf-truncated key from input order
  // (the keys are sorted on every digit here: such leaves come with a large ncrit, which plans no
  // levels, or lie on the last level)
  int* blev = s.idx.p;
  k_leaf_levels<<<ceil_div(nnodes, TB), TB, 0, s.stream>>>(nnodes, s.nchildn.p, s.nbegin.p,
                                                           s.ncount.p, s.nlevel.p, blev);
  FMM_LAUNCH_CHECK();
  k_tkey<<<ceil_div(n, TB), TB, 0, s.stream>>>(n, s.keys2.p, s.idx2.p, blev, s.keys.p, s.order.p);
  FMM_LAUNCH_CHECK();
  // s.order holds 0..n-1 (input positions); sort them by truncated key within each root
  FMM_CUDA(cudaMemcpyAsync(s.idx.p, s.order.p, n * sizeof(int), cudaMemcpyDeviceToDevice,
                           s.stream));
  forest_sort(s, s.keys.p, s.keys2.p, s.idx.p, s.order.p, n, nroots, 3 * kMaxLevel);
  k_permute<T><<<ceil_div(n, TB), TB, 0, s.stream>>>(n, s.bodies_in.p, s.order.p, s.bodies.p);
  FMM_LAUNCH_CHECK();
}

// The bodies of part `part` of nparts: [t0, t1) with t = floor(k n / nparts), each bound
// moved down to the first body of the leaf that holds it, so that every leaf belongs to one
// part.  One leaf holds each bound below n and writes it; the leaf that ends at n writes
// the bound n.
__global__ void k_part_range(int nleaves, const int* __restrict__ leaves,
                             const int* __restrict__ ibody, const int* __restrict__ nbody, int n,
                             int t0, int t1, int* __restrict__ range) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nleaves) return;
  const int c = leaves[i];
  const int b = ibody[c], e = b + nbody[c];
  if (b <= t0 && t0 < e) range[0] = b;
  if (b <= t1 && t1 < e) range[1] = b;
  if (t1 >= n && e == n) range[1] = n;
}

void partition_range(SolverBase& s) {
  if (s.nparts <= 1) return;
  if (s.nroots > 1 || s.ij)
    throw FmmError(FMM_ERR_NOT_SUPPORTED, "a partitioned solve is one solve of one tree");
  if (s.cfg.mutual && s.cfg.images == 0)
    throw FmmError(FMM_ERR_NOT_SUPPORTED, "a partitioned solve with the mutual traversal");
  s.part_range.ensure(2);
  if (s.n == 0 || s.nleaves == 0) return;
  const int t0 = (int)((long long)s.part * s.n / s.nparts);
  const int t1 = (int)((long long)(s.part + 1) * s.n / s.nparts);
  k_part_range<<<ceil_div(s.nleaves, 256), 256, 0, s.stream>>>(
      s.nleaves, s.leaves.p, s.c_ibody.p, s.c_nbody.p, s.n, t0, t1, s.part_range.p);
  FMM_LAUNCH_CHECK();
}

template void build_tree<float>(Solver<float>&, bool);
template void build_tree<double>(Solver<double>&, bool);

}  // namespace fmmb200
