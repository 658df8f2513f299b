// Dual-tree traversal on the device (Traversal::dualTreeTraversal, include/traversal.h).
//
// The reference recurses from (root, root) (:248): a pair is far (M2L) when
// |Xi - Xj|^2 > (Ri + Rj)^2 (:40), two leaves interact directly (P2P, :44-58), and
// otherwise splitCell (:188-212) descends into the children of the leaf-less side, of both
// sides when NBODY_i + NBODY_j >= nspawn (TraverseRange :65-124, which for mutual = false
// visits every child pair), or of the larger cell (ties split Ci).  The set of emitted
// pairs depends only on each pair, so here a few steps breadth first make a frontier of pairs
// (k_trav_step), whose subtrees of pairs the blocks of one kernel then walk, each with a stack
// of its own (k_traverse).  Counts beyond a buffer's size are reported and the walk is done
// again on larger buffers.  Lists are then grouped by target (per-target CSR for the M2L and
// P2P kernels) and sorted by source within each target.
#include <algorithm>
#include <climits>
#include <vector>

#include "fmm_solver.cuh"

namespace fmmb200 {

enum {
  PAIR_DROP = -1,  // a partitioned solve: the target cell holds none of the part's bodies
  PAIR_M2L = 0, PAIR_P2P = 1, PAIR_SPLIT_I = 2, PAIR_SPLIT_J = 3, PAIR_SPLIT_IJ = 4,
  PAIR_SPLIT_SELF = 5  // mutual: a cell against itself, its children pairs (a, b), a <= b
};

// cj: source cell with the periodic image of the source tree in its top bits (pair_cell,
// pair_img); the distance is (Xi - Xj) - Xperiodic as the reference rounds it (:38)
// mutual (dualTreeTraversal's flag, open boundary): each unordered pair is visited once
// (TraverseRange drops the (latter, former) quarter of a range against itself, :108-113),
// a cell against itself always splits both sides (:200), and an M2L or a P2P between two
// different cells is emitted in both directions (the mutual kernels update both cells);
// *nout counts those outputs
// The pair's cell data (centres with radii, and (NCHILD, ICHILD, NBODY, IBODY)) are loaded
// together, so that a pair costs one round trip to memory rather than one per decision.
// A partitioned solve drops the pairs whose target cell holds none of the bodies [b0, b1):
// every pair below them has a target inside that cell, so the pairs kept are exactly the
// whole traversal's pairs of the part's targets (b0 = INT_MIN, b1 = INT_MAX keep all).
template <typename T>
__device__ __forceinline__ int classify_data(int ci, int cjp, const vec4<T>& a, const vec4<T>& b,
                                             const int4& fi, const int4& fj, int nspawn, T cycle,
                                             int mutual, int b0, int b1, int* nout) {
  const int cj = pair_cell((unsigned)cjp);
  T px, py, pz;
  img_shift<T>(pair_img((unsigned)cjp), cycle, px, py, pz);
  if (!(fi.w < b1 && fi.w + fi.z > b0)) {
    *nout = 0;
    return PAIR_DROP;
  }
  T R2 = norm_rn(sub_rn(sub_rn(a.x, b.x), px), sub_rn(sub_rn(a.y, b.y), py),
                 sub_rn(sub_rn(a.z, b.z), pz));
  T Rs = add_rn(a.w, b.w);
  if (R2 > mul_rn(Rs, Rs)) {
    *nout = mutual ? 2 : 1;
    return PAIR_M2L;
  }
  const int ni = fi.x, nj = fj.x;
  if (ni == 0 && nj == 0) {
    *nout = mutual && ci != cj ? 2 : 1;
    return PAIR_P2P;
  }
  if (nj == 0) {
    *nout = ni;
    return PAIR_SPLIT_I;
  }
  if (ni == 0) {
    *nout = nj;
    return PAIR_SPLIT_J;
  }
  if (mutual && ci == cj) {
    *nout = ni * (ni + 1) / 2;
    return PAIR_SPLIT_SELF;
  }
  if (fi.z + fj.z >= nspawn) {
    *nout = ni * nj;
    return PAIR_SPLIT_IJ;
  }
  if (a.w >= b.w) {
    *nout = ni;
    return PAIR_SPLIT_I;
  }
  *nout = nj;
  return PAIR_SPLIT_J;
}
// the part's body range [range[0], range[1]) of a partitioned solve, else everything
__device__ __forceinline__ void part_bounds(const int* __restrict__ range, int& b0, int& b1) {
  b0 = INT_MIN;
  b1 = INT_MAX;
  if (range) {
    b0 = range[0];
    b1 = range[1];
  }
}

// One traversal step.  Each lane takes kTravItems consecutive frontier pairs (their loads are
// independent); output slots come from a warp-wide scan of the lanes' packed (M2L, P2P,
// children) counts, the block's warps' totals and three atomics per block and 512 pairs.  (Three
// per warp, all on the same addresses, and four pairs a lane at 126 registers: traverse phase of
// Plummer 2^20 0.89 ms, now 0.79; sphere of 2^22 1.13 -> 0.93; 256 solves 4.18 -> 3.79.  One
// pair a lane 0.81, 1.03 and 4.18; four in 80 registers 0.94, 1.12 and 4.42; the children of a
// split written by the whole warp 0.99, 1.33 and 4.65.)  Writes beyond a buffer's capacity are
// skipped but every slot below it is written and all are counted, so the host can tell an
// overflow from the counts and run the traversal again on larger buffers.
constexpr int kTravItems = 2, kTravStepThreads = 256;
constexpr int kTravMaxSteps = 2 * (kMaxLevel + 1) + 2;

template <typename T> struct TravArgs {
  int2 *front, *front2;  // the first frontier in front
  unsigned long long front_cap, nfront0, m2l_cap, p2p_cap;
  const vec4<T>* X;
  const int4* info;
  int nspawn, mutual, ncells;
  T cycle;
  const int* range;  // the part's bodies, or null
  // [0] M2L, [1] P2P, [2] bad index, [3] pairs of the last frontier taken by k_traverse's
  // blocks, [4] a stack overflowed, [5 + l] frontier size after step l; zero at the start
  unsigned long long* ctr;
  unsigned long long *m2l, *p2p;
  int2* stacks;  // kTravStack pairs per block of k_traverse
};

// the first n pairs that a split of p puts in its place
__device__ __forceinline__ void trav_children(const int4* __restrict__ info, int ty, int2 p, int n,
                                              int2* out) {
  const int4 fi = info[p.x], fj = info[pair_cell((unsigned)p.y)];
  const int img = (int)((unsigned)p.y & ~kCellMask);
  if (ty == PAIR_SPLIT_SELF) {
    int w = 0;
    for (int a = 0; a < fi.x; a++)
      for (int b = a; b < fi.x; b++, w++)
        if (w < n) out[w] = make_int2(fi.y + a, fi.y + b);
  } else if (ty == PAIR_SPLIT_I) {
    for (int i = 0; i < n; i++) out[i] = make_int2(fi.y + i, p.y);
  } else if (ty == PAIR_SPLIT_J) {
    for (int j = 0; j < n; j++) out[j] = make_int2(p.x, (fj.y + j) | img);
  } else {
    for (int i = 0; i < n; i++) out[i] = make_int2(fi.y + i / fj.x, (fj.y + i % fj.x) | img);
  }
}

template <typename T>
__device__ __forceinline__ void trav_step(const TravArgs<T>& g, const vec4<T>* __restrict__ X,
                                          const int4* __restrict__ info, const int2* front,
                                          long long nfront, int2* next,
                                          unsigned long long* next_count, int b0, int b1) {
  const int nspawn = g.nspawn, mutual = g.mutual, ncells = g.ncells;
  const T cycle = g.cycle;
  unsigned long long *ctr = g.ctr, *m2l = g.m2l, *p2p = g.p2p;
  const unsigned long long m2l_cap = g.m2l_cap, p2p_cap = g.p2p_cap, next_cap = g.front_cap;
  const int lane = lane_id();
  constexpr int WARPS = kTravStepThreads / 32;
  __shared__ unsigned wtot[WARPS];
  __shared__ unsigned long long at[3];
  const int wl = threadIdx.x >> 5;
  const long long stride = (long long)gridDim.x * kTravStepThreads * kTravItems;
  const long long base = (long long)blockIdx.x * kTravStepThreads * kTravItems;
  for (long long w = base; w < nfront; w += stride) {  // block-uniform trip count
    const long long t0 = w + (long long)threadIdx.x * kTravItems;
    int ty[kTravItems], k[kTravItems];
    int2 p[kTravItems];
    unsigned v = 0;  // packed: M2L in bits 0-8, P2P in 9-17, children in 18-31 (warp totals:
                     // <= 128, <= 128, <= 4096)
#pragma unroll
    for (int u = 0; u < kTravItems; u++) {
      ty[u] = -1;
      k[u] = 0;
      p[u] = t0 + u < nfront ? front[t0 + u] : make_int2(0, 0);
    }
    bool okp[kTravItems];
#pragma unroll
    for (int u = 0; u < kTravItems; u++)
      okp[u] = t0 + u < nfront && (unsigned)p[u].x < (unsigned)ncells &&
               (unsigned)pair_cell((unsigned)p[u].y) < (unsigned)ncells &&
               pair_img((unsigned)p[u].y) < 27;
    if constexpr (sizeof(T) == 4) {
      // FP32: all the items' cell data loaded before any is classified, so that the gathers
      // of the pairs are in flight together (FP64 cells take twice the registers: one pair at
      // a time)
      vec4<T> ca[kTravItems], cb[kTravItems];
      int4 fa[kTravItems], fb[kTravItems];
#pragma unroll
      for (int u = 0; u < kTravItems; u++)
        if (okp[u]) {
          const int cj = pair_cell((unsigned)p[u].y);
          ca[u] = X[p[u].x];
          cb[u] = X[cj];
          fa[u] = info[p[u].x];
          fb[u] = info[cj];
        }
#pragma unroll
      for (int u = 0; u < kTravItems; u++)
        if (okp[u])
          ty[u] = classify_data<T>(p[u].x, p[u].y, ca[u], cb[u], fa[u], fb[u], nspawn, cycle,
                                   mutual, b0, b1, &k[u]);
    } else {
#pragma unroll
      for (int u = 0; u < kTravItems; u++)
        if (okp[u]) {
          const int cj = pair_cell((unsigned)p[u].y);
          ty[u] = classify_data<T>(p[u].x, p[u].y, X[p[u].x], X[cj], info[p[u].x], info[cj],
                                   nspawn, cycle, mutual, b0, b1, &k[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < kTravItems; u++) {
      if (t0 + u < nfront && !okp[u])
        atomicOr(&ctr[2], 1ULL);  // never expected: reported to the host, pair skipped
      v += (ty[u] == PAIR_M2L ? (unsigned)k[u] : 0u) |
           (ty[u] == PAIR_P2P ? (unsigned)k[u] << 9 : 0u) |
           (ty[u] >= PAIR_SPLIT_I ? (unsigned)k[u] << 18 : 0u);
    }
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) wtot[wl] = incl;
    __syncthreads();
    // bits of a field in the packed totals: M2L, P2P, children
    auto field = [](unsigned x, int f) { return f == 0 ? x & 0x1ffu : f == 1 ? x >> 9 & 0x1ffu : x >> 18; };
    unsigned long long bm = 0, bp = 0, bn = 0;  // of the block's earlier warps
    for (int k = 0; k < wl; k++) {
      bm += field(wtot[k], 0);
      bp += field(wtot[k], 1);
      bn += field(wtot[k], 2);
    }
    if (threadIdx.x < 3) {
      unsigned sum = 0;
      for (int k = 0; k < WARPS; k++) sum += field(wtot[k], threadIdx.x);
      at[threadIdx.x] =
          sum ? atomicAdd(threadIdx.x < 2 ? &ctr[threadIdx.x] : next_count, (unsigned long long)sum)
              : 0;
    }
    __syncthreads();
    bm += at[0] + field(incl - v, 0);
    bp += at[1] + field(incl - v, 1);
    bn += at[2] + field(incl - v, 2);
#pragma unroll
    for (int u = 0; u < kTravItems; u++) {
      const unsigned long long packed =
          ((unsigned long long)(unsigned)p[u].x << 32) | (unsigned)p[u].y;
      const unsigned long long rev =
          ((unsigned long long)(unsigned)p[u].y << 32) | (unsigned)p[u].x;
      if (ty[u] == PAIR_M2L) {
        if (bm < m2l_cap) m2l[bm] = packed;
        if (k[u] == 2 && bm + 1 < m2l_cap) m2l[bm + 1] = rev;
        bm += k[u];
      } else if (ty[u] == PAIR_P2P) {
        if (bp < p2p_cap) p2p[bp] = packed;
        if (k[u] == 2 && bp + 1 < p2p_cap) p2p[bp + 1] = rev;
        bp += k[u];
      } else if (ty[u] >= PAIR_SPLIT_I) {
        // every slot below the capacity is written (the next step reads up to it)
        const unsigned long long o = bn;
        const int kw = o >= next_cap ? 0 : (int)min((unsigned long long)k[u], next_cap - o);
        trav_children(info, ty[u], p[u], kw, next + o);
        bn += k[u];
      }
    }
  }
}

// Step l as a launch of its own, its frontier's size read on the device.
template <typename T>
__global__ void __launch_bounds__(kTravStepThreads, 4) k_trav_step(TravArgs<T> g, int l) {
  int b0, b1;
  part_bounds(g.range, b0, b1);
  const unsigned long long n = l == 0 ? g.nfront0 : min(g.ctr[4 + l], g.front_cap);
  trav_step<T>(g, g.X, g.info, (l & 1) ? g.front2 : g.front, (long long)n,
               (l & 1) ? g.front : g.front2, &g.ctr[5 + l], b0, b1);
}

// The pairs below the frontier that l0 steps left.  A block takes pairs of the frontier a few
// at a time and walks all that comes of them: up to kTravThreads pairs from the top of its
// stack per round, one per thread, whose children go back on the stack and whose M2L and P2P
// pairs go through shared memory to the lists a few hundred at a time.  No block waits for
// another: a launch per step costs 5-6 us however few pairs it has.
constexpr int kTravThreads = 128, kTravBlocks = 8;  // per block; blocks per SM
constexpr int kTravBuf = 512;     // pairs of either list that a block holds back
constexpr int kTravStack = 4096;  // pairs

template <typename T>
__global__ void __launch_bounds__(kTravThreads, kTravBlocks) k_traverse(TravArgs<T> g, int l0) {
  __shared__ unsigned long long mbuf[kTravBuf], pbuf[kTravBuf], mat, pat, taken;
  __shared__ int nm, np, kids[2];
  const int tid = threadIdx.x, lane = lane_id();
  int b0, b1;
  part_bounds(g.range, b0, b1);
  const int2* front = (l0 & 1) ? g.front2 : g.front;
  const unsigned long long n = l0 == 0 ? g.nfront0 : min(g.ctr[4 + l0], g.front_cap);
  // pairs taken at a time: few enough that every block comes to the frontier several times
  const int chunk =
      (int)min(n / (4 * gridDim.x) + 4, (unsigned long long)kTravThreads);
  int2* stack = g.stacks + (size_t)blockIdx.x * kTravStack;
  if (tid == 0) nm = np = kids[0] = kids[1] = 0;
  auto flush = [&](int cm, int cp) {
    __syncthreads();  // (all have read the counts)
    if (tid == 0) {
      mat = cm ? atomicAdd(&g.ctr[0], (unsigned long long)cm) : 0;
      nm = 0;
    }
    if (tid == 32) {
      pat = cp ? atomicAdd(&g.ctr[1], (unsigned long long)cp) : 0;
      np = 0;
    }
    __syncthreads();
    for (int i = tid; i < cm; i += kTravThreads)
      if (mat + i < g.m2l_cap) g.m2l[mat + i] = mbuf[i];
    for (int i = tid; i < cp; i += kTravThreads)
      if (pat + i < g.p2p_cap) g.p2p[pat + i] = pbuf[i];
  };
  int top = 0;
  bool more = true;
  for (int it = 0;; it++) {
    __syncthreads();
    top = min(top + kids[(it + 1) & 1], kTravStack);
    const int cm = nm, cp = np;
    if (max(cm, cp) > kTravBuf - 2 * kTravThreads) flush(cm, cp);
    int got = 0;
    unsigned long long from = 0;
    if (top < kTravThreads && more) {
      const int want = min(chunk, kTravThreads - top);
      if (tid == 0) taken = atomicAdd(&g.ctr[3], (unsigned long long)want);
      __syncthreads();
      from = taken;
      got = from < n ? (int)min((unsigned long long)want, n - from) : 0;
      more = from + want < n;
    }
    const int own = min(top, kTravThreads);
    if (own + got == 0) {
      if (max(cm, cp) <= kTravBuf - 2 * kTravThreads) flush(cm, cp);
      return;
    }
    int2 p = make_int2(0, 0);
    int ty = -1, k = 0;
    if (tid < own + got) {
      p = tid < own ? stack[top - 1 - tid] : front[from + (tid - own)];
      const int cj = pair_cell((unsigned)p.y);
      if ((unsigned)p.x < (unsigned)g.ncells && (unsigned)cj < (unsigned)g.ncells &&
          pair_img((unsigned)p.y) < 27)
        ty = classify_data<T>(p.x, p.y, g.X[p.x], g.X[cj], g.info[p.x], g.info[cj], g.nspawn,
                              g.cycle, g.mutual, b0, b1, &k);
      else
        atomicOr(&g.ctr[2], 1ULL);  // never expected: reported to the host, pair skipped
    }
    top -= own;
    // M2L in bits 0-7, P2P in 8-15, children in 16-31 (warp totals: <= 64, <= 64, <= 2048)
    const unsigned v = ty == PAIR_M2L ? (unsigned)k
                       : ty == PAIR_P2P ? (unsigned)k << 8
                       : ty >= PAIR_SPLIT_I ? (unsigned)k << 16 : 0u;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    __syncthreads();  // every thread has its pair
    if (tid == 0) kids[(it + 1) & 1] = 0;
    int bm = 0, bp = 0, bn = 0;
    if (lane == 31) {
      if (incl & 0xffu) bm = atomicAdd(&nm, (int)(incl & 0xffu));
      if ((incl >> 8) & 0xffu) bp = atomicAdd(&np, (int)((incl >> 8) & 0xffu));
      if (incl >> 16) bn = atomicAdd(&kids[it & 1], (int)(incl >> 16));
    }
    const unsigned excl = incl - v;
    bm = __shfl_sync(0xffffffffu, bm, 31) + (int)(excl & 0xffu);
    bp = __shfl_sync(0xffffffffu, bp, 31) + (int)((excl >> 8) & 0xffu);
    bn = __shfl_sync(0xffffffffu, bn, 31) + (int)(excl >> 16) + top;
    const unsigned long long packed = (unsigned long long)(unsigned)p.x << 32 | (unsigned)p.y;
    const unsigned long long rev = (unsigned long long)(unsigned)p.y << 32 | (unsigned)p.x;
    if (ty == PAIR_M2L) {
      mbuf[bm] = packed;
      if (k == 2) mbuf[bm + 1] = rev;
    } else if (ty == PAIR_P2P) {
      pbuf[bp] = packed;
      if (k == 2) pbuf[bp + 1] = rev;
    } else if (ty >= PAIR_SPLIT_I) {
      const int room = min(k, kTravStack - bn);
      if (room < k) g.ctr[4] = 1;
      trav_children(g.info, ty, p, room, stack + bn);
    }
  }
}

// ---------------------------------------------------------------- grouping by target
// A list leaves the traversal in the order its pairs were found (atomic slots).  It is
// grouped by target with a count per target (warp-aggregated atomics), an exclusive scan
// of the counts into the CSR offsets, and a scatter of every pair's source key
// (image << b | cell) into its target's range; each range is then sorted in shared memory
// and written back as (target << 32 | image << 27 | cell).  The result is the order of a
// global sort of the packed pairs (target, then image, then source cell), so it does not
// depend on the order in which the traversal emitted them.
constexpr int kSegWarpCap = 1024;   // keys one warp sorts in its registers
constexpr int kSegBlockCap = 8192;  // keys one block sorts; longer ranges: global sort
constexpr int kSegWarps = 8;
constexpr int kSegBlock = 512;
constexpr int kSegBothCells = 2048;  // trees whose two lists are grouped together

struct SegList {
  unsigned long long* pairs;
  long long n;
  int *cnt, *off;      // counts per target (zeros at the start), CSR offsets
  unsigned* keys;      // n keys of scratch
  int* overflow;       // set if a range is too long for k_seg_sort_block
};
struct SegLists {
  SegList l[2];
  __device__ __forceinline__ SegList at(int k) const { return k ? l[1] : l[0]; }
};
// (blockIdx.y: the list)

__global__ void k_seg_count(SegLists g) {
  const unsigned long long* __restrict__ pairs = g.at(blockIdx.y).pairs;
  const long long n = g.at(blockIdx.y).n;
  int* __restrict__ cnt = g.at(blockIdx.y).cnt;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t0 = blockIdx.x * (long long)blockDim.x; t0 < n; t0 += stride) {
    const long long t = t0 + threadIdx.x;
    const unsigned act = __ballot_sync(0xffffffffu, t < n);
    if (t >= n) continue;
    const int tgt = (int)(pairs[t] >> 32);
    const unsigned grp = __match_any_sync(act, tgt);
    if (lane_id() == __ffs(grp) - 1) atomicAdd(&cnt[tgt], __popc(grp));
  }
}

// cnt holds the counts on entry and zeros on exit; each warp's pairs of one target take
// consecutive slots from the top of the target's remaining range
__global__ void k_seg_scatter(SegLists g, int b) {
  const unsigned long long* __restrict__ pairs = g.at(blockIdx.y).pairs;
  const long long n = g.at(blockIdx.y).n;
  const int* __restrict__ off = g.at(blockIdx.y).off;
  int* __restrict__ cnt = g.at(blockIdx.y).cnt;
  unsigned* __restrict__ keys = g.at(blockIdx.y).keys;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int lane = lane_id();
  for (long long t0 = blockIdx.x * (long long)blockDim.x; t0 < n; t0 += stride) {
    const long long t = t0 + threadIdx.x;
    const unsigned act = __ballot_sync(0xffffffffu, t < n);
    if (t >= n) continue;
    const unsigned long long v = pairs[t];
    const int tgt = (int)(v >> 32);
    const unsigned src = (unsigned)v;
    const unsigned grp = __match_any_sync(act, tgt);
    const int leader = __ffs(grp) - 1, k = __popc(grp);
    int top = 0;
    if (lane == leader) top = atomicSub(&cnt[tgt], k);
    top = __shfl_sync(grp, top, leader);
    const int rank = __popc(grp & ((1u << lane) - 1));
    keys[off[tgt] + top - k + rank] = ((unsigned)pair_img(src) << b) | (unsigned)pair_cell(src);
  }
}

__device__ __forceinline__ unsigned long long seg_pair(int c, unsigned key, int b) {
  const unsigned src = ((key >> b) << kImgShift) | (key & ((1u << b) - 1));
  return ((unsigned long long)(unsigned)c << 32) | src;
}

// ascending bitonic sort of a[0, n2), n2 a power of two, by the block's nt threads (tid)
__device__ __forceinline__ void bitonic_sort(unsigned* a, int n2, int tid, int nt) {
  for (int k = 2; k <= n2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int p = tid; p < (n2 >> 1); p += nt) {
        const int i = ((p & ~(j - 1)) << 1) | (p & (j - 1));  // bit j of i clear
        const int l = i | j;
        const unsigned x = a[i], y = a[l];
        if ((x > y) == ((i & k) == 0)) {
          a[i] = y;
          a[l] = x;
        }
      }
      __syncthreads();
    }
}

// A warp's range of n <= 32 K keys sorted in registers: lane l holds keys l K .. l K + K - 1
// (padded with 0xffffffff), the bitonic network's stages of partner distance j < K run
// within each lane, those with j >= K pair the lanes l and l ^ (j / K) by shuffles; every
// index and, for k < K, every direction is a compile-time constant.
template <int K>
__device__ __forceinline__ void warp_sort_range(const unsigned* __restrict__ keys, int n, int c,
                                                int b, unsigned long long* __restrict__ out) {
  const int lane = lane_id();
  unsigned v[K];
#pragma unroll
  for (int r = 0; r < K; r++) {
    const int e = lane * K + r;
    v[r] = e < n ? keys[e] : 0xffffffffu;
  }
#pragma unroll
  for (int k = 2; k <= 32 * K; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j < K) {
#pragma unroll
        for (int r = 0; r < K; r++) {
          if (r & j) continue;
          const bool up = k < K ? (r & k) == 0 : (lane & (k / K)) == 0;
          const unsigned x = v[r], y = v[r | j];
          const unsigned lo = min(x, y), hi = max(x, y);
          v[r] = up ? lo : hi;
          v[r | j] = up ? hi : lo;
        }
      } else {
        const bool keep_min = ((lane & (j / K)) == 0) == ((lane & (k / K)) == 0);
#pragma unroll
        for (int r = 0; r < K; r++) {
          const unsigned y = __shfl_xor_sync(0xffffffffu, v[r], j / K);
          v[r] = keep_min ? min(v[r], y) : max(v[r], y);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < K; r++) {
    const int e = lane * K + r;
    if (e < n) out[e] = seg_pair(c, v[r], b);
  }
}

// one warp per target with at most kSegWarpCap pairs
__global__ void __launch_bounds__(32 * kSegWarps, 5)
    k_seg_sort_warp(int ncells, SegLists g, int b) {
  const int* __restrict__ off = g.at(blockIdx.y).off;
  const unsigned* __restrict__ keys = g.at(blockIdx.y).keys;
  unsigned long long* __restrict__ out = g.at(blockIdx.y).pairs;
  const int c = blockIdx.x * kSegWarps + (threadIdx.x >> 5);
  if (c >= ncells) return;
  const int s0 = off[c], n = off[c + 1] - s0;
  if (n == 0 || n > kSegWarpCap) return;
  keys += s0;
  out += s0;
  if (n <= 32) warp_sort_range<1>(keys, n, c, b, out);
  else if (n <= 64) warp_sort_range<2>(keys, n, c, b, out);
  else if (n <= 128) warp_sort_range<4>(keys, n, c, b, out);
  else if (n <= 256) warp_sort_range<8>(keys, n, c, b, out);
  else if (n <= 512) warp_sort_range<16>(keys, n, c, b, out);
  else warp_sort_range<32>(keys, n, c, b, out);
}

// the longer ranges, one block at a time; a range above kSegBlockCap is written unsorted and
// flagged for the global sort
__global__ void __launch_bounds__(kSegBlock)
    k_seg_sort_block(int ncells, SegLists g, int b) {
  const int* __restrict__ off = g.at(blockIdx.y).off;
  const unsigned* __restrict__ keys = g.at(blockIdx.y).keys;
  unsigned long long* __restrict__ out = g.at(blockIdx.y).pairs;
  int* __restrict__ overflow = g.at(blockIdx.y).overflow;
  __shared__ unsigned a[kSegBlockCap];
  __shared__ int todo[kSegBlock];
  __shared__ int ntodo;
  for (int base = blockIdx.x * kSegBlock; base < ncells; base += gridDim.x * kSegBlock) {
    if (threadIdx.x == 0) ntodo = 0;
    __syncthreads();
    const int cc = base + threadIdx.x;
    if (cc < ncells && off[cc + 1] - off[cc] > kSegWarpCap) todo[atomicAdd(&ntodo, 1)] = cc;
    __syncthreads();
    const int m = ntodo;
    for (int q = 0; q < m; q++) {
      const int c = todo[q];
      const int s0 = off[c], n = off[c + 1] - s0;
      if (n > kSegBlockCap) {
        for (int i = threadIdx.x; i < n; i += kSegBlock) out[s0 + i] = seg_pair(c, keys[s0 + i], b);
        if (threadIdx.x == 0) atomicExch(overflow, 1);
        continue;
      }
      int n2 = 32;
      while (n2 < n) n2 <<= 1;
      for (int i = threadIdx.x; i < n2; i += kSegBlock) a[i] = i < n ? keys[s0 + i] : 0xffffffffu;
      __syncthreads();
      bitonic_sort(a, n2, threadIdx.x, kSegBlock);
      for (int i = threadIdx.x; i < n; i += kSegBlock) out[s0 + i] = seg_pair(c, a[i], b);
      __syncthreads();
    }
    __syncthreads();
  }
}

// M2L targets (cells with at least one source) by descending pair count in buckets of 2^shift
// pairs, so that the warps of an M2L block have about the same amount of work: the spherical
// kernel takes sources in batches of 32 (shift 5), the Cartesian one a thread per target (shift
// 0: exact counts, even warps); cells without pairs last.  A radix sort on 8 bits (counts
// above the last bucket share the first place), stable, so that neighbouring targets of a
// bucket, and so their shared sources, stay together: in the order of a counting sort by
// atomics, which saves the sort's launches, the Cartesian M2L of 2^22 bodies took 0.87 ms
// instead of 0.79, the spherical one of 2^20 1.50 ms instead of 1.47.
constexpr int kTgtKeyBits = 8, kTgtKeyMax = (1 << kTgtKeyBits) - 1;
__device__ __forceinline__ unsigned tgt_key(int n, int shift) {
  const int b = (n + (1 << shift) - 1) >> shift;
  return n ? (unsigned)(kTgtKeyMax - 1 - min(kTgtKeyMax - 1, b)) : (unsigned)kTgtKeyMax;
}
__global__ void k_m2l_targets(int ncells, const int* __restrict__ off, int shift,
                              unsigned* __restrict__ key, int* __restrict__ cell,
                              int* __restrict__ count) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = c < ncells ? off[c + 1] - off[c] : 0;
  const unsigned m = __ballot_sync(0xffffffffu, n > 0);
  if (m && lane_id() == 0) atomicAdd(count, __popc(m));
  if (c >= ncells) return;
  key[c] = tgt_key(n, shift);
  cell[c] = c;
}

// Small trees: the offsets of both lists by a block each, and the M2L list's target keys as
// k_m2l_targets writes them.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads)
    k_seg_scan(int ncells, SegLists g, int shift, unsigned* __restrict__ key,
               int* __restrict__ cell, int* __restrict__ count) {
  __shared__ int wsum[kScanThreads / 32];
  const int* __restrict__ cnt = g.at(blockIdx.x).cnt;
  int* __restrict__ off = g.at(blockIdx.x).off;
  const int lane = lane_id(), wl = threadIdx.x >> 5;
  const int per = (ncells + kScanThreads) / kScanThreads;  // of ncells + 1 offsets
  const int lo = min(ncells + 1, (int)threadIdx.x * per), hi = min(ncells + 1, lo + per);
  int sum = 0, used = 0;
  for (int i = lo; i < hi; i++) {
    const int n = cnt[i];
    sum += n;
    if (blockIdx.x == 0 && i < ncells) {
      used += n > 0;
      key[i] = tgt_key(n, shift);
      cell[i] = i;
    }
  }
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += u;
  }
  if (lane == 31) wsum[wl] = incl;
  used = __reduce_add_sync(0xffffffffu, used);
  if (lane == 0 && used) atomicAdd(count, used);
  __syncthreads();
  int run = incl - sum;
  for (int k = 0; k < wl; k++) run += wsum[k];
  for (int i = lo; i < hi; i++) {
    off[i] = run;
    run += cnt[i];
  }
}

// body-pair count of the P2P list: sum over pairs of nbody(target) * nbody(source)
__global__ void k_p2p_bodypairs(const unsigned long long* __restrict__ pairs, long long n,
                                const int* __restrict__ nbody,
                                unsigned long long* __restrict__ out) {
  unsigned long long s = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    unsigned long long p = pairs[t];
    s += (unsigned long long)nbody[p >> 32] * (unsigned long long)nbody[pair_cell((unsigned)p)];
  }
  s = warp_sum(s);
  if (lane_id() == 0 && s) atomicAdd(out, s);
}

// (target << 32 | image << 27 | cell) <-> (target << (b + ib) | image << b | cell): sort keys
// of 2 b + ib bits (ib = 5 with periodic images, else 0)
__global__ void k_pack_pairs(unsigned long long* __restrict__ a, long long n, int b, int ib,
                             int pack) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const unsigned long long v = a[t];
    if (pack) {
      const unsigned src = (unsigned)v;
      a[t] = ((v >> 32) << (b + ib)) | ((unsigned long long)pair_img(src) << b) |
             (unsigned long long)pair_cell(src);
    } else {
      const unsigned long long src = ((v >> b) & ((1ULL << ib) - 1)) << kImgShift |
                                     (v & ((1ULL << b) - 1));
      a[t] = ((v >> (b + ib)) << 32) | src;
    }
  }
}

static int bits_for(int n) {
  int b = 1;
  while ((1LL << b) < (long long)n) b++;
  return b;
}

// group a list, or both, by target (k_seg_*): CSR offsets into off[0, ncells], pairs sorted
// within each target's range; `scan`: the counts into the offsets
template <typename F>
static void group_by_target(SolverBase& s, const SegLists& g, int lists, int b, F&& scan) {
  const int TB = 256;
  const long long n = lists == 1 ? g.l[0].n : std::max(g.l[0].n, g.l[1].n);
  const dim3 grid((int)std::max(1LL, std::min<long long>(ceil_div(n, TB), 148 * 16)), lists);
  if (n > 0) {
    k_seg_count<<<grid, TB, 0, s.stream>>>(g);
    FMM_LAUNCH_CHECK();
  }
  scan();
  if (n == 0) return;
  k_seg_scatter<<<grid, TB, 0, s.stream>>>(g, b);
  FMM_LAUNCH_CHECK();
  k_seg_sort_warp<<<dim3(ceil_div(s.ncells, kSegWarps), lists), 32 * kSegWarps, 0, s.stream>>>(
      s.ncells, g, b);
  FMM_LAUNCH_CHECK();
  // (a target has a pair per cell and image at most)
  if ((long long)s.ncells * (s.cfg.images > 0 ? 27 : 1) <= kSegWarpCap) return;
  k_seg_sort_block<<<dim3(std::min(ceil_div(s.ncells, kSegBlock), 148), lists), kSegBlock, 0,
                     s.stream>>>(s.ncells, g, b);
  FMM_LAUNCH_CHECK();
}
// one list; scratch for the counts' scan: tmp, or s.cub_tmp if null
static void group_one(SolverBase& s, const SegList& l, int b, DevArr<char>* tmp) {
  FMM_CUDA(cudaMemsetAsync(l.cnt, 0, (s.ncells + 1) * sizeof(int), s.stream));
  group_by_target(s, SegLists{{l, l}}, 1, b,
                  [&] { exclusive_sum_int(s, l.cnt, l.off, s.ncells + 1, tmp); });
}

// a whole list sorted on (target << (b + ib) | image << b | source), 2 b + ib key bits:
// the targets whose ranges were too long for k_seg_sort_block
static void global_sort_list(SolverBase& s, unsigned long long* lst, long long n, int b, int ib) {
  const int TB = 256;
  const int grid = (int)std::min<long long>(ceil_div(n, TB), 148 * 16);
  k_pack_pairs<<<grid, TB, 0, s.stream>>>(lst, n, b, ib, 1);
  FMM_LAUNCH_CHECK();
  sort_keys_u64(s, lst, s.list_tmp.p, (int)n, 2 * b + ib);
  k_pack_pairs<<<grid, TB, 0, s.stream>>>(s.list_tmp.p, n, b, ib, 0);
  FMM_LAUNCH_CHECK();
  FMM_CUDA(cudaMemcpyAsync(lst, s.list_tmp.p, 8 * (size_t)n, cudaMemcpyDeviceToDevice, s.stream));
}

// the mutual traversal applies to one tree with an open boundary, as in the reference (the
// image traversals and dualTreeTraversal(cells, jcells) run with mutual = false)
static int mutual_of(const SolverBase& s) {
  return s.cfg.mutual && s.cfg.images == 0 && !s.ij ? 1 : 0;
}

// pairs of the first frontier at most
static int root_count(const SolverBase& s) {
  return s.ij ? s.nroots == 2 : s.nroots * (s.cfg.images > 0 ? 27 : 1);
}
// the first frontier, s.nfront0 pairs, to `front`
template <typename T> static void upload_roots(Solver<T>& s, int2* front) {
  // one (root, root) pair per solve of the batch (lists never cross solves); with periodic
  // images one per shift of the source tree, in the reference's image order (:250-260)
  std::vector<int2> roots;
  if (s.ij) {
    // dualTreeTraversal(cells, jcells): the target root against the source root
    if (s.nroots == 2) roots.push_back(make_int2(s.root_cell[0], s.root_cell[1]));
  }
  for (int r = 0; r < s.nroots && !s.ij; r++) {
    if (s.cfg.images == 0) {
      roots.push_back(make_int2(s.root_cell[r], s.root_cell[r]));
      continue;
    }
    for (int ix = -1; ix <= 1; ix++)
      for (int iy = -1; iy <= 1; iy++)
        for (int iz = -1; iz <= 1; iz++)
          roots.push_back(make_int2(s.root_cell[r],
                                    s.root_cell[r] | (img_code(ix, iy, iz) << kImgShift)));
  }
  s.nfront0 = (int)roots.size();
  if (roots.empty()) return;
  if (roots.size() > s.roots_cap) {
    if (s.roots_host) s.roots_retired.push_back(s.roots_host);
    s.roots_host = nullptr;
    s.roots_cap = 0;
    const size_t cap = std::max<size_t>(2 * roots.size(), 64);
    FMM_CUDA(cudaMallocHost((void**)&s.roots_host, sizeof(int2) * cap));
    s.roots_cap = cap;
  }
  std::copy(roots.begin(), roots.end(), s.roots_host);
  FMM_CUDA(cudaMemcpyAsync(front, s.roots_host, sizeof(int2) * roots.size(),
                           cudaMemcpyHostToDevice, s.stream));
}

// The traversal on the handle's buffers, run again on larger ones while any was too small.  The
// lists of small trees start at lengths per cell that most inputs stay below; on a larger tree a
// handle's first traversal counts them.  The stacks and the frontiers lie in the array that the
// grouping takes its keys from afterwards.  (With arrays of their own, twice as long as needed,
// and lists sized by cells on every tree, a new handle held 111 MB after a solve of 31,607 bodies
// and 3.28 GB after one of 2^22 on a sphere; now 63 MB and 2.49 GB, and the first solves take 5.0
// instead of 6.6 ms and 21.4 instead of 21.6.)  Trees of up to kTravStackCells cells: steps
// until the frontier is some four times as long as there are cells (a step makes about 20 pairs
// of one; from a frontier a quarter as long the blocks' shares differ by far more: 30,003 bodies
// in images 0.37 ms against 0.26), then k_traverse; should one of its stacks overflow, this and
// the handle's next kTravBySteps traversals take steps only.  Larger trees: steps only, as many as
// the last traversal took, two more per level that the tree has grown by since, and two to spare (at
// first as many as any tree needs).  Against all steps in one cooperative kernel with a barrier
// between them the traverse phase of 1,000 bodies takes 0.16 instead of 0.19 ms, of 200,003 0.26
// instead of 0.31, of 250,007 in the uniform tree 0.25 instead of 0.27; 2^22 on a sphere (361,000
// cells) took 1.26 ms in k_traverse, whose blocks end far apart there, and 1.14 by steps (0.93
// since).
constexpr int kTravStackCells = 8192;
constexpr int kTravBySteps = 16;

template <typename T>
static void traverse_lists(Solver<T>& s, long long& nm2l, long long& np2p) {
  unsigned long long* ctr = (unsigned long long*)s.scal.p + 32;
  unsigned long long* hctr = (unsigned long long*)s.scal_host + 32;
  constexpr int NC = kTravMaxSteps + 5;
  const bool small = s.ncells <= kTravStackCells;
  size_t m2l = small ? 192 * (size_t)s.ncells + 1024 : 0;
  size_t p2p = small ? 64 * (size_t)s.ncells + 1024 : 0;
  size_t front = std::max((small ? 128 : 96) * (size_t)s.ncells + 1024, (size_t)root_count(s));
  bool stacks = small && s.trav_by_steps == 0, all = false;
  if (small && !stacks) s.trav_by_steps--;
  const int blocks = std::max(16, std::min(148 * kTravBlocks, s.ncells / 2));
  for (;;) {
    s.m2l.ensure(m2l, !small);
    s.p2p.ensure(p2p, !small);
    const size_t stack = stacks ? (size_t)blocks * kTravStack : 0;
    s.list_tmp.ensure(stack + 2 * front, false);
    int2* scratch = (int2*)s.list_tmp.p;
    front = (s.list_tmp.cap - stack) / 2;
    upload_roots(s, scratch + stack);
    FMM_CUDA(cudaMemsetAsync(ctr, 0, sizeof(unsigned long long) * NC, s.stream));
    TravArgs<T> g{};
    g.stacks = scratch;
    g.front = scratch + stack;
    g.front2 = g.front + front;
    g.front_cap = front;
    g.nfront0 = s.nfront0;
    g.m2l_cap = s.m2l.cap;
    g.p2p_cap = s.p2p.cap;
    g.X = s.cX.p;
    g.info = s.c_info.p;
    g.nspawn = s.cfg.nspawn;
    g.mutual = mutual_of(s);
    g.ncells = s.ncells;
    g.cycle = (T)s.cfg.cycle;
    g.range = s.part_ptr();
    g.ctr = ctr;
    g.m2l = s.m2l.p;
    g.p2p = s.p2p.p;
    int steps = kTravMaxSteps;
    if (stacks) {
      steps = 0;
      for (long long e = std::max(s.nfront0, 1); e < 4LL * s.ncells; e *= 20) steps++;
    } else if (s.trav_steps > 0 && !all) {
      steps = std::min(steps, s.trav_steps + 2 * std::max(0, s.maxlevel - s.trav_maxlevel) + 2);
    }
    for (int l = 0; l < steps; l++) {
      k_trav_step<T><<<std::min(148 * 8, std::max(1, s.ncells / 8)), kTravStepThreads, 0,
                       s.stream>>>(g, l);
      FMM_LAUNCH_CHECK();
    }
    if (stacks) {
      k_traverse<T><<<blocks, kTravThreads, 0, s.stream>>>(g, steps);
      FMM_LAUNCH_CHECK();
    }
    FMM_CUDA(cudaMemcpyAsync(hctr, ctr, sizeof(unsigned long long) * NC, cudaMemcpyDeviceToHost,
                             s.stream));
    FMM_CUDA(cudaStreamSynchronize(s.stream));
    if (hctr[2]) throw FmmError(FMM_ERR_DEVICE, "traversal read a cell index out of range");
    bool walked = true;  // to the end: the counts are exact
    int used = 0;        // steps with pairs to classify
    for (int l = 0; l < steps; l++) {
      if (hctr[5 + l]) used = l + 2;
      if (hctr[5 + l] > g.front_cap) {
        walked = false;
        front = std::max<size_t>(2 * front, hctr[5 + l]);
      }
    }
    if (hctr[4]) {
      walked = stacks = false;
      s.trav_by_steps = kTravBySteps;
    }
    if (!stacks && hctr[4 + steps]) {  // more steps than planned
      walked = false;
      all = true;
    }
    if (walked && !stacks) {
      s.trav_steps = std::max(used, 1);
      s.trav_maxlevel = s.maxlevel;
    }
    if (walked && hctr[0] <= s.m2l.cap && hctr[1] <= s.p2p.cap) {
      nm2l = (long long)hctr[0];
      np2p = (long long)hctr[1];
      return;
    }
    m2l = std::max<size_t>(s.m2l.cap, hctr[0]);
    p2p = std::max<size_t>(s.p2p.cap, hctr[1]);
  }
}

// the P2P list of a build_lists(s, true): wait (on the host) for its grouping on the side
// stream, sort it globally if a target's range was too long for the blocks, and make the
// main stream wait for it
void finish_p2p_list(SolverBase& s) {
  if (!s.p2p_pending) return;
  s.p2p_pending = false;
  FMM_CUDA(cudaEventSynchronize(s.p2p_ready));
  const int* hflow = (const int*)((unsigned long long*)s.scal_host + 5);
  if (hflow[1]) {
    FMM_CUDA(cudaStreamWaitEvent(s.stream, s.p2p_ready, 0));
    global_sort_list(s, s.p2p.p, s.np2p, bits_for(s.ncells), s.cfg.images > 0 ? 5 : 0);
    order_p2p_targets(s);
    FMM_CUDA(cudaStreamSynchronize(s.stream));
  } else {
    FMM_CUDA(cudaStreamWaitEvent(s.stream, s.p2p_ready, 0));
  }
}

template <typename T> void build_lists(Solver<T>& s, bool defer_p2p) {
  const int TB = 256;
  s.nm2l = s.np2p = s.p2p_body_pairs = 0;
  if (s.ncells == 0) return;
  if (s.ncells > (int)kCellMask)
    throw FmmError(FMM_ERR_NOT_SUPPORTED, "more than 2^27 - 1 cells (list pairs hold 27-bit cells)");
  unsigned long long* cnt = (unsigned long long*)s.scal.p;  // [0..2] counts, [3] body pairs
  unsigned long long* hc = (unsigned long long*)s.scal_host;
  long long nm2l = 0, np2p = 0;
  traverse_lists(s, nm2l, np2p);
  s.nm2l = nm2l;
  s.np2p = np2p;
  const int b = bits_for(s.ncells), ib = s.cfg.images > 0 ? 5 : 0;
  if (std::max(nm2l, np2p) > (long long)INT_MAX)
    throw FmmError(FMM_ERR_NOT_SUPPORTED, "more than 2^31 - 1 pairs in an interaction list");
  s.list_tmp.ensure(std::max<long long>(std::max(nm2l, np2p), 1));
  s.m2l_off.ensure(s.ncells + 1);
  s.p2p_off.ensure(s.ncells + 1);
  s.m2l_tgt.ensure(s.ncells);
  s.tgt_key.ensure(2 * (size_t)s.ncells);
  s.idx.ensure(s.ncells);
  int* ntgt = (int*)(cnt + 4);
  int* overflow = (int*)(cnt + 5);  // per list: a target range too long for the blocks
  const int shift = s.cfg.basis == FMM_SPHERICAL ? 5 : 0;
  FMM_CUDA(cudaMemsetAsync(cnt + 4, 0, 2 * sizeof(unsigned long long), s.stream));
  // Small trees: both lists by the same launches, one after the other with the P2P order on the
  // main stream.  Their kernels take 2-10 us, about what the host needs to queue them: 14
  // launches and copies instead of 33 take 1,000 bodies from 0.49 to 0.44 ms, 16,384 in FP64
  // from 0.66 to 0.61 (118 and 585 cells).  Larger ones group the P2P list beside the M2L:
  // at 5,137 cells 1.60 ms against 1.63 together.
  const bool both = s.ncells <= kSegBothCells;
  s.seg_cnt.ensure((both ? 2 : 1) * (size_t)(s.ncells + 1));
  const SegList lm{s.m2l.p, nm2l, s.seg_cnt.p, s.m2l_off.p, (unsigned*)s.list_tmp.p, overflow};
  SegList lp{s.p2p.p, np2p, s.seg_cnt.p, s.p2p_off.p, (unsigned*)s.list_tmp.p, overflow + 1};
  s.p2p_pending = !both && defer_p2p && s.side != nullptr;
  if (both) {
    lp.cnt += s.ncells + 1;
    lp.keys += nm2l;
    const SegLists g{{lm, lp}};
    FMM_CUDA(cudaMemsetAsync(s.seg_cnt.p, 0, 2 * (size_t)(s.ncells + 1) * sizeof(int), s.stream));
    group_by_target(s, g, 2, b, [&] {
      k_seg_scan<<<2, kScanThreads, 0, s.stream>>>(s.ncells, g, shift, s.tgt_key.p, s.idx.p, ntgt);
      FMM_LAUNCH_CHECK();
    });
    order_p2p_targets(s);
  } else {
    group_one(s, lm, b, nullptr);
  }
  if (s.p2p_pending) {
    // the P2P list is grouped on the side stream with scratch of its own, beside M2L; its
    // overflow flag reaches the host through the pinned mirror (finish_p2p_list)
    s.seg_cnt2.ensure(s.ncells + 1);
    s.seg_keys2.ensure(std::max<long long>(np2p, 1));
    lp.cnt = s.seg_cnt2.p;
    lp.keys = s.seg_keys2.p;
    if (!s.p2p_ready) FMM_CUDA(cudaEventCreateWithFlags(&s.p2p_ready, cudaEventDisableTiming));
    FMM_CUDA(cudaEventRecord(s.fork, s.stream));
    FMM_CUDA(cudaStreamWaitEvent(s.side, s.fork, 0));
    cudaStream_t main = s.stream;
    s.stream = s.side;
    try {
      group_one(s, lp, b, &s.cub_tmp2);
      order_p2p_targets(s);
      FMM_CUDA(cudaMemcpyAsync((int*)(hc + 5) + 1, overflow + 1, sizeof(int),
                               cudaMemcpyDeviceToHost, s.stream));
      FMM_CUDA(cudaEventRecord(s.p2p_ready, s.stream));
    } catch (...) {
      s.stream = main;
      throw;
    }
    s.stream = main;
  } else if (!both) {
    group_one(s, lp, b, nullptr);
    order_p2p_targets(s);
  }
  // M2L target order: by descending pair count in buckets (stable in cell index)
  if (!both) {
    k_m2l_targets<<<ceil_div(s.ncells, TB), TB, 0, s.stream>>>(s.ncells, s.m2l_off.p, shift,
                                                               s.tgt_key.p, s.idx.p, ntgt);
    FMM_LAUNCH_CHECK();
  }
  sort_pairs_u32(s, s.tgt_key.p, s.tgt_key.p + s.ncells, s.idx.p, s.m2l_tgt.p, s.ncells,
                 kTgtKeyBits);
  // body pairs, targets and the overflow flags (the P2P list's on its own while it is pending)
  FMM_CUDA(cudaMemcpyAsync(hc + 3, cnt + 3,
                           2 * sizeof(unsigned long long) + (s.p2p_pending ? 1 : 2) * sizeof(int),
                           cudaMemcpyDeviceToHost, s.stream));
  FMM_CUDA(cudaStreamSynchronize(s.stream));
  const int* hflow = (const int*)(hc + 5);
  if (hflow[0] || (!s.p2p_pending && hflow[1])) {
    if (hflow[0]) global_sort_list(s, s.m2l.p, nm2l, b, ib);
    if (!s.p2p_pending && hflow[1]) {
      global_sort_list(s, s.p2p.p, np2p, b, ib);
      order_p2p_targets(s);
    }
    FMM_CUDA(cudaStreamSynchronize(s.stream));
  }
  s.p2p_body_pairs = -1;  // counted when asked for (count_p2p_body_pairs)
  s.m2l_ntgt = *(const int*)(hc + 4);
}

// the body pairs of the P2P list, for the statistics (not needed by the solve itself)
long long count_p2p_body_pairs(SolverBase& s) {
  if (s.np2p == 0) return 0;
  const int TB = 256;
  unsigned long long* cnt = (unsigned long long*)s.scal.p;
  unsigned long long* hc = (unsigned long long*)s.scal_host;
  FMM_CUDA(cudaMemsetAsync(cnt + 3, 0, sizeof(unsigned long long), s.stream));
  k_p2p_bodypairs<<<std::max(1, std::min(ceil_div(s.np2p, TB), 148 * 8)), TB, 0, s.stream>>>(
      s.p2p.p, s.np2p, s.c_nbody.p, cnt + 3);
  FMM_LAUNCH_CHECK();
  FMM_CUDA(cudaMemcpyAsync(hc + 3, cnt + 3, sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                           s.stream));
  FMM_CUDA(cudaStreamSynchronize(s.stream));
  return (long long)hc[3];
}

template void build_lists<float>(Solver<float>&, bool);
template void build_lists<double>(Solver<double>&, bool);

}  // namespace fmmb200
