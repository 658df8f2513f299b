// Near-field P2P over the per-target-leaf source lists (kernel::P2P,
// kernels/LaplaceP2PCPU.cxx:4-170 and the self form :172-331).
//
// A team of 1, 2, 4 or 8 warps of one block owns a target leaf and shares out the bodies of
// its source list evenly; the warps' sums meet in shared memory in warp order.  The size of
// the team follows from the leaf's own list (p2p_class), so a leaf's result does not depend
// on what else the launch holds.  (One warp per leaf left a launch of a few thousand leaves
// with a long tail: 1.4 waves of warps at 4,096 leaves, and 512 leaves a third of the GPU:
// cube of 16,384 bodies in FP64 0.43 ms, now 0.12 ms.)
//
// A warp's lanes hold up to TPL = 3 targets each (FP64: 2), spread over G = 1 .. 8 lanes that
// take every G-th source (p2p_lanes).  Sources stream through shared memory 32 bodies at a
// time, a chunk running on across source leaves; FP32 takes them two at a time with the
// packed two-wide instructions of sm_100, 13 packed instructions and two MUFU rsqrt for two
// pairs.  Every lane reads every staged source, 16 bytes a source, and the shared-memory
// pipe returns 128 bytes a cycle and SM: at one target per lane that return path would bound
// the kernel, not the FMA pipe (4 cycles a source and warp against 3.25), so a source has to
// serve several targets of its lane.  FP32 folds the sums of up to 32 of a lane's sources
// (p2p_folds) into a compensated (TwoSum) accumulator, so the accumulation error does not grow
// with the length of the list; FP64 sums plainly.
//
// Bound: the FMA pipe (FP64: the FP64 pipe), 26 cycles a source pair and target, at 50-65 %
// of it: the rest is idle target slots, the chunks' staging and latency at 16 warps per SM.
// FP32, one warp per leaf and one to two targets per lane before: Plummer 2^20, P = 10
// (0.99 G pairs, 18 bodies a leaf) 1.08 -> 0.89 ms; 256 solves (14.4 G pairs) 14.4 -> 12.1 ms;
// cube of 200,003 (1.28 G, 49 a leaf) 1.19 -> 0.89 ms; sphere of 2^22 (1.23 G, 13 a leaf) 1.98
// -> 1.90 ms.  Measured beside it on the 256 solves: four targets per lane 13.8 ms against
// 13.6 (128 registers either way), two at 24 warps per SM 14.4 ms; accumulators in registers
// 15.6 ms; chunks of 64 bodies 14.1 ms; teams twice as large 12.9 ms.
//
// Away from the target leaf itself the pairs take no r^2 == 0 test and an FTZ rsqrt.  If a
// warp's potential then is not finite (two bodies of different leaves in one place, or
// closer than the normal range), it sums its part of the list again with the exact form
// throughout.  Pairs with r^2 == 0 are skipped, as the reference does (:149); the result is
// per unit target charge (the reference multiplies by q_i in P2P and divides again in L2P /
// normalize).
#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "fmm_solver.cuh"

namespace fmmb200 {

// 1/sqrt with subnormal inputs flushed to zero (PTX rsqrt.approx.ftz.f32): no handling of
// subnormal inputs and no r^2 == 0 test, for the source leaves where neither can occur
__device__ __forceinline__ float rsqrt_ftz(float a) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ double rsqrt_ftz(double a) { return rsqrt(a); }

// Most targets of a lane, and the lanes G that share one: 32 TPL / G slots for the leaf's
// targets (64 at a time; FP32 without images: p2p_width).  FP32 at the default limits g4 = 8,
// g2 = 16: G = 8 up to 12 bodies, 4 up to 24, 2 up to 48, so slots come in steps of 4, 8 and 16
// and few stay idle; FP64, whose arithmetic and not its reads bounds it, takes G = 4, 2, 1 (fewer
// sums to merge).  So do solves with periodic images, whose sums are also folded after every
// chunk by one warp per leaf: in that order their results keep every bit they had (30,003 bodies:
// 0.05 ms either way).
template <typename T> __host__ __device__ constexpr int p2p_tpl() { return sizeof(T) == 4 ? 3 : 2; }
template <typename T> __device__ __forceinline__ int p2p_lanes(int nb, int g4, int g2, int images) {
  if (sizeof(T) == 8 || images) return nb <= g4 ? 4 : nb <= g2 ? 2 : 1;
  constexpr int X = p2p_tpl<T>();
  return nb <= X * g4 / 2 ? 8 : nb <= X * g2 / 2 ? 4 : nb <= 16 * X ? 2 : 1;
}

// FP32: chunks of a leaf of nb bodies between folds.  A lane sums 32 sources plainly in between
// (16 in each half of its packed sums), 8 and 16 for targets of leaves up to g4 and g2 bodies: as
// many as when those had 4 and 2 lanes and every chunk was folded.  With 32 throughout, the near
// field's error against 64 bits grew by a quarter (30,000 bodies of either sign, 7 a leaf:
// potential 9.9e-8 of its norm against 7.8e-8).
__device__ __forceinline__ int p2p_folds(int nb, int G, int g4, int g2) {
  return G / (nb <= g4 ? 4 : nb <= g2 ? 2 : 1);
}

// FP32: targets of the next pass of a leaf with `left` to go, 96 at most, and as many as fill
// their slots (48 at G = 2, the rest by its own size, where one pass at G = 1 would hold
// 96 slots: leaves of 65-80 bodies take 65-80 slots instead of 96; uniform tree of 250,007
// bodies, 61 a leaf, 0.79 -> 0.70 ms).  Up to 64 bodies stay one pass: 48 and the rest apart
// for leaves of 49-56 made the 256 solves 1 % slower.
__device__ __forceinline__ int p2p_width(int left) {
  constexpr int X = p2p_tpl<float>();
  return left >= 32 * X ? 32 * X : left > 64 ? 16 * X : left;
}

constexpr int kP2PWindow = 512;  // source bodies whose indices a warp lists ahead

// two staged sources of a row: FP32 (x, x', y, y') and (z, z', q, q'); FP64 one source, (x, y)
// and (z, q)
template <typename T> struct Row;
template <> struct Row<float> {
  float4 a[16], b[16];
  int idx[kP2PWindow];
  __device__ __forceinline__ void put(int i, const float4& v) {
    float* p = reinterpret_cast<float*>(&a[i >> 1]) + (i & 1);
    float* q = reinterpret_cast<float*>(&b[i >> 1]) + (i & 1);
    p[0] = v.x;
    p[2] = v.y;
    q[0] = v.z;
    q[2] = v.w;
  }
};
template <> struct Row<double> {
  double2 a[32], b[32];
  int idx[kP2PWindow];
  __device__ __forceinline__ void put(int i, const double4& v) {
    a[i] = make_double2(v.x, v.y);
    b[i] = make_double2(v.z, v.w);
  }
};

// A target and its sums over some sources.  FP32: the coordinates negated, in both halves;
// the halves of a sum take the even and the odd sources.
template <typename T> struct Target;
template <> struct Target<float> {
  float2 nx, ny, nz, p, x, y, z;
  __device__ __forceinline__ void set(const float4& v) {
    nx = make_float2(-v.x, -v.x);
    ny = make_float2(-v.y, -v.y);
    nz = make_float2(-v.z, -v.z);
  }
  __device__ __forceinline__ void zero() { p = x = y = z = make_float2(0.f, 0.f); }
  __device__ __forceinline__ void sums(float* v) const {
    v[0] = p.x + p.y;
    v[1] = x.x + x.y;
    v[2] = y.x + y.y;
    v[3] = z.x + z.y;
  }
};
template <> struct Target<double> {
  double nx, ny, nz, p, x, y, z;
  __device__ __forceinline__ void set(const double4& v) { nx = -v.x, ny = -v.y, nz = -v.z; }
  __device__ __forceinline__ void zero() { p = x = y = z = 0; }
  __device__ __forceinline__ void sums(double* v) const { v[0] = p, v[1] = x, v[2] = y, v[3] = z; }
};

// The first `cnt` sources of a staged row (the rest of it charges nothing) on the lane's TPL
// targets, every G-th entry from `sub` on.
// EXACT: skip r^2 == 0 and take subnormal r^2 as it is (the reference's arithmetic);
// otherwise an r^2 of zero or below the normal range makes the potential non-finite.
// SHIFT: the source is a periodic image shifted by (px, py, pz); the offset is formed as
// (xj - xi) + p, the negation of the reference's (xi - xj) - Xperiodic
template <int TPL, bool EXACT, bool SHIFT>
__device__ __forceinline__ void p2p_row(const Row<float>& row, int sub, int G, int cnt, float eps2,
                                        const float* shift, Target<float>* t) {
  const int np = (cnt + 1) >> 1;
  const float2 e2 = make_float2(eps2, eps2);
  constexpr int UNROLL = TPL <= 2 ? 2 : 1;
#pragma unroll UNROLL
  for (int i = 0; i < np; i += G) {
    const float4 a = row.a[i + sub], c = row.b[i + sub];
    const float2 x2 = make_float2(a.x, a.y), y2 = make_float2(a.z, a.w);
    const float2 z2 = make_float2(c.x, c.y), q2 = make_float2(c.z, c.w);
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      float2 dx = __fadd2_rn(x2, t[u].nx), dy = __fadd2_rn(y2, t[u].ny),
             dz = __fadd2_rn(z2, t[u].nz);
      if (SHIFT) {
        dx = __fadd2_rn(dx, make_float2(shift[0], shift[0]));
        dy = __fadd2_rn(dy, make_float2(shift[1], shift[1]));
        dz = __fadd2_rn(dz, make_float2(shift[2], shift[2]));
      }
      const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
      float2 inv;
      inv.x = EXACT ? (r2.x > 0.f ? rsqrt_(r2.x) : 0.f) : rsqrt_ftz(r2.x);
      inv.y = EXACT ? (r2.y > 0.f ? rsqrt_(r2.y) : 0.f) : rsqrt_ftz(r2.y);
      const float2 qinv = __fmul2_rn(q2, inv);
      const float2 inv3 = __fmul2_rn(__fmul2_rn(qinv, inv), inv);
      t[u].p = __fadd2_rn(t[u].p, qinv);
      t[u].x = __ffma2_rn(dx, inv3, t[u].x);
      t[u].y = __ffma2_rn(dy, inv3, t[u].y);
      t[u].z = __ffma2_rn(dz, inv3, t[u].z);
    }
  }
}
template <int TPL, bool EXACT, bool SHIFT>
__device__ __forceinline__ void p2p_row(const Row<double>& row, int sub, int G, int cnt,
                                        double eps2, const double* shift, Target<double>* t) {
#pragma unroll(4 / TPL)
  for (int i = 0; i < cnt; i += G) {
    const double2 a = row.a[i + sub], c = row.b[i + sub];
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      double dx = a.x + t[u].nx, dy = a.y + t[u].ny, dz = c.x + t[u].nz;
      if (SHIFT) {
        dx += shift[0];
        dy += shift[1];
        dz += shift[2];
      }
      const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
      const double inv = EXACT ? (r2 > 0 ? rsqrt_(r2) : 0) : rsqrt_ftz(r2);
      const double qinv = c.y * inv;
      const double inv3 = qinv * inv * inv;
      t[u].p += qinv;
      t[u].x = fma(dx, inv3, t[u].x);
      t[u].y = fma(dy, inv3, t[u].y);
      t[u].z = fma(dz, inv3, t[u].z);
    }
  }
}

// A lane's accumulators in shared memory: potential and gradient of target u in s[u][lane],
// in FP32 the sums' rounding errors in e[u][lane] (in registers they would cost 8 per target
// and spill).
template <typename T, bool COMP> struct Accum {
  vec4<T> s[p2p_tpl<T>()][32], e[COMP ? p2p_tpl<T>() : 1][COMP ? 32 : 1];
};

// the targets' sums into their accumulators, and zero again
template <typename T, bool COMP, int TPL>
__device__ __forceinline__ void p2p_fold(Target<T>* t, Accum<T, COMP>& acc, int lane) {
#pragma unroll
  for (int u = 0; u < TPL; u++) {
    T v[4];
    t[u].sums(v);
    vec4<T> s = acc.s[u][lane];
    if constexpr (COMP) {
      vec4<T> e = acc.e[u][lane];
      Comp<T> a[4] = {{s.x, e.x}, {s.y, e.y}, {s.z, e.z}, {s.w, e.w}};
#pragma unroll
      for (int d = 0; d < 4; d++) comp_add(a[d], v[d]);
      acc.s[u][lane] = make_v4<T>(a[0].s, a[1].s, a[2].s, a[3].s);
      acc.e[u][lane] = make_v4<T>(a[0].e, a[1].e, a[2].e, a[3].e);
    } else {
      acc.s[u][lane] = make_v4<T>(s.x + v[0], s.y + v[1], s.z + v[2], s.w + v[3]);
    }
    t[u].zero();
  }
}

// A source leaf as k_p2p reads it: first body in bits 0-30, image in 31-35, bodies above.
__host__ __device__ __forceinline__ unsigned long long p2p_leaf(int body, int n, int img) {
  return (unsigned long long)(unsigned)body | (unsigned long long)img << 31 |
         (unsigned long long)(unsigned)n << 36;
}

// Positions [p0, p1) of the target leaf's source bodies (the bodies of its source leaves in
// list order) on the targets of one warp.  Source leaves' descriptors (first body, count,
// image) are read 32 at a time, one per lane, and scanned; each lane then writes the indices
// of its leaf's bodies into the warp's window in shared memory, from which the chunks are
// loaded, the next one while the staged one is summed.
template <typename T, bool COMP, int TPL>
__device__ __forceinline__ void p2p_segment(int lane, Row<T>& row, int b0, int nb, int sub, int G,
                                            int s0, int s1, int p0, int p1, bool whole, int folds,
                                            const unsigned long long* __restrict__ srcs,
                                            const vec4<T>* __restrict__ bodies, T eps2, T cycle,
                                            bool exact, Target<T>* t, Accum<T, COMP>& acc) {
  const unsigned full = 0xffffffffu;
  int pending = 0;  // chunks since the last fold
  int cum = 0;
  for (int sb = s0; sb < s1 && cum < p1; sb += 32) {
    // lane k: source leaf sb + k
    int dj0 = 0, dnj = 0, dimg = -1;
    if (sb + lane < s1) {
      const unsigned long long d = srcs[sb + lane];
      dj0 = (int)(d & 0x7fffffffu);
      dimg = (int)(d >> 31) & 31;
      dnj = (int)(d >> 36);
    }
    // the leaves of one image at a time: lanes k0 .. cut - 1
    for (int k0 = 0; k0 < 32;) {
      const int img = __shfl_sync(full, dimg, k0);
      if (img < 0) break;
      const unsigned other = __ballot_sync(full, dimg != img) & (full << k0);
      const int cut = other ? __ffs(other) - 1 : 32;
      const int cnj = lane >= k0 && lane < cut ? dnj : 0;
      int incl = cnj;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(full, incl, d);
        if (lane >= d) incl += v;
      }
      const int total = __shfl_sync(full, incl, 31), excl = incl - cnj;
      const int lo = max(0, min(total, p0 - cum)), hi = max(0, min(total, p1 - cum));
      T shift[3] = {0, 0, 0};
      if (img > 0) img_shift<T>(img, cycle, shift[0], shift[1], shift[2]);
      for (int w0 = lo; w0 < hi; w0 += kP2PWindow) {
        const int w1 = min(hi, w0 + kP2PWindow);
        // every lane lists the bodies of its leaf that lie in the window
        for (int p = max(excl, w0); p < min(incl, w1); p++) row.idx[p - w0] = dj0 - excl + p;
        __syncwarp();
        vec4<T> b;
        bool own;
        auto load = [&](int q) {
          const int bj = q + lane < w1 ? row.idx[q - w0 + lane] : -1;
          b = make_v4<T>(T(1e30), T(1e30), T(1e30), T(0));
          if (bj >= 0) b = bodies[bj];
          own = bj >= b0 && bj < b0 + nb;
        };
        load(w0);
        for (int q = w0; q < w1; q += 32) {
          const int cnt = min(32, w1 - q);
          const bool self = __any_sync(full, own) && img == 0;  // (orders the last reads, too)
          row.put(lane, b);
          __syncwarp();
          if (q + 32 < w1) load(q + 32);
          if (self || exact) p2p_row<TPL, true, true>(row, sub, G, cnt, eps2, shift, t);
          else if (img > 0) p2p_row<TPL, false, true>(row, sub, G, cnt, eps2, shift, t);
          else p2p_row<TPL, false, false>(row, sub, G, cnt, eps2, shift, t);
          __syncwarp();
          if (++pending >= folds) {
            p2p_fold<T, COMP, TPL>(t, acc, lane);
            pending = 0;
          }
        }
      }
      if (!whole) cum += total;  // (a whole list has no end to reach)
      k0 = cut;
    }
  }
  if (pending) p2p_fold<T, COMP, TPL>(t, acc, lane);
}

// one warp's part of a target leaf: its targets from body b0 + base on
struct P2PTeam {
  int base, G, s0, s1, S, p0, p1;
  int folds;  // chunks between folds
};
template <typename T, bool COMP, int TPL>
__device__ __forceinline__ void p2p_targets(const P2PTeam& w, int lane, Row<T>& row,
                                            Accum<T, COMP>& mem, int b0, int nb,
                                            const unsigned long long* __restrict__ srcs,
                                            const vec4<T>* __restrict__ bodies, T eps2, T cycle,
                                            vec4<T>* __restrict__ trg_s,
                                            vec4<T>* __restrict__ trg_e) {
  const int sub = lane % w.G, step = 32 / w.G;
  const vec4<T> zero4 = make_v4<T>(0, 0, 0, 0);
  Target<T> t[TPL];
#pragma unroll
  for (int u = 0; u < TPL; u++) {
    const int i = w.base + u * step + lane / w.G;
    t[u].set(i < nb ? bodies[b0 + i] : zero4);
  }
  for (int exact = 0; exact < 2; exact++) {
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      t[u].zero();
      mem.s[u][lane] = zero4;
      if constexpr (COMP) mem.e[u][lane] = zero4;
    }
    p2p_segment<T, COMP, TPL>(lane, row, b0, nb, sub, w.G, w.s0, w.s1, w.p0, w.p1, w.S == 1, w.folds, srcs,
                              bodies, eps2, cycle, exact != 0, t, mem);
    bool bad = false;
#pragma unroll
    for (int u = 0; u < TPL; u++)
      bad |= w.base + u * step + lane / w.G < nb && !isfinite(mem.s[u][lane].x);
    if (!__any_sync(0xffffffffu, bad)) break;
  }
  Comp<T> acc[TPL][4];
#pragma unroll
  for (int u = 0; u < TPL; u++) {
    const vec4<T> s = mem.s[u][lane];
    vec4<T> e = zero4;
    if constexpr (COMP) e = mem.e[u][lane];
    acc[u][0] = Comp<T>{s.x, e.x};
    acc[u][1] = Comp<T>{s.y, e.y};
    acc[u][2] = Comp<T>{s.z, e.z};
    acc[u][3] = Comp<T>{s.w, e.w};
  }
  for (int o = 1; o < w.G; o <<= 1) {
#pragma unroll
    for (int u = 0; u < TPL; u++)
#pragma unroll
      for (int d = 0; d < 4; d++) {
        Comp<T> r = {0, 0};
        r.s = __shfl_xor_sync(0xffffffffu, acc[u][d].s, o);
        if constexpr (COMP) {
          r.e = __shfl_xor_sync(0xffffffffu, acc[u][d].e, o);
          comp_merge(acc[u][d], r);
        } else {
          acc[u][d].s += r.s;
        }
      }
  }
  __syncwarp();
  if (sub == 0) {
#pragma unroll
    for (int u = 0; u < TPL; u++) {
      const int i = u * step + lane / w.G;
      const vec4<T> s = make_v4<T>(acc[u][0].s, acc[u][1].s, acc[u][2].s, acc[u][3].s),
                    e = make_v4<T>(acc[u][0].e, acc[u][1].e, acc[u][2].e, acc[u][3].e);
      if (w.S > 1) {
        mem.s[i >> 5][i & 31] = s;  // (every lane has taken its own accumulators out)
        if constexpr (COMP) mem.e[i >> 5][i & 31] = e;
      } else if (w.base + i < nb) {
        trg_s[b0 + w.base + i] = s;
        trg_e[b0 + w.base + i] = e;
      }
    }
  }
}

constexpr int kP2PWarps = 8;  // per block, and of the largest team


// order[i]: (first body, bodies, list begin, list end) of target leaf i in launch order, the
// leaves of teams of 8 warps first, then 4, 2 and 1 (counts n8 .. n1); nsrc[i]: its source
// bodies; srcs: the list's source leaves (p2p_leaf)
template <typename T, bool COMP>
__global__ void __launch_bounds__(32 * kP2PWarps, sizeof(T) == 4 ? 2 : 3)
    k_p2p(const int4* __restrict__ order, const int* __restrict__ nsrc, int n8, int n4, int n2,
          int n1, const unsigned long long* __restrict__ srcs,
          const vec4<T>* __restrict__ bodies, T eps2, T cycle, vec4<T>* __restrict__ trg_s,
          vec4<T>* __restrict__ trg_e, int g4, int g2, int images) {
  __shared__ Row<T> rows[kP2PWarps];
  __shared__ Accum<T, COMP> mem[kP2PWarps];
  const int wl = threadIdx.x >> 5, lane = lane_id();
  // the block's class: S warps per leaf, kP2PWarps / S leaves of the block
  int blk = blockIdx.x, first = 0, cls = n8, S = 8;
  const int rest[3] = {n4, n2, n1};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int blocks = (cls * S + kP2PWarps - 1) / kP2PWarps;
    if (blk >= blocks) {
      blk -= blocks;
      first += cls;
      cls = rest[k];
      S >>= 1;
    } else {
      break;
    }
  }
  const int at = blk * (kP2PWarps / S) + wl / S, seg = wl % S;
  if (at >= cls) return;  // the whole team
  const int4 leaf = order[first + at];
  const int b0 = leaf.x, nb = leaf.y, s0 = leaf.z, s1 = leaf.w;
  const int ns = nsrc[first + at];
  const int per = (ns + 32 * S - 1) / (32 * S) * 32;
  const int p0 = S == 1 ? 0 : min(ns, per * seg), p1 = S == 1 ? INT_MAX : min(ns, p0 + per);
  const int G = p2p_lanes<T>(nb, g4, g2, images);
  P2PTeam w{0, G, s0, s1, S, p0, p1,
            images ? 1 : sizeof(T) == 8 ? G : p2p_folds(nb, G, g4, g2)};
  const int team = wl / S, bar = 1 + team, thr = 32 * S;
  for (int base = 0, width = 64; base < nb; base += width) {
    if (sizeof(T) == 4 && !images && nb > 64) {
      width = p2p_width(nb - base);
      w.folds = w.G = p2p_lanes<T>(width, g4, g2, 0);
    }
    w.base = base;
    const int tpl = (min(width, nb - base) * w.G + 31) / 32;
    auto run = [&](auto n) {
      p2p_targets<T, COMP, decltype(n)::value>(w, lane, rows[wl], mem[wl], b0, nb, srcs,
                                               bodies, eps2, cycle, trg_s, trg_e);
    };
    if (tpl == 1) run(std::integral_constant<int, 1>());
    else if (tpl == 2 || p2p_tpl<T>() == 2) run(std::integral_constant<int, 2>());
    else if constexpr (p2p_tpl<T>() > 2) {
      run(std::integral_constant<int, 3>());
    }
    if (S == 1) continue;
    // the team's warps: partial sums through shared memory, added in warp order
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(thr) : "memory");
    for (int t = seg * 32 + lane; t < min(width, nb - base); t += thr) {
      vec4<T> s = mem[team * S].s[t >> 5][lane], e = make_v4<T>(0, 0, 0, 0);
      if constexpr (COMP) e = mem[team * S].e[t >> 5][lane];
      Comp<T> a[4] = {{s.x, e.x}, {s.y, e.y}, {s.z, e.z}, {s.w, e.w}};
      for (int k = 1; k < S; k++) {
        const vec4<T> u = mem[team * S + k].s[t >> 5][lane];
        if constexpr (COMP) {
          const vec4<T> d = mem[team * S + k].e[t >> 5][lane];
          comp_merge(a[0], Comp<T>{u.x, d.x});
          comp_merge(a[1], Comp<T>{u.y, d.y});
          comp_merge(a[2], Comp<T>{u.z, d.z});
          comp_merge(a[3], Comp<T>{u.w, d.w});
        } else {
          a[0].s += u.x, a[1].s += u.y, a[2].s += u.z, a[3].s += u.w;
        }
      }
      trg_s[b0 + base + t] = make_v4<T>(a[0].s, a[1].s, a[2].s, a[3].s);
      trg_e[b0 + base + t] = make_v4<T>(a[0].e, a[1].e, a[2].e, a[3].e);
    }
    if (base + width < nb) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(thr) : "memory");
  }
}

// ---------------------------------------------------------------- launch order
// Target leaves by team size, within a size by descending work (the longest start first, so
// that none is left alone at the end): a counting sort on (class, quarter octaves of source
// bodies times targets).  The order inside a bucket follows the atomics; no result depends
// on it.
constexpr int kSubBuckets = 192;
constexpr int kP2PBuckets = 4 * kSubBuckets;

// Class (0 .. 3: a team of 8, 4, 2, 1 warps) of a leaf of nb bodies with `src` source bodies:
// `share` pairs per lane of a warp or more, so that the team's start and its merge (about 500
// instructions a warp) stay small beside its pairs.  One warp for a count that no int holds, and
// with periodic images (see p2p_lanes).
__host__ __device__ __forceinline__ int p2p_class(unsigned long long src, int nb, int share) {
  if (src > INT_MAX / 2) return 3;
  const unsigned long long w = src * (unsigned long long)(nb < 61 ? (nb + 3) / 4 * 4 : 64) / 32;
  return w >= 8ULL * share ? 0 : w >= 4ULL * share ? 1 : w >= 2ULL * share ? 2 : 3;
}

__global__ void __launch_bounds__(256)
    k_p2p_work(int nleaves, const int* __restrict__ leaves, const int* __restrict__ off,
               const unsigned long long* __restrict__ pairs, const int4* __restrict__ info,
               unsigned long long* __restrict__ srcs, int* __restrict__ bucket,
               int* __restrict__ work, int* __restrict__ hist, int share) {
  __shared__ int h[kP2PBuckets];
  for (int i = threadIdx.x; i < kP2PBuckets; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const int lane = lane_id(), nw = gridDim.x * (blockDim.x >> 5);
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nleaves; i += nw) {
    const int c = leaves[i];
    unsigned long long src = 0;
    for (int k = off[c] + lane; k < off[c + 1]; k += 32) {
      const unsigned p = (unsigned)pairs[k];
      const int4 f = info[pair_cell(p)];
      src += (unsigned)f.z;
      srcs[k] = p2p_leaf(f.w, f.z, pair_img(p));
    }
    src = warp_sum(src);
    if (lane == 0) {
      const unsigned long long w = src * (unsigned long long)max(8, info[c].z) | 4ULL;
      const int e = 63 - __clzll(w);
      const int q = 4 * e + (int)((w >> (e - 2)) & 3);
      const int b = p2p_class(src, info[c].z, share) * kSubBuckets + kSubBuckets - 1 - min(q, kSubBuckets - 1);
      bucket[i] = b;
      work[i] = (int)min(src, (unsigned long long)INT_MAX);
      atomicAdd(&h[b], 1);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kP2PBuckets; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

// cursor: kP2PBuckets zeros on entry; teams[0..3]: leaves of teams of 8, 4, 2, 1 warps
__global__ void __launch_bounds__(256)
    k_p2p_place(int nleaves, const int* __restrict__ leaves, const int* __restrict__ bucket,
                const int* __restrict__ work, const int* __restrict__ hist,
                const int* __restrict__ off, const int4* __restrict__ info,
                int* __restrict__ cursor, int* __restrict__ teams, int4* __restrict__ order,
                int* __restrict__ nsrc) {
  constexpr int PER = kP2PBuckets / 256;
  __shared__ int start[kP2PBuckets], wsum[8];
  const int lane = lane_id(), wl = threadIdx.x >> 5;
  int v[PER], sum = 0;
#pragma unroll
  for (int k = 0; k < PER; k++) {
    v[k] = hist[threadIdx.x * PER + k];
    sum += v[k];
  }
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += u;
  }
  if (lane == 31) wsum[wl] = incl;
  __syncthreads();
  int run = incl - sum;
  for (int k = 0; k < wl; k++) run += wsum[k];
#pragma unroll
  for (int k = 0; k < PER; k++) {
    start[threadIdx.x * PER + k] = run;
    run += v[k];
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x < 4) {
    const int k = threadIdx.x;
    teams[k] = (k < 3 ? start[(k + 1) * kSubBuckets] : nleaves) - start[k * kSubBuckets];
  }
  for (int i0 = blockIdx.x * blockDim.x; i0 < nleaves; i0 += gridDim.x * blockDim.x) {
    const int i = i0 + threadIdx.x;
    const unsigned act = __ballot_sync(0xffffffffu, i < nleaves);
    if (i >= nleaves) continue;
    const int b = bucket[i];
    const unsigned grp = __match_any_sync(act, b);
    const int leader = __ffs(grp) - 1;
    int pos = 0;
    if (lane == leader) pos = atomicAdd(&cursor[b], __popc(grp));
    pos = __shfl_sync(grp, pos, leader) + start[b] + __popc(grp & ((1u << lane) - 1));
    const int c = leaves[i];
    order[pos] = make_int4(info[c].w, info[c].z, off[c], off[c + 1]);
    nsrc[pos] = work[i];
  }
}

static int p2p_share(const SolverBase& s) {
  return s.cfg.images > 0 ? INT_MAX : s.cfg.precision == FMM_FP32 ? 512 : 192;
}

// The launch order of a few pairs that the host lists (a single-operator call: CSR offsets per
// cell, the cells' bodies in kc_ibody and kc_nbody), worked out there: no kernel and no wait for
// the team counts (one pair of leaves 0.060 ms a call with the device's order, 0.038 now).  The
// targets follow their source counts in p2p_nsrc; inside a team size they keep call order.
void order_p2p_pairs(SolverBase& s, const std::vector<unsigned long long>& pairs,
                     const std::vector<int>& off, const std::vector<int>& targets) {
  const size_t np = pairs.size(), nt = targets.size();
  std::vector<unsigned long long> srcs(np);
  std::vector<int4> order(nt);
  std::vector<int> nsrc(nt), cls(nt), sorted(2 * nt);
  int* teams = s.scal_host + kP2PTeamsHost;
  std::fill(teams, teams + 4, 0);
  for (size_t t = 0; t < nt; t++) {
    const int c = targets[t];
    unsigned long long src = 0;
    for (int k = off[c]; k < off[c + 1]; k++) {
      const unsigned p = (unsigned)pairs[k];
      const int j = pair_cell(p);
      src += (unsigned)s.kc_nbody[j];
      srcs[k] = p2p_leaf(s.kc_ibody[j], s.kc_nbody[j], pair_img(p));
    }
    cls[t] = p2p_class(src, s.kc_nbody[c], p2p_share(s));
    nsrc[t] = (int)std::min<unsigned long long>(src, INT_MAX);
    teams[cls[t]]++;
  }
  int at[4] = {0, teams[0], teams[0] + teams[1], teams[0] + teams[1] + teams[2]};
  for (size_t t = 0; t < nt; t++) {
    const int c = targets[t], i = at[cls[t]]++;
    order[i] = make_int4(s.kc_ibody[c], s.kc_nbody[c], off[c], off[c + 1]);
    sorted[i] = nsrc[t];
    sorted[nt + t] = c;
  }
  s.p2p_srcs.ensure(np);
  s.p2p_order.ensure(nt);
  s.p2p_nsrc.ensure(2 * nt);
  auto up = [&](void* dst, const void* src, size_t bytes) {
    FMM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s.stream));
  };
  up(s.p2p_srcs.p, srcs.data(), np * sizeof(srcs[0]));
  up(s.p2p_order.p, order.data(), nt * sizeof(order[0]));
  up(s.p2p_nsrc.p, sorted.data(), 2 * nt * sizeof(int));
}

// the launch order of the current P2P lists, on the solver's current stream; the team counts
// reach s.scal_host (kP2PTeamsHost) once that stream has been waited for
void order_p2p_targets(SolverBase& s) {
  const int nl = s.nleaves;
  if (nl <= 0) return;
  s.p2p_srcs.ensure(std::max<long long>(s.np2p, 1));
  s.p2p_bucket.ensure(nl);
  s.p2p_work.ensure(nl);
  s.p2p_order.ensure(nl);
  s.p2p_nsrc.ensure(nl);
  s.p2p_hist.ensure(2 * kP2PBuckets + 4);
  int *hist = s.p2p_hist.p, *cursor = hist + kP2PBuckets, *teams = cursor + kP2PBuckets;
  FMM_CUDA(cudaMemsetAsync(hist, 0, 2 * kP2PBuckets * sizeof(int), s.stream));
  k_p2p_work<<<std::min(ceil_div(nl, 8), 148 * 4), 256, 0, s.stream>>>(
      nl, s.leaves.p, s.p2p_off.p, s.p2p.p, s.c_info.p, s.p2p_srcs.p,
      s.p2p_bucket.p, s.p2p_work.p, hist, p2p_share(s));
  FMM_LAUNCH_CHECK();
  k_p2p_place<<<std::min(ceil_div(nl, 256), 148 * 4), 256, 0, s.stream>>>(
      nl, s.leaves.p, s.p2p_bucket.p, s.p2p_work.p, hist, s.p2p_off.p, s.c_info.p, cursor, teams,
      s.p2p_order.p, s.p2p_nsrc.p);
  FMM_LAUNCH_CHECK();
  FMM_CUDA(cudaMemcpyAsync(s.scal_host + kP2PTeamsHost, teams, 4 * sizeof(int),
                           cudaMemcpyDeviceToHost, s.stream));
}

template <typename T> void run_p2p(Solver<T>& s) {
  if (s.nleaves == 0) return;
  constexpr bool comp = sizeof(T) == 4;
  const int* t = s.scal_host + kP2PTeamsHost;
  const long long blocks = (long long)t[0] + ceil_div(4LL * t[1], kP2PWarps) +
                           ceil_div(2LL * t[2], kP2PWarps) + ceil_div(t[3], kP2PWarps);
  k_p2p<T, comp><<<(int)blocks, 32 * kP2PWarps, 0, s.stream>>>(
      s.p2p_order.p, s.p2p_nsrc.p, t[0], t[1], t[2], t[3], s.p2p_srcs.p,
      s.bodies.p, (T)s.cfg.eps2, (T)s.cfg.cycle, s.trg_s.p, s.trg_e.p, std::min(s.p2p_g4, 8),
      std::min(s.p2p_g2, 16), s.cfg.images > 0);
  FMM_LAUNCH_CHECK();
}

template void run_p2p<float>(Solver<float>&);
template void run_p2p<double>(Solver<double>&);

}  // namespace fmmb200
