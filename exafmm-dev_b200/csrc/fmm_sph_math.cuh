// Spherical-harmonic translation operators of the Laplace FMM, P known at compile time.
//
// Restates kernels/LaplaceSphericalCPU.cxx (evalMultipole :29-65, evalLocal :68-101,
// P2M :103-118, M2M :120-147, M2L :149-191, L2L :193-224, L2P :226-256) for the device:
//   * angles come straight from the Cartesian offset: cos(alpha) = dz / r,
//     sin(alpha) = |(dx, dy)| / r, e^(i beta) = (dx + i dy) / |(dx, dy)|, in place of the
//     reference's acos / atan2 / cos / sin round trip (same values up to rounding);
//   * harmonics are stored for m >= 0 only, Y[n, -m] = conj(Y[n, m]) (the reference keeps
//     both halves, :41-42), at index n (n + 1) / 2 + m, the layout of the expansions;
//   * the M2L sum over m < 0 and m >= 0 is folded into per-(n, |m|) terms with the signs
//     of :158-185 resolved at compile time.
// Every function is __host__ __device__ so the CPU tests run the exact device arithmetic.
#pragma once
#include <cmath>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace fmmb200 {
namespace sph {

__host__ __device__ constexpr int NT(int P) { return P * (P + 1) / 2; }
__host__ __device__ constexpr int sidx(int n, int m) { return n * (n + 1) / 2 + m; }

template <typename T> struct Angles {
  T r, x, y, cb, sb;  // |dX|, cos(alpha), sin(alpha), cos(beta), sin(beta)
};

template <typename T> __host__ __device__ __forceinline__ T hsqrt(T v) { return std::sqrt(v); }

// cart2sph (:9-13): alpha = acos(dz / r) (0 when r = 0), beta = atan2(dy, dx)
template <typename T> __host__ __device__ __forceinline__ Angles<T> angles(T dx, T dy, T dz) {
  Angles<T> a;
  T rxy2 = dx * dx + dy * dy;
  a.r = hsqrt(rxy2 + dz * dz);
  T rxy = hsqrt(rxy2);
  if (a.r > T(0)) {
    T inv = T(1) / a.r;
    a.x = dz * inv;
    a.y = rxy * inv;
  } else {
    a.x = T(1);
    a.y = T(0);
  }
  if (rxy > T(0)) {
    T inv = T(1) / rxy;
    a.cb = dx * inv;
    a.sb = dy * inv;
  } else {
    a.cb = dx < T(0) ? T(-1) : T(1);  // atan2(+-0, x) = 0 or pi
    a.sb = T(0);
  }
  return a;
}

// 1 / sqrt(v): the device's reciprocal square root (rsqrtf, rsqrt), the quotient on the host
template <typename T> __host__ __device__ __forceinline__ T hrsqrt(T v) {
#ifdef __CUDA_ARCH__
  if constexpr (sizeof(T) == 4) return rsqrtf(v);
  else return rsqrt(v);
#else
  return T(1) / std::sqrt(v);
#endif
}

// angles() for an offset of nonzero length with reciprocal square roots instead of two
// square roots and two divisions (r = r^2 / sqrt(r^2)); invr = 1 / r.  For the M2L pairs,
// whose cells are well separated.
template <typename T>
__host__ __device__ __forceinline__ Angles<T> angles_rs(T dx, T dy, T dz, T& invr) {
  Angles<T> a;
  const T rxy2 = dx * dx + dy * dy, r2 = rxy2 + dz * dz;
  invr = hrsqrt(r2);
  a.r = r2 * invr;
  a.x = dz * invr;
  if (rxy2 > T(0)) {
    const T ixy = hrsqrt(rxy2);
    a.y = rxy2 * ixy * invr;
    a.cb = dx * ixy;
    a.sb = dy * ixy;
  } else {
    a.y = T(0);
    a.cb = dx < T(0) ? T(-1) : T(1);
    a.sb = T(0);
  }
  return a;
}

// evalMultipole (:29-65) without the theta derivative: Y[n, m] = rho^n P_n^m e^(i m beta)
// / (-1)^n (n + m)!-style normalisation of the reference; its divisions by -(n + m) and
// (2m + 2)(2m + 1) are multiplications by the reciprocals here.
template <typename T, int P>
__host__ __device__ __forceinline__ void multipole(const Angles<T>& a, T rho, T* yr, T* yi) {
  T fact = 1, pn = 1, rhom = 1;
  T er = 1, ei = 0;
#pragma unroll
  for (int m = 0; m < P; m++) {
    T p = pn;
    yr[sidx(m, m)] = rhom * p * er;
    yi[sidx(m, m)] = rhom * p * ei;
    T p1 = p;
    p = a.x * (2 * m + 1) * p1;
    rhom *= rho;
    T rhon = rhom;
#pragma unroll
    for (int n = m + 1; n < P; n++) {
      rhon *= T(-1) / T(n + m);
      yr[sidx(n, m)] = rhon * p * er;
      yi[sidx(n, m)] = rhon * p * ei;
      T p2 = p1;
      p1 = p;
      p = (a.x * (2 * n + 1) * p1 - (n + m) * p2) * (T(1) / T(n - m + 1));
      rhon *= rho;
    }
    rhom *= T(-1) / T((2 * m + 2) * (2 * m + 1));
    pn = -pn * fact * a.y;
    fact += 2;
    T t = er * a.cb - ei * a.sb;
    ei = er * a.sb + ei * a.cb;
    er = t;
  }
}

// evalLocal (:68-101): singular harmonics y[n, m] = (-1)^n r^-(n+1) (n - m)! P_n^m e^(i m beta)
// with the reference's P_n^m.  Q[n] = (n - m)! P_n^m follows
//   Q[m] = P_m^m,   Q[n + 1] = (2n + 1) x Q[n] - (n + m)(n - m) Q[n - 1]
// (the reference's recurrence times (n + 1 - m)!), so each term costs one multiply and one
// fused multiply-add, and the radial factor is a table of P powers of -1/r.
template <typename T, int P>
__host__ __device__ __forceinline__ void local(const Angles<T>& a, T* yr, T* yi) {
  const T ninvr = -T(1) / a.r;
  T fact = 1, pn = 1;
  T rpm = -ninvr;  // (-1)^m / r^(m+1)
  T er = 1, ei = 0;
#pragma unroll
  for (int m = 0; m < P; m++) {
    T q = pn, qm1 = 0;  // Q[m] = P_m^m
    {
      const T t = q * rpm;
      yr[sidx(m, m)] = t * er;
      yi[sidx(m, m)] = t * ei;
    }
    T rpn = rpm;
#pragma unroll
    for (int n = m + 1; n < P; n++) {
      // Q[n] = (2n - 1) x Q[n-1] - (n - 1 + m)(n - 1 - m) Q[n-2]
      const T qn = fma(T(2 * n - 1) * a.x, q, T(-(n - 1 + m) * (n - 1 - m)) * qm1);
      qm1 = q;
      q = qn;
      rpn *= ninvr;
      const T t = q * rpn;
      yr[sidx(n, m)] = t * er;
      yi[sidx(n, m)] = t * ei;
    }
    rpm *= ninvr;
    pn = -pn * fact * a.y;
    fact += 2;
    const T tt = er * a.cb - ei * a.sb;
    ei = er * a.sb + ei * a.cb;
    er = tt;
  }
}

// M2L of one source multipole into a register local expansion (:149-191, mutual = false,
// unnormalised multipoles), for the output degrees j in [J0, J1) only (the FP32 kernel
// splits the outputs into passes).  Mj holds NT (re, im) pairs.  The loop bounds are
// compile-time after unrolling, so the whole contraction resolves to register operands.
// (re, im) of one coefficient; on the device one 8-byte (float) or 16-byte (double) load,
// for a row that starts on a multiple of 2 reals (every expansion row does: its length is
// even)
__host__ __device__ __forceinline__ void load_pair(const float* p, float& a, float& b) {
#ifdef __CUDA_ARCH__
  const float2 v = *reinterpret_cast<const float2*>(p);
  a = v.x;
  b = v.y;
#else
  a = p[0];
  b = p[1];
#endif
}
__host__ __device__ __forceinline__ void load_pair(const double* p, double& a, double& b) {
#ifdef __CUDA_ARCH__
  const double2 v = *reinterpret_cast<const double2*>(p);
  a = v.x;
  b = v.y;
#else
  a = p[0];
  b = p[1];
#endif
}

template <typename T, int P, int J0 = 0, int J1 = P>
__host__ __device__ __forceinline__ void m2l_pair(const T* yr, const T* yi, const T* Mj, T* Lr,
                                                  T* Li) {
  // Every product goes straight into its accumulator as one fused multiply-add; the signs
  // ((-1)^j of :189, (-1)^min(k, mu) of the m > 0 half, the conjugations) are compile-time
  // after unrolling and become operand negations.
#pragma unroll
  for (int n = 0; n < P - J0; n++) {
#pragma unroll
    for (int mu = 0; mu <= n; mu++) {
      T mr, mi;
      load_pair(Mj + 2 * sidx(n, mu), mr, mi);
#pragma unroll
      for (int j = J0; j < J1; j++) {
        if (j + n >= P) break;
        const int a = j + n;
        const T sr = (j & 1) ? -mr : mr, si = (j & 1) ? -mi : mi;  // (-1)^j M[n, mu]
#pragma unroll
        for (int k = 0; k <= j; k++) {
          const int t = sidx(j, k);
          if (mu == 0) {
            // M[n,0] conj(Y[a,k])
            const T ur = yr[sidx(a, k)], ui = yi[sidx(a, k)];
            Lr[t] = fma(sr, ur, Lr[t]);
            Lr[t] = fma(si, ui, Lr[t]);
            Li[t] = fma(si, ur, Li[t]);
            Li[t] = fma(-sr, ui, Li[t]);
          } else {
            // m = -mu: conj(M[n,mu] Y[a, k+mu])
            const T ur = yr[sidx(a, k + mu)], ui = yi[sidx(a, k + mu)];
            Lr[t] = fma(sr, ur, Lr[t]);
            Lr[t] = fma(-si, ui, Lr[t]);
            Li[t] = fma(-sr, ui, Li[t]);
            Li[t] = fma(-si, ur, Li[t]);
            // m = +mu: (-1)^(k < mu ? k : mu) M[n,mu] Y[a, mu-k] (conj Y[a, k-mu] if k > mu)
            const bool neg = ((k < mu ? k : mu) & 1) != 0;
            const T br = neg ? -sr : sr, bi = neg ? -si : si;
            if (mu >= k) {
              const T wr = yr[sidx(a, mu - k)], wi = yi[sidx(a, mu - k)];
              Lr[t] = fma(br, wr, Lr[t]);
              Lr[t] = fma(-bi, wi, Lr[t]);
              Li[t] = fma(br, wi, Li[t]);
              Li[t] = fma(bi, wr, Li[t]);
            } else {
              const T wr = yr[sidx(a, k - mu)], wi = yi[sidx(a, k - mu)];
              Lr[t] = fma(br, wr, Lr[t]);
              Lr[t] = fma(bi, wi, Lr[t]);
              Li[t] = fma(bi, wr, Li[t]);
              Li[t] = fma(-br, wi, Li[t]);
            }
          }
        }
      }
    }
  }
}

// The local harmonics split into a real factor and an azimuthal phase: Y[n, m] =
// rho[n, m] e^(i m beta) for m >= 0 (rho = the t of local(), the same arithmetic given
// invr = 1 / r).  rho is stored for the degrees n >= A0 only, at sidx(n, m) - sidx(A0, 0);
// (cr[m], ci[m]) = e^(i m beta) for m < P.
template <typename T, int P, int A0>
__host__ __device__ __forceinline__ void local_rho(const Angles<T>& a, T invr, T* rho, T* cr,
                                                   T* ci) {
  const T ninvr = -invr;
  T fact = 1, pn = 1;
  T rpm = -ninvr;  // (-1)^m / r^(m+1)
  T er = 1, ei = 0;
#pragma unroll
  for (int m = 0; m < P; m++) {
    cr[m] = er;
    ci[m] = ei;
    T q = pn, qm1 = 0;  // Q[m] = P_m^m
    if (m >= A0) rho[sidx(m, m) - sidx(A0, 0)] = q * rpm;
    T rpn = rpm;
#pragma unroll
    for (int n = m + 1; n < P; n++) {
      const T qn = fma(T(2 * n - 1) * a.x, q, T(-(n - 1 + m) * (n - 1 - m)) * qm1);
      qm1 = q;
      q = qn;
      rpn *= ninvr;
      if (n >= A0) rho[sidx(n, m) - sidx(A0, 0)] = q * rpn;
    }
    rpm *= ninvr;
    pn = -pn * fact * a.y;
    fact += 2;
    const T tt = er * a.cb - ei * a.sb;
    ei = er * a.sb + ei * a.cb;
    er = tt;
  }
}

// The M2L of m2l_pair in the source's azimuthal frame.  Every term of output (j, k) carries
// the phase e^(i (m - k) beta) of its harmonic, so with M'[n, mu] = M[n, mu] e^(i mu beta)
//   L[j, k] += e^(-i k beta) A[j, k],   A[j, k] = sum over (n, mu) of real rho times M' or
//   conj(M'),
// and each term of A is two real multiply-adds instead of a complex one (four): the
// source is rotated once on entry (one complex product per mu > 0 coefficient) and each
// output once on exit.  Terms and signs as m2l_pair: mu = 0: (-1)^j rho[a, k] M';
// m = -mu: (-1)^j rho[a, k + mu] conj(M'); m = +mu: (-1)^(j + min(k, mu)) rho[a, |mu - k|] M'.
template <typename T, int P, int J0, int J1>
__host__ __device__ __forceinline__ void m2l_pair_rot(const T* rho, const T* cr, const T* ci,
                                                      const T* Mj, T* Lr, T* Li) {
  constexpr int O0 = sidx(J0, 0), NO = sidx(J1, 0) - sidx(J0, 0);
  T Ar[NO], Ai[NO];
#pragma unroll
  for (int t = 0; t < NO; t++) Ar[t] = Ai[t] = T(0);
#pragma unroll
  for (int n = 0; n < P - J0; n++) {
#pragma unroll
    for (int mu = 0; mu <= n; mu++) {
      T mr, mi;
      load_pair(Mj + 2 * sidx(n, mu), mr, mi);
      if (mu > 0) {
        const T r = mr * cr[mu] - mi * ci[mu];
        mi = mr * ci[mu] + mi * cr[mu];
        mr = r;
      }
#pragma unroll
      for (int j = J0; j < J1; j++) {
        if (j + n >= P) break;
        const int a = j + n;
        const bool oj = (j & 1) != 0;
#pragma unroll
        for (int k = 0; k <= j; k++) {
          const int t = sidx(j, k) - O0;
          if (mu == 0) {
            const T p = rho[sidx(a, k) - O0];
            const T ps = oj ? -p : p;
            Ar[t] = fma(ps, mr, Ar[t]);
            Ai[t] = fma(ps, mi, Ai[t]);
          } else {
            const T p1 = rho[sidx(a, k + mu) - O0];
            const T s1 = oj ? -p1 : p1;
            Ar[t] = fma(s1, mr, Ar[t]);
            Ai[t] = fma(-s1, mi, Ai[t]);
            const T p2 = rho[sidx(a, mu >= k ? mu - k : k - mu) - O0];
            const bool o2 = oj != (((k < mu ? k : mu) & 1) != 0);
            const T s2 = o2 ? -p2 : p2;
            Ar[t] = fma(s2, mr, Ar[t]);
            Ai[t] = fma(s2, mi, Ai[t]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int j = J0; j < J1; j++)
#pragma unroll
    for (int k = 0; k <= j; k++) {
      const int t = sidx(j, k) - O0, g = sidx(j, k);
      if (k == 0) {
        Lr[g] += Ar[t];
        Li[g] += Ai[t];
      } else {
        Lr[g] = fma(cr[k], Ar[t], fma(ci[k], Ai[t], Lr[g]));
        Li[g] = fma(cr[k], Ai[t], fma(-ci[k], Ar[t], Li[g]));
      }
    }
}

// m2l_pair_rot with the loops the other way round: the rotated source coefficients of the
// degrees n < P - J0 held in registers and each output's sum A[j, k] finished and rotated
// before the next (the same terms in the same order, so the same results); for the
// passes of high output degree, which take few source coefficients and many outputs.
template <typename T, int P, int J0, int J1>
__host__ __device__ __forceinline__ void m2l_pair_rot_out(const T* rho, const T* cr,
                                                          const T* ci, const T* Mj, T* Lr,
                                                          T* Li) {
  constexpr int O0 = sidx(J0, 0), NIN = sidx(P - J0, 0);
  T Mr[NIN], Mi[NIN];
#pragma unroll
  for (int n = 0; n < P - J0; n++)
#pragma unroll
    for (int mu = 0; mu <= n; mu++) {
      T mr, mi;
      load_pair(Mj + 2 * sidx(n, mu), mr, mi);
      if (mu > 0) {
        const T r = mr * cr[mu] - mi * ci[mu];
        mi = mr * ci[mu] + mi * cr[mu];
        mr = r;
      }
      Mr[sidx(n, mu)] = mr;
      Mi[sidx(n, mu)] = mi;
    }
  // outputs by order k, then degree: e^(i k beta) advances by one rotation per k, so the
  // phases need not stay live in registers
  T er = T(1), ei = T(0);
#pragma unroll
  for (int k = 0; k < J1; k++) {
#pragma unroll
    for (int j = (k > J0 ? k : J0); j < J1; j++) {
      const bool oj = (j & 1) != 0;
      T ar = T(0), ai = T(0);
#pragma unroll
      for (int n = 0; n < P - j; n++) {
        const int a = j + n;
#pragma unroll
        for (int mu = 0; mu <= n; mu++) {
          const T mr = Mr[sidx(n, mu)], mi = Mi[sidx(n, mu)];
          if (mu == 0) {
            const T p = rho[sidx(a, k) - O0];
            const T ps = oj ? -p : p;
            ar = fma(ps, mr, ar);
            ai = fma(ps, mi, ai);
          } else {
            const T p1 = rho[sidx(a, k + mu) - O0];
            const T s1 = oj ? -p1 : p1;
            ar = fma(s1, mr, ar);
            ai = fma(-s1, mi, ai);
            const T p2 = rho[sidx(a, mu >= k ? mu - k : k - mu) - O0];
            const bool o2 = oj != (((k < mu ? k : mu) & 1) != 0);
            const T s2 = o2 ? -p2 : p2;
            ar = fma(s2, mr, ar);
            ai = fma(s2, mi, ai);
          }
        }
      }
      const int g = sidx(j, k);
      if (k == 0) {
        Lr[g] += ar;
        Li[g] += ai;
      } else {
        Lr[g] = fma(er, ar, fma(ei, ai, Lr[g]));
        Li[g] = fma(er, ai, fma(-ei, ar, Li[g]));
      }
    }
    const T tt = er * cr[1] - ei * ci[1];
    ei = er * ci[1] + ei * cr[1];
    er = tt;
  }
}

// The real harmonic factors of local_rho (up to rounding), all degrees n < P at sidx(n, m),
// with the radial power inside the recurrence
//   rho[n, m] = (2n - 1) (-x / r) rho[n-1, m] - (n - 1 + m)(n - 1 - m) / r^2 rho[n-2, m],
// three operations per term (the factors (2n - 1)(-x / r) are shared by all m).
template <typename T, int P>
__host__ __device__ __forceinline__ void fold_rho(const Angles<T>& a, T invr, T* rho) {
  const T xi = -a.x * invr, w = invr * invr, yi = a.y * invr;
  T X[P];
#pragma unroll
  for (int n = 1; n < P; n++) X[n] = T(2 * n - 1) * xi;
  T d = invr;  // rho[m, m] = (-1)^m P_m^m / r^(m+1)
#pragma unroll
  for (int m = 0; m < P; m++) {
    T q = d, qm1 = 0;
    rho[sidx(m, m)] = q;
#pragma unroll
    for (int n = m + 1; n < P; n++) {
      const int c = (n - 1 + m) * (n - 1 - m);
      const T qn = c ? fma(X[n], q, T(-c) * (w * qm1)) : X[n] * q;
      qm1 = q;
      q = qn;
      rho[sidx(n, m)] = q;
    }
    // P_{m+1}^{m+1} = -(2m + 1) sin(alpha) P_m^m
    d *= T(2 * m + 1) * yi;
  }
}

// a complex value (a pair of registers the packed two-wide FP32 instructions take together)
template <typename T> struct Cx {
  T r, i;
};
// a.r += u m.r, a.i += v m.i, each rounded once; FP32 on the device: one packed instruction
template <typename T>
__host__ __device__ __forceinline__ void fold_fma(T u, T v, const Cx<T>& m, Cx<T>& a) {
#ifdef __CUDA_ARCH__
  if constexpr (sizeof(T) == 4) {
    const float2 t = __ffma2_rn(make_float2(u, v), make_float2(m.r, m.i), make_float2(a.r, a.i));
    a.r = t.x;
    a.i = t.y;
    return;
  }
#endif
  a.r = fma(u, m.r, a.r);
  a.i = fma(v, m.i, a.i);
}

// The M2L of m2l_pair in the source's azimuthal frame, the terms of m = +mu and m = -mu
// folded.  Every term of output (j, k) carries the phase e^(i (m - k) beta) of its harmonic,
// so with M'[n, mu] = M[n, mu] e^(i mu beta)
//   L[j, k] += (-1)^j e^(-i k beta) A[j, k],
//   A[j, k] = sum over n of rho[j+n, k] M'[n, 0]
//           + sum over n, mu > 0 of (s rho[j+n, |k-mu|] + rho[j+n, k+mu]) Re M'[n, mu]
//                               + i (s rho[j+n, |k-mu|] - rho[j+n, k+mu]) Im M'[n, mu],
// s = (-1)^min(k, mu).  The two real factors depend on (j + n, k, mu) only, so they are formed
// once for all (j, n) of one sum: a term costs two multiply-adds (the unfolded form takes
// four), one for k = 0, whose factors are 2 rho[j+n, mu] and 0.
// Outputs of the orders k in [K0, K1) into A at fold_idx; the phases of the source by one
// rotation per mu; Mj the source's row by order (col_idx).
__host__ __device__ constexpr int fold_idx(int P, int K0, int k, int j) {
  int t = j - k;
  for (int q = K0; q < k; q++) t += P - q;
  return t;
}
// hide where a value came from (device): the compiler then forms values that depend on it
// again instead of keeping them in registers across a long unrolled sum
template <typename U> __host__ __device__ __forceinline__ void launder(U& v) {
#ifdef __CUDA_ARCH__
  if constexpr (sizeof(U) == 4) asm volatile("" : "+f"(v));
  else asm volatile("" : "+d"(v));
#endif
}
template <typename U> __host__ __device__ __forceinline__ void launder(const U*& v) {
#ifdef __CUDA_ARCH__
  asm volatile("" : "+l"(v));
#endif
}

// Source coefficients by order: the coefficients (n, mu), n = mu .. P - 1, of one order mu
// contiguous, each order padded to an even number, so that the sum over one mu reads whole
// 16-byte pairs.  Offset of (n, mu) in reals, and a row's length (a multiple of 16 bytes).
__host__ __device__ constexpr int col_idx(int P, int n, int mu) {
  int t = 0;
  for (int q = 0; q < mu; q++) t += (P - q + 1) / 2 * 2;
  return 2 * (t + n - mu);
}
__host__ __device__ constexpr int col_len(int P) { return col_idx(P, P, P); }
// coefficients p[0], p[1] (16 bytes in FP32 from a 16-byte boundary, two such in FP64)
template <typename T>
__host__ __device__ __forceinline__ void load_pair2(const T* p, Cx<T>& a, Cx<T>& b) {
#ifdef __CUDA_ARCH__
  if constexpr (sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a.r = v.x, a.i = v.y, b.r = v.z, b.i = v.w;
    return;
  }
#endif
  load_pair(p, a.r, a.i);
  load_pair(p + 2, b.r, b.i);
}

// the terms of the source orders MU, MU + 1, ... (a recursion over compile-time mu, so that
// every index below is a constant however long the unrolled sum); (er, ei) = e^(i MU beta)
template <typename T, int P, int K0, int K1, int MU>
__host__ __device__ __forceinline__ void m2l_fold_from(const T* rho, T cb, T sb, T er, T ei,
                                                       const T* Mj, Cx<T>* A) {
  constexpr int NS = P - K0;  // source degrees n < NS reach these outputs
  if constexpr (MU < NS) {
    Cx<T> m[NS - MU + 1];  // (and the pad of an odd column)
#pragma unroll
    for (int n = MU; n < NS; n += 2) {
      if (n + 1 < NS || sizeof(T) == 4) load_pair2(Mj + col_idx(P, n, MU), m[n - MU], m[n - MU + 1]);
      else load_pair(Mj + col_idx(P, n, MU), m[n - MU].r, m[n - MU].i);
    }
    if (MU > 0) {
#pragma unroll
      for (int n = 0; n < NS - MU; n++) {
        const T mr = m[n].r, mi = m[n].i;
        m[n].r = mr * er - mi * ei;
        m[n].i = mr * ei + mi * er;
      }
    }
#pragma unroll
    for (int k = K0; k < K1; k++) {
#pragma unroll
      for (int a = k + MU; a < P; a++) {
        if (MU == 0) {
          // (k = 0: half the term, doubled below with the terms of mu > 0)
          const T p = k == 0 ? T(0.5) * rho[sidx(a, 0)] : rho[sidx(a, k)];
#pragma unroll
          for (int n = 0; n <= a - k; n++) fold_fma(p, p, m[n], A[fold_idx(P, K0, k, a - n)]);
        } else if (k == 0) {
          const T p = rho[sidx(a, MU)];
#pragma unroll
          for (int n = MU; n <= a; n++) {
            Cx<T>& o = A[fold_idx(P, K0, 0, a - n)];
            o.r = fma(p, m[n - MU].r, o.r);
          }
        } else {
          const T p1 = rho[sidx(a, k + MU)], p2 = rho[sidx(a, MU >= k ? MU - k : k - MU)];
          const bool neg = ((k < MU ? k : MU) & 1) != 0;
          const T u = neg ? p1 - p2 : p1 + p2, v = neg ? -p2 - p1 : p2 - p1;
#pragma unroll
          for (int n = MU; n <= a - k; n++)
            fold_fma(u, v, m[n - MU], A[fold_idx(P, K0, k, a - n)]);
        }
      }
    }
    m2l_fold_from<T, P, K0, K1, MU + 1>(rho, cb, sb, er * cb - ei * sb, er * sb + ei * cb, Mj,
                                        A);
  }
}
template <typename T, int P, int K0, int K1>
__host__ __device__ __forceinline__ void m2l_fold(const T* rho, T cb, T sb, const T* Mj,
                                                  Cx<T>* A) {
#pragma unroll
  for (int t = 0; t < fold_idx(P, K0, K1, K1); t++) A[t].r = A[t].i = T(0);
  m2l_fold_from<T, P, K0, K1, 0>(rho, cb, sb, T(1), T(0), Mj, A);
  if (K0 == 0) {
#pragma unroll
    for (int j = 0; j < P; j++) {
      A[j].r += A[j].r;
      A[j].i += A[j].i;
    }
  }
}

// The regular harmonics' real factors: Y[n, m] of multipole() = reg[n, m] e^(i m beta).
template <typename T, int P>
__host__ __device__ __forceinline__ void multipole_rho(const Angles<T>& a, T rho, T* reg) {
  T fact = 1, pn = 1, rhom = 1;
#pragma unroll
  for (int m = 0; m < P; m++) {
    T p = pn, p1 = p;
    reg[sidx(m, m)] = rhom * p;
    p = a.x * (2 * m + 1) * p1;
    rhom *= rho;
    T rhon = rhom;
#pragma unroll
    for (int n = m + 1; n < P; n++) {
      rhon *= T(-1) / T(n + m);
      reg[sidx(n, m)] = rhon * p;
      const T p2 = p1;
      p1 = p;
      p = (a.x * (2 * n + 1) * p1 - (n + m) * p2) * (T(1) / T(n - m + 1));
      rhon *= rho;
    }
    rhom *= T(-1) / T((2 * m + 2) * (2 * m + 1));
    pn = -pn * fact * a.y;
    fact += 2;
  }
}

// M2M (UP) and L2L of m2m_term / l2l_term in the azimuthal frame of the shift, folded as
// m2l_fold: with the source (the child's M, the parent's L) rotated, S'[l, mu] = S[l, mu]
// e^(i mu beta), each output is e^(-i k beta) A[j, k] and
//   A[j, k] = sum over mu and d of (s2 reg[d, |k-mu|] + s1 reg[d, k+mu]) Re S'[l, mu]
//                             + i (s2 reg[d, |k-mu|] - s1 reg[d, k+mu]) Im S'[l, mu],
// l = j - d (M2M) or j + d (L2L), a harmonic of order above its degree d being none, and the
// two real factors shared by all (j, l) of one d.  M2M: s2 = (-1)^d, times (-1)^(k-mu) for
// k < mu (none at mu = 0), s1 = (-1)^(d+mu); L2L: s2 = (-1)^(k-mu) for mu < k, else 1,
// s1 = (-1)^k (none at mu = 0).  S: the row in the layout of the expansions.
template <typename T, int P, int K0, int K1, int MU, bool UP>
__host__ __device__ __forceinline__ void shift_fold_from(const T* reg, T cb, T sb, T er, T ei,
                                                         const T* S, Cx<T>* A) {
  if constexpr (MU < P) {
    Cx<T> m[P - MU];
#pragma unroll
    for (int l = MU; l < P; l++) {
      const T mr = S[2 * sidx(l, MU)], mi = S[2 * sidx(l, MU) + 1];
      m[l - MU].r = MU > 0 ? mr * er - mi * ei : mr;
      m[l - MU].i = MU > 0 ? mr * ei + mi * er : mi;
    }
#pragma unroll
    for (int k = K0; k < K1; k++) {
#pragma unroll
      for (int d = 0; d < P; d++) {
        const int q = MU >= k ? MU - k : k - MU;
        const bool has2 = q <= d && !(UP && MU == 0), has1 = k + MU <= d && !(!UP && MU == 0);
        if (!has2 && !has1) continue;
        const bool neg2 = UP ? (d & 1) != (k < MU && (q & 1)) : MU < k && (q & 1);
        const bool neg1 = UP ? ((d + MU) & 1) != 0 : (k & 1) != 0;
        T u = T(0), v = T(0);  // factors of the real and the imaginary part
        if (has2) u = v = neg2 ? -reg[sidx(d, q)] : reg[sidx(d, q)];
        if (has1) {
          const T p1 = neg1 ? -reg[sidx(d, k + MU)] : reg[sidx(d, k + MU)];
          v = has2 ? v - p1 : -p1;
          u = has2 ? u + p1 : p1;
        }
        // k = 0, mu > 0: both terms are there with the same sign, and v is zero
        const bool real = k == 0 && MU > 0;
#pragma unroll
        for (int l = MU; l < P; l++) {
          const int j = UP ? l + d : l - d;
          if (j < k || j >= P) continue;
          Cx<T>& o = A[fold_idx(P, K0, k, j)];
          if (real) o.r = fma(u, m[l - MU].r, o.r);
          else fold_fma(u, v, m[l - MU], o);
        }
      }
    }
    shift_fold_from<T, P, K0, K1, MU + 1, UP>(reg, cb, sb, er * cb - ei * sb, er * sb + ei * cb,
                                              S, A);
  }
}
// the outputs of the orders [K0, K1), rotated back, at fold_idx
template <typename T, int P, int K0, int K1, bool UP>
__host__ __device__ __forceinline__ void shift_fold(const T* reg, T cb, T sb, const T* S,
                                                    Cx<T>* A) {
#pragma unroll
  for (int t = 0; t < fold_idx(P, K0, K1, K1); t++) A[t].r = A[t].i = T(0);
  shift_fold_from<T, P, K0, K1, 0, UP>(reg, cb, sb, T(1), T(0), S, A);
  T er = T(1), ei = T(0);
#pragma unroll
  for (int k = 0; k < K1; k++) {
#pragma unroll
    for (int j = k; j < P && k >= K0 && k > 0; j++) {
      Cx<T>& o = A[fold_idx(P, K0, k, j)];
      const T r = fma(er, o.r, ei * o.i);
      o.i = fma(er, o.i, -ei * o.r);
      o.r = r;
    }
    const T t = er * cb - ei * sb;
    ei = er * sb + ei * cb;
    er = t;
  }
}

// Y[a, b] for any sign of b from the m >= 0 store (real parts yr, imaginary parts yi)
template <typename T>
__host__ __device__ __forceinline__ void yget(const T* yr, const T* yi, int a, int b, T& r,
                                              T& i) {
  if (b >= 0) {
    r = yr[sidx(a, b)];
    i = yi[sidx(a, b)];
  } else {
    r = yr[sidx(a, -b)];
    i = -yi[sidx(a, -b)];
  }
}

// M2M output coefficient (j, k) from one child (:127-144); Y (yr, yi) from multipole() at
// Xparent - Xchild, Mc the child's NT (re, im) pairs.  Runtime indices when (j, k) are
// runtime values, register operands when they are unrolled constants.
template <typename T>
__host__ __device__ __forceinline__ void m2m_term(int j, int k, const T* yr, const T* yi,
                                                  const T* Mc, T& outr, T& outi) {
  T sr = 0, si = 0;
#pragma unroll
  for (int n = 0; n <= j; n++) {
    // m in [max(-n, -j+k+n), min(k-1, n)]
#pragma unroll
    for (int m = -n; m <= n; m++) {
      if (m < -j + k + n) continue;
      if (m > k - 1) break;
      // Cj->M[(j-n)(j-n+1)/2 + k - m] * Ynm[n*n+n-m] * IPOW2N(m) * ODDEVEN(n)
      const int q = (j - n) * (j - n + 1) / 2 + k - m;
      const T Mr = Mc[2 * q], Mi = Mc[2 * q + 1];
      T ur, ui;
      yget(yr, yi, n, -m, ur, ui);
      const T pr = Mr * ur - Mi * ui, pi = Mr * ui + Mi * ur;
      const int sgn = ((m < 0 && (m & 1)) ? -1 : 1) * ((n & 1) ? -1 : 1);
      sr += sgn * pr;
      si += sgn * pi;
    }
    // m in [k, min(n, j+k-n)]
#pragma unroll
    for (int m = k; m <= n; m++) {
      if (m > j + k - n) break;
      // conj(Cj->M[(j-n)(j-n+1)/2 - k + m]) * Ynm[n*n+n-m] * ODDEVEN(k+n+m)
      const int q = (j - n) * (j - n + 1) / 2 - k + m;
      const T Mr = Mc[2 * q], Mi = -Mc[2 * q + 1];
      T ur, ui;
      yget(yr, yi, n, -m, ur, ui);
      const T pr = Mr * ur - Mi * ui, pi = Mr * ui + Mi * ur;
      const int sgn = ((k + n + m) & 1) ? -1 : 1;
      sr += sgn * pr;
      si += sgn * pi;
    }
  }
  outr = sr;
  outi = si;
}

// L2L output coefficient (j, k) from the parent (:203-222); Y (yr, yi) from multipole() at
// Xchild - Xparent, Lp the parent's NT (re, im) pairs.
template <typename T>
__host__ __device__ __forceinline__ void l2l_term(int P, int j, int k, const T* yr,
                                                  const T* yi, const T* Lp, T& outr, T& outi) {
  T sr = 0, si = 0;
#pragma unroll
  for (int n = j; n < P; n++) {
    // m in [j+k-n, -1]
#pragma unroll
    for (int m = -n; m < 0; m++) {
      if (m < j + k - n) continue;
      // conj(Cj->L[n(n+1)/2 - m]) * Ynm[(n-j)^2 + n-j + m-k] * ODDEVEN(k)
      const int q = n * (n + 1) / 2 - m;
      const T Lr = Lp[2 * q], Li = -Lp[2 * q + 1];
      T ur, ui;
      yget(yr, yi, n - j, m - k, ur, ui);
      const T pr = Lr * ur - Li * ui, pi = Lr * ui + Li * ur;
      const int sgn = (k & 1) ? -1 : 1;
      sr += sgn * pr;
      si += sgn * pi;
    }
#pragma unroll
    for (int m = 0; m <= n; m++) {
      const int d = m - k;
      if (n - j < (d < 0 ? -d : d)) continue;
      // Cj->L[n(n+1)/2 + m] * Ynm[(n-j)^2 + n-j + m-k] * ODDEVEN((m-k)(m<k))
      const int q = n * (n + 1) / 2 + m;
      const T Lr = Lp[2 * q], Li = Lp[2 * q + 1];
      T ur, ui;
      yget(yr, yi, n - j, d, ur, ui);
      const T pr = Lr * ur - Li * ui, pi = Lr * ui + Li * ur;
      const int sgn = (d < 0 && (d & 1)) ? -1 : 1;
      sr += sgn * pr;
      si += sgn * pi;
    }
  }
  outr = sr;
  outi = si;
}

// Whole M2M / L2L translations for the output degrees j in [J0, J1) with compile-time
// indices (register operands); out[t - sidx(J0, 0)] holds output t as (re, im).
template <typename T, int P, int J0 = 0, int J1 = P>
__host__ __device__ __forceinline__ void m2m_range(const T* yr, const T* yi, const T* Mc,
                                                   T* out) {
#pragma unroll
  for (int j = J0; j < J1; j++)
#pragma unroll
    for (int k = 0; k <= j; k++) {
      T r, i;
      m2m_term<T>(j, k, yr, yi, Mc, r, i);
      out[2 * (sidx(j, k) - sidx(J0, 0))] += r;
      out[2 * (sidx(j, k) - sidx(J0, 0)) + 1] += i;
    }
}
template <typename T, int P, int J0 = 0, int J1 = P>
__host__ __device__ __forceinline__ void l2l_range(const T* yr, const T* yi, const T* Lp,
                                                   T* out) {
#pragma unroll
  for (int j = J0; j < J1; j++)
#pragma unroll
    for (int k = 0; k <= j; k++) {
      T r, i;
      l2l_term<T>(P, j, k, yr, yi, Lp, r, i);
      out[2 * (sidx(j, k) - sidx(J0, 0))] += r;
      out[2 * (sidx(j, k) - sidx(J0, 0)) + 1] += i;
    }
}

// L2P of one body (:226-256): potential and gradient of the local expansion L (NT (re, im)
// pairs) at offset dX from the cell centre.  Harmonics and their theta derivatives are
// generated column by column and consumed on the fly.
template <typename T, int P>
__host__ __device__ __forceinline__ void l2p_body(T dx, T dy, T dz, const T* L, T& pot, T& gx,
                                                  T& gy, T& gz) {
  // the divisions of the reference (by rho per term, by -(n+m) and (2m+2)(2m+1) per
  // step) are multiplications by reciprocals here: one division per body
  Angles<T> a = angles(dx, dy, dz);
  const T rho = a.r, invrho = T(1) / rho;
  T s0 = 0, s1 = 0, s2 = 0, ph = 0;
  T fact = 1, pn = 1, rhom = 1;
  T er = 1, ei = 0;
  const T invy = T(1) / a.y;
#pragma unroll
  for (int m = 0; m < P; m++) {
    const T w = m == 0 ? T(1) : T(2);
    T p = pn;
    T p1 = p;
    p = a.x * (2 * m + 1) * p1;
    {
      // Y[m,m] and its theta derivative
      const T yv = rhom * p1;
      const T tv = rhom * (p - (m + 1) * a.x * p1) * invy;
      const T Lr = L[2 * sidx(m, m)], Li = L[2 * sidx(m, m) + 1];
      const T re = Lr * er - Li * ei, im = Lr * ei + Li * er;  // L * e^(i m beta)
      ph += w * yv * re;
      s0 += w * yv * re * invrho * m;
      s1 += w * tv * re;
      s2 -= w * yv * im * m;
    }
    rhom *= rho;
    T rhon = rhom;
#pragma unroll
    for (int n = m + 1; n < P; n++) {
      rhon *= T(-1) / T(n + m);
      const T yv = rhon * p;
      T p2 = p1;
      p1 = p;
      p = (a.x * (2 * n + 1) * p1 - (n + m) * p2) * (T(1) / T(n - m + 1));
      const T tv = rhon * ((n - m + 1) * p - (n + 1) * a.x * p1) * invy;
      const T Lr = L[2 * sidx(n, m)], Li = L[2 * sidx(n, m) + 1];
      const T re = Lr * er - Li * ei, im = Lr * ei + Li * er;
      ph += w * yv * re;
      s0 += w * yv * re * invrho * n;
      s1 += w * tv * re;
      s2 -= w * yv * im * m;
      rhon *= rho;
    }
    rhom *= T(-1) / T((2 * m + 2) * (2 * m + 1));
    pn = -pn * fact * a.y;
    fact += 2;
    T t = er * a.cb - ei * a.sb;
    ei = er * a.sb + ei * a.cb;
    er = t;
  }
  // sph2cart (:17-26)
  pot = ph;
  gx = a.y * a.cb * s0 + a.x * a.cb * invrho * s1 - a.sb * invrho * invy * s2;
  gy = a.y * a.sb * s0 + a.x * a.sb * invrho * s1 + a.cb * invrho * invy * s2;
  gz = a.x * s0 - a.y * invrho * s1;
}

}  // namespace sph
}  // namespace fmmb200
