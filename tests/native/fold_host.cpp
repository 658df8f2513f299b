// Host build of the folded M2L contraction (exafmm-dev_b200/csrc/fmm_sph_math.cuh: fold_rho,
// m2l_fold, shift_fold) for tests/test_fold_math.py: one pair's M2L in FP64 with the output
// orders taken in one group or split, the source row laid out by order as the kernel reads it,
// and one shift of an M2M or an L2L.
#include <vector>

#include "fmm_sph_math.cuh"

using namespace fmmb200;

namespace {

template <int P, int K0, int K1>
void group(const double* rho, const sph::Angles<double>& a, const double* row, double* Li) {
  sph::Cx<double> A[sph::fold_idx(P, K0, K1, K1)];
  sph::m2l_fold<double, P, K0, K1>(rho, a.cb, a.sb, row, A);
  double er = 1, ei = 0;
  for (int k = 0; k < K1; k++) {
    for (int j = k; j < P && k >= K0; j++) {
      const sph::Cx<double> o = A[sph::fold_idx(P, K0, k, j)];
      const double s = j & 1 ? -1 : 1;
      Li[2 * sph::sidx(j, k)] += s * (er * o.r + ei * o.i);
      Li[2 * sph::sidx(j, k) + 1] += s * (er * o.i - ei * o.r);
    }
    const double t = er * a.cb - ei * a.sb;
    ei = er * a.sb + ei * a.cb;
    er = t;
  }
}

template <int P> void pair(int split, const double* Xi, const double* Xj, const double* Mj,
                           double* Li) {
  double rho[sph::NT(P)], invr;
  const sph::Angles<double> a =
      sph::angles_rs(Xi[0] - Xj[0], Xi[1] - Xj[1], Xi[2] - Xj[2], invr);
  sph::fold_rho<double, P>(a, invr, rho);
  std::vector<double> row(sph::col_len(P), 0.0);
  for (int mu = 0; mu < P; mu++)
    for (int n = mu; n < P; n++)
      for (int c = 0; c < 2; c++) row[sph::col_idx(P, n, mu) + c] = Mj[2 * sph::sidx(n, mu) + c];
  if (split == 0) {
    group<P, 0, P>(rho, a, row.data(), Li);
  } else if (split == 1) {
    group<P, 0, 1>(rho, a, row.data(), Li);
    group<P, 1, P>(rho, a, row.data(), Li);
  } else {
    group<P, 0, P / 2>(rho, a, row.data(), Li);
    group<P, P / 2, P - 1>(rho, a, row.data(), Li);
    group<P, P - 1, P>(rho, a, row.data(), Li);
  }
}

// The folded M2M (up) and L2L of one shift, the outputs in one group or split at order 1 or P / 2.
template <int P, int K0, int K1, bool UP>
void shift_group(const double* reg, const sph::Angles<double>& a, const double* in, double* out) {
  sph::Cx<double> A[sph::fold_idx(P, K0, K1, K1)];
  sph::shift_fold<double, P, K0, K1, UP>(reg, a.cb, a.sb, in, A);
  for (int k = K0; k < K1; k++)
    for (int j = k; j < P; j++) {
      out[2 * sph::sidx(j, k)] += A[sph::fold_idx(P, K0, k, j)].r;
      out[2 * sph::sidx(j, k) + 1] += A[sph::fold_idx(P, K0, k, j)].i;
    }
}
template <int P, bool UP>
void shift(int split, const double* d, const double* in, double* out) {
  double reg[sph::NT(P)];
  const sph::Angles<double> a = sph::angles(d[0], d[1], d[2]);
  sph::multipole_rho<double, P>(a, a.r, reg);
  if (split == 0) {
    shift_group<P, 0, P, UP>(reg, a, in, out);
  } else if (split == 1) {
    shift_group<P, 0, 1, UP>(reg, a, in, out);
    shift_group<P, 1, P, UP>(reg, a, in, out);
  } else {
    shift_group<P, 0, P / 2, UP>(reg, a, in, out);
    shift_group<P, P / 2, P, UP>(reg, a, in, out);
  }
}

}  // namespace

extern "C" int fold_m2l(int P, int split, const double* Xi, const double* Xj, const double* Mj,
                        double* Li) {
#define CASE(p)                       \
  if (P == p) {                       \
    pair<p>(split, Xi, Xj, Mj, Li);   \
    return 0;                         \
  }
  CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10) CASE(12)
  return 1;
}

// d: parent - child (M2M, up) or child - parent (L2L)
extern "C" int fold_shift(int P, int up, int split, const double* d, const double* in,
                          double* out) {
#define SHIFT(p)                                  \
  if (P == p) {                                   \
    if (up) shift<p, true>(split, d, in, out);    \
    else shift<p, false>(split, d, in, out);      \
    return 0;                                     \
  }
  SHIFT(4) SHIFT(5) SHIFT(6) SHIFT(7) SHIFT(8) SHIFT(9) SHIFT(10) SHIFT(12)
  return 1;
}
