// Two-electron integrals of super-shell pairs (host and device code).
//
// The quartets of a molecule are ordered by pair type (0: s x s, 1: s x sp, 2: sp x sp), the
// smaller type as bra.  A sp x sp bra is cut into slices F x sp (F = s: like type 1; F = p: three
// slices, axes permuted so that F lies along axis 0), so a bra has 1 or 4 functions and a ket 1,
// 4 or 16.  With the Hermite expansion (r-A) = PA + u d/dP, u = 1/(2 zeta), of the
// McMurchie-Davidson scheme (J. Comput. Phys. 26, 218 (1978)) a bra function is a polynomial in
// d/dX (X = P - Q) acting on f = pref F_0(rho X^2).  For a fixed ket primitive the ket's
// polynomial (QC - v d), (QD - v d) is fixed too, so one lane sums, over the bra's primitives,
//   Phi_b = sum_p [bra polynomial of function b] f   and its derivatives up to the ket's order
// (1, 4 or 10 values per bra function) and applies the ket's polynomial once at the end: the cost
// per primitive quartet is the derivative tensor and the bra's polynomial, not the up to 64
// integrals.
#pragma once
#include "boys.cuh"
#include "super.cuh"

// a bra slice's primitive: coefficients of F x s and F x p, u, (P - A)_F, P - B, zeta, P
template <typename T> struct __align__(16) B2EriBra { T kS, kP, u, FA, B[3], z, P[3], pad; };
// a ket primitive: eta, v = 1/(2 eta), Q, Q - C, Q - D, coefficients
template <typename T> struct B2EriKet { T z, v, Q[3], C[3], D[3], kss, ksp, kps, kpp; };

// bra primitive from a pair record; f: axis of F (p slices), AB: A - B (original axes)
B2_HD void b2es_bra(const B2gPrim &r, bool p, int f, const double *AB, B2EriBra<double> &o) {
  o.kS = p ? r.kps : r.kss;
  o.kP = p ? r.kpp : r.ksp;
  o.u = r.u; o.z = r.z; o.pad = 0.0;
  for (int k = 0; k < 3; ++k) {
    const int x = f + k >= 3 ? f + k - 3 : f + k;
    o.B[k] = r.ra * AB[x];
    o.P[k] = r.P[x];
  }
  o.FA = (r.ra - 1.0) * AB[f];
}
B2_HD void b2es_bra(const B2gPrim32 &r, bool p, int f, const double *, B2EriBra<float> &o) {
  o.kS = p ? r.kps : r.kss;
  o.kP = p ? r.kpp : r.ksp;
  o.u = r.u; o.z = r.z; o.pad = 0.f;
  for (int k = 0; k < 3; ++k) {
    const int x = f + k >= 3 ? f + k - 3 : f + k;
    o.B[k] = r.B[x];
    o.P[k] = r.P[x];
  }
  o.FA = r.A[f];
}
// ket primitive, axes permuted by f
B2_HD void b2es_ket(const B2gPrim &r, int f, const double *CD, B2EriKet<double> &o) {
  o.z = r.z; o.v = r.u; o.kss = r.kss; o.ksp = r.ksp; o.kps = r.kps; o.kpp = r.kpp;
  for (int k = 0; k < 3; ++k) {
    const int x = f + k >= 3 ? f + k - 3 : f + k;
    const double cd = x == 0 ? CD[0] : (x == 1 ? CD[1] : CD[2]);
    o.Q[k] = x == 0 ? r.P[0] : (x == 1 ? r.P[1] : r.P[2]);
    o.C[k] = (r.ra - 1.0) * cd;
    o.D[k] = r.ra * cd;
  }
}
B2_HD void b2es_ket(const B2gPrim32 &r, int f, const double *, B2EriKet<float> &o) {
  o.z = r.z; o.v = r.u; o.kss = r.kss; o.ksp = r.ksp; o.kps = r.kps; o.kpp = r.kpp;
  for (int k = 0; k < 3; ++k) {
    const int x = f + k >= 3 ? f + k - 3 : f + k;
    o.Q[k] = x == 0 ? r.P[0] : (x == 1 ? r.P[1] : r.P[2]);
    o.C[k] = x == 0 ? r.A[0] : (x == 1 ? r.A[1] : r.A[2]);
    o.D[k] = x == 0 ? r.B[0] : (x == 1 ? r.B[1] : r.B[2]);
  }
}

// TB: bra slice 0 (s x s), 1 (s x sp), 2 (p x sp); TK: ket pair type
template <typename T, int TB, int TK>
struct B2Es {
  static constexpr bool BF = TB == 2;
  static constexpr int NB = TB ? 4 : 1, NK = TK == 0 ? 1 : (TK == 1 ? 4 : 16);
  static constexpr int L = TK + (TB ? 1 : 0) + (BF ? 1 : 0);        // Boys and tensor order
  static constexpr int NP = b2g_ncart(TK);                           // derivatives kept per bra function

  B2_HD static void zero(T phi[NB][NP]) {
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int k = 0; k < NP; ++k) phi[b][k] = (T)0;
  }

  // one primitive quartet added to phi
  B2_HD static void quartet(const B2EriBra<T> &p, const B2EriKet<T> &q, const T *btab, T phi[NB][NP]) {
    const T X[3] = {p.P[0] - q.Q[0], p.P[1] - q.Q[1], p.P[2] - q.Q[2]};
    T rho, rs;
    b2_rho_rs<T>(p.z * q.z, p.z + q.z, rho, rs);
    const T tt = rho * (X[0] * X[0] + X[1] * X[1] + X[2] * X[2]);
    T F[L + 1], f[L + 1];
    b2_boys<T, L, T>(tt, btab, F);
    {
      const T m2r = (T)-2 * rho;
      T s = rs;
#pragma unroll
      for (int n = 0; n <= L; ++n) { f[n] = s * F[n]; s *= m2r; }
    }
    T R[b2g_ncart(L)];
    b2gs_rtensor<L>(X, f, R);
    if constexpr (TB == 0) {
#pragma unroll
      for (int k = 0; k < NP; ++k) phi[0][k] += p.kS * R[k];
    } else {
      T w[b2g_ncart(TK + 1)];                                      // F's polynomial applied
      if constexpr (BF) b2gs_shift<TK + 1, 0>(p.FA, p.u, R, w);
      else b2gs_copy<TK + 1>(R, w);
      const T uP = p.kP * p.u;
#pragma unroll
      for (int l = 0; l <= TK; ++l)
#pragma unroll
        for (int i = l; i >= 0; --i)
#pragma unroll
          for (int j = l - i; j >= 0; --j) {
            const int k = l - i - j, e = b2g_cidx(i, j, k);
            const T kw = p.kP * w[e];
            phi[0][e] += p.kS * w[e];
            // (r-P)_F (r-P)_b meets at one point for b = F (axis 0)
            phi[1][e] += p.B[0] * kw + uP * (BF ? w[b2g_cidx(i + 1, j, k)] + R[e] : w[b2g_cidx(i + 1, j, k)]);
            phi[2][e] += p.B[1] * kw + uP * w[b2g_cidx(i, j + 1, k)];
            phi[3][e] += p.B[2] * kw + uP * w[b2g_cidx(i, j, k + 1)];
          }
    }
  }

  // integrals of bra function b with every ket function: out[d] (TK 1: second function s, x, y, z)
  // or out[4 c + d] (TK 2)
  B2_HD static void ket(const B2EriKet<T> &q, const T *phi, T *out) {
    if constexpr (TK == 0) {
      out[0] = q.kss * phi[0];
    } else {
      const T v = q.v;
      out[0] = q.kss * phi[0];
#pragma unroll
      for (int d = 0; d < 3; ++d) out[1 + d] = q.ksp * (q.D[d] * phi[0] - v * phi[1 + d]);
      if constexpr (TK == 2) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          T psi[4];                                              // (QC - v d_c) phi and its gradient
          psi[0] = q.C[c] * phi[0] - v * phi[1 + c];
#pragma unroll
          for (int d = 0; d < 3; ++d)
            psi[1 + d] = q.C[c] * phi[1 + d] -
                         v * phi[b2g_cidx((c == 0) + (d == 0), (c == 1) + (d == 1), (c == 2) + (d == 2))];
          out[4 * (1 + c)] = q.kps * psi[0];
#pragma unroll
          for (int d = 0; d < 3; ++d)
            out[4 * (1 + c) + 1 + d] =
                q.kpp * (q.D[d] * psi[0] - v * psi[1 + d] + (c == d ? v * phi[0] : (T)0));
        }
      }
    }
  }
};

// Work of one class: bra slices i, each with the ket pairs k < limit(i).  Pair indices follow
// b2gs_pair's storage: s x s, s x sp, sp x sp.
B2_HD int b2es_npair(int ns, int np, int type) {
  return type == 0 ? ns * (ns + 1) / 2 : type == 1 ? ns * np : np * (np + 1) / 2;
}
B2_HD int b2es_first(int ns, int np, int type) {
  return type == 0 ? 0 : type == 1 ? ns * (ns + 1) / 2 : ns * (ns + 1) / 2 + ns * np;
}
// bra slices of class (TB, TK): s x s; s x sp pairs and, for sp x sp kets, the s slices of sp x sp
// pairs; the p slices of sp x sp pairs (axis minor)
B2_HD int b2es_nbra(int ns, int np, int TB, int TK) {
  return TB == 0 ? b2es_npair(ns, np, 0)
                 : TB == 1 ? ns * np + (TK == 2 ? b2es_npair(ns, np, 2) : 0) : 3 * b2es_npair(ns, np, 2);
}
// pair of bra slice i and the number of its kets (each unordered pair of pairs once)
B2_HD void b2es_bra_of(int ns, int np, int TB, int TK, int i, int &pair, int &limit) {
  const int nk = b2es_npair(ns, np, TK);
  if (TB == 0) { pair = i; limit = TK == 0 ? i + 1 : nk; return; }
  if (TB == 1 && i < ns * np) { pair = b2es_first(ns, np, 1) + i; limit = TK == 1 ? i + 1 : nk; return; }
  const int p = TB == 1 ? i - ns * np : i / 3;
  pair = b2es_first(ns, np, 2) + p;
  limit = p + 1;
}

// one integral (i j | k l) into the molecule's s8 list.  same1 / same2: both functions of the
// pair come from one super shell (every ordered pair occurs, one is kept); same: bra and ket are
// one pair.  AO index -1: a super shell without that function.
template <typename TO>
B2_HD void b2es_put(TO *out, int i, int j, int k, int l, bool same1, bool same2, bool same, TO v) {
  if (i < 0 || j < 0 || k < 0 || l < 0 || (same1 && j > i) || (same2 && l > k)) return;
  const int ij = i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
  const int kl = k >= l ? k * (k + 1) / 2 + l : l * (l + 1) / 2 + k;
  if (same && kl > ij) return;
  const int r = ij >= kl ? ij : kl, c = ij >= kl ? kl : ij;
  out[(long long)(r * (r + 1) / 2) + c] = v;
}
