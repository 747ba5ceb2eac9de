// Two-electron part of the RKS nuclear gradient over super shells (host and device code).
//
// Super-shell pairs (super.cuh) are cut into slices F x {s} or F x {s, px, py, pz}: one function F
// on the first centre and every function of the second shell, so a slice has 1 or 4 components:
//   type 0  s x s;  type 1  s x sp;  type 2  p x sp (three slices per pair, one per axis).
// All functions of a slice share the primitive pair, so one Boys evaluation and one derivative
// tensor serve up to 16 integrals, and the integrals themselves are never formed: with
// Gamma_{Fb,F'd} the symmetrised density factors of a slice quartet, its energy is
//   E = sum_{bd} Gamma_bd (F b | F' d) = C(d/dX) f(X),   X = P - Q,  f = pref F_0(rho X^2),
// C a polynomial in the derivatives (Hermite expansion of the McMurchie-Davidson scheme,
// J. Comput. Phys. 26, 218 (1978); (r-A) = PA + u d/dP acting on the Gaussian at P, u = 1/(2
// zeta)).  The gradient needs E, dE/dP = -dE/dQ and the derivatives of E with respect to the
// displacements P - A, P - B, Q - C, Q - D, which C holds explicitly; the chain rule through
// P = (a A + b B)/zeta and K = exp(-mu |A-B|^2) then gives the four centres:
//   dE/dA = (a/zeta) dE/dP + g,  dE/dB = (b/zeta) dE/dP - g,
//   g = -2 mu (A-B) E - (b/zeta) dE/d(P-A) + (a/zeta) dE/d(P-B).
#pragma once
#include "boys.cuh"
#include "super.cuh"

// component d of the gradient of W at the derivative index (i, j, k)
B2_HD double b2gs_at(const double *W, int i, int j, int k) { return W[b2g_cidx(i, j, k)]; }

// a slice's data on one primitive pair, axes permuted so that a p function F lies along axis 0
struct B2gBraPrim {
  double kS, kP, u, FA, B[3];      // coefficients, 1/(2 zeta), (P - A)_F, P - B
};
// the ket primitive with the density factors contracted over its second shell, per bra function
// b = s, x, y, z:  gs_b = kS Gamma_bs + kP sum_d (Q - D)_d Gamma_bd;  g_bd = kP Gamma_bd
template <int NB, int NK>
struct B2gKet {
  double gs[NB ? 4 : 1], g[NB ? 4 : 1][3], v, FC;
};
// sums of one ket primitive over bra primitives, or of one evaluation
struct B2gOut {
  double E, dP[3], A, B[3], C, D[3];       // dE/d(P-A)_F, dE/d(P-B), dE/d(Q-C)_F', dE/d(Q-D)
};

// One primitive quartet.  BF: the bra's F is a p function (axis 0); KF: the ket's F' is s (-1)
// or the p function along axis KF; NB / NK: the second shell has p functions.
template <bool BF, int NB, int KF, int NK>
B2_HD void b2gs_quartet(const B2gBraPrim &b, const B2gKet<NB, NK> &q, const double *X, const double *f,
                        B2gOut &o) {
  constexpr int LH = (NB ? 1 : 0) + (NK ? 1 : 0);               // order of the second shells' part
  constexpr int L = 1 + LH + (BF ? 1 : 0) + (KF >= 0 ? 1 : 0);
  double R[b2g_ncart(L)];
  b2gs_rtensor<L>(X, f, R);
  // wK = (PA + u d_F) f, wB = (QC - v d_F') f, w = both
  constexpr int LW = 1 + LH;                                     // orders used of w
  double w[b2g_ncart(LW)], wB[b2g_ncart(LW)], wK[b2g_ncart(LW + (KF >= 0 ? 1 : 0))];
  if constexpr (BF) b2gs_shift<LW + (KF >= 0 ? 1 : 0), 0>(b.FA, b.u, R, wK);
  else b2gs_copy<LW + (KF >= 0 ? 1 : 0)>(R, wK);
  if constexpr (KF >= 0) {
    b2gs_shift<LW, KF>(q.FC, -q.v, wK, w);
    b2gs_shift<LW, KF>(q.FC, -q.v, R, wB);
  } else {
    b2gs_copy<LW>(wK, w);
    b2gs_copy<LW>(R, wB);
  }
  const double uP = b.u * b.kP;
  double H0, h[3] = {0, 0, 0}, qd[3] = {0, 0, 0}, M[6] = {0, 0, 0, 0, 0, 0};   // xx xy xz yy yz zz
  if constexpr (NB) {
    H0 = b.kS * q.gs[0] + b.kP * (b.B[0] * q.gs[1] + b.B[1] * q.gs[2] + b.B[2] * q.gs[3]);
#pragma unroll
    for (int d = 0; d < 3; ++d) h[d] = uP * q.gs[1 + d];
  } else {
    H0 = b.kS * q.gs[0];
  }
  if constexpr (NK) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if constexpr (NB)
        qd[d] = b.kS * q.g[0][d] + b.kP * (b.B[0] * q.g[1][d] + b.B[1] * q.g[2][d] + b.B[2] * q.g[3][d]);
      else
        qd[d] = b.kS * q.g[0][d];
      h[d] -= q.v * qd[d];
    }
    if constexpr (NB) {
      const double c = -uP * q.v;
      M[0] = c * q.g[1][0];
      M[1] = c * (q.g[1][1] + q.g[2][0]);
      M[2] = c * (q.g[1][2] + q.g[3][0]);
      M[3] = c * q.g[2][1];
      M[4] = c * (q.g[2][2] + q.g[3][1]);
      M[5] = c * q.g[3][2];
    }
  }
  // the operator H0 + h.d + M:dd applied to a field at derivative index (i, j, k)
  auto apply = [&](const double *W, int i, int j, int k) -> double {
    double e = H0 * b2gs_at(W, i, j, k);
    if constexpr (NB || NK)
      e += h[0] * b2gs_at(W, i + 1, j, k) + h[1] * b2gs_at(W, i, j + 1, k) + h[2] * b2gs_at(W, i, j, k + 1);
    if constexpr (NB && NK)
      e += M[0] * b2gs_at(W, i + 2, j, k) + M[1] * b2gs_at(W, i + 1, j + 1, k) + M[2] * b2gs_at(W, i + 1, j, k + 1) +
           M[3] * b2gs_at(W, i, j + 2, k) + M[4] * b2gs_at(W, i, j + 1, k + 1) + M[5] * b2gs_at(W, i, j, k + 2);
    return e;
  };
  // (r-P)_F (r-P)_b also meets at one point: u d_Fb; its ket part, and the bra part of the ket's
  auto braX = [&](const double *W, int i, int j, int k) -> double {     // u kP (gs_F - v g_F.d) W
    double e = q.gs[1] * b2gs_at(W, i, j, k);
    if constexpr (NK)
      e -= q.v * (q.g[1][0] * b2gs_at(W, i + 1, j, k) + q.g[1][1] * b2gs_at(W, i, j + 1, k) +
                  q.g[1][2] * b2gs_at(W, i, j, k + 1));
    return uP * e;
  };
  auto ketX = [&](const double *W, int i, int j, int k) -> double {     // v (q_F' + u kP g_.F'.d) W
    double e = qd[KF < 0 ? 0 : KF] * b2gs_at(W, i, j, k);
    if constexpr (NB)
      e += uP * (q.g[1][KF < 0 ? 0 : KF] * b2gs_at(W, i + 1, j, k) + q.g[2][KF < 0 ? 0 : KF] * b2gs_at(W, i, j + 1, k) +
                 q.g[3][KF < 0 ? 0 : KF] * b2gs_at(W, i, j, k + 1));
    return q.v * e;
  };
  double e4[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int i = m == 1, j = m == 2, k = m == 3;
    double e = apply(w, i, j, k);
    if constexpr (BF) e += braX(wB, i, j, k);
    if constexpr (KF >= 0) e += ketX(wK, i, j, k);
    if constexpr (BF && KF >= 0) e += uP * q.v * q.g[1][KF] * b2gs_at(R, i, j, k);
    e4[m] = e;
  }
  o.E = e4[0];
  o.dP[0] = e4[1]; o.dP[1] = e4[2]; o.dP[2] = e4[3];
  if constexpr (BF) {
    o.A = apply(wB, 0, 0, 0);
    if constexpr (KF >= 0) o.A += ketX(R, 0, 0, 0);
  }
  if constexpr (KF >= 0) {
    o.C = apply(wK, 0, 0, 0);
    if constexpr (BF) o.C += braX(R, 0, 0, 0);
  }
  if constexpr (NB) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double e = q.gs[1 + d] * w[0];
      if constexpr (NK) e -= q.v * (q.g[1 + d][0] * w[1] + q.g[1 + d][1] * w[2] + q.g[1 + d][2] * w[3]);
      if constexpr (KF >= 0) e += q.v * q.g[1 + d][KF] * wK[0];
      o.B[d] = b.kP * e;
    }
  }
  if constexpr (NK) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double e = qd[d] * w[0];
      if constexpr (NB) e += uP * (q.g[1][d] * w[1] + q.g[2][d] * w[2] + q.g[3][d] * w[3]);
      if constexpr (BF) e += uP * q.g[1][d] * wB[0];
      o.D[d] = e;
    }
  }
}

// the highest Boys order of a class
template <int TB, int TK> struct B2gsClass {
  static constexpr bool BF = TB == 2;
  static constexpr int NB = TB ? 1 : 0, NK = TK ? 1 : 0;
  static constexpr int L = 1 + NB + NK + (BF ? 1 : 0) + (TK == 2 ? 1 : 0);
};

// density factors of a slice quartet contracted over the ket's second shell.  D: the molecule's
// matrix (row-major, stride N); F / b: the bra's functions, F2 / d: the ket's; wt: the number of
// index orderings.  Gamma_bd = wt [D_Fb D_F'd / 2 - hyb/8 (D_Fd D_bF' + D_FF' D_bd)], zero where
// a shell lacks the function (AO index -1).
template <int NB, int NK>
B2_HD void b2gs_ket(const double *D, int N, double hyb, double wt, int F, const int *bi, int F2, const int *di,
                    double kS, double kP, const double *QD, B2gKet<NB, NK> &q) {
  const double h8 = 0.125 * hyb * wt, hw = 0.5 * wt;
  const bool ok = F >= 0 && F2 >= 0;
  const double DFF = ok ? D[F * N + F2] : 0.0;
  double DFd[NK ? 4 : 1], DF2d[NK ? 4 : 1];
#pragma unroll
  for (int d = 0; d < (NK ? 4 : 1); ++d) {
    DFd[d] = ok && di[d] >= 0 ? D[F * N + di[d]] : 0.0;
    DF2d[d] = ok && di[d] >= 0 ? D[F2 * N + di[d]] : 0.0;
  }
#pragma unroll
  for (int b = 0; b < (NB ? 4 : 1); ++b) {
    const bool bo = ok && bi[b] >= 0;
    const double DFb = bo ? hw * D[F * N + bi[b]] : 0.0, DbF2 = bo ? h8 * D[bi[b] * N + F2] : 0.0;
    double G[NK ? 4 : 1];
#pragma unroll
    for (int d = 0; d < (NK ? 4 : 1); ++d)
      G[d] = DFb * DF2d[d] - DbF2 * DFd[d] - (bo && di[d] >= 0 ? h8 * DFF * D[bi[b] * N + di[d]] : 0.0);
    double s = kS * G[0];
    if constexpr (NK) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        q.g[b][d] = kP * G[1 + d];
        s += QD[d] * q.g[b][d];
      }
    }
    q.gs[b] = s;
  }
}

// a bra slice's primitive pair, axes permuted by the slice's axis
struct __align__(16) B2gBraRec {
  B2gBraPrim b;
  double P[3], z, ra, mu2, pad;
};
// AB: A - B in the permuted axes; f: axis of F (0 for types 0 and 1)
B2_HD void b2gs_bra(const B2gPrim &r, int type, int f, const double *AB, B2gBraRec &o) {
  o.b.kS = type == 2 ? r.kps : r.kss;
  o.b.kP = type == 2 ? r.kpp : r.ksp;
  o.b.u = r.u;
  o.b.FA = (r.ra - 1.0) * AB[0];
  for (int k = 0; k < 3; ++k) {
    o.b.B[k] = r.ra * AB[k];
    o.P[k] = r.P[(f + k) % 3];
  }
  o.z = r.z;
  o.ra = r.ra;
  o.mu2 = r.mu2;
  o.pad = 0.0;
}

B2_HD double b2gs_rsqrt(double x) {
#ifdef __CUDA_ARCH__
  return rsqrt(x);
#else
  return 1.0 / sqrt(x);
#endif
}

// one primitive quartet of the slices: Boys values, derivative tensor, energy and derivatives
template <int TB, int TK, int KF>
B2_HD void b2gs_eval(const B2gBraRec &r, const B2gKet<B2gsClass<TB, TK>::NB, B2gsClass<TB, TK>::NK> &q,
                     const double *Q, double eta, const double *btab, B2gOut &o) {
  using C = B2gsClass<TB, TK>;
  constexpr int L = C::L;
  const double X[3] = {r.P[0] - Q[0], r.P[1] - Q[1], r.P[2] - Q[2]};
  const double rs = b2gs_rsqrt(r.z + eta), rho = r.z * eta * rs * rs;
  double F[L + 1], f[L + 1];
  b2_boys<double, L, double>(rho * (X[0] * X[0] + X[1] * X[1] + X[2] * X[2]), btab, F);
  double s = rs;
#pragma unroll
  for (int n = 0; n <= L; ++n) { f[n] = s * F[n]; s *= -2.0 * rho; }
  b2gs_quartet<C::BF, C::NB, KF, C::NK>(r.b, q, X, f, o);
}

// the bra's centres: gA, gB += the quartet's derivatives (permuted axes)
template <int TB>
B2_HD void b2gs_add_bra(const B2gBraRec &r, const double *AB, const B2gOut &o, double *gA, double *gB) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double g = -r.mu2 * AB[k] * o.E;
    if (TB) g += r.ra * o.B[k];
    if (TB == 2 && k == 0) g += (r.ra - 1.0) * o.A;
    gA[k] += r.ra * o.dP[k] + g;
    gB[k] += (1.0 - r.ra) * o.dP[k] - g;
  }
}
// the ket primitive's sums over bra primitives (E, dP, C, D) to its centres
template <int TK, int KF>
B2_HD void b2gs_add_ket(double ra, double mu2, const double *CD, const B2gOut &s, double *gC, double *gD) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double g = -mu2 * CD[k] * s.E;
    if (TK) g += ra * s.D[k];
    if (TK == 2 && k == KF) g += (ra - 1.0) * s.C;
    gC[k] += g - ra * s.dP[k];
    gD[k] -= g + (1.0 - ra) * s.dP[k];
  }
}

// a bra primitive pair against a point charge at C: b2gs_eval in the limit eta -> infinity,
// f_n = (-2 zeta)^n F_n(zeta |P - C|^2); the charge and constants are in q.gs
template <int TB>
B2_HD void b2gs_eval_point(const B2gBraRec &r, const B2gKet<B2gsClass<TB, 0>::NB, 0> &q, const double *C,
                           const double *btab, B2gOut &o) {
  constexpr int L = B2gsClass<TB, 0>::L;
  const double X[3] = {r.P[0] - C[0], r.P[1] - C[1], r.P[2] - C[2]};
  double F[L + 1], f[L + 1];
  b2_boys<double, L, double>(r.z * (X[0] * X[0] + X[1] * X[1] + X[2] * X[2]), btab, F);
  double s = 1.0;
#pragma unroll
  for (int n = 0; n <= L; ++n) { f[n] = s * F[n]; s *= -2.0 * r.z; }
  b2gs_quartet<TB == 2, B2gsClass<TB, 0>::NB, -1, 0>(r.b, q, X, f, o);
}

// overlap and kinetic energy of one primitive pair of a slice, derivative with respect to the
// first centre (the second's is its negative).  With the slice's second shell contracted with
// the density factors, l0 + l.(r - P) (l0 = kS g_s + kP g.PB, l = kP g), and the first function
// sa + (r - P)_F:
//   <1> = sa l0 + u l_F,   <r_B^2> = sa l0 PB^2 + u (l_F PB^2 + 2 l0 PB_F + 2 sa l.PB + 3 sa l0) + 5 u^2 l_F,
//   T = -1/2 (4 b^2 <r_B^2> - 2 b (3 <1>_s + 5 <1>_p))  (Laplacian on the second function).
// dg: factors of T, wg: factors of S.
template <int TB>
B2_HD void b2gs_st(const B2gBraRec &r, const double *dg, const double *wg, const double *AB, double *gA) {
  constexpr bool BF = TB == 2;
  constexpr int NB = TB ? 1 : 0;
  const double be = (1.0 - r.ra) * r.z, u = r.b.u, sa = BF ? r.b.FA : 1.0;
  // (pi / zeta)^(3/2) over the pair constant sqrt(2) pi^(5/4) / zeta
  const double c3 = 0.94139626377671481 / sqrt(r.z);
  const double *PB = r.b.B;
  double l0 = r.b.kS * dg[0], w0 = r.b.kS * wg[0], l[3] = {0, 0, 0}, wl[3] = {0, 0, 0};
  const double ls = l0;                                   // the second shell's s part
  double PB2 = 0, lPB = 0;
  for (int k = 0; k < 3; ++k) PB2 += PB[k] * PB[k];
  if (NB)
    for (int k = 0; k < 3; ++k) {
      l[k] = r.b.kP * dg[k + (NB ? 1 : 0)];
      wl[k] = r.b.kP * wg[k + (NB ? 1 : 0)];
      l0 += l[k] * PB[k];
      w0 += wl[k] * PB[k];
      lPB += l[k] * PB[k];
    }
  const double b2 = -2.0 * be * be;
  const double lF = BF ? l[0] : 0.0, wF = BF ? wl[0] : 0.0, pF = BF ? PB[0] : 0.0;
  const double r2 = sa * l0 * PB2 + u * (lF * PB2 + 2.0 * l0 * pF + 2.0 * sa * lPB + 3.0 * sa * l0) + 5.0 * u * u * lF;
  const double E = b2 * r2 + 5.0 * be * (sa * l0 + u * lF) - 2.0 * be * sa * ls + sa * w0 + u * wF;
  double EA = 0;
  if (BF) EA = b2 * (l0 * PB2 + u * (2.0 * lPB + 3.0 * l0)) + 5.0 * be * l0 - 2.0 * be * ls + w0;
  for (int k = 0; k < 3; ++k) {
    const double r2B = sa * l[k] * PB2 + 2.0 * sa * l0 * PB[k] +
                       u * (2.0 * lF * PB[k] + 2.0 * l[k] * pF + (BF && k == 0 ? 2.0 * l0 : 0.0) + 5.0 * sa * l[k]);
    const double EB = b2 * r2B + 5.0 * be * sa * l[k] + sa * wl[k];
    double g = -r.mu2 * AB[k] * E + r.ra * EB;
    if (BF && k == 0) g += (r.ra - 1.0) * EA;
    gA[k] = c3 * g;
  }
}
