// Super shells and their pairs: the basis as the integral and gradient kernels see it.
//
// A super shell is an s shell, or an s and a p shell of one atom with the same exponents
// (STO-3G's 2s / 2p), or a p shell alone.  All functions of a pair of super shells share the
// pair's primitives, so one Boys evaluation and one derivative tensor serve up to 256 integrals.
#pragma once
#include "common.cuh"
#include "plan_host.hpp"

// Cartesian components of order l: first index of order l, number of components of 0..l, index
B2_HD constexpr int b2g_cstart(int l) { return l * (l + 1) * (l + 2) / 6; }
B2_HD constexpr int b2g_ncart(int l) { return (l + 1) * (l + 2) * (l + 3) / 6; }   // components of 0..l
// index of the Cartesian (x, y, z) among all components of l = 0..3 (order within a shell:
// x descending, then y descending)
B2_HD constexpr int b2g_cidx(int x, int y, int z) {
  const int l = x + y + z;
  return b2g_cstart(l) + (l - x) * (l - x + 1) / 2 + z;
}

struct B2gSuper {                  // super shell: centre, exponents, s and p coefficients
  double R[3], ex[B2_MAXPRIM], cs[B2_MAXPRIM], cp[B2_MAXPRIM];
  int nprim, atom, ao_s, ao_p;     // first AO of the s / p part (-1: absent)
};

// primitive pair of two super shells: a/zeta, zeta, P, 2 mu, u = 1/(2 zeta) and the
// coefficient products K c c' sqrt(2) pi^(5/4) / zeta (so that the quartet's prefactor is
// K_bra K_ket / sqrt(zeta + eta))
struct __align__(16) B2gPrim {
  double ra, z, P[3], mu2, u, kss, ksp, kps, kpp, pad;
};

// primitive pair (p, q); returns the size that screening looks at: the largest |c c' K| over the
// pair's functions (K = exp(-mu R^2))
B2_HD double b2gs_prim(const B2gSuper &a, const B2gSuper &b, int p, int q, B2gPrim &o) {
  const double al = a.ex[p], be = b.ex[q], z = al + be, iz = 1.0 / z, mu = al * be * iz;
  double R2 = 0;
  for (int d = 0; d < 3; ++d) {
    R2 += (a.R[d] - b.R[d]) * (a.R[d] - b.R[d]);
    o.P[d] = (al * a.R[d] + be * b.R[d]) * iz;
  }
  const double K = exp(-mu * R2);
  const double ca = fmax(fabs(a.cs[p]), fabs(a.cp[p])), cb = fmax(fabs(b.cs[q]), fabs(b.cp[q]));
  const double k0 = 5.914967172795613 * iz * K;              // sqrt(2) pi^(5/4)
  o.ra = al * iz;
  o.z = z;
  o.mu2 = 2.0 * mu;
  o.u = 0.5 * iz;
  o.kss = k0 * a.cs[p] * b.cs[q];
  o.ksp = k0 * a.cs[p] * b.cp[q];
  o.kps = k0 * a.cp[p] * b.cs[q];
  o.kpp = k0 * a.cp[p] * b.cp[q];
  o.pad = 0.0;
  return K * ca * cb;
}

// float32 copy for the float32 integral kernels, with P - A and P - B
struct __align__(16) B2gPrim32 {
  float z, P[3], u, kss, ksp, kps, kpp, A[3], B[3], pad;
};
B2_HD void b2gs_prim32(const B2gPrim &r, const double *AB, B2gPrim32 &o) {
  o.z = (float)r.z;
  o.u = (float)r.u;
  o.kss = (float)r.kss; o.ksp = (float)r.ksp; o.kps = (float)r.kps; o.kpp = (float)r.kpp;
  for (int d = 0; d < 3; ++d) {
    o.P[d] = (float)r.P[d];
    o.A[d] = (float)((r.ra - 1.0) * AB[d]);
    o.B[d] = (float)(r.ra * AB[d]);
  }
  o.pad = 0.f;
}

// Screening of a pair's primitive pairs (surviving ones packed first):
//   gradient  |c c' K| >= 1e-20;
//   integrals |c c' K| sqrt(2) pi^(5/4) / zeta >= 1e-15 (float64) or 1e-11 (float32): what is
//   dropped contributes less than 1e-12 / 1e-8 to any integral, below the accuracy of each form
//   (the reference drops primitive pairs below exp(-60), libcint's expcutoff).
// pr64: the float64 integrals' n.y first, then the gradient's further ones up to n.z; pr32: n.x.
struct B2gCount { unsigned char x, y, z, w; };
B2_HD B2gCount b2gs_pair_prims(const B2gSuper &a, const B2gSuper &b, B2gPrim *pr64, B2gPrim32 *pr32) {
  B2gCount n = {0, 0, 0, 0};
  const double AB[3] = {a.R[0] - b.R[0], a.R[1] - b.R[1], a.R[2] - b.R[2]};
  for (int pass = 0; pass < 2; ++pass)
    for (int p = 0; p < a.nprim; ++p)
      for (int q = 0; q < b.nprim; ++q) {
        B2gPrim r;
        const double k = b2gs_prim(a, b, p, q, r), s = k * (2.0 * 5.914967172795613) * r.u;
        if (pass == 0 && s >= B2_PP_SCREEN64) {
          pr64[n.y++] = r;
          n.z = n.y;
          if (s >= B2_PP_SCREEN32) b2gs_prim32(r, AB, pr32[n.x++]);
        }
        if (pass == 1 && !(s >= B2_PP_SCREEN64) && k >= 1e-20) pr64[n.z++] = r;
      }
  return n;
}

// super shells of one molecule from its shells: s shells without a partner first, then the p
// shells with their s partner (same atom, same exponents; the first unused one).  Returns the
// number of s-only ones, *ntot the total.
B2_HD int b2gs_supers(const B2Shell *S, int nbas, B2gSuper *out, int *ntot) {
  unsigned long long taken[2] = {0, 0};          // s shells merged into a p shell (nbas <= 72)
  int n = 0;
  for (int pass = 0; pass < 2; ++pass)
    for (int s = 0; s < nbas; ++s) {
      const B2Shell &a = S[s];
      if (pass == 0) {
        // s-only: no p shell takes it; the merge itself is found from the p side below
        if (a.l != 1) continue;
        for (int t = 0; t < nbas; ++t) {
          const B2Shell &b = S[t];
          if (b.l != 0 || b.atom != a.atom || b.nprim != a.nprim || (taken[t >> 6] >> (t & 63) & 1)) continue;
          bool same = true;
          for (int k = 0; k < a.nprim; ++k) same = same && b.exp[k] == a.exp[k];
          if (same) { taken[t >> 6] |= 1ull << (t & 63); break; }
        }
      } else if (a.l == 0 && !(taken[s >> 6] >> (s & 63) & 1)) {
        B2gSuper &o = out[n++];
        for (int d = 0; d < 3; ++d) o.R[d] = a.R[d];
        for (int k = 0; k < B2_MAXPRIM; ++k) { o.ex[k] = a.exp[k]; o.cs[k] = a.coef[k]; o.cp[k] = 0.0; }
        o.nprim = a.nprim; o.atom = a.atom; o.ao_s = a.ao0; o.ao_p = -1;
      }
    }
  const int ns = n;
  taken[0] = taken[1] = 0;
  for (int s = 0; s < nbas; ++s) {
    const B2Shell &a = S[s];
    if (a.l != 1) continue;
    B2gSuper &o = out[n++];
    for (int d = 0; d < 3; ++d) o.R[d] = a.R[d];
    for (int k = 0; k < B2_MAXPRIM; ++k) { o.ex[k] = a.exp[k]; o.cp[k] = a.coef[k]; o.cs[k] = 0.0; }
    o.nprim = a.nprim; o.atom = a.atom; o.ao_s = -1; o.ao_p = a.ao0;
    for (int t = 0; t < nbas; ++t) {             // same search order as above: the same partners
      const B2Shell &b = S[t];
      if (b.l != 0 || b.atom != a.atom || b.nprim != a.nprim || (taken[t >> 6] >> (t & 63) & 1)) continue;
      bool same = true;
      for (int k = 0; k < a.nprim; ++k) same = same && b.exp[k] == a.exp[k];
      if (same) {
        taken[t >> 6] |= 1ull << (t & 63);
        for (int k = 0; k < B2_MAXPRIM; ++k) o.cs[k] = b.coef[k];
        o.ao_s = b.ao0;
        break;
      }
    }
  }
  *ntot = n;
  return ns;
}

// pair storage of a molecule with ns s-only and np sp super shells (s-only first):
// [s s] I >= J, then [s sp] (s index major), then [sp sp] I >= J
B2_HD int b2gs_npair(int ns, int np) { return (ns + np) * (ns + np + 1) / 2; }
B2_HD void b2gs_pair(int ns, int np, int idx, int &A, int &B) {
  const int nss = ns * (ns + 1) / 2;
  if (idx < nss) {
    A = (int)b2_untri(idx);
    B = idx - (int)b2_tri(A);
    return;
  }
  idx -= nss;
  if (idx < ns * np) {
    A = idx / np;
    B = ns + idx - (idx / np) * np;
    return;
  }
  idx -= ns * np;
  const int i = (int)b2_untri(idx);
  A = ns + i;
  B = ns + idx - (int)b2_tri(i);
}
// slices of a type, and a slice's pair and axis (type 2: axis minor, so that kets of one pair
// are neighbours); type 2 as a ket is counted per pair (its three axes run together)
B2_HD int b2gs_nslice(int ns, int np, int type) {
  return type == 0 ? ns * (ns + 1) / 2 : type == 1 ? ns * np + np * (np + 1) / 2 : 3 * (np * (np + 1) / 2);
}
B2_HD int b2gs_nket(int ns, int np, int type) {
  return type == 2 ? np * (np + 1) / 2 : b2gs_nslice(ns, np, type);
}
B2_HD int b2gs_ket_pair(int ns, int np, int type, int k) {
  const int nss = ns * (ns + 1) / 2;
  return type == 0 ? k : type == 1 ? nss + k : nss + ns * np + k;
}


struct B2gsMol {                   // a molecule's super shells
  int ns, np, su_off, pad;         // s-only and sp super shells, first super shell
  long long pr_off;                // first super-shell pair
};

// derivative tensor R_{ijk} = d^i/dX^i d^j/dY^j d^k/dZ^k f, i + j + k <= L, at b2g_cidx(i, j, k),
// from f_n = (-2 rho)^n pref F_n: R^n_{t+1} = X R^{n+1}_t + t R^{n+1}_{t-1}, in place from n = L
template <int L, typename T>
B2_HD void b2gs_rtensor(const T *X, const T *f, T *R) {
  R[0] = f[L];
#pragma unroll
  for (int n = L - 1; n >= 0; --n) {
#pragma unroll
    for (int l = L - n; l >= 1; --l)
#pragma unroll
      for (int i = l; i >= 0; --i)
#pragma unroll
        for (int j = l - i; j >= 0; --j) {
          const int k = l - i - j;
          T r;
          if (i == 1 || (i > 1 && j != 1 && k != 1)) {
            r = X[0] * R[b2g_cidx(i - 1, j, k)];
            if (i > 1) r += (T)(i - 1) * R[b2g_cidx(i - 2, j, k)];
          } else if (j == 1 || (j > 1 && k != 1)) {
            r = X[1] * R[b2g_cidx(i, j - 1, k)];
            if (j > 1) r += (T)(j - 1) * R[b2g_cidx(i, j - 2, k)];
          } else {
            r = X[2] * R[b2g_cidx(i, j, k - 1)];
            if (k > 1) r += (T)(k - 1) * R[b2g_cidx(i, j, k - 2)];
          }
          R[b2g_cidx(i, j, k)] = r;
        }
    R[0] = f[n];
  }
}

// W = c0 R + c1 d_axis R up to order L
template <int L, int AX, typename T>
B2_HD void b2gs_shift(T c0, T c1, const T *R, T *W) {
#pragma unroll
  for (int l = 0; l <= L; ++l)
#pragma unroll
    for (int i = l; i >= 0; --i)
#pragma unroll
      for (int j = l - i; j >= 0; --j) {
        const int k = l - i - j;
        W[b2g_cidx(i, j, k)] = c0 * R[b2g_cidx(i, j, k)] + c1 * R[b2g_cidx(i + (AX == 0), j + (AX == 1), k + (AX == 2))];
      }
}
template <int L, typename T>
B2_HD void b2gs_copy(const T *R, T *W) {
#pragma unroll
  for (int t = 0; t < b2g_ncart(L); ++t) W[t] = R[t];
}
