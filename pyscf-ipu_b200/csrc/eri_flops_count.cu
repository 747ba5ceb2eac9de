// Per-class arithmetic of one primitive quartet of the float32 ERI kernels, counted on the host
// by running the kernels' own code (eri_su.cuh, B2Es<T,...>::quartet with its Boys evaluation and
// B2Es<T,...>::ket) on a counting number type.  Writes eri_flops.h, which bench.py's ERI roofline uses:
//
//   nvcc -std=c++17 -I. -I../../include -x cu eri_flops_count.cu -o /tmp/eri_flops && /tmp/eri_flops > eri_flops.h
//
// Counting rules: +, -, * and / count one flop each (a fused multiply-add is two); sqrt, exp and
// the reciprocal square root count one each (special-function unit); operations whose operands
// are compile-time constants of the template (the zeros and ones the class's angular momenta fix)
// are folded, as the compiler folds them, and not counted; comparisons and index arithmetic are
// not counted.  The Boys function is counted on its table branch (T < 40), the common one, and
// F_0 alone on its error-function branch (erf counts as one special function).
#include <cstdio>
#include <cmath>
#include "eri_su.cuh"

static long long g_flops = 0, g_special = 0;

struct CF {                   // value (for the branches) + "is a folded constant" flag
  double v = 0;
  bool k = false;
  CF() = default;
  CF(int x) : v(x), k(true) {}
  CF(double x) : v(x), k(true) {}
  CF(float x) : v(x), k(true) {}
  static CF var(double x) { CF c; c.v = x; c.k = false; return c; }
  explicit operator int() const { return (int)v; }
};
static CF op(double v, bool both_const) {
  CF c;
  c.v = v;
  c.k = both_const;
  if (!both_const) ++g_flops;
  return c;
}
inline CF operator+(CF a, CF b) {
  if (a.k && a.v == 0) return b;
  if (b.k && b.v == 0) return a;
  return op(a.v + b.v, a.k && b.k);
}
inline CF operator-(CF a, CF b) {
  if (b.k && b.v == 0) return a;
  return op(a.v - b.v, a.k && b.k);
}
inline CF operator-(CF a) { CF c = a; c.v = -a.v; return c; }     // sign flips fold into the next op
inline CF operator*(CF a, CF b) {
  if ((a.k && a.v == 0) || (b.k && b.v == 0)) return CF(0);
  if (a.k && a.v == 1) return b;
  if (b.k && b.v == 1) return a;
  return op(a.v * b.v, a.k && b.k);
}
inline CF operator/(CF a, CF b) { return op(a.v / b.v, a.k && b.k); }
inline CF &operator+=(CF &a, CF b) { a = a + b; return a; }
inline CF &operator-=(CF &a, CF b) { a = a - b; return a; }
inline CF &operator*=(CF &a, CF b) { a = a * b; return a; }
inline bool operator<(CF a, CF b) { return a.v < b.v; }
inline bool operator>(CF a, CF b) { return a.v > b.v; }
inline bool operator==(CF a, CF b) { return a.v == b.v; }
inline bool operator!=(CF a, CF b) { return a.v != b.v; }
inline CF sqrt(CF a) { if (!a.k) ++g_special; CF c = a; c.v = std::sqrt(a.v); return c; }
inline CF exp(CF a) { if (!a.k) ++g_special; CF c = a; c.v = std::exp(a.v); return c; }
inline CF erf(CF a) { if (!a.k) ++g_special; CF c = a; c.v = std::erf(a.v); return c; }

// the float32 kernels' Taylor length of the Boys table branch, and their error-function F_0
template <> struct B2BoysTerms<CF> { static constexpr int n = B2BoysTerms<float>::n; };
template <> struct B2BoysErfF0<CF> { static constexpr bool value = B2BoysErfF0<float>::value; };
template <> struct B2BoysOddLow<CF> { static constexpr bool value = B2BoysOddLow<float>::value; };

template <int TB, int TK>
static void count(long long &fl, long long &sp, long long &kf) {
  using S = B2Es<CF, TB, TK>;
  static CF tab[B2_BOYS_NT * B2_BOYS_NM];
  static bool filled = false;
  if (!filled) {
    static double t64[B2_BOYS_NT * B2_BOYS_NM];
    b2_boys_fill_table(t64);
    for (int i = 0; i < B2_BOYS_NT * B2_BOYS_NM; ++i) tab[i] = CF::var(t64[i]);
    filled = true;
  }
  B2EriBra<CF> A;
  B2EriKet<CF> B;
  const double a[12] = {1.3, 0.4, 0.2, -0.1, 0.3, 0.25, -0.2, 0.1, 0.9, 0.35, 0.7, 0.6};
  CF *pa = &A.kS, *pb = &B.z;                  // the structs are runs of T fields
  for (int i = 0; i < (int)(sizeof(A) / sizeof(CF)); ++i) pa[i] = CF::var(a[i % 12] + 0.01 * i);
  for (int i = 0; i < (int)(sizeof(B) / sizeof(CF)); ++i) pb[i] = CF::var(a[(i + 5) % 12] + 0.02 * i);
  CF phi[S::NB][S::NP], out[S::NK];
  for (int b = 0; b < S::NB; ++b)
    for (int k = 0; k < S::NP; ++k) phi[b][k] = CF::var(0.0);
  g_flops = g_special = 0;
  S::quartet(A, B, tab, phi);
  fl = g_flops;
  sp = g_special;
  g_flops = 0;
  for (int b = 0; b < S::NB; ++b) S::ket(B, phi[b], out);
  kf = g_flops;
}

int main() {
  long long f[6], s[6], k[6];
  count<0, 0>(f[0], s[0], k[0]);
  count<0, 1>(f[1], s[1], k[1]);
  count<1, 1>(f[2], s[2], k[2]);
  count<0, 2>(f[3], s[3], k[3]);
  count<1, 2>(f[4], s[4], k[4]);
  count<2, 2>(f[5], s[5], k[5]);
  printf("// Generated by eri_flops_count.cu from eri_su.cuh: arithmetic of one primitive quartet of the\n");
  printf("// float32 ERI kernels per class (bra slice type, ket pair type) = (0,0) (0,1) (1,1) (0,2) (1,2) (2,2)\n");
  printf("// (flops: +, -, *, /; special: sqrt, exp, erf, reciprocal square root), and of the ket's polynomial\n");
  printf("// per bra slice and ket primitive, constants folded as the compiler folds them.\n");
  printf("#pragma once\n");
  auto row = [](const char *name, const long long *v) {
    printf("static const int %s[6] = {", name);
    for (int g = 0; g < 6; ++g) printf("%lld%s", v[g], g < 5 ? ", " : "};\n");
  };
  row("B2_ERI_FLOPS", f);
  row("B2_ERI_SPECIAL", s);
  row("B2_ERI_KET_FLOPS", k);
  return 0;
}
