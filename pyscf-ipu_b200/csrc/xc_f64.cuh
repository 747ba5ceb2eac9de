// Float64 exchange-correlation tiles: the phases that the XC evaluation (xc_direct.cu) and its
// nuclear gradient (grad.cu) share.  A CTA of 8 warps works on tiles of 32 points (lane = point
// wherever work is per point) of one molecule whose orbitals fill the bucket N <= 16 Q.
//
// Orbital planes live in shared memory point-contiguous, sA[plane][orbital][36]; the strides 36
// and 16 Q + 4 (4 modulo 16 doubles) keep every MMA fragment load free of bank conflicts.
// Products run over the molecule's orbitals rounded up to 8, not the bucket's 16 Q.
#pragma once
#include "device_plan.cuh"
#include "dmma.cuh"
#include "xc_math.cuh"

#define B2_XF_LDP 36
template <int Q> struct B2Xf {
  static constexpr int NB = 16 * Q, LDD = NB + 4, PL = NB * B2_XF_LDP, NX = (2 * Q + 3) / 4;
  // D, four planes, partial densities of four warp pairs, three functional parts
  static constexpr size_t SMEM = sizeof(double) * (NB * LDD + 4 * PL + 16 * 32 + 9 * 32);
};
// CTAs per SM that shared memory allows (116 / 82 / 53 / 26 KB for Q = 4 / 3 / 2 / 1)
#define B2_XF_CTAS(Q) ((Q) <= 2 ? 4 : ((Q) <= 4 ? 2 : 1))

__device__ __forceinline__ int b2_xf_find(const long long *off, int n, long long x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// AO values and gradients of the tile's points into the four planes; warp = super shell, so a
// shell's s and p functions share their exponentials and nothing diverges.  on: the lane's point
// exists (others get zeros)
template <int PL>
__device__ __forceinline__ void b2_xf_ao(const B2gSuper *__restrict__ su, int nsu, bool on, double px, double py,
                                         double pz, double *sA) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int s = w; s < nsu; s += 8) {
    const B2gSuper &S = su[s];
    const double dx = px - S.R[0], dy = py - S.R[1], dz = pz - S.R[2], r2 = dx * dx + dy * dy + dz * dz;
    double sa = 0, sb = 0, pa = 0, pb = 0;            // sum c e, sum -2 a c e of the s and p parts
    for (int k = 0; k < S.nprim; ++k) {
      const double al = S.ex[k], ax = al * r2;
      if (!on || ax > 60.0) continue;
      const double ev = exp(-ax), es = S.cs[k] * ev, ep = S.cp[k] * ev;
      sa += es;
      sb += -2.0 * al * es;
      pa += ep;
      pb += -2.0 * al * ep;
    }
    if (S.ao_s >= 0) {
      double *o = sA + S.ao_s * B2_XF_LDP + lane;
      o[0] = sa;
      o[PL] = sb * dx;
      o[2 * PL] = sb * dy;
      o[3 * PL] = sb * dz;
    }
    if (S.ao_p >= 0) {
      double *o = sA + S.ao_p * B2_XF_LDP + lane;
      const double dd[3] = {dx, dy, dz};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        o[c * B2_XF_LDP] = dd[c] * pa;
#pragma unroll
        for (int k = 0; k < 3; ++k) o[(1 + k) * PL + c * B2_XF_LDP] = (c == k ? pa : 0.0) + dd[c] * dd[k] * pb;
      }
    }
  }
}

// x = P^T M for the plane P (rows = points of this warp's half, columns 8 j, j = (w >> 1) + 4 i)
template <int Q>
__device__ __forceinline__ void b2_xf_mm(const double *P, const double *sD, int n8, double (&x)[B2Xf<Q>::NX][4]) {
  constexpr int LDD = B2Xf<Q>::LDD;
  const int w = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
  const int r0 = 16 * (w & 1), j0 = w >> 1;
#pragma unroll
  for (int i = 0; i < B2Xf<Q>::NX; ++i) x[i][0] = x[i][1] = x[i][2] = x[i][3] = 0.0;
  for (int k0 = 0; k0 < 8 * n8; k0 += 8) {
    double a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = P[(k0 + t + 4 * (i >> 1)) * B2_XF_LDP + r0 + g + 8 * (i & 1)];
#pragma unroll
    for (int i = 0; i < B2Xf<Q>::NX; ++i) {
      const int j = j0 + 4 * i;
      if (j < n8) {
        const double b[2] = {sD[(k0 + t) * LDD + 8 * j + g], sD[(k0 + t + 4) * LDD + 8 * j + g]};
        b2_dmma(x[i], a, b);
      }
    }
  }
}

// partial rho_c = sum_n x AO_c of this warp's columns into sR[warp pair][c][point]
template <int Q>
__device__ __forceinline__ void b2_xf_rho(const double *sA, int n8, const double (&x)[B2Xf<Q>::NX][4], double *sR) {
  constexpr int PL = B2Xf<Q>::PL;
  const int w = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
  const int r0 = 16 * (w & 1), j0 = w >> 1;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    double s0 = 0, s1 = 0;
#pragma unroll
    for (int i = 0; i < B2Xf<Q>::NX; ++i) {
      const int j = j0 + 4 * i;
      if (j < n8) {
        const double *o = sA + c * PL + (8 * j + 2 * t) * B2_XF_LDP + r0 + g;
        s0 += x[i][0] * o[0] + x[i][1] * o[B2_XF_LDP];
        s1 += x[i][2] * o[8] + x[i][3] * o[B2_XF_LDP + 8];
      }
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (t == 0) {
      sR[(j0 * 4 + c) * 32 + r0 + g] = s0;
      sR[(j0 * 4 + c) * 32 + r0 + g + 8] = s1;
    }
  }
}

// rho of the lane's point (every warp) and B3LYP: Slater + B88, VWN and LYP on three warps, one
// point per lane; two CTA barriers (partial densities in, parts out)
struct B2XfPoint { double rho[4], exc, vrho, vgamma; };
__device__ __forceinline__ void b2_xf_func(const double *sR, double *sF, B2XfPoint &o) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 4; ++c)
    o.rho[c] = (sR[c * 32 + lane] + sR[(4 + c) * 32 + lane]) + (sR[(8 + c) * 32 + lane] + sR[(12 + c) * 32 + lane]);
  if (w < 3) {
    const B2XcPoint<double> p = w == 0   ? b2_b3lyp_x<double>(o.rho[0], o.rho[1], o.rho[2], o.rho[3])
                                : w == 1 ? b2_b3lyp_vwn<double>(o.rho[0], o.rho[1], o.rho[2], o.rho[3])
                                         : b2_b3lyp_lyp<double>(o.rho[0], o.rho[1], o.rho[2], o.rho[3]);
    sF[(3 * w) * 32 + lane] = p.exc;
    sF[(3 * w + 1) * 32 + lane] = p.vrho;
    sF[(3 * w + 2) * 32 + lane] = p.vgamma;
  }
  __syncthreads();
  o.exc = sF[lane] + sF[3 * 32 + lane] + sF[6 * 32 + lane];
  o.vrho = sF[32 + lane] + sF[4 * 32 + lane] + sF[7 * 32 + lane];
  o.vgamma = sF[2 * 32 + lane] + sF[5 * 32 + lane] + sF[8 * 32 + lane];
}
