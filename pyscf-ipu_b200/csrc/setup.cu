// Per-molecule setup on the device (sm_100a): one-electron matrices, Becke grid, guess,
// nuclear repulsion.  These replace the host PySCF calls of the reference
// (int1e_ovlp/kin/nuc dft.py:225-227, Grids.build dft.py:214-216 / build_grid.py:109-135,
// minao dft.py:223, energy_nuc dft.py:202) and follow the same formulas as the package's
// host versions (b200dft/int1e.py, b200dft/grids.py, b200dft/guess.py), so the device
// setup reproduces the host setup to rounding.
#include <algorithm>
#include <vector>
#include "device_plan.cuh"
#include "devmem.cuh"
#include "setup.cuh"

// ------------------------------------------------------------------ one-electron matrices
// Every s/p primitive is d.(r-P) + s times the Gaussian product at P (d = 0, s = 1 for s):
//   overlap  <fa fb> = sa sb + (da.db) u,                           u = 1/(2 zeta)
//   r_B^2    <fa fb |r-B|^2> = sa sb |PB|^2 + u[(da.db)|PB|^2 + 2 sb da.PB + 2 sa db.PB + 3 sa sb]
//                              + 5 u^2 (da.db)
//   kinetic  T = -1/2 [4 b^2 <r_B^2> - 2 b (3 + 2 l_b) <1>]
//   nuclear  V = sum_C -Z_C (2 pi / zeta) K [E0 f0 + u (sb Xa + sa Xb) f1 + u^2 (da.db f1 + Xa Xb f2)]
__device__ __forceinline__ int b2_find_ll(const long long *off, int lo, int hi, long long x) {
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// One warp per super-shell pair (super.cuh; primitives screened at 1e-20), all of the pair's 1, 4 or
// 16 components: overlap and kinetic energy with a primitive per lane, nuclear attraction with the
// lanes over (nucleus, primitive), one Boys evaluation for every component, and the sums over lanes
// by a transposing butterfly that leaves component c on lane c.  Pairs of one type are neighbours, so
// the warps of a CTA run the same code.  The Boys table sits in shared memory (its rows are gathered
// at random); CTAs stay resident and stride over chunks of consecutive pairs.
// Bound by FP64 latency at 16 warps per SM.  1500 molecules: 2.45 ms with one AO pair per thread
// (own Boys evaluations and exponentials, one CTA per molecule), 0.83 ms now.

// v[0..NC) summed over the warp, component c on lanes c, c + NC, ...
template <int NC>
__device__ __forceinline__ double b2_i1_sum(double (&v)[NC], int lane) {
#pragma unroll
  for (int h = NC / 2, o = 1; h >= 1; h >>= 1, o <<= 1) {
    // lanes differing in bit o: one keeps the even components, the other the odd ones
    const bool odd = lane & o;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const double keep = odd ? v[2 * k + 1] : v[2 * k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, odd ? v[2 * k] : v[2 * k + 1], o);
    }
  }
#pragma unroll
  for (int o = NC; o < 32; o <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// TA / TB: the first / second shell has p functions (component a * (TB ? 4 : 1) + b; 0 is s)
template <bool TA, bool TB>
__device__ __forceinline__ void b2_i1_pair(const B2gSuper &A, const B2gSuper &B, bool same, const B2gPrim *__restrict__ pr,
                                           int np, const double *tab, const double *__restrict__ xyz,
                                           const int *__restrict__ Z, int natm, int N, double *__restrict__ S,
                                           double *__restrict__ T, double *__restrict__ V, int lane) {
  constexpr int NA = TA ? 4 : 1, NB = TB ? 4 : 1, NC = NA * NB;
  const double AB[3] = {A.R[0] - B.R[0], A.R[1] - B.R[1], A.R[2] - B.R[2]};
  const double k0 = 5.914967172795613;                 // the coefficients carry sqrt(2) pi^(5/4) / zeta
  double s[NC], t[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) s[k] = t[k] = 0.0;
  if (lane < np) {
    const B2gPrim p = pr[lane];
    const double be = (1.0 - p.ra) * p.z, u = p.u, c3 = (M_PI / k0) * sqrt(M_PI / p.z);   // (pi/zeta)^(3/2) zeta / k0
    double PA[3], PB[3], PB2 = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      PA[d] = (p.ra - 1.0) * AB[d];
      PB[d] = p.ra * AB[d];
      PB2 += PB[d] * PB[d];
    }
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const double cc = c3 * (a ? (b ? p.kpp : p.kps) : (b ? p.ksp : p.kss));
        const double sa = a ? PA[a ? a - 1 : 0] : 1.0, sb = b ? PB[b ? b - 1 : 0] : 1.0, dab = a && a == b ? 1.0 : 0.0;
        const double daPB = a ? PB[a ? a - 1 : 0] : 0.0, dbPB = b ? PB[b ? b - 1 : 0] : 0.0;
        const double ov = sa * sb + dab * u;
        const double r2 = sa * sb * PB2 + u * (dab * PB2 + 2 * sb * daPB + 2 * sa * dbPB + 3 * sa * sb) + 5 * u * u * dab;
        s[a * NB + b] = cc * ov;
        t[a * NB + b] = cc * (-0.5) * (4 * be * be * r2 - 2 * be * (b ? 5 : 3) * ov);
      }
  }
  const double sv = b2_i1_sum<NC>(s, lane), tv = b2_i1_sum<NC>(t, lane);
  double v[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) v[k] = 0.0;
#pragma unroll 1
  for (int e = lane; e < np * natm; e += 32) {
    const int c = e / np;
    const B2gPrim p = pr[e - c * np];
    const double X[3] = {p.P[0] - xyz[3 * c], p.P[1] - xyz[3 * c + 1], p.P[2] - xyz[3 * c + 2]};
    double F[3] = {0, 0, 0};
    b2_boys<double, (TA ? 1 : 0) + (TB ? 1 : 0)>(p.z * (X[0] * X[0] + X[1] * X[1] + X[2] * X[2]), tab, F);
    const double q = -(double)Z[c] * (2.0 * M_PI / k0), u = p.u;
    const double f0 = q * F[0], f1 = -2 * p.z * q * F[1], f2 = 4 * p.z * p.z * q * F[2];
    double PA[3], PB[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      PA[d] = (p.ra - 1.0) * AB[d];
      PB[d] = p.ra * AB[d];
    }
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const double cc = a ? (b ? p.kpp : p.kps) : (b ? p.ksp : p.kss);
        const int da = a ? a - 1 : 0, db = b ? b - 1 : 0;
        double x;
        if (!a && !b) x = f0;
        else if (!b) x = PA[da] * f0 + u * X[da] * f1;
        else if (!a) x = PB[db] * f0 + u * X[db] * f1;
        else {
          x = PA[da] * PB[db] * f0 + u * (PB[db] * X[da] + PA[da] * X[db]) * f1 + u * u * X[da] * X[db] * f2;
          if (a == b) x += u * f0 + u * u * f1;
        }
        v[a * NB + b] += cc * x;
      }
  }
  const double vv = b2_i1_sum<NC>(v, lane);
  if (lane < NC) {
    const int a = lane / NB, b = lane - (lane / NB) * NB;
    const int i = a ? (A.ao_p < 0 ? -1 : A.ao_p + a - 1) : A.ao_s, j = b ? (B.ao_p < 0 ? -1 : B.ao_p + b - 1) : B.ao_s;
    if (i >= 0 && j >= 0 && !(same && j > i)) {        // a shell with itself: one of the two orders
      S[i * N + j] = sv; S[j * N + i] = sv;
      T[i * N + j] = tv; T[j * N + i] = tv;
      V[i * N + j] = vv; V[j * N + i] = vv;
    }
  }
}

__global__ void __launch_bounds__(256, 2)
k_int1e(const B2MolDev *__restrict__ mols, const B2gsMol *__restrict__ gms, const long long *__restrict__ poff, int nmol,
        int chunk, const B2gSuper *__restrict__ su, const B2gPrim *__restrict__ prims, const B2gCount *__restrict__ pn,
        const double *__restrict__ atom_xyz, const int *__restrict__ atom_z, const double *__restrict__ btab,
        double *__restrict__ S, double *__restrict__ T, double *__restrict__ V) {
  __shared__ double tab[B2_BOYS_NT * B2_BOYS_NM];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < B2_BOYS_NT * B2_BOYS_NM; e += blockDim.x) tab[e] = btab[e];
  __syncthreads();
  const long long n = poff[nmol];
  for (long long c0 = ((long long)blockIdx.x * 8 + w) * chunk; c0 < n; c0 += (long long)gridDim.x * 8 * chunk) {
    int m = b2_find_ll(poff, 0, nmol - 1, c0);         // molecule of pair c0
    const long long c1 = min(n, c0 + chunk);
    for (long long t = c0; t < c1; ++t) {
      while (poff[m + 1] <= t) ++m;
      const B2MolDev &md = mols[m];
      const B2gsMol g = gms[m];
      int A, B;
      b2gs_pair(g.ns, g.np, (int)(t - g.pr_off), A, B);
      const B2gSuper &a = su[g.su_off + A], &b = su[g.su_off + B];
      const B2gPrim *pr = prims + t * B2_MAXPP;
      const int np = pn[t].z;
      const double *xyz = atom_xyz + 3ll * md.atm_off;
      const int *Z = atom_z + md.atm_off;
      double *s = S + md.mat_off, *tt = T + md.mat_off, *v = V + md.mat_off;
      if (B < g.ns) b2_i1_pair<false, false>(a, b, A == B, pr, np, tab, xyz, Z, md.natm, md.nao, s, tt, v, lane);
      else if (A < g.ns) b2_i1_pair<false, true>(a, b, false, pr, np, tab, xyz, Z, md.natm, md.nao, s, tt, v, lane);
      else b2_i1_pair<true, true>(a, b, A == B, pr, np, tab, xyz, Z, md.natm, md.nao, s, tt, v, lane);
    }
  }
}

// ------------------------------------------------------------------ Becke grid
__constant__ double c_bragg_sqrt[10];     // sqrt of Bragg-Slater radius (Angstrom), by Z

// One CTA per block of 128 grid points of one molecule, one thread per point: coordinate from
// the owning atom's template, weight = template weight * Becke cell function (3-fold
// polynomial, size-adjusted, build_grid.py:34-100) normalised over atoms.  The CTA tabulates
// 1/R_ij and the size adjustments a_ij of its molecule in shared memory; each unordered atom
// pair is evaluated once per point, using a_ji = -a_ij and the odd polynomial, so
// s(nu_ji) = 1 - s(nu_ij).  The factors are taken twice their size, 1 -+ g instead of
// (1 -+ g) / 2: every cell has the same number of factors, so the power of two cancels in the
// normalisation.  Eight atoms at a time sit in registers (distance and product); for each later
// atom j its distance is formed again (one reciprocal square root for eight pairs) and only its
// product makes a round trip through shared memory.  Stored distances bounded the kernel by
// shared-memory capacity (8 warps per SM for molecules of 17-32 atoms: 30% of the FP64 pipe).  One
// launch for molecules up to 16 atoms and one above, so that small molecules do not hold shared
// memory for the largest.  1500 molecules, 1.4e7 points: 4.9 ms with one pair per 4 loads and a store,
// 3.4 ms now.
#define B2_GRID_MAXATM 32
#define B2_GRID_BLK 8
__global__ void __launch_bounds__(128)
k_grid(const B2MolDev *__restrict__ mols, int nmol, const long long *__restrict__ gblk_off, int natm_lo, int natm_hi,
       const long long *__restrict__ grid_off, const long long *__restrict__ atom_pt_off,
       const double *__restrict__ atom_xyz, const int *__restrict__ atom_z,
       const double *__restrict__ tmpl, const long long *__restrict__ tmpl_off,
       double *__restrict__ coords, double *__restrict__ weights) {
  constexpr int BK = B2_GRID_BLK;
  __shared__ double sA[B2_GRID_MAXATM][3];
  extern __shared__ __align__(16) double sgrid[];   // [na][na] (1/R, a), [na][128] products
  const int m = b2_find_ll(gblk_off, 0, nmol - 1, blockIdx.x);
  const B2MolDev md = mols[m];
  const int na = md.natm, tid = threadIdx.x;
  if (na < natm_lo || na > natm_hi) return;
  double2 *sIA = reinterpret_cast<double2 *>(sgrid);
  double (*sP)[128] = reinterpret_cast<double (*)[128]>(sIA + na * na);
  for (int e = tid; e < na; e += blockDim.x) {
    sA[e][0] = atom_xyz[3 * (md.atm_off + e)];
    sA[e][1] = atom_xyz[3 * (md.atm_off + e) + 1];
    sA[e][2] = atom_xyz[3 * (md.atm_off + e) + 2];
  }
  __syncthreads();
  for (int e = tid; e < na * na; e += blockDim.x) {
    const int i = e / na, j = e - (e / na) * na;
    double inv = 0.0, a = 0.0;
    if (i != j) {
      const double rx = sA[i][0] - sA[j][0], ry = sA[i][1] - sA[j][1], rz = sA[i][2] - sA[j][2];
      inv = 1.0 / sqrt(rx * rx + ry * ry + rz * rz);
      const double chi = c_bragg_sqrt[atom_z[md.atm_off + i]] / c_bragg_sqrt[atom_z[md.atm_off + j]];
      const double uu = (chi - 1) / (chi + 1);
      a = fmin(0.5, fmax(-0.5, uu / (uu * uu - 1)));
    }
    sIA[e] = make_double2(inv, a);
  }
  __syncthreads();
  const long long G = grid_off[m + 1] - grid_off[m];
  const long long lp = (blockIdx.x - gblk_off[m]) * 128 + tid;    // point index in the molecule
  if (lp >= G) return;
  const long long gp = grid_off[m] + lp;
  const int ia = b2_find_ll(atom_pt_off, md.atm_off, md.atm_off + na - 1, gp) - md.atm_off;
  const int z = atom_z[md.atm_off + ia];
  const long long t = tmpl_off[z] + (gp - atom_pt_off[md.atm_off + ia]);
  const double x = sA[ia][0] + tmpl[4 * t], y = sA[ia][1] + tmpl[4 * t + 1], zc = sA[ia][2] + tmpl[4 * t + 2];
  coords[3 * gp] = x; coords[3 * gp + 1] = y; coords[3 * gp + 2] = zc;
  auto dist = [&](int i) {
    const double dx = x - sA[i][0], dy = y - sA[i][1], dz = zc - sA[i][2], r2 = dx * dx + dy * dy + dz * dz;
    return r2 > 0.0 ? r2 * rsqrt(r2) : 0.0;
  };
  auto pair = [](double di, double dj, double2 ia2, double &pi, double &pj) {
    const double mu = (di - dj) * ia2.x;
    double g = fma(ia2.y, fma(-mu, mu, 1.0), mu);
#pragma unroll
    for (int k = 0; k < 3; ++k) g *= fma(-0.5 * g, g, 1.5);       // (3 - g^2) g / 2
    pi = fma(-pi, g, pi);
    pj = fma(pj, g, pj);
  };
  double psum = 0, pown = 0;
  for (int i0 = 0; i0 < na; i0 += BK) {
    double di[BK], pi[BK];
#pragma unroll
    for (int k = 0; k < BK; ++k)
      if (i0 + k < na) {
        di[k] = dist(i0 + k);
        pi[k] = i0 ? sP[i0 + k][tid] : 1.0;
      }
#pragma unroll
    for (int k = 0; k < BK - 1; ++k)
#pragma unroll
      for (int l = k + 1; l < BK; ++l)
        if (i0 + l < na) pair(di[k], di[l], sIA[(i0 + k) * na + i0 + l], pi[k], pi[l]);
    for (int j = i0 + BK; j < na; ++j) {           // every atom of the block exists here
      const double dj = dist(j);
      double pj[2] = {i0 ? sP[j][tid] : 1.0, 1.0};  // two chains
#pragma unroll
      for (int k = 0; k < BK; ++k) pair(di[k], dj, sIA[(i0 + k) * na + j], pi[k], pj[k & 1]);
      sP[j][tid] = pj[0] * pj[1];
    }
#pragma unroll
    for (int k = 0; k < BK; ++k)
      if (i0 + k < na) {
        psum += pi[k];
        if (i0 + k == ia) pown = pi[k];
      }
  }
  weights[gp] = tmpl[4 * t + 3] * pown / psum;
}

// ------------------------------------------------------------------ guess + E_nuc
// MINAO-style occupations on the diagonal: H 1s 1; heavy 1s 2, 2s 2, 2p (Z-4)/3 each
__global__ void k_guess(const B2MolDev *__restrict__ mols, const B2Shell *__restrict__ shells,
                        const int *__restrict__ ao2sh, const int *__restrict__ atom_z,
                        double *__restrict__ D) {
  const B2MolDev md = mols[blockIdx.x];
  const int N = md.nao;
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int a = e / N, b = e - (e / N) * N;
    double v = 0;
    if (a == b) {
      const int s = ao2sh[md.ao_off + a];
      const B2Shell sh = shells[md.sh_off + s];
      const int z = atom_z[md.atm_off + sh.atom];
      if (z <= 2) v = (double)z;
      else if (sh.l == 0) v = 2.0;
      else v = (z - 4) / 3.0;
    }
    D[md.mat_off + e] = v;
  }
}

// one warp per molecule, lanes over the atom pairs
__global__ void __launch_bounds__(128)
k_enuc(const B2MolDev *__restrict__ mols, int nmol, const double *__restrict__ atom_xyz,
       const int *__restrict__ atom_z, double *__restrict__ enuc) {
  const int m = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (m >= nmol) return;                            // whole warp
  const B2MolDev md = mols[m];
  const double *A = atom_xyz + 3 * md.atm_off;
  const int npair = md.natm * (md.natm - 1) / 2;
  double e = 0;
  for (int p = lane; p < npair; p += 32) {
    const int k = (int)b2_untri(p), i = k + 1, j = p - (int)b2_tri(k);     // i > j
    const double dx = A[3 * i] - A[3 * j], dy = A[3 * i + 1] - A[3 * j + 1], dz = A[3 * i + 2] - A[3 * j + 2];
    e += (double)atom_z[md.atm_off + i] * atom_z[md.atm_off + j] / sqrt(dx * dx + dy * dy + dz * dz);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if (lane == 0) enuc[m] = e;
}

// s8 entries with |v| <= threshold become 0 (the ERI threshold of nanoDFT.py:280-288); the
// molecules' padding entries are never read, so the whole buffer is swept
template <typename T>
__global__ void k_threshold(long long n, T *__restrict__ x, double thr) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (fabs((double)x[i]) <= thr) x[i] = (T)0;
}

int b2_launch_eri_threshold(const B2PlanDev &P, int precision, void *eri, double thr, cudaStream_t st) {
  if (!eri || (precision != 32 && precision != 64) || !(thr >= 0.0)) return B2_ERR_ARG;
  const long long n = P.h.n_eri;
  if (n > 0) {
    const unsigned nb = (unsigned)std::min<long long>((n + 255) / 256, 148ll * 32);
    if (precision == 64) k_threshold<double><<<nb, 256, 0, st>>>(n, (double *)eri, thr);
    else k_threshold<float><<<nb, 256, 0, st>>>(n, (float *)eri, thr);
    b2_count_launches(1);
  }
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

int b2_launch_int1e(const B2PlanDev &P, double *S, double *T, double *V, cudaStream_t st) {
  const long long n = P.su.n_pair;
  if (n <= 0) return B2_OK;
  // up to 8 consecutive pairs per warp (one molecule search for all) once every resident warp has work
  const int chunk = (int)std::max(1ll, std::min(8ll, n / (148ll * 4 * 8)));
  const long long nb = (n + 8ll * chunk - 1) / (8ll * chunk);
  k_int1e<<<(unsigned)std::min<long long>(nb, 148ll * 4), 256, 0, st>>>(
      P.mols, P.su.mol, P.su.off + B2_SU_PAIRS * (P.h.nmol + 1ll), P.h.nmol, chunk, P.su.su, P.su.pr64, P.su.pn,
      P.atom_xyz, P.atom_z, P.boys, S, T, V);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

int b2_launch_grid_build(B2PlanDev &P, int nz, const double *tmpl_host, const long long *tmpl_off_host,
                         double *coords, double *weights, cudaStream_t st) {
  if (!P.g.grid_off || nz < 10) return B2_ERR_ARG;
  if (P.h.max_natm > B2_GRID_MAXATM) return B2_ERR_SIZE;
  // per-atom point offsets from the templates; must agree with the registered grid layout
  std::vector<long long> apo(P.h.n_atm + 1, 0);
  long long tot = 0;
  for (int m = 0; m < P.h.nmol; ++m) {
    const B2MolDev &md = P.h.mols[m];
    if (tot != P.g.grid_off_h[m]) return B2_ERR_ARG;
    for (int a = 0; a < md.natm; ++a) {
      const int z = P.h.atom_z[md.atm_off + a];
      if (z < 0 || z >= nz) return B2_ERR_UNSUPPORTED;
      apo[md.atm_off + a] = tot;
      tot += tmpl_off_host[z + 1] - tmpl_off_host[z];
    }
  }
  apo[P.h.n_atm] = tot;
  if (tot != P.g.n_points) return B2_ERR_ARG;
  const long long ntm = tmpl_off_host[nz];
  b2_dfree(P.g.tmpl); b2_dfree(P.g.tmpl_off); b2_dfree(P.g.atom_pt_off);
  B2_CUDA_TRY(b2_dmalloc_t(&P.g.tmpl, sizeof(double) * 4 * std::max(1ll, ntm)));
  B2_CUDA_TRY(b2_dmalloc_t(&P.g.tmpl_off, sizeof(long long) * (nz + 1)));
  B2_CUDA_TRY(b2_dmalloc_t(&P.g.atom_pt_off, sizeof(long long) * apo.size()));
  B2_CUDA_TRY(cudaMemcpy(P.g.tmpl, tmpl_host, sizeof(double) * 4 * ntm, cudaMemcpyHostToDevice));
  B2_CUDA_TRY(cudaMemcpy(P.g.tmpl_off, tmpl_off_host, sizeof(long long) * (nz + 1), cudaMemcpyHostToDevice));
  B2_CUDA_TRY(cudaMemcpy(P.g.atom_pt_off, apo.data(), sizeof(long long) * apo.size(), cudaMemcpyHostToDevice));
  const double br[10] = {0.35, 0.35, 0, 0, 0, 0, 0.70, 0.65, 0.60, 0.50};
  double brs[10];
  for (int i = 0; i < 10; ++i) brs[i] = br[i] > 0 ? sqrt(br[i]) : 1.0;
  B2_CUDA_TRY(cudaMemcpyToSymbol(c_bragg_sqrt, brs, sizeof(brs)));
  if (P.g.n_points > 0) {
    auto smem = [](int na) { return sizeof(double) * (size_t)(2 * na * na + 128 * na); };
    B2_CUDA_TRY(cudaFuncSetAttribute(k_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem(P.h.max_natm)));
    bool small = false, large = false;
    for (int m = 0; m < P.h.nmol; ++m) (P.h.mols[m].natm <= 16 ? small : large) = true;
    for (int part = 0; part < 2; ++part) {
      if (!(part ? large : small)) continue;
      const int lo = part ? 17 : 0, hi = part ? B2_GRID_MAXATM : 16;
      k_grid<<<(unsigned)P.g.n_gblk, 128, smem(std::min(hi, P.h.max_natm)), st>>>(
          P.mols, P.h.nmol, P.g.gblk_off, lo, hi, P.g.grid_off, P.g.atom_pt_off, P.atom_xyz, P.atom_z, P.g.tmpl,
          P.g.tmpl_off, coords, weights);
      b2_count_launches(1);
    }
  }
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

int b2_launch_guess(const B2PlanDev &P, double *D, cudaStream_t st) {
  k_guess<<<P.h.nmol, 256, 0, st>>>(P.mols, P.shells, P.ao2sh, P.atom_z, D);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

int b2_launch_enuc(const B2PlanDev &P, double *enuc, cudaStream_t st) {
  k_enuc<<<(P.h.nmol + 3) / 4, 128, 0, st>>>(P.mols, P.h.nmol, P.atom_xyz, P.atom_z, enuc);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

