// Nuclear gradients of converged RKS SCFs on the GPU, batched over a plan's molecules: the
// reference's grad(mol, coords, weight, mo_coeff, mo_energy) = grad_elec + grad_nuc
// (nanoDFT.py:403-477), which builds int2e_ip1 / int1e_ip* on the host and contracts them with
// einsums.  Here every term is contracted as it is generated, in float64:
//
//   k_grad_dm   dm0 = 2 C_occ C_occ^T, dme0 = 2 C_occ eps_occ C_occ^T (nanoDFT.py:405-406);
//   k_grad_sp   d/dR of 1/2 <D, J> - hyb/4 <D, K> (the vj / vk terms, nanoDFT.py:416-418): one
//               warp per super-shell slice x 32 ket pairs of one class, one ket primitive per
//               lane (grad_sp.cuh);
//   k_grad_1e   d/dR of <D, T + V_nuc> - <dme0, S> (h1aos and s1, nanoDFT.py:420-424): one warp
//               per super-shell slice, lanes over nuclei;
//   k_grad_xc   d/dR of E_xc at fixed density and grid (V_xc, nanoDFT.py:408-415): tiles of 32
//               points of one molecule, products with D by float64 MMA;
//   k_grad_nuc  nuclear repulsion (grad_nuc, nanoDFT.py:428-438).
//
// The two- and one-electron math is grad_sp.cuh, which the host-check build runs too and compares with
// the Obara-Saika forms of grad_math.cuh; those are compared with the finite-difference oracle.
#include <algorithm>
#include "device_plan.cuh"
#include "grad_sp.cuh"
#include "xc_f64.cuh"

__global__ void __launch_bounds__(256)
k_grad_dm(const B2MolDev *__restrict__ mols, const double *__restrict__ C, const double *__restrict__ eps,
          double *__restrict__ D, double *__restrict__ W) {
  const int m = blockIdx.x;
  const B2MolDev md = mols[m];
  const int N = md.nao, NN = N * N;
  const double *Cm = C + md.mat_off;
  const double *em = eps + (long long)m * B2_MAXNAO;
  for (int e = threadIdx.x; e < NN; e += blockDim.x) {
    const int a = e / N, b = e - (e / N) * N;
    double s = 0, t = 0;
    for (int k = 0; k < md.nocc; ++k) {
      const double p = Cm[a * N + k] * Cm[b * N + k];
      s += p;
      t += p * em[k];
    }
    D[md.mat_off + e] = 2.0 * s;
    W[md.mat_off + e] = 2.0 * t;
  }
}

// ---- two-electron and one-electron parts: super-shell slices (grad_sp.cuh)
//
// The tables (super shells, screened primitive pairs, task prefixes) are the plan's.
#define B2GS_TABLE (B2_BOYS_NT * B2_BOYS_NM)

__device__ __forceinline__ int b2gs_find(const long long *__restrict__ off, int n, long long x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// per-warp shared memory of the two-electron kernel
struct __align__(16) B2gsWarp {
  B2gBraRec bra[B2_MAXPP];
  double CD[32][3], wt[32], acc[32][6];
  int ao[32][4], off[32], pair[32];
  unsigned char map[32 * B2_MAXPP];
};

// density factors, bra loop and centre sums of one ket primitive (axis KF of the ket's p
// function relative to the bra's)
template <int TB, int TK, int KF>
__device__ __forceinline__ void b2gs_lane(const B2gsWarp &W, int nb, int k, const B2gPrim &r, const double *AB, int f,
                                          int F, const int *bi, const double *__restrict__ Dm, int N, double hyb,
                                          const double *tab, double *gA, double *gB, double *gC, double *gD) {
  using C = B2gsClass<TB, TK>;
  const int cs = W.ao[k][0], cp = W.ao[k][1], ds = W.ao[k][2], dp = W.ao[k][3];
  const int F2 = TK == 2 ? (cp < 0 ? -1 : cp + (f + KF) % 3) : cs;
  int di[4] = {ds, -1, -1, -1};
  double CD[3], QD[3], Q[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const int px = f + x >= 3 ? f + x - 3 : f + x;
    if (TK && dp >= 0) di[1 + x] = dp + px;
    CD[x] = W.CD[k][x];
    QD[x] = r.ra * CD[x];
    Q[x] = px == 0 ? r.P[0] : (px == 1 ? r.P[1] : r.P[2]);
  }
  B2gKet<C::NB, C::NK> q;
  b2gs_ket<C::NB, C::NK>(Dm, N, hyb, W.wt[k], F, bi, F2, di, TK == 2 ? r.kps : r.kss, TK == 2 ? r.kpp : r.ksp, QD, q);
  q.v = r.u;
  q.FC = (r.ra - 1.0) * CD[KF < 0 ? 0 : KF];
  B2gOut s;
  s.E = s.C = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) s.dP[x] = s.D[x] = 0.0;
#pragma unroll 1
  for (int p = 0; p < nb; ++p) {
    B2gOut o;
    b2gs_eval<TB, TK, KF>(W.bra[p], q, Q, r.z, tab, o);
    b2gs_add_bra<TB>(W.bra[p], AB, o, gA, gB);
    s.E += o.E;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      s.dP[x] += o.dP[x];
      if (TK) s.D[x] += o.D[x];
    }
    if (TK == 2) s.C += o.C;
  }
  b2gs_add_ket<TK, KF>(r.ra, r.mu2, CD, s, gC, gD);
}

// Two-electron part of one class (bra slices of type TB, ket slices of type TK <= TB; each
// unordered slice quartet once).  One warp per task (molecule, bra slice, 32 kets): the kets'
// surviving primitive pairs are packed over the lanes; a lane contracts its ket primitive with the
// density factors once and runs over the bra's primitive pairs in shared memory, so a lane holds
// one primitive quartet's derivative tensor (up to 56 values) in registers and no integral is ever
// stored.  The bra centres' sums stay in registers for the whole task; the ket centres' are summed
// over the lanes of a ket by a segmented scan.  CTAs stay resident and stride over the tasks; the
// Boys table sits in shared memory (its rows are gathered at random: from global memory those
// gathers took longer than the arithmetic of the small classes).
// Bound by FP64 issue and latency (118-255 registers: 8-16 warps per SM); the whole gradient of
// 160 uneven molecules takes 24 ms, of one molecule with 5 heavy atoms 0.24 ms.  Before (one warp
// per shell quartet and l class in 16 kernels, contracted Obara-Saika [e0|f0] arrays through
// shared memory and a horizontal recursion per quartet): 732 ms and 65 ms.
template <int TB, int TK>
__global__ void __launch_bounds__(128)
k_grad_sp(const long long *__restrict__ toff, int nmol, const B2gsMol *__restrict__ gms,
          const B2MolDev *__restrict__ mols, const B2gSuper *__restrict__ su, const B2gPrim *__restrict__ pr,
          const B2gCount *__restrict__ pn, const double *__restrict__ btab, const double *__restrict__ D,
          double hyb, double *__restrict__ grad) {
  extern __shared__ __align__(16) unsigned char gs_smem[];
  double *tab = reinterpret_cast<double *>(gs_smem);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  B2gsWarp &W = reinterpret_cast<B2gsWarp *>(gs_smem + sizeof(double) * B2GS_TABLE)[w];
  for (int e = threadIdx.x; e < B2GS_TABLE; e += blockDim.x) tab[e] = btab[e];
  __syncthreads();
  const long long ntask = toff[nmol];
  for (long long task = (long long)blockIdx.x * 4 + w; task < ntask; task += (long long)gridDim.x * 4) {
    const int m = b2gs_find(toff, nmol, task);
    const B2gsMol g = gms[m];
    const int nket = b2gs_nket(g.ns, g.np, TK), nch = (nket + 31) >> 5;
    const int r0 = (int)(task - toff[m]), i = r0 / nch, k0 = (r0 - i * nch) * 32;
    const int bpr = TB == 2 ? i / 3 : i, f = TB == 2 ? i - 3 * (i / 3) : 0;
    const int cnt = min(32, (TB == TK ? bpr + 1 : nket) - k0);
    if (cnt <= 0) continue;                        // whole warp: beyond the diagonal
    const B2MolDev md = mols[m];
    const B2gSuper *sm = su + g.su_off;
    const double *Dm = D + md.mat_off;
    const int N = md.nao;
    int A, B;
    const int pb = b2gs_ket_pair(g.ns, g.np, TB, bpr);
    b2gs_pair(g.ns, g.np, pb, A, B);
    double AB[3];
    int bi[4] = {sm[B].ao_s, -1, -1, -1};
    const int F = TB == 2 ? (sm[A].ao_p < 0 ? -1 : sm[A].ao_p + f) : sm[A].ao_s;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const int px = f + x >= 3 ? f + x - 3 : f + x;
      AB[x] = sm[A].R[px] - sm[B].R[px];
      if (TB && sm[B].ao_p >= 0) bi[1 + x] = sm[B].ao_p + px;
    }
    const int nb = pn[g.pr_off + pb].z;
    __syncwarp();                                  // the previous task's shared memory is consumed
    if (lane < nb) b2gs_bra(pr[(g.pr_off + pb) * B2_MAXPP + lane], TB, f, AB, W.bra[lane]);
    int nq = 0, ca = 0, da = 0;
    if (lane < cnt) {
      int c, d;
      const int pk = b2gs_ket_pair(g.ns, g.np, TK, k0 + lane);
      b2gs_pair(g.ns, g.np, pk, c, d);
      const B2gSuper &sc = sm[c], &sd = sm[d];
      nq = pn[g.pr_off + pk].z;
      ca = sc.atom;
      da = sd.atom;
      W.pair[lane] = pk;
      W.ao[lane][0] = sc.ao_s;
      W.ao[lane][1] = sc.ao_p;
      W.ao[lane][2] = sd.ao_s;
      W.ao[lane][3] = sd.ao_p;
      W.wt[lane] = (A == B ? 1.0 : 2.0) * (c == d ? 1.0 : 2.0) * (TB == TK && k0 + lane == bpr ? 1.0 : 2.0);
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const int px = f + x >= 3 ? f + x - 3 : f + x;
        W.CD[lane][x] = sc.R[px] - sd.R[px];
      }
    }
#pragma unroll
    for (int x = 0; x < 6; ++x) W.acc[lane][x] = 0.0;
    int inc = nq;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    const int E = __shfl_sync(0xffffffffu, inc, 31);
    W.off[lane] = inc - nq;
    for (int j = 0; j < nq; ++j) W.map[inc - nq + j] = (unsigned char)lane;
    __syncwarp();
    double gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0};
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const bool valid = e < E;
      const int k = valid ? (int)W.map[e] : -1 - lane;      // entries past the end: unique keys
      double gk[6] = {0, 0, 0, 0, 0, 0};
      if (valid) {
        const B2gPrim r = pr[(g.pr_off + W.pair[k]) * B2_MAXPP + (e - W.off[k])];
        if constexpr (TK == 2) {
          b2gs_lane<TB, TK, 0>(W, nb, k, r, AB, f, F, bi, Dm, N, hyb, tab, gA, gB, gk, gk + 3);
          b2gs_lane<TB, TK, 1>(W, nb, k, r, AB, f, F, bi, Dm, N, hyb, tab, gA, gB, gk, gk + 3);
          b2gs_lane<TB, TK, 2>(W, nb, k, r, AB, f, F, bi, Dm, N, hyb, tab, gA, gB, gk, gk + 3);
        } else {
          b2gs_lane<TB, TK, -1>(W, nb, k, r, AB, f, F, bi, Dm, N, hyb, tab, gA, gB, gk, gk + 3);
        }
      }
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {                     // same-ket inclusive scan (<= 9 lanes)
        const int ko = __shfl_up_sync(0xffffffffu, k, o);
        const bool take = lane >= o && ko == k;
#pragma unroll
        for (int x = 0; x < 6; ++x) {
          const double y = __shfl_up_sync(0xffffffffu, gk[x], o);
          if (take) gk[x] += y;
        }
      }
      const int kn = __shfl_down_sync(0xffffffffu, k, 1);
      if (valid && (lane == 31 || kn != k))
#pragma unroll
        for (int x = 0; x < 6; ++x) W.acc[k][x] += gk[x];
      __syncwarp();
    }
    double *gm = grad + 3ll * md.atm_off;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const int px = f + x >= 3 ? f + x - 3 : f + x;
      if (lane < cnt) {
        atomicAdd(gm + 3 * ca + px, W.acc[lane][x]);
        atomicAdd(gm + 3 * da + px, W.acc[lane][3 + x]);
      }
      double u = gA[x], t = gB[x];
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, o);
        t += __shfl_xor_sync(0xffffffffu, t, o);
      }
      if (lane == 0) {
        atomicAdd(gm + 3 * sm[A].atom + px, u);
        atomicAdd(gm + 3 * sm[B].atom + px, t);
      }
    }
  }
}

// One-electron part: one warp per bra slice of a molecule.  Overlap and kinetic energy: one
// primitive pair per lane; nuclear attraction: lanes over (primitive pair, nucleus), the nuclei
// of a molecule padded to 8, 16 or 32 lanes, so every lane keeps its nucleus' gradient in
// registers over the primitive pairs.  Before: one thread per ordered shell pair with all
// primitive pairs and nuclei in its local-memory recursion tables, one CTA per molecule.
template <int TB>
__device__ __forceinline__ void b2gs_one(const B2gsMol &g, int i, const B2MolDev &md, const B2gSuper *__restrict__ sm,
                                         const B2gPrim *__restrict__ prm, const B2gCount *__restrict__ pnm,
                                         const double *__restrict__ xyz, const int *__restrict__ Z,
                                         const double *tab, const double *__restrict__ Dm,
                                         const double *__restrict__ Wm, double *__restrict__ gm, int lane) {
  constexpr int NB = TB ? 1 : 0;
  const int bpr = TB == 2 ? i / 3 : i, f = TB == 2 ? i - 3 * (i / 3) : 0, N = md.nao;
  const int pb = b2gs_ket_pair(g.ns, g.np, TB, bpr);
  int A, B;
  b2gs_pair(g.ns, g.np, pb, A, B);
  const B2gSuper &sa = sm[A], &sb = sm[B];
  const int F = TB == 2 ? (sa.ao_p < 0 ? -1 : sa.ao_p + f) : sa.ao_s;
  const double wt = A == B ? 1.0 : 2.0;
  double AB[3], dg[NB ? 4 : 1], wg[NB ? 4 : 1];            // density factors of T / V and of S
#pragma unroll
  for (int b = 0; b < (NB ? 4 : 1); ++b) {
    const int bb = b == 0 ? sb.ao_s : (sb.ao_p < 0 ? -1 : sb.ao_p + (f + b - 1) % 3);
    const bool ok = F >= 0 && bb >= 0;
    dg[b] = ok ? wt * Dm[F * N + bb] : 0.0;
    wg[b] = ok ? -wt * Wm[F * N + bb] : 0.0;
  }
#pragma unroll
  for (int x = 0; x < 3; ++x) AB[x] = sa.R[(f + x) % 3] - sb.R[(f + x) % 3];
  const int nb = pnm[pb].z;
  double gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0};
  if (lane < nb) {
    B2gBraRec r;
    b2gs_bra(prm[(long long)pb * B2_MAXPP + lane], TB, f, AB, r);
    double gk[3];
    b2gs_st<TB>(r, dg, wg, AB, gk);
#pragma unroll
    for (int x = 0; x < 3; ++x) { gA[x] += gk[x]; gB[x] -= gk[x]; }
  }
  const int lg = md.natm <= 8 ? 3 : (md.natm <= 16 ? 4 : 5), G = 1 << lg, step = 32 >> lg;
  for (int c0 = 0; c0 < md.natm; c0 += G) {
    const int c = c0 + (lane & (G - 1));
    double gN[3] = {0, 0, 0};
    if (c < md.natm) {
      const double q0 = -(double)Z[c] * (6.283185307179586 / 5.914967172795613);   // 2 pi over the pair constant
      const double C[3] = {xyz[3 * c + f], xyz[3 * c + (f + 1) % 3], xyz[3 * c + (f + 2) % 3]};
      B2gKet<NB, 0> q;
#pragma unroll
      for (int b = 0; b < (NB ? 4 : 1); ++b) q.gs[b] = q0 * dg[b];
      q.v = q.FC = 0.0;
      for (int p = lane >> lg; p < nb; p += step) {
        B2gBraRec r;
        b2gs_bra(prm[(long long)pb * B2_MAXPP + p], TB, f, AB, r);
        B2gOut o;
        b2gs_eval_point<TB>(r, q, C, tab, o);
        b2gs_add_bra<TB>(r, AB, o, gA, gB);
#pragma unroll
        for (int x = 0; x < 3; ++x) gN[x] -= o.dP[x];
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      double v = gN[x];
      for (int o = G; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < G && c < md.natm) atomicAdd(gm + 3 * c + (f + x) % 3, v);
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    double u = gA[x], t = gB[x];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      u += __shfl_xor_sync(0xffffffffu, u, o);
      t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (lane == 0) {
      atomicAdd(gm + 3 * sa.atom + (f + x) % 3, u);
      atomicAdd(gm + 3 * sb.atom + (f + x) % 3, t);
    }
  }
}

__global__ void __launch_bounds__(128)
k_grad_1e(const long long *__restrict__ toff, int nmol, const B2gsMol *__restrict__ gms,
          const B2MolDev *__restrict__ mols, const B2gSuper *__restrict__ su, const B2gPrim *__restrict__ pr,
          const B2gCount *__restrict__ pn, const double *__restrict__ atom_xyz, const int *__restrict__ atom_z,
          const double *__restrict__ btab, const double *__restrict__ D, const double *__restrict__ Wd,
          double *__restrict__ grad) {
  extern __shared__ __align__(16) unsigned char gs_smem[];
  double *tab = reinterpret_cast<double *>(gs_smem);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < B2GS_TABLE; e += blockDim.x) tab[e] = btab[e];
  __syncthreads();
  const long long ntask = toff[nmol];
  for (long long task = (long long)blockIdx.x * 4 + w; task < ntask; task += (long long)gridDim.x * 4) {
    const int m = b2gs_find(toff, nmol, task);
    const B2gsMol g = gms[m];
    const B2MolDev md = mols[m];
    int i = (int)(task - toff[m]);
    const int n0 = b2gs_nslice(g.ns, g.np, 0), n1 = b2gs_nslice(g.ns, g.np, 1);
    const B2gSuper *sm = su + g.su_off;
    const B2gPrim *prm = pr + g.pr_off * B2_MAXPP;
    const B2gCount *pnm = pn + g.pr_off;
    const double *xyz = atom_xyz + 3ll * md.atm_off, *Dm = D + md.mat_off, *Wm = Wd + md.mat_off;
    const int *Z = atom_z + md.atm_off;
    double *gm = grad + 3ll * md.atm_off;
    if (i < n0) b2gs_one<0>(g, i, md, sm, prm, pnm, xyz, Z, tab, Dm, Wm, gm, lane);
    else if ((i -= n0) < n1) b2gs_one<1>(g, i, md, sm, prm, pnm, xyz, Z, tab, Dm, Wm, gm, lane);
    else b2gs_one<2>(g, i - n1, md, sm, prm, pnm, xyz, Z, tab, Dm, Wm, gm, lane);
  }
}

// Exchange-correlation part.  With phi the AO values, u = D phi and, per point, a = w vrho and
// b = 2 w vgamma grad rho, moving atom A moves its orbitals (d phi_i / dR_A = -grad phi_i):
//   dE/dR_A,x = -2 sum_g sum_{i on A} [d_x phi_i t_i + u_i sum_k b_k d_x d_k phi_i],
//   t = D (a phi + sum_k b_k d_k phi).
// So two products with D per tile (u and t; the form before made four, u and D d_k phi), by
// float64 MMA in the phases of xc_f64.cuh; u and t replace the AO planes, and the last phase takes
// the orbitals' derivatives from the radial sums again, one super shell per warp, its three sums
// in registers over the CTA's tiles.  160 molecules, 1.45e6 points: 9.5 ms before (CUDA-core
// products in 160 KB CTAs, the functional on one warp), 2.8 ms now.
template <int Q>
__global__ void __launch_bounds__(256, Q <= 4 ? 2 : 1)       // more registers than CTAs: the sums stay in them
k_grad_xc(const B2MolDev *__restrict__ mols, const B2gsMol *__restrict__ gms, const B2gSuper *__restrict__ su,
          const long long *__restrict__ xblk_off, const long long *__restrict__ grid_off, int nmol, int tpc,
          const double *__restrict__ coords, const double *__restrict__ weights, const double *__restrict__ D,
          double *__restrict__ grad) {
  using X = B2Xf<Q>;
  constexpr int NB = X::NB, LDD = X::LDD, LDP = B2_XF_LDP, PL = X::PL;
  constexpr int NS = 2 * Q + 1;                  // super shells per warp: at most 16 Q / 8, rounded up
  extern __shared__ __align__(16) unsigned char gx_smem[];
  const int m = b2_xf_find(xblk_off, nmol, blockIdx.x);
  const B2MolDev md = mols[m];
  const int N = md.nao;
  if ((N + 15) / 16 != Q) return;
  const B2gsMol gm = gms[m];
  const B2gSuper *sm = su + gm.su_off;
  const int nsu = gm.ns + gm.np;
  double *sD = reinterpret_cast<double *>(gx_smem), *sA = sD + NB * LDD, *sR = sA + 4 * PL, *sF = sR + 16 * 32;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  for (int e = tid; e < NB * LDD; e += 256) {
    const int a = e / LDD, b = e - (e / LDD) * LDD;
    sD[e] = (a < N && b < N) ? D[md.mat_off + b * N + a] : 0.0;      // u_i = sum_j D_ij phi_j
  }
  for (int e = tid; e < 4 * PL; e += 256) sA[e] = 0.0;         // rows beyond N stay zero
  const long long G = grid_off[m + 1] - grid_off[m], t0 = (blockIdx.x - xblk_off[m]) * (long long)tpc;
  const double *cm = coords + 3 * grid_off[m], *wm = weights + grid_off[m];
  const int n8 = (N + 7) >> 3, r0 = 16 * (w & 1), j0 = w >> 1;
  double acc[NS][3];
#pragma unroll
  for (int k = 0; k < NS; ++k) acc[k][0] = acc[k][1] = acc[k][2] = 0.0;
  // a product's accumulators to a plane
  auto put = [&](const double (&x)[X::NX][4], double *P) {
#pragma unroll
    for (int i = 0; i < X::NX; ++i) {
      const int j = j0 + 4 * i;
      if (j < n8) {
        double *o = P + (8 * j + 2 * t) * LDP + r0 + g;
        o[0] = x[i][0];
        o[LDP] = x[i][1];
        o[8] = x[i][2];
        o[LDP + 8] = x[i][3];
      }
    }
  };
  for (int tt = 0; tt < tpc; ++tt) {
    const long long g0 = (t0 + tt) * 32;
    if (g0 >= G) break;
    const bool pt = g0 + lane < G;
    double px = 0, py = 0, pz = 0, wg = 0;
    if (pt) {
      px = cm[3 * (g0 + lane)]; py = cm[3 * (g0 + lane) + 1]; pz = cm[3 * (g0 + lane) + 2];
      wg = wm[g0 + lane];
    }
    __syncthreads();                                           // tables filled / previous tile consumed
    b2_xf_ao<PL>(sm, nsu, pt, px, py, pz, sA);
    __syncthreads();
    double x[X::NX][4];
    b2_xf_mm<Q>(sA, sD, n8, x);
    b2_xf_rho<Q>(sA, n8, x, sR);
    B2XfPoint f;
    b2_xf_func(sR, sF, f);
    // points beyond the grid add nothing; grad rho = 2 rho[1..3]
    const double a = pt ? wg * f.vrho : 0.0;
    const double b[3] = {pt ? 4.0 * wg * f.vgamma * f.rho[1] : 0.0, pt ? 4.0 * wg * f.vgamma * f.rho[2] : 0.0,
                         pt ? 4.0 * wg * f.vgamma * f.rho[3] : 0.0};
    for (int n = w; n < 8 * n8; n += 8) {
      double *o = sA + n * LDP + lane;
      o[PL] = a * o[0] + b[0] * o[PL] + b[1] * o[2 * PL] + b[2] * o[3 * PL];
    }
    __syncthreads();                                           // planes 2 and 3 are free now
    put(x, sA + 2 * PL);
    b2_xf_mm<Q>(sA + PL, sD, n8, x);
    put(x, sA + 3 * PL);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NS; ++k) {
      const int s = w + 8 * k;
      if (s < nsu) {
        const B2gSuper &S = sm[s];
        const double d[3] = {px - S.R[0], py - S.R[1], pz - S.R[2]}, r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        double s1 = 0, s2 = 0, p0 = 0, p1 = 0, p2 = 0;         // sums of c e, -2 a c e, 4 a^2 c e
        for (int q = 0; q < S.nprim; ++q) {
          const double al = S.ex[q], ax = al * r2;
          if (!pt || ax > 60.0) continue;
          const double ev = exp(-ax), es = S.cs[q] * ev, ep = S.cp[q] * ev;
          s1 -= 2.0 * al * es;
          s2 += 4.0 * al * al * es;
          p0 += ep;
          p1 -= 2.0 * al * ep;
          p2 += 4.0 * al * al * ep;
        }
        const double bd = b[0] * d[0] + b[1] * d[1] + b[2] * d[2];
        if (S.ao_s >= 0) {
          const double *o = sA + S.ao_s * LDP + lane;
          const double ui = o[2 * PL], ti = o[3 * PL], c = s1 * ti + s2 * bd * ui;
#pragma unroll
          for (int y = 0; y < 3; ++y) acc[k][y] += c * d[y] + s1 * ui * b[y];
        }
        if (S.ao_p >= 0) {
          const double *o = sA + S.ao_p * LDP + lane;
          double ui[3], ti[3], T = 0, U = 0, bU = 0;
#pragma unroll
          for (int y = 0; y < 3; ++y) {
            ui[y] = o[2 * PL + y * LDP];
            ti[y] = o[3 * PL + y * LDP];
            T += d[y] * ti[y];
            U += d[y] * ui[y];
            bU += b[y] * ui[y];
          }
          const double c = p1 * (T + bU) + p2 * bd * U;
#pragma unroll
          for (int y = 0; y < 3; ++y) acc[k][y] += p0 * ti[y] + p1 * bd * ui[y] + p1 * U * b[y] + c * d[y];
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    const int s = w + 8 * k;
    if (s < nsu) {
#pragma unroll
      for (int y = 0; y < 3; ++y) {
        double v = acc[k][y];
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) atomicAdd(grad + 3ll * (md.atm_off + sm[s].atom) + y, -2.0 * v);
      }
    }
  }
}

// nuclear repulsion: g_a = -sum_{b != a} Z_a Z_b (R_a - R_b) / |R_a - R_b|^3 (coincident atoms
// contribute nothing, as in the reference)
__global__ void __launch_bounds__(128)
k_grad_nuc(const B2MolDev *__restrict__ mols, const double *__restrict__ atom_xyz, const int *__restrict__ atom_z,
           double *__restrict__ grad) {
  const B2MolDev md = mols[blockIdx.x];
  const double *R = atom_xyz + 3ll * md.atm_off;
  const int *Z = atom_z + md.atm_off;
  for (int a = threadIdx.x; a < md.natm; a += blockDim.x) {
    double g[3] = {0, 0, 0};
    for (int b = 0; b < md.natm; ++b) {
      const double d[3] = {R[3 * a] - R[3 * b], R[3 * a + 1] - R[3 * b + 1], R[3 * a + 2] - R[3 * b + 2]};
      const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
      if (b == a || r2 == 0.0) continue;
      const double f = (double)Z[a] * Z[b] / (r2 * sqrt(r2));
      for (int x = 0; x < 3; ++x) g[x] -= f * d[x];
    }
    for (int x = 0; x < 3; ++x) atomicAdd(grad + 3ll * (md.atm_off + a) + x, g[x]);
  }
}

// resident CTAs of 4 warps, tasks strided over them
static unsigned b2gs_grid(long long ntask) { return (unsigned)std::min<long long>((ntask + 3) / 4, 148ll * 8); }

template <int C>
static int b2gs_launch_2e(const B2PlanDev &P, const double *D, double hyb, double *grad, cudaStream_t st) {
  constexpr int TB = C < 3 ? 2 : (C < 5 ? 1 : 0), TK = C == 0 ? 2 : (C == 1 || C == 3 ? 1 : 0);
  const long long n = P.su.n_task[B2_SU_GRAD + C];
  if (n > 0) {
    const size_t smem = sizeof(double) * B2GS_TABLE + 4 * sizeof(B2gsWarp);
    B2_CUDA_TRY(cudaFuncSetAttribute(k_grad_sp<TB, TK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_grad_sp<TB, TK><<<b2gs_grid(n), 128, smem, st>>>(P.su.off + (B2_SU_GRAD + C) * (P.h.nmol + 1ll), P.h.nmol,
                                                       P.su.mol, P.mols, P.su.su, P.su.pr64, P.su.pn, P.boys, D, hyb,
                                                       grad);
    b2_count_launches(1);
  }
  return B2_OK;
}

// the six two-electron classes and the one-electron part side by side on the plan's streams
// (forked from and joined back to `st`): every kernel adds to grad with atomics
static int b2gs_launch(const B2PlanDev &P, int parts, double hyb, const double *D,
                       const double *W, double *grad, cudaStream_t st) {
  const bool fork = P.bkt_stream[0] != nullptr;
  cudaStream_t s[B2_NBKT];
  if (fork) B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[B2_NBKT], st));
  for (int b = 0; b < B2_NBKT; ++b) {
    s[b] = fork ? P.bkt_stream[b] : st;
    if (fork) B2_CUDA_TRY(cudaStreamWaitEvent(s[b], P.bkt_ev[B2_NBKT], 0));
  }
  int rc = B2_OK;
  if (parts & 2) {
    rc = b2gs_launch_2e<0>(P, D, hyb, grad, s[0]);
    if (!rc) rc = b2gs_launch_2e<1>(P, D, hyb, grad, s[1]);
    if (!rc) rc = b2gs_launch_2e<3>(P, D, hyb, grad, s[2]);
    if (!rc) rc = b2gs_launch_2e<4>(P, D, hyb, grad, s[3]);
    if (!rc) rc = b2gs_launch_2e<2>(P, D, hyb, grad, s[4]);
    if (!rc) rc = b2gs_launch_2e<5>(P, D, hyb, grad, s[2]);
  }
  const long long n1 = P.su.n_task[B2_SU_GRAD1];
  if (!rc && (parts & 1) && n1 > 0) {
    k_grad_1e<<<b2gs_grid(n1), 128, sizeof(double) * B2GS_TABLE, s[0]>>>(
        P.su.off + B2_SU_GRAD1 * (P.h.nmol + 1ll), P.h.nmol, P.su.mol, P.mols, P.su.su, P.su.pr64, P.su.pn, P.atom_xyz,
        P.atom_z, P.boys, D, W, grad);
    b2_count_launches(1);
  }
  if (fork)
    for (int b = 0; b < B2_NBKT; ++b) {
      cudaEventRecord(P.bkt_ev[b], s[b]);
      cudaStreamWaitEvent(st, P.bkt_ev[b], 0);
    }
  if (!rc) B2_CUDA_TRY(cudaGetLastError());
  return rc;
}

// one launch per orbital bucket that holds molecules, on the bucket streams; CTAs of other buckets'
// molecules return at once
template <int Q>
static int b2g_launch_xc(const B2PlanDev &P, const double *coords, const double *weights, const double *D, double *grad,
                         cudaStream_t st) {
  if (P.bkt_off_h[Q] > P.bkt_off_h[Q - 1]) {
    const cudaStream_t s = P.bkt_stream[Q - 1];
    B2_CUDA_TRY(cudaStreamWaitEvent(s, P.bkt_ev[B2_NBKT], 0));
    B2_CUDA_TRY(cudaFuncSetAttribute(k_grad_xc<Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B2Xf<Q>::SMEM));
    k_grad_xc<Q><<<(unsigned)P.g.n_xblk64, 256, B2Xf<Q>::SMEM, s>>>(P.mols, P.su.mol, P.su.su, P.g.xblk64, P.g.grid_off,
                                                                    P.h.nmol, P.g.tpc64, coords, weights, D, grad);
    b2_count_launches(1);
    B2_CUDA_TRY(cudaGetLastError());
    B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[Q - 1], s));
    B2_CUDA_TRY(cudaStreamWaitEvent(st, P.bkt_ev[Q - 1], 0));
  }
  if constexpr (Q > 1) return b2g_launch_xc<Q - 1>(P, coords, weights, D, grad, st);
  return B2_OK;
}

int b2_launch_grad(B2PlanDev &P, int parts, double hyb, const double *C, const double *mo_energy,
                   const double *coords, const double *weights, double *D, double *W, double *grad,
                   cudaStream_t st) {
  if (!D || !W || !grad || (parts & ~15)) return B2_ERR_ARG;
  if ((parts & 4) && (!coords || !weights || !P.g.grid_off)) return B2_ERR_ARG;
  const int nmol = P.h.nmol;
  B2_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(double) * 3 * std::max(1, P.h.n_atm), st));
  if (nmol == 0) return B2_OK;
  if (C) {
    if (!mo_energy) return B2_ERR_ARG;
    k_grad_dm<<<nmol, 256, 0, st>>>(P.mols, C, mo_energy, D, W);
    b2_count_launches(1);
  }
  if (parts & 3) {
    const int rc = b2gs_launch(P, parts, hyb, D, W, grad, st);
    if (rc) return rc;
  }
  if ((parts & 4) && P.g.n_xblk64 > 0) {
    if (P.g.n_xblk64 >= (1ll << 31)) return B2_ERR_SIZE;
    B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[B2_NBKT], st));
    const int rc = b2g_launch_xc<B2_NBKT>(P, coords, weights, D, grad, st);
    if (rc) return rc;
  }
  if (parts & 8) {
    k_grad_nuc<<<nmol, 128, 0, st>>>(P.mols, P.atom_xyz, P.atom_z, grad);
    b2_count_launches(1);
  }
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}
