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
//   k_grad_xc   d/dR of E_xc at fixed density and grid (V_xc, nanoDFT.py:408-415): one CTA per
//               32 grid points of one molecule, AO values, D-products and B3LYP staged in
//               shared memory;
//   k_grad_nuc  nuclear repulsion (grad_nuc, nanoDFT.py:428-438).
//
// The per-term math is grad_sp.cuh and grad_math.cuh, the same code the host-check build tests
// against the finite-difference oracle.
#include <algorithm>
#include <vector>
#include "device_plan.cuh"
#include "devmem.cuh"
#include "grad_math.cuh"
#include "grad_sp.cuh"

#define B2G_TP 32                  // grid points per XC tile (one warp's lanes)
#define B2G_XC_THREADS 256

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
// 160 uneven molecules takes 31 ms, of one molecule with 5 heavy atoms 0.26 ms.  Before (one warp
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

// Exchange-correlation part on 32 grid points of one molecule (tile t of molecule m, tile_off:
// per-molecule tile prefix).  With phi the AO values and u = D phi, U_k = D d_k phi:
//   rho = phi.u, grad rho = 2 (d phi).u, and moving atom A moves its orbitals, so
//   dE/dR_A,x = -2 sum_g w sum_{i on A} [vrho d_x phi_i u_i
//                                        + 2 vgamma sum_k g_k (d_x d_k phi_i u_i + d_x phi_i U_k,i)].
// Shared memory: D (N x N), phi and its gradient (4 x N x 32), u and U (4 x N x 32), the
// points' weighted vrho / vgamma and grad rho, and the molecule's atom sums.
__host__ __device__ inline long long b2g_xc_smem_doubles(int N, int natm) {
  return (long long)N * N + 8ll * N * B2G_TP + 5 * B2G_TP + 3ll * natm;
}

__global__ void __launch_bounds__(B2G_XC_THREADS)
k_grad_xc(const B2MolDev *__restrict__ mols, int nmol, const B2Shell *__restrict__ shells,
          const long long *__restrict__ grid_off, const long long *__restrict__ tile_off,
          const double *__restrict__ coords, const double *__restrict__ weights, const double *__restrict__ D,
          double *__restrict__ grad) {
  extern __shared__ double sm[];
  const long long bt = blockIdx.x;
  int lo = 0, hi = nmol - 1;                      // molecule: last m with tile_off[m] <= bt
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_off[mid] <= bt) lo = mid; else hi = mid - 1;
  }
  const int m = lo;
  const B2MolDev md = mols[m];
  const int N = md.nao, nbas = md.nbas, natm = md.natm;
  const long long p0 = grid_off[m] + (bt - tile_off[m]) * B2G_TP;
  const int np = (int)min((long long)B2G_TP, grid_off[m + 1] - p0);
  double *sD = sm;
  double *phi = sD + N * N;                       // [4][N][TP]
  double *u = phi + 4 * N * B2G_TP;               // [4][N][TP]
  double *vr = u + 4 * N * B2G_TP, *vg = vr + B2G_TP, *gr = vg + B2G_TP;   // gr [3][TP]
  double *sG = gr + 3 * B2G_TP;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < N * N; e += blockDim.x) sD[e] = D[md.mat_off + e];
  for (int e = tid; e < 3 * natm; e += blockDim.x) sG[e] = 0.0;
  // AO values and gradients; item = shell * 32 + point, so a warp shares one shell
  for (int it = tid; it < nbas * B2G_TP; it += blockDim.x) {
    const int s = it / B2G_TP, p = it - s * B2G_TP;
    const B2Shell &S = shells[md.sh_off + s];
    double f[3] = {0, 0, 0}, df[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, hf[3][6];
    if (p < np) b2g_ao2<double>(S, coords + 3 * (p0 + p), f, df, hf);
    for (int c = 0; c < 2 * S.l + 1; ++c) {
      const int i = S.ao0 + c;
      phi[i * B2G_TP + p] = f[c];
      for (int x = 0; x < 3; ++x) phi[((1 + x) * N + i) * B2G_TP + p] = df[c][x];
    }
  }
  __syncthreads();
  for (int it = tid; it < N * B2G_TP; it += blockDim.x) {
    const int i = it / B2G_TP, p = it - i * B2G_TP;
    double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
    for (int j = 0; j < N; ++j) {
      const double dij = sD[i * N + j];
      s0 += dij * phi[j * B2G_TP + p];
      s1 += dij * phi[(N + j) * B2G_TP + p];
      s2 += dij * phi[(2 * N + j) * B2G_TP + p];
      s3 += dij * phi[(3 * N + j) * B2G_TP + p];
    }
    u[i * B2G_TP + p] = s0;
    u[(N + i) * B2G_TP + p] = s1;
    u[(2 * N + i) * B2G_TP + p] = s2;
    u[(3 * N + i) * B2G_TP + p] = s3;
  }
  __syncthreads();
  if (tid < B2G_TP) {
    const int p = tid;
    double rho = 0, r1[3] = {0, 0, 0};
    for (int i = 0; i < N; ++i) {
      const double ui = u[i * B2G_TP + p];
      rho += phi[i * B2G_TP + p] * ui;
      for (int x = 0; x < 3; ++x) r1[x] += phi[((1 + x) * N + i) * B2G_TP + p] * ui;
    }
    double a = 0, b = 0;
    if (p < np) {
      const B2XcPoint<double> o = b2_b3lyp_point<double>(rho, r1[0], r1[1], r1[2]);
      const double wt = weights[p0 + p];
      a = wt * o.vrho;
      b = wt * o.vgamma;
    }
    vr[p] = a;
    vg[p] = b;
    for (int x = 0; x < 3; ++x) gr[x * B2G_TP + p] = 2.0 * r1[x];
  }
  __syncthreads();
  const int hidx[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  for (int it = tid; it < nbas * B2G_TP; it += blockDim.x) {    // warp-uniform shell
    const int s = it / B2G_TP, p = it - s * B2G_TP;
    const B2Shell &S = shells[md.sh_off + s];
    double acc[3] = {0, 0, 0};
    if (p < np) {
      double f[3], df[3][3], hf[3][6];
      b2g_ao2<double>(S, coords + 3 * (p0 + p), f, df, hf);
      const double a = vr[p], b2 = 2.0 * vg[p];
      const double g0 = gr[p], g1 = gr[B2G_TP + p], g2 = gr[2 * B2G_TP + p];
      for (int c = 0; c < 2 * S.l + 1; ++c) {
        const int i = S.ao0 + c;
        const double u0 = u[i * B2G_TP + p];
        const double uk[3] = {u[(N + i) * B2G_TP + p], u[(2 * N + i) * B2G_TP + p], u[(3 * N + i) * B2G_TP + p]};
        const double gk[3] = {g0, g1, g2};
        for (int x = 0; x < 3; ++x) {
          double q = 0;
          for (int k = 0; k < 3; ++k) q += gk[k] * (hf[c][hidx[x][k]] * u0 + df[c][x] * uk[k]);
          acc[x] += a * df[c][x] * u0 + b2 * q;
        }
      }
    }
    for (int x = 0; x < 3; ++x) {
      double v = acc[x];
#pragma unroll
      for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) atomicAdd(&sG[3 * S.atom + x], -2.0 * v);
    }
  }
  __syncthreads();
  for (int e = tid; e < 3 * natm; e += blockDim.x) atomicAdd(grad + 3ll * md.atm_off + e, sG[e]);
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
  if (parts & 4) {
    std::vector<long long> toff(nmol + 1, 0);
    for (int m = 0; m < nmol; ++m) {
      const long long G = P.g.grid_off_h[m + 1] - P.g.grid_off_h[m];
      toff[m + 1] = toff[m] + (G + B2G_TP - 1) / B2G_TP;
    }
    if (toff[nmol] > 0) {
      if (toff[nmol] >= (1ll << 31)) return B2_ERR_SIZE;
      const size_t smem = sizeof(double) * (size_t)b2g_xc_smem_doubles(P.h.max_nao, P.h.max_natm);
      B2_CUDA_TRY(cudaFuncSetAttribute(k_grad_xc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      long long *dtoff = nullptr;
      B2_CUDA_TRY(b2_dmalloc_t(&dtoff, sizeof(long long) * (nmol + 1), st));
      // pageable source: the call returns once the data is staged, so toff may go out of scope
      cudaError_t e = cudaMemcpyAsync(dtoff, toff.data(), sizeof(long long) * (nmol + 1),
                                      cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) {
        k_grad_xc<<<(unsigned)toff[nmol], B2G_XC_THREADS, smem, st>>>(P.mols, nmol, P.shells, P.g.grid_off,
                                                                       dtoff, coords, weights, D, grad);
        b2_count_launches(1);
        e = cudaGetLastError();
      }
      b2_dfree(dtoff, st);
      if (e != cudaSuccess) return B2_ERR_CUDA;
    }
  }
  if (parts & 8) {
    k_grad_nuc<<<nmol, 128, 0, st>>>(P.mols, P.atom_xyz, P.atom_z, grad);
    b2_count_launches(1);
  }
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}
