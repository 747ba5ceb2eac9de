// Exchange-correlation without a stored AO tensor (sm_100a).
//
// Same result as b2_xc (exchange_correlation, nanoDFT.py:105-123) but the AO values and
// gradients of each tile of points are generated in shared memory from the basis (the
// reference evaluates them once on the host with eval_gto, dft.py:220, and streams the
// (4, G, N) tensor every iteration).  Per tile of PT points:
//   AO, dAO/dx,y,z  -> shared memory            (thread per (point, shell))
//   X = AO0 D       -> registers                (thread (tx,ty): points ty+16r, orbitals tx+16q)
//   rho_c = sum_n X AO_c                        (shuffle reduction over the 16 tx lanes)
//   B3LYP per point -> rt = [vrho/2, 4 vgamma rho_1..3] * w
//   Y = sum_c AO_c rt_c, V += AO0^T Y            (registers across the CTA's tiles)
// The orbital dimension is padded to the molecule's bucket NB = 16*Q (Q = 1..5), a
// compile-time choice per CTA, so small molecules do not pay for nao = 70.  float64 runs k_xc_f64
// (matrix instructions), float32 on request k_xc_direct (CUDA cores).
#include "device_plan.cuh"
#include "xc_math.cuh"
#include "xc.cuh"
#include "xc_f64.cuh"

#define B2_XD_MAXSH 48

template <typename T, int PT, int Q>
__device__ __forceinline__ void b2_xd_body(const B2MolDev &md, const B2Shell *sh, T *sD, T *sA,
                                           T (*sRt)[4], double *sC, const double *__restrict__ coords,
                                           const double *__restrict__ w, long long G, long long t0,
                                           int tpc, double *__restrict__ V, double &e_part) {
  constexpr int R = PT / 16, NB = 16 * Q, LD = NB + 1;
  const int N = md.nao, nbas = md.nbas;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  T vacc[Q][Q];
#pragma unroll
  for (int r = 0; r < Q; ++r)
#pragma unroll
    for (int q = 0; q < Q; ++q) vacc[r][q] = (T)0;
  for (int tt = 0; tt < tpc; ++tt) {
    const long long g0 = (t0 + tt) * PT;
    if (g0 >= G) break;
    const int np = (int)min((long long)PT, G - g0);
    __syncthreads();                                   // previous tile consumed
    for (int e = threadIdx.x; e < PT * 3; e += blockDim.x) {
      const int p = e / 3, d = e - (e / 3) * 3;
      sC[e] = (p < np) ? coords[3 * (g0 + p) + d] : 1e30;
    }
    for (int e = threadIdx.x; e < 4 * PT * NB; e += blockDim.x) {   // clear (pads stay zero)
      const int cp = e / NB, n = e - (e / NB) * NB;
      sA[cp * LD + n] = (T)0;
    }
    __syncthreads();
    // AO values + gradients
    for (int e = threadIdx.x; e < PT * nbas; e += blockDim.x) {
      const int p = e / nbas, s = e - (e / nbas) * nbas;
      if (p >= np) continue;
      const B2Shell &S = sh[s];
      const T dx = (T)(sC[3 * p] - S.R[0]), dy = (T)(sC[3 * p + 1] - S.R[1]), dz = (T)(sC[3 * p + 2] - S.R[2]);
      const T r2 = dx * dx + dy * dy + dz * dz;
      T ga = 0, gb = 0;
      for (int k = 0; k < S.nprim; ++k) {
        const T ax = (T)S.exp[k] * r2;
        if (ax > (T)60) continue;
        const T ev = (T)S.coef[k] * exp(-ax);
        ga += ev;
        gb += (T)(-2.0 * S.exp[k]) * ev;
      }
      if (S.l == 0) {
        sA[(0 * PT + p) * LD + S.ao0] = ga;
        sA[(1 * PT + p) * LD + S.ao0] = gb * dx;
        sA[(2 * PT + p) * LD + S.ao0] = gb * dy;
        sA[(3 * PT + p) * LD + S.ao0] = gb * dz;
      } else {
        const T dd[3] = {dx, dy, dz};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          sA[(0 * PT + p) * LD + S.ao0 + c] = dd[c] * ga;
#pragma unroll
          for (int k = 0; k < 3; ++k)
            sA[((1 + k) * PT + p) * LD + S.ao0 + c] = (c == k ? ga : (T)0) + dd[c] * dd[k] * gb;
        }
      }
    }
    __syncthreads();
    // X = AO0 * D
    T x[R][Q];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int q = 0; q < Q; ++q) x[r][q] = (T)0;
    for (int k = 0; k < N; ++k) {
      T a[R], d[Q];
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = sA[(ty + 16 * r) * LD + k];
#pragma unroll
      for (int q = 0; q < Q; ++q) d[q] = sD[k * NB + tx + 16 * q];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < Q; ++q) x[r][q] += a[r] * d[q];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int p = ty + 16 * r;
      T rc[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        T s = 0;
#pragma unroll
        for (int q = 0; q < Q; ++q) s += x[r][q] * sA[(c * PT + p) * LD + tx + 16 * q];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        rc[c] = s;
      }
      if (tx == 0) {
        T rt0 = 0, f4 = 0;
        if (p < np) {
          const B2XcPoint<T> o = b2_b3lyp_point<T>(rc[0], rc[1], rc[2], rc[3]);
          const double wg = w[g0 + p];
          e_part += (double)rc[0] * wg * (double)o.exc;
          rt0 = o.vrho * (T)0.5 * (T)wg;
          f4 = (T)4 * o.vgamma * (T)wg;
        }
        sRt[p][0] = rt0;
        sRt[p][1] = f4 * rc[1];
        sRt[p][2] = f4 * rc[2];
        sRt[p][3] = f4 * rc[3];
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < PT * NB; e += blockDim.x) {
      const int p = e / NB, n = e - (e / NB) * NB;
      sA[(PT + p) * LD + n] = sA[p * LD + n] * sRt[p][0] + sA[(PT + p) * LD + n] * sRt[p][1] +
                              sA[(2 * PT + p) * LD + n] * sRt[p][2] + sA[(3 * PT + p) * LD + n] * sRt[p][3];
    }
    __syncthreads();
    for (int p = 0; p < np; ++p) {
      T a[Q], y[Q];
#pragma unroll
      for (int r = 0; r < Q; ++r) a[r] = sA[p * LD + ty + 16 * r];
#pragma unroll
      for (int q = 0; q < Q; ++q) y[q] = sA[(PT + p) * LD + tx + 16 * q];
#pragma unroll
      for (int r = 0; r < Q; ++r)
#pragma unroll
        for (int q = 0; q < Q; ++q) vacc[r][q] += a[r] * y[q];
    }
  }
#pragma unroll
  for (int r = 0; r < Q; ++r)
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int a = ty + 16 * r, b = tx + 16 * q;
      if (a < N && b < N && vacc[r][q] != (T)0) atomicAdd(&V[md.mat_off + a * N + b], (double)vacc[r][q]);
    }
}

template <typename T, int PT>
__global__ void __launch_bounds__(256)
k_xc_direct(const B2MolDev *__restrict__ mols, const B2Shell *__restrict__ shells,
            const long long *__restrict__ xblk_off, const long long *__restrict__ grid_off, int nmol,
            int tpc, const int *__restrict__ active, const double *__restrict__ coords,
            const double *__restrict__ w, const double *__restrict__ D, double *__restrict__ V,
            double *__restrict__ exc, const int *__restrict__ mol_map) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ B2Shell sh[B2_XD_MAXSH];
  __shared__ T sRt[PT][4];
  __shared__ double sC[PT * 3];
  __shared__ double red[8];
  const int lo = b2_xf_find(xblk_off, nmol, blockIdx.x);
  const int m = mol_map ? mol_map[lo] : lo;
  if (active && !active[m]) return;
  const B2MolDev md = mols[m];
  const int N = md.nao;
  const int Q = (N + 15) / 16, NB = 16 * Q;
  T *sD = reinterpret_cast<T *>(smem_raw);                  // [NB][NB]
  T *sA = sD + NB * NB;                                      // [4][PT][NB+1]
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
    const int a = e / NB, b = e - (e / NB) * NB;
    sD[e] = (a < N && b < N) ? (T)D[md.mat_off + a * N + b] : (T)0;
  }
  for (int s = threadIdx.x; s < md.nbas; s += blockDim.x) sh[s] = shells[md.sh_off + s];
  const long long G = grid_off[m + 1] - grid_off[m];
  const long long t0 = (blockIdx.x - xblk_off[lo]) * (long long)tpc;
  const double *cm = coords + 3 * grid_off[m];
  const double *wm = w + grid_off[m];
  double e_part = 0;
  switch (Q) {
    case 1: b2_xd_body<T, PT, 1>(md, sh, sD, sA, sRt, sC, cm, wm, G, t0, tpc, V, e_part); break;
    case 2: b2_xd_body<T, PT, 2>(md, sh, sD, sA, sRt, sC, cm, wm, G, t0, tpc, V, e_part); break;
    case 3: b2_xd_body<T, PT, 3>(md, sh, sD, sA, sRt, sC, cm, wm, G, t0, tpc, V, e_part); break;
    case 4: b2_xd_body<T, PT, 4>(md, sh, sD, sA, sRt, sC, cm, wm, G, t0, tpc, V, e_part); break;
    default: b2_xd_body<T, PT, 5>(md, sh, sD, sA, sRt, sC, cm, wm, G, t0, tpc, V, e_part); break;
  }
  for (int o = 16; o > 0; o >>= 1) e_part += __shfl_down_sync(0xffffffffu, e_part, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e_part;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int i = 0; i < 8; ++i) s += red[i];
    atomicAdd(&exc[m], s);
  }
}

// ------------------------------------------------------------------ float64 form
// Per tile of 32 points (xc_f64.cuh): AO values, X = AO0^T D by float64 MMA with rho reduced from
// the accumulators, B3LYP on three warps, Y = sum_c AO_c rt_c over plane 1, V += AO0 Y^T by MMA
// into registers over the CTA's tiles.  One launch per orbital bucket sizes shared memory for
// that bucket (2 CTAs per SM at 64 orbitals, 4 up to 32).
// 272 000 points x 62 orbitals: 1117 us per evaluation with CUDA-core products in one 134 KB CTA
// per SM and the functional on one lane in 16; 610 us with MMA products, one CTA per SM resident
// and every l shell's own exponentials; 436 us before runs of tiles filled the rounds of CTAs, 383 us now.
template <int Q>
__global__ void __launch_bounds__(256, B2_XF_CTAS(Q))
k_xc_f64(const B2MolDev *__restrict__ mols, const B2gsMol *__restrict__ gms, const B2gSuper *__restrict__ su,
         const long long *__restrict__ xblk_off, const long long *__restrict__ grid_off, int nmol, int tpc,
         const int *__restrict__ active, const double *__restrict__ coords, const double *__restrict__ wt,
         const double *__restrict__ D, double *__restrict__ V, double *__restrict__ exc,
         const int *__restrict__ mol_map) {
  using X = B2Xf<Q>;
  constexpr int NB = X::NB, LDD = X::LDD, LDP = B2_XF_LDP, PL = X::PL, NV = (2 * Q * Q + 7) / 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lo = b2_xf_find(xblk_off, nmol, blockIdx.x);
  const int m = mol_map ? mol_map[lo] : lo;
  const B2MolDev md = mols[m];
  const int N = md.nao;
  if ((N + 15) / 16 != Q || (active && !active[m])) return;
  const B2gsMol gm = gms[m];
  double *sD = reinterpret_cast<double *>(smem_raw), *sA = sD + NB * LDD, *sR = sA + 4 * PL, *sF = sR + 16 * 32;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  for (int e = tid; e < NB * LDD; e += 256) {
    const int a = e / LDD, b = e - (e / LDD) * LDD;
    sD[e] = (a < N && b < N) ? D[md.mat_off + a * N + b] : 0.0;
  }
  for (int e = tid; e < 4 * PL; e += 256) sA[e] = 0.0;         // rows beyond N stay zero
  const long long G = grid_off[m + 1] - grid_off[m], t0 = (blockIdx.x - xblk_off[lo]) * (long long)tpc;
  const double *cm = coords + 3 * grid_off[m], *wm = wt + grid_off[m];
  const int n8 = (N + 7) >> 3, m16 = (n8 + 1) >> 1, per = (m16 * n8 + 7) >> 3;
  double vacc[NV][4];
#pragma unroll
  for (int j = 0; j < NV; ++j) vacc[j][0] = vacc[j][1] = vacc[j][2] = vacc[j][3] = 0.0;
  double e_part = 0.0;
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
    b2_xf_ao<PL>(su + gm.su_off, gm.ns + gm.np, pt, px, py, pz, sA);
    __syncthreads();
    {
      double x[X::NX][4];
      b2_xf_mm<Q>(sA, sD, n8, x);
      b2_xf_rho<Q>(sA, n8, x, sR);
    }
    B2XfPoint f;
    b2_xf_func(sR, sF, f);
    {
      if (w == 0 && pt) e_part += f.rho[0] * wg * f.exc;
      const double f4 = 4.0 * f.vgamma * wg;                   // points beyond the grid add nothing
      const double rt0 = pt ? f.vrho * 0.5 * wg : 0.0, rt1 = pt ? f4 * f.rho[1] : 0.0, rt2 = pt ? f4 * f.rho[2] : 0.0,
                   rt3 = pt ? f4 * f.rho[3] : 0.0;
      for (int n = w; n < 8 * n8; n += 8) {
        double *o = sA + n * LDP + lane;
        o[PL] = o[0] * rt0 + o[PL] * rt1 + o[2 * PL] * rt2 + o[3 * PL] * rt3;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 8) {
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const int i = w * per + j;
        if (j < per && i < m16 * n8) {
          const int mi = i / n8, ni = i - (i / n8) * n8;
          const double *oa = sA + (16 * mi + g) * LDP + k0 + t, *ob = sA + PL + (8 * ni + g) * LDP + k0 + t;
          const double a[4] = {oa[0], oa[8 * LDP], oa[4], oa[8 * LDP + 4]};
          const double b[2] = {ob[0], ob[4]};
          b2_dmma(vacc[j], a, b);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = w * per + j;
    if (j < per && i < m16 * n8) {
      const int mi = i / n8, ni = i - (i / n8) * n8;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int a = 16 * mi + g + 8 * (c >> 1), b = 8 * ni + 2 * t + (c & 1);
        if (a < N && b < N && vacc[j][c] != 0.0) atomicAdd(&V[md.mat_off + a * N + b], vacc[j][c]);
      }
    }
  }
  if (w == 0) {
    for (int o = 16; o > 0; o >>= 1) e_part += __shfl_down_sync(0xffffffffu, e_part, o);
    if (lane == 0) atomicAdd(&exc[m], e_part);
  }
}

// V and E_xc of the active molecules (all without a mask) <- 0
__global__ void k_zero_xc(const B2MolDev *__restrict__ mols, const int *__restrict__ active,
                          double *__restrict__ V, double *__restrict__ exc) {
  const int m = blockIdx.x;
  if (active && !active[m]) return;
  const B2MolDev md = mols[m];
  for (int e = threadIdx.x; e < md.nao * md.nao; e += blockDim.x) V[md.mat_off + e] = 0.0;
  if (threadIdx.x == 0) exc[m] = 0.0;
}

__global__ void k_sym2(const B2MolDev *__restrict__ mols, const int *__restrict__ active,
                       double *__restrict__ V) {
  if (active && !active[blockIdx.x]) return;
  const B2MolDev md = mols[blockIdx.x];
  const int N = md.nao;
  double *v = V + md.mat_off;
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int a = e / N, b = e - (e / N) * N;
    if (a < b) {
      const double s = v[a * N + b] + v[b * N + a];
      v[a * N + b] = s;
      v[b * N + a] = s;
    } else if (a == b) {
      v[e] *= 2.0;
    }
  }
}

int b2_zero_xc(const B2PlanDev &P, const int *active, double *V, double *exc, cudaStream_t st) {
  k_zero_xc<<<P.h.nmol, 256, 0, st>>>(P.mols, active, V, exc);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}
int b2_sym_v(const B2PlanDev &P, const int *active, double *V, cudaStream_t st) {
  k_sym2<<<P.h.nmol, 256, 0, st>>>(P.mols, active, V);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

// one float64 launch per orbital bucket that holds molecules (largest first), on the bucket
// streams forked from and joined back to `st`; every launch covers all CTAs, and those of other
// buckets' molecules return at once
template <int Q>
static int b2_xf_bucket(const B2PlanDev &P, bool one, const int *active, const double *coords, const double *w,
                        const double *D, double *V, double *exc, cudaStream_t st) {
  const bool sub = P.sub.n > 0;
  const std::vector<int> &off = sub ? P.sub.bkt_off_h : P.bkt_off_h;
  const long long nblk = sub ? P.sub.n_x64 : P.g.n_xblk64;
  if (off[Q] > off[Q - 1] && nblk > 0) {
    const cudaStream_t s = one ? st : P.bkt_stream[Q - 1];
    if (!one) B2_CUDA_TRY(cudaStreamWaitEvent(s, P.bkt_ev[B2_NBKT], 0));
    B2_CUDA_TRY(cudaFuncSetAttribute(k_xc_f64<Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B2Xf<Q>::SMEM));
    k_xc_f64<Q><<<(unsigned)nblk, 256, B2Xf<Q>::SMEM, s>>>(
        P.mols, P.su.mol, P.su.su, sub ? P.sub.x64 : P.g.xblk64, P.g.grid_off, sub ? P.sub.n : P.h.nmol, P.g.tpc64, active,
        coords, w, D, V, exc, sub ? P.sub.mol_map : nullptr);
    b2_count_launches(1);
    B2_CUDA_TRY(cudaGetLastError());
    if (!one) {
      B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[Q - 1], s));
      B2_CUDA_TRY(cudaStreamWaitEvent(st, P.bkt_ev[Q - 1], 0));
    }
  }
  if constexpr (Q > 1) return b2_xf_bucket<Q - 1>(P, one, active, coords, w, D, V, exc, st);
  return B2_OK;
}

// the shell limit is k_xc_direct's table; the float64 kernel keeps none, but accepts the same molecules
static int b2_xcd_zero(const B2PlanDev &P, const int *active, double *V, double *exc, cudaStream_t st) {
  if (P.h.max_nbas > B2_XD_MAXSH) return B2_ERR_SIZE;
  return b2_zero_xc(P, active, V, exc, st);
}

static int b2_xc_f64(const B2PlanDev &P, const int *active, const double *coords, const double *w, const double *D,
                     double *V, double *exc, cudaStream_t st, bool sym) {
  int rc = b2_xcd_zero(P, active, V, exc, st);
  if (rc) return rc;
  const std::vector<int> &off = P.sub.n > 0 ? P.sub.bkt_off_h : P.bkt_off_h;
  int used = 0;
  for (int b = 0; b < B2_NBKT; ++b) used += off[b + 1] > off[b];
  if (used > 1) B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[B2_NBKT], st));
  rc = b2_xf_bucket<B2_NBKT>(P, used <= 1, active, coords, w, D, V, exc, st);
  return rc || !sym ? rc : b2_sym_v(P, active, V, st);
}

// float32 on the CUDA cores (implementation 1)
static int b2_xcd_f32(const B2PlanDev &P, const int *active, const double *coords, const double *w, const double *D,
                      double *V, double *exc, cudaStream_t st, bool sym) {
  constexpr int PT = 64, NBmax = 80;
  const bool sub = P.sub.n > 0;
  const long long nblk = sub ? P.sub.n_x32 : P.g.n_xblk32;
  const int rc = b2_xcd_zero(P, active, V, exc, st);
  if (rc) return rc;
  const size_t sm = sizeof(float) * (NBmax * NBmax + 4 * PT * (NBmax + 1));
  B2_CUDA_TRY(cudaFuncSetAttribute(k_xc_direct<float, PT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  if (nblk > 0) {
    k_xc_direct<float, PT><<<(unsigned)nblk, 256, sm, st>>>(
        P.mols, P.shells, sub ? P.sub.x32 : P.g.xblk32, P.g.grid_off, sub ? P.sub.n : P.h.nmol, P.g.tpc32, active,
        coords, w, D, V, exc, sub ? P.sub.mol_map : nullptr);
    b2_count_launches(1);
    B2_CUDA_TRY(cudaGetLastError());
  }
  return sym ? b2_sym_v(P, active, V, st) : B2_OK;
}

int b2_launch_xc_direct(const B2PlanDev &P, int precision, const int *active, const double *coords,
                        const double *w, const double *D, double *V, double *exc, cudaStream_t st,
                        bool sym) {
  if (!P.g.grid_off) return B2_ERR_ARG;
  if (precision == 64) return b2_xc_f64(P, active, coords, w, D, V, exc, st, sym);
  if (precision == 32 && P.xc_impl == 0)
    return b2_launch_xc_tq(P, active, coords, w, D, V, exc, st, sym);
  if (precision == 32 && P.xc_impl == 2)
    return b2_launch_xc_tc(P, active, coords, w, D, V, exc, st, sym);
  if (precision == 32) return b2_xcd_f32(P, active, coords, w, D, V, exc, st, sym);
  return B2_ERR_ARG;
}
