// s8 ERI generator kernel (sm_100a).  Replaces the reference's per-quartet IPU vertex
// ``poplar_int2e_sph_forloop`` (int2e_sph.cpp:7180-7254) driven by ``integrals_v1``
// (direct.py:584-707), and writes straight into the tril-of-tril s8 layout of
// ``mol.intor('int2e_sph', aosym='s8')`` (nanoDFT.py:285).
//
// Batch plans: super-shell pairs (super.cuh, eri_su.cuh).  A class is a bra slice type and a ket
// pair type; a warp task is one bra slice x 32 ket pairs of one molecule, found from prefix sums
// of the molecules' task counts (no work list in memory).  The allocation-free single-molecule
// entry at the end of this file keeps the shell-pair kernels k_eri_sq and their host work list.
#include <type_traits>
#include "eri_sq.cuh"
#include "eri_su.cuh"
#include "device_plan.cuh"
#include "devmem.cuh"
#include "eri_flops.h"

template <typename T, int LI, int LJ, int LK, int LL>
__global__ void __launch_bounds__(128)
k_eri_sq(const B2EriTask *__restrict__ tasks, long long ntask, const B2MolDev *__restrict__ mols,
         const B2PairInfo *__restrict__ pinfo, const B2PairPrim<T> *__restrict__ pp,
         const int *__restrict__ cls_list, const T *__restrict__ btab, T *__restrict__ out) {
  __shared__ B2PairPrim<T> sbra[4][B2_MAXPP];
  __shared__ int s_nb[4];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long ti = (long long)blockIdx.x * 4 + w;
  if (ti >= ntask) return;                        // whole warp
  const B2EriTask tk = tasks[ti];
  const B2MolDev md = mols[tk.mol];
  const B2PairInfo bp = pinfo[md.sp_off + tk.IJ];
  if (lane == 0) {
    const B2PairPrim<T> *src = pp + (size_t)(md.sp_off + tk.IJ) * B2_MAXPP;
    int nb = 0;
    for (int x = 0; x < B2_MAXPP; ++x)
      if (src[x].K != (T)0) sbra[w][nb++] = src[x];
    s_nb[w] = nb;
  }
  __syncwarp();
  const int nb = s_nb[w];
  for (int k = lane; k < tk.count; k += 32) {
    const int KL = cls_list[md.sp_off + md.cls_start[tk.cls] + tk.start + k];
    const B2PairInfo kp = pinfo[md.sp_off + KL];
    b2_sq_sub<T, LI, LJ, LK, LL, T>(tk.sub, sbra[w], nb, pp + (size_t)(md.sp_off + KL) * B2_MAXPP,
                                    btab, out + md.eri_off, bp, kp);
  }
}

// ------------------------------------------------------------------ batch plans
template <typename T> struct B2EriPrimOf { using type = B2gPrim; };
template <> struct B2EriPrimOf<float> { using type = B2gPrim32; };
__device__ __forceinline__ int b2_eri_n(const B2gCount &n, const B2gPrim *) { return n.y; }
__device__ __forceinline__ int b2_eri_n(const B2gCount &n, const B2gPrim32 *) { return n.x; }

__device__ __forceinline__ int b2_eri_find(const long long *__restrict__ off, int n, long long x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// one warp task: the bra slice's data and its ket range
struct B2EriTaskSu {
  int m, pair, f, cnt, k0, A, B;
};
template <int TB, int TK>
__device__ __forceinline__ bool b2_eri_task(const long long *__restrict__ toff, int nmol,
                                            const B2gsMol *__restrict__ gms, long long task, B2gsMol &g,
                                            B2EriTaskSu &t) {
  t.m = b2_eri_find(toff, nmol, task);
  g = gms[t.m];
  const int nch = (b2es_npair(g.ns, g.np, TK) + 31) >> 5;
  const int r0 = (int)(task - toff[t.m]), i = r0 / nch;
  int limit;
  b2es_bra_of(g.ns, g.np, TB, TK, i, t.pair, limit);
  t.f = TB == 2 ? i - 3 * (i / 3) : 0;
  t.k0 = (r0 - i * nch) * 32;
  t.cnt = min(32, limit - t.k0);
  if (t.cnt <= 0) return false;
  b2gs_pair(g.ns, g.np, t.pair, t.A, t.B);
  return true;
}

// (ss|ss) pairs: lanes over the chunk's (ket, ket primitive) entries packed by a prefix sum of the
// kets' surviving primitives; each lane sums its entry over the bra's primitives, a same-ket
// segmented scan (segments <= 9 lanes) combines the entries of a ket.  The sums are float64 in the
// float32 form too: this class holds the core integrals, of magnitude 4-9, whose float32 sums were
// the largest errors of the list: 1.06e-6, 2.3e-7 so (2048 molecules, all classes: 36.1 -> 36.5 ms).
template <typename T>
__global__ void __launch_bounds__(128)
k_eri_ss(const long long *__restrict__ toff, int nmol, const B2gsMol *__restrict__ gms,
         const B2MolDev *__restrict__ mols, const B2gSuper *__restrict__ su,
         const typename B2EriPrimOf<T>::type *__restrict__ pr, const B2gCount *__restrict__ pn,
         const T *__restrict__ btab, T *__restrict__ out) {
  using S = B2Es<T, 0, 0>;
  __shared__ B2EriBra<T> sbra[4][B2_MAXPP];
  __shared__ int s_off[4][32];
  __shared__ unsigned char s_map[4][32 * B2_MAXPP];
  __shared__ double s_acc[4][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long ntask = toff[nmol];
  for (long long task = (long long)blockIdx.x * 4 + w; task < ntask; task += (long long)gridDim.x * 4) {
    B2gsMol g;
    B2EriTaskSu t;
    if (!b2_eri_task<0, 0>(toff, nmol, gms, task, g, t)) continue;   // whole warp: beyond the diagonal
    const long long p0 = g.pr_off;
    const int nb = b2_eri_n(pn[p0 + t.pair], pr);
    __syncwarp();                                    // the previous task's shared memory is consumed
    const double zero[3] = {0, 0, 0};
    if (lane < nb) b2es_bra(pr[(p0 + t.pair) * B2_MAXPP + lane], false, 0, zero, sbra[w][lane]);
    const int nq = lane < t.cnt ? b2_eri_n(pn[p0 + t.k0 + lane], pr) : 0;
    int inc = nq;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    const int E = __shfl_sync(0xffffffffu, inc, 31);
    s_off[w][lane] = inc - nq;
    for (int j = 0; j < nq; ++j) s_map[w][inc - nq + j] = (unsigned char)lane;
    s_acc[w][lane] = 0.0;
    __syncwarp();
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const bool valid = e < E;
      const int k = valid ? (int)s_map[w][e] : -1 - lane;   // entries past the end: unique keys
      double a = 0.0;
      if (valid) {
        B2EriKet<T> q;
        b2es_ket(pr[(p0 + t.k0 + k) * B2_MAXPP + (e - s_off[w][k])], 0, zero, q);
        for (int p = 0; p < nb; ++p) {
          T phi[1][1] = {{(T)0}};
          S::quartet(sbra[w][p], q, btab, phi);
          a += (double)phi[0][0];
        }
        a *= (double)q.kss;
      }
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {                     // same-ket inclusive scan
        const int ko = __shfl_up_sync(0xffffffffu, k, o);
        const double y = __shfl_up_sync(0xffffffffu, a, o);
        if (lane >= o && ko == k) a += y;
      }
      const int kn = __shfl_down_sync(0xffffffffu, k, 1);
      if (valid && (lane == 31 || kn != k)) s_acc[w][k] += a;
      __syncwarp();
    }
    if (lane < t.cnt) {
      int c, d;
      b2gs_pair(g.ns, g.np, t.k0 + lane, c, d);
      const B2gSuper *sm = su + g.su_off;
      b2es_put(out + mols[t.m].eri_off, sm[t.A].ao_s, sm[t.B].ao_s, sm[c].ao_s, sm[d].ao_s, t.A == t.B, c == d,
               t.pair == t.k0 + lane, (T)s_acc[w][lane]);
    }
  }
}

// The other classes: a ket pair's primitives are cut into units of four, one per lane of a group of
// four lanes, and the task's units are packed over the warp's eight groups (with whole ket pairs per
// group and as many passes as the longest pair of a pass needs, 19-21 of 32 lanes worked).  A lane
// sums, over the bra's primitives (shared memory), the derivatives Phi of the class (up to 40 values
// in registers).  The ket's polynomial turns them into up to 16 integrals per bra function, which a
// two-step transposing butterfly sums over the group: lane li ends with the integrals of ket function
// li.  A pair's further units (at most three in all) sit in the next groups, or at the next pass's
// start: a segmented scan over groups and a carry combine them, and the pair's last group writes.
// Bound by FP32 issue (float32) and by the chain of a quartet at 8 warps per SM (float64, 242
// registers).  Before: 16 kernels, one per l class over the unmerged shells, every integral
// accumulated per primitive quartet: 2.2 times the quartets, each with its own Boys evaluation.
// All classes and the exchange list, 2048 molecules float32: 67.6 -> 38.2 ms, 36.0 ms with the units
// packed (36.4 ms with the float64 (ss|ss) sums and unbiased Boys values); 50 molecules float64: 5.21 -> 2.06 ms.
template <typename T> struct __align__(16) B2EriWarp {
  B2EriBra<T> bra[B2_MAXPP];
  double CD[32][3];
  int ao[32][4];
  unsigned char n[32], same[32], off[32], map[96];
};
template <typename T, int TB, int TK>
__global__ void __launch_bounds__(128)
k_eri_su(const long long *__restrict__ toff, int nmol, const B2gsMol *__restrict__ gms,
         const B2MolDev *__restrict__ mols, const B2gSuper *__restrict__ su,
         const typename B2EriPrimOf<T>::type *__restrict__ pr, const B2gCount *__restrict__ pn,
         const T *__restrict__ btab, T *__restrict__ out) {
  using S = B2Es<T, TB, TK>;
  constexpr int NB = S::NB, NO = TK == 2 ? 4 : 1;      // integrals a lane ends with per bra function
  extern __shared__ __align__(16) unsigned char es_smem[];
  T *tab = reinterpret_cast<T *>(es_smem);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, qd = lane >> 2, li = lane & 3;
  B2EriWarp<T> &W = reinterpret_cast<B2EriWarp<T> *>(es_smem + sizeof(T) * B2_BOYS_NT * B2_BOYS_NM)[w];
  for (int e = threadIdx.x; e < B2_BOYS_NT * B2_BOYS_NM; e += blockDim.x) tab[e] = btab[e];
  __syncthreads();
  const long long ntask = toff[nmol];
  for (long long task = (long long)blockIdx.x * 4 + w; task < ntask; task += (long long)gridDim.x * 4) {
    B2gsMol g;
    B2EriTaskSu t;
    if (!b2_eri_task<TB, TK>(toff, nmol, gms, task, g, t)) continue;
    const B2gSuper *sm = su + g.su_off;
    const long long p0 = g.pr_off;
    const int nb = b2_eri_n(pn[p0 + t.pair], pr), kf = b2es_first(g.ns, g.np, TK) + t.k0;
    __syncwarp();                                    // the previous task's shared memory is consumed
    if (lane < nb) {
      double AB[3];
#pragma unroll
      for (int x = 0; x < 3; ++x) AB[x] = sm[t.A].R[x] - sm[t.B].R[x];
      b2es_bra(pr[(p0 + t.pair) * B2_MAXPP + lane], TB == 2, t.f, AB, W.bra[lane]);
    }
    int nu = 0;                                      // units of this lane's ket (a pair without primitives has one)
    if (lane < t.cnt) {
      int c, d;
      b2gs_pair(g.ns, g.np, kf + lane, c, d);
      const int n = b2_eri_n(pn[p0 + kf + lane], pr);
      nu = max(1, (n + 3) >> 2);
      W.n[lane] = (unsigned char)n;
      W.same[lane] = (unsigned char)((c == d) + 2 * (t.pair == kf + lane));
      W.ao[lane][0] = sm[c].ao_s; W.ao[lane][1] = sm[c].ao_p; W.ao[lane][2] = sm[d].ao_s; W.ao[lane][3] = sm[d].ao_p;
#pragma unroll
      for (int x = 0; x < 3; ++x) W.CD[lane][x] = sm[c].R[x] - sm[d].R[x];
    }
    int inc = nu;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    const int U = __shfl_sync(0xffffffffu, inc, 31);
    W.off[lane] = (unsigned char)(inc - nu);
    for (int j = 0; j < nu; ++j) W.map[inc - nu + j] = (unsigned char)lane;
    const int F = TB == 2 ? (sm[t.A].ao_p < 0 ? -1 : sm[t.A].ao_p + t.f) : sm[t.A].ao_s;
    const int bs = sm[t.B].ao_s, bp = sm[t.B].ao_p;
    T *o = out + mols[t.m].eri_off;
    __syncwarp();
    auto perm = [&](int x) { return t.f + x >= 3 ? t.f + x - 3 : t.f + x; };
    T carry[NB][NO];
    int kc = -1;                                     // ket of the last pass's last group
#pragma unroll 1
    for (int u0 = 0; u0 < U; u0 += 8) {
      const int u = u0 + qd;
      const int kk = u < U ? (int)W.map[u] : -2 - qd;  // groups past the end: unique keys
      const int sub = kk >= 0 ? u - (int)W.off[kk] : 0, j = 4 * sub + li;
      const bool act = kk >= 0 && j < (int)W.n[max(kk, 0)];
      T acc[NB][NO];
      {
        T phi[NB][S::NP];
        S::zero(phi);
        B2EriKet<T> q;
        if (act) {
          b2es_ket(pr[(p0 + kf + kk) * B2_MAXPP + j], t.f, W.CD[kk], q);
#pragma unroll 1
          for (int p = 0; p < nb; ++p) S::quartet(W.bra[p], q, tab, phi);
        }
        const bool hi = li & 2, od = li & 1;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          T v[S::NK];
#pragma unroll
          for (int e = 0; e < S::NK; ++e) v[e] = (T)0;
          if (act) S::ket(q, phi[b], v);
          T h[S::NK / 2];
#pragma unroll
          for (int e = 0; e < S::NK / 2; ++e) {
            const T keep = hi ? v[S::NK / 2 + e] : v[e];
            h[e] = keep + __shfl_xor_sync(0xffffffffu, hi ? v[e] : v[S::NK / 2 + e], 2);
          }
#pragma unroll
          for (int e = 0; e < NO; ++e) {
            const T keep = od ? h[NO + e] : h[e];
            acc[b][e] = keep + __shfl_xor_sync(0xffffffffu, od ? h[e] : h[NO + e], 1);
          }
        }
      }
      // the carry, then an inclusive scan over the groups of one ket (at most three)
      const bool cont = qd == 0 && kk == kc;
      const bool s1 = __shfl_up_sync(0xffffffffu, kk, 4) == kk && qd >= 1;
      const bool s2 = __shfl_up_sync(0xffffffffu, kk, 8) == kk && qd >= 2;
      if (__any_sync(0xffffffffu, cont || s1)) {
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
          for (int e = 0; e < NO; ++e) {
            if (cont) acc[b][e] += carry[b][e];
            const T y = __shfl_up_sync(0xffffffffu, acc[b][e], 4);
            if (s1) acc[b][e] += y;
            const T z = __shfl_up_sync(0xffffffffu, acc[b][e], 8);
            if (s2) acc[b][e] += z;
          }
      }
      const bool last = kk >= 0 && 4 * (sub + 1) >= (int)W.n[max(kk, 0)];
      kc = __shfl_sync(0xffffffffu, last ? -1 : kk, 28);   // a ket that goes on in the next pass
      if (kc >= 0) {
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
          for (int e = 0; e < NO; ++e) carry[b][e] = __shfl_sync(0xffffffffu, acc[b][e], 28 + li);
      }
      if (last) {
        const int cs = W.ao[kk][0], cp = W.ao[kk][1], ds = W.ao[kk][2], dp = W.ao[kk][3];
        const bool same2 = W.same[kk] & 1, same = W.same[kk] & 2;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const int jb = b == 0 ? bs : (bp < 0 ? -1 : bp + perm(b - 1));
          if constexpr (TK == 1) {
            const int l = li == 0 ? ds : (dp < 0 ? -1 : dp + perm(li - 1));
            b2es_put(o, F, jb, cs, l, t.A == t.B, same2, same, acc[b][0]);
          } else {
            const int k = li == 0 ? cs : (cp < 0 ? -1 : cp + perm(li - 1));
#pragma unroll
            for (int d = 0; d < 4; ++d) {
              const int l = d == 0 ? ds : (dp < 0 ? -1 : dp + perm(d - 1));
              b2es_put(o, F, jb, k, l, t.A == t.B, same2, same, acc[b][d]);
            }
          }
        }
      }
    }
  }
}

template <typename T> static const T *b2_boys_table(const B2PlanDev &P);
template <> const double *b2_boys_table<double>(const B2PlanDev &P) { return P.boys; }
template <> const float *b2_boys_table<float>(const B2PlanDev &P) { return P.boys32; }

template <typename T, int LI, int LJ, int LK, int LL>
static void b2_eri_group(const B2PlanDev &P, const B2EriTask *tasks, long long n,
                         const B2PairPrim<T> *pp, T *out, cudaStream_t st) {
  const long long maxg = 4 * ((1ll << 31) - 1);    // 4 tasks (one per warp) per CTA
  for (long long t0 = 0; t0 < n; t0 += maxg) {
    const long long nt = std::min(maxg, n - t0);
    k_eri_sq<T, LI, LJ, LK, LL><<<(unsigned)((nt + 3) / 4), 128, 0, st>>>(
        tasks + t0, nt, P.mols, P.pinfo, pp, P.cls_list, b2_boys_table<T>(P), out);
    b2_count_launches(1);
  }
}

// The six class kernels write disjoint entries of the s8 lists, so they run side by side on the
// plan's bucket streams (forked from and joined back to `st` with events), the largest first.
template <typename T, int TB, int TK>
static int b2_eri_class(const B2PlanDev &P, int cls, const typename B2EriPrimOf<T>::type *pr, T *out, cudaStream_t st) {
  const long long n = P.su.n_task[cls];
  if (n <= 0) return B2_OK;
  const unsigned nb = (unsigned)std::min<long long>((n + 3) / 4, 148ll * 8);
  const long long *off = P.su.off + cls * (P.h.nmol + 1ll);
  if constexpr (TB == 0 && TK == 0) {
    k_eri_ss<T><<<nb, 128, 0, st>>>(off, P.h.nmol, P.su.mol, P.mols, P.su.su, pr, P.su.pn, b2_boys_table<T>(P), out);
  } else {
    const size_t sm = sizeof(T) * B2_BOYS_NT * B2_BOYS_NM + 4 * sizeof(B2EriWarp<T>);
    B2_CUDA_TRY(cudaFuncSetAttribute(k_eri_su<T, TB, TK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_eri_su<T, TB, TK><<<nb, 128, sm, st>>>(off, P.h.nmol, P.su.mol, P.mols, P.su.su, pr, P.su.pn,
                                             b2_boys_table<T>(P), out);
  }
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

template <typename T>
static int b2_eri_all(const B2PlanDev &P, const typename B2EriPrimOf<T>::type *pr, T *out, cudaStream_t st) {
  cudaStream_t s[B2_NBKT];
  const bool fork = P.bkt_stream[0] != nullptr;
  if (fork) B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[B2_NBKT], st));
  for (int b = 0; b < B2_NBKT; ++b) {
    s[b] = fork ? P.bkt_stream[b] : st;
    if (fork) B2_CUDA_TRY(cudaStreamWaitEvent(s[b], P.bkt_ev[B2_NBKT], 0));
  }
  int rc = b2_eri_class<T, 1, 2>(P, 4, pr, out, s[0]);
  if (!rc) rc = b2_eri_class<T, 0, 1>(P, 1, pr, out, s[1]);
  if (!rc) rc = b2_eri_class<T, 1, 1>(P, 2, pr, out, s[2]);
  if (!rc) rc = b2_eri_class<T, 0, 0>(P, 0, pr, out, s[3]);
  if (!rc) rc = b2_eri_class<T, 2, 2>(P, 5, pr, out, s[4]);
  if (!rc) rc = b2_eri_class<T, 0, 2>(P, 3, pr, out, s[4]);
  if (fork)
    for (int b = 0; b < B2_NBKT; ++b) {
      cudaEventRecord(P.bkt_ev[b], s[b]);
      cudaStreamWaitEvent(st, P.bkt_ev[b], 0);
    }
  return rc;
}

int b2_launch_eri_s8(B2PlanDev &P, int precision, void *out, cudaStream_t st) {
  if (precision == 64) return b2_eri_all<double>(P, P.su.pr64, (double *)out, st);
  if (precision == 32) return b2_eri_all<float>(P, P.su.pr32, (float *)out, st);
  return B2_ERR_ARG;
}

// ------------------------------------------------------------------ super-shell tables
// primitive pairs of every super-shell pair, one thread per pair
__global__ void __launch_bounds__(128)
k_su_prims(const B2gsMol *__restrict__ gm, const long long *__restrict__ poff, int nmol,
           const B2gSuper *__restrict__ su, B2gPrim *__restrict__ pr64, B2gPrim32 *__restrict__ pr32,
           B2gCount *__restrict__ pn) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= poff[nmol]) return;
  const int m = b2_eri_find(poff, nmol, t);
  const B2gsMol g = gm[m];
  int A, B;
  b2gs_pair(g.ns, g.np, (int)(t - g.pr_off), A, B);
  pn[t] = b2gs_pair_prims(su[g.su_off + A], su[g.su_off + B], pr64 + t * B2_MAXPP, pr32 + t * B2_MAXPP);
}

// host tables: super shells, molecules, and the prefixes over molecules of the tasks of the six
// integral classes, of the pairs, of the six gradient classes' tasks and of the one-electron
// gradient's slices
static const int b2_eri_tb[6] = {0, 0, 1, 0, 1, 2}, b2_eri_tk[6] = {0, 1, 1, 2, 2, 2};

void b2_su_host(const B2PlanHost &h, std::vector<B2gSuper> &su, std::vector<B2gsMol> &gm,
                std::vector<long long> &off) {
  const int nmol = h.nmol;
  gm.resize(nmol);
  off.assign((size_t)B2_SU_NOFF * (nmol + 1), 0);
  su.clear();
  su.reserve(h.n_sh);
  std::vector<B2gSuper> tmp(std::max(1, h.max_nbas));
  for (int m = 0; m < nmol; ++m) {
    const B2MolDev &md = h.mols[m];
    int nt = 0;
    const int ns = b2gs_supers(h.shells.data() + md.sh_off, md.nbas, tmp.data(), &nt), np = nt - ns;
    auto add = [&](int k, long long n) {
      long long *o = off.data() + k * (nmol + 1ll) + m;
      o[1] = o[0] + n;
      return o[0];
    };
    for (int c = 0; c < 6; ++c)
      add(c, (long long)b2es_nbra(ns, np, b2_eri_tb[c], b2_eri_tk[c]) * ((b2es_npair(ns, np, b2_eri_tk[c]) + 31) / 32));
    const long long pr0 = add(B2_SU_PAIRS, b2gs_npair(ns, np));
    for (int c = 0; c < 6; ++c)
      add(B2_SU_GRAD + c, (long long)b2gs_nslice(ns, np, b2gs_tb[c]) * ((b2gs_nket(ns, np, b2gs_tk[c]) + 31) / 32));
    add(B2_SU_GRAD1, b2gs_nslice(ns, np, 0) + b2gs_nslice(ns, np, 1) + b2gs_nslice(ns, np, 2));
    gm[m] = B2gsMol{ns, np, (int)su.size(), 0, pr0};
    su.insert(su.end(), tmp.begin(), tmp.begin() + nt);
  }
}

// ============================================================================================
// Allocation-free single-molecule ERI entry (b2_int2e_sph_s8_noalloc).
//
// For callers that must not call cudaMalloc: processes whose device memory is handed out by
// another allocator or a pool with a fixed budget (a cudaMalloc there would fail or take memory
// the pool has promised elsewhere), and loops with a latency budget, where cudaMalloc/cudaFree
// can block and synchronise the device.  The per-molecule tables the ERI kernels read (molecule
// descriptor, shell-pair primitive data, class lists, work list, Boys table) live in one
// file-scope __device__ array of B2_NOALLOC_BYTES (2.5 MiB) that every GPU loading this library
// keeps until the process exits; the host side fills a static buffer of the same size and copies
// it with one cudaMemcpyAsync (pageable source: the copy has left the buffer when the call
// returns).  Limits: nbas <= 48 shells, nao <= 70, s/p shells with <= 3 primitives.  The s8
// output is written completely, so no part of the array has to start at zero.
// The call is asynchronous on `stream`: the output is ready, and kernel faults are reported,
// only once the caller synchronises that stream.  All calls share the device array and the
// host staging buffer: calls from several host threads must be serialised by the caller, and
// calls whose work overlaps on the GPU (different streams) race; calls on one stream are
// ordered.  The first call on a device looks up the array's device address
// (cudaGetSymbolAddress) with that device current; make it before any stream capture.
#define B2_NOALLOC_MAXBAS 48
#define B2_NOALLOC_MAXSP (B2_NOALLOC_MAXBAS * (B2_NOALLOC_MAXBAS + 1) / 2)
#define B2_NOALLOC_MAXTASK (B2_NOALLOC_MAXSP * 42)
#define B2_NOALLOC_BYTES (2621440)

static __device__ __align__(256) unsigned char g_b2_noalloc_scratch[B2_NOALLOC_BYTES];
static __align__(256) unsigned char g_b2_noalloc_stage[B2_NOALLOC_BYTES];
static unsigned char *g_b2_noalloc_dev[128];     // device address of the array, per device

static size_t b2_na_align(size_t x) { return (x + 255) & ~(size_t)255; }

// class-group launch over a fixed-size group table (no container)
template <typename T>
static void b2_eri_all_na(const B2PlanDev &P, const B2EriTask *tasks, const long long *g,
                          const B2PairPrim<T> *pp, T *out, cudaStream_t st) {
#define B2_G(grp, LI, LJ, LK, LL)                                                            \
  if (g[grp + 1] > g[grp])                                                                   \
    b2_eri_group<T, LI, LJ, LK, LL>(P, tasks + g[grp], g[grp + 1] - g[grp], pp, out, st);
  B2_G(0, 0, 0, 0, 0) B2_G(1, 0, 0, 1, 0) B2_G(2, 0, 0, 0, 1) B2_G(3, 0, 0, 1, 1)
  B2_G(4, 1, 0, 0, 0) B2_G(5, 1, 0, 1, 0) B2_G(6, 1, 0, 0, 1) B2_G(7, 1, 0, 1, 1)
  B2_G(8, 0, 1, 0, 0) B2_G(9, 0, 1, 1, 0) B2_G(10, 0, 1, 0, 1) B2_G(11, 0, 1, 1, 1)
  B2_G(12, 1, 1, 0, 0) B2_G(13, 1, 1, 1, 0) B2_G(14, 1, 1, 0, 1) B2_G(15, 1, 1, 1, 1)
#undef B2_G
}

extern "C" int b2_int2e_sph_s8_noalloc(const int *atm, int natm, const int *bas, int nbas,
                                       const double *env, int n_env, int precision, void *eri_out,
                                       void *stream) {
  if (!atm || !bas || !env || !eri_out || natm <= 0 || nbas <= 0 || n_env <= 0) return B2_ERR_ARG;
  if (precision != 64 && precision != 32) return B2_ERR_ARG;
  if (nbas > B2_NOALLOC_MAXBAS) return B2_ERR_SIZE;
  unsigned char *H = g_b2_noalloc_stage;
  // ---- host tables in the static staging buffer (same layout as the device array) ----
  const size_t o_mol = 0;
  const size_t o_pi = b2_na_align(o_mol + sizeof(B2MolDev));
  const size_t o_pp = b2_na_align(o_pi + sizeof(B2PairInfo) * B2_NOALLOC_MAXSP);
  const size_t pp_bytes = (precision == 64 ? sizeof(B2PairPrim<double>) : sizeof(B2PairPrim<float>)) *
                          B2_NOALLOC_MAXSP * B2_MAXPP;
  const size_t o_cls = b2_na_align(o_pp + pp_bytes);
  const size_t o_task = b2_na_align(o_cls + sizeof(int) * B2_NOALLOC_MAXSP);
  const size_t o_boys = b2_na_align(o_task + sizeof(B2EriTask) * B2_NOALLOC_MAXTASK);
  const size_t total = b2_na_align(o_boys + sizeof(double) * B2_BOYS_NT * B2_BOYS_NM);
  if (total > B2_NOALLOC_BYTES) return B2_ERR_SIZE;
  B2Shell S[B2_NOALLOC_MAXBAS];
  int nao = 0;
  for (int s = 0; s < nbas; ++s) {
    const int *b = bas + s * B2_BAS_SLOTS;
    const int l = b[B2_ANG_OF], np = b[B2_NPRIM_OF], ia = b[B2_ATOM_OF];
    if (l > B2_MAXL || np < 1 || np > B2_MAXPRIM || b[B2_NCTR_OF] != 1) return B2_ERR_UNSUPPORTED;
    if (ia < 0 || ia >= natm) return B2_ERR_ARG;
    const int pc = atm[ia * B2_ATM_SLOTS + B2_PTR_COORD];
    if (pc < 0 || pc + 3 > n_env || b[B2_PTR_EXP] < 0 || b[B2_PTR_COEFF] < 0 ||
        b[B2_PTR_EXP] + np > n_env || b[B2_PTR_COEFF] + np > n_env)
      return B2_ERR_ARG;
    memset(&S[s], 0, sizeof(B2Shell));
    for (int d = 0; d < 3; ++d) S[s].R[d] = env[pc + d];
    const double fac = l == 0 ? B2_FAC_S : B2_FAC_P;
    for (int k = 0; k < np; ++k) {
      S[s].exp[k] = env[b[B2_PTR_EXP] + k];
      S[s].coef[k] = env[b[B2_PTR_COEFF] + k] * fac;
    }
    S[s].l = l; S[s].ao0 = nao; S[s].nprim = np; S[s].atom = ia;
    nao += 2 * l + 1;
  }
  if (nao > B2_MAXNAO - 2) return B2_ERR_SIZE;
  const int nsp = nbas * (nbas + 1) / 2;
  B2MolDev *md = (B2MolDev *)(H + o_mol);
  memset(md, 0, sizeof(B2MolDev));
  md->nao = nao; md->nbas = nbas; md->natm = natm; md->nsp = nsp;
  const long long n2 = (long long)nao * (nao + 1) / 2;
  md->n4 = n2 * (n2 + 1) / 2;
  B2PairInfo *PI = (B2PairInfo *)(H + o_pi);
  static int cls[B2_NOALLOC_MAXSP];
  for (int I = 0; I < nbas; ++I)
    for (int J = 0; J <= I; ++J) {
      const int sp = (int)b2_tri(I) + J;
      const B2Shell &a = S[I], &b = S[J];
      PI[sp] = B2PairInfo{I, J, a.l, b.l, a.ao0, b.ao0, a.nprim * b.nprim, 0};
      cls[sp] = a.l + 2 * b.l;
      B2PairPrim<double> q64[B2_MAXPP];
      B2PairPrim<float> q32[B2_MAXPP];
      b2_pair_prims_packed(a, b, q64, q32);              // same screening as the batch plan
      for (int x = 0; x < B2_MAXPP; ++x) {
        if (precision == 64) ((B2PairPrim<double> *)(H + o_pp))[(size_t)sp * B2_MAXPP + x] = q64[x];
        else ((B2PairPrim<float> *)(H + o_pp))[(size_t)sp * B2_MAXPP + x] = q32[x];
      }
    }
  int *CL = (int *)(H + o_cls);
  int start = 0;
  for (int c = 0; c < 4; ++c) {
    md->cls_start[c] = start;
    for (int sp = 0; sp < nsp; ++sp)
      if (cls[sp] == c) CL[start++] = sp;
  }
  md->cls_start[4] = start;
  // work list grouped by class combination, kets in chunks of 128 (as b2_eri_tasks)
  B2EriTask *TK = (B2EriTask *)(H + o_task);
  long long goff[17];
  long long nt = 0;
  for (int grp = 0; grp < 16; ++grp) {
    goff[grp] = nt;
    const int bc = grp / 4, c = grp % 4;
    for (int IJ = 0; IJ < nsp; ++IJ) {
      if (PI[IJ].lI + 2 * PI[IJ].lJ != bc) continue;
      const int spcut = (int)b2_tri(PI[IJ].I) + PI[IJ].I;
      int cnt = 0;                                      // class-c members KL <= spcut
      for (int e = md->cls_start[c]; e < md->cls_start[c + 1]; ++e) cnt += (CL[e] <= spcut);
      const int nsub = (precision == 64 && PI[IJ].lI) ? 3 : 1;
      for (int s0 = 0; s0 < cnt; s0 += 128)
        for (int sub = 0; sub < nsub; ++sub) {
          if (nt >= B2_NOALLOC_MAXTASK) return B2_ERR_SIZE;
          TK[nt++] = B2EriTask{0, IJ, c, s0, cnt - s0 < 128 ? cnt - s0 : 128, nsub > 1 ? sub : -1};
        }
    }
  }
  goff[16] = nt;
  b2_boys_fill_table((double *)(H + o_boys));
  if (precision == 32) {                          // float32 kernels read a float table
    const double *bd = (const double *)(H + o_boys);
    float *bf = (float *)(H + o_boys);
    for (int i = 0; i < B2_BOYS_NT * B2_BOYS_NM; ++i) bf[i] = (float)bd[i];   // in place, ascending
  }
  // ---- stage to the device array and launch (no device allocation anywhere) ----
  // arguments are all checked above, before any CUDA call; first call on a device: set-up
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return B2_ERR_CUDA;
  if (!g_b2_noalloc_dev[dev]) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_b2_noalloc_scratch) != cudaSuccess || !p) return B2_ERR_CUDA;
    g_b2_noalloc_dev[dev] = (unsigned char *)p;
  }
  unsigned char *Dv = g_b2_noalloc_dev[dev];
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemcpyAsync(Dv, H, total, cudaMemcpyHostToDevice, st) != cudaSuccess) return B2_ERR_CUDA;
  B2PlanDev P;                                           // view onto the static array
  P.mols = (B2MolDev *)(Dv + o_mol);
  P.pinfo = (B2PairInfo *)(Dv + o_pi);
  P.cls_list = (int *)(Dv + o_cls);
  P.boys = (double *)(Dv + o_boys);
  P.boys32 = (float *)(Dv + o_boys);
  B2EriTask *tasks = (B2EriTask *)(Dv + o_task);
  if (precision == 64)
    b2_eri_all_na<double>(P, tasks, goff, (const B2PairPrim<double> *)(Dv + o_pp), (double *)eri_out, st);
  else
    b2_eri_all_na<float>(P, tasks, goff, (const B2PairPrim<float> *)(Dv + o_pp), (float *)eri_out, st);
  P.mols = nullptr; P.pinfo = nullptr; P.cls_list = nullptr; P.boys = nullptr; P.boys32 = nullptr;
  if (cudaGetLastError() != cudaSuccess) return B2_ERR_CUDA;
  return B2_OK;
}

// device tables of a plan that kernels build: the super-shell pairs' primitives
int b2_build_pairs(B2PlanDev &P, cudaStream_t st) {
  const long long np = P.su.n_pair;
  B2_CUDA_TRY(b2_dmalloc_t(&P.su.pr64, sizeof(B2gPrim) * B2_MAXPP * (size_t)std::max(1ll, np), st));
  B2_CUDA_TRY(b2_dmalloc_t(&P.su.pr32, sizeof(B2gPrim32) * B2_MAXPP * (size_t)std::max(1ll, np), st));
  B2_CUDA_TRY(b2_dmalloc_t(&P.su.pn, sizeof(B2gCount) * (size_t)std::max(1ll, np), st));
  if (np > 0) {
    k_su_prims<<<(unsigned)((np + 127) / 128), 128, 0, st>>>(P.su.mol, P.su.off + B2_SU_PAIRS * (P.h.nmol + 1ll),
                                                             P.h.nmol, P.su.su, P.su.pr64, P.su.pr32, P.su.pn);
    b2_count_launches(1);
    B2_CUDA_TRY(cudaGetLastError());
  }
  return B2_OK;
}

// Work the float32 ERI kernels do for a plan: primitive quartets evaluated (bra survivors x ket
// survivors of every slice quartet) and their arithmetic by the per-class counts of eri_flops.h
// (generated from eri_su.cuh by eri_flops_count.cu): per primitive quartet, and per bra slice and
// ket primitive for the ket's polynomial.  One thread per task.
template <int TB, int TK>
__global__ void __launch_bounds__(256)
k_eri_count(const long long *__restrict__ toff, int nmol, const B2gsMol *__restrict__ gms,
            const B2gCount *__restrict__ pn, double fl, double sp, double kf, double *__restrict__ out) {
  __shared__ double red[3][8];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double q = 0, e = 0;
  B2gsMol g;
  B2EriTaskSu tk;
  if (t < toff[nmol] && b2_eri_task<TB, TK>(toff, nmol, gms, t, g, tk)) {
    const int k0 = b2es_first(g.ns, g.np, TK) + tk.k0;
    for (int k = 0; k < tk.cnt; ++k) e += pn[g.pr_off + k0 + k].x;
    q = e * pn[g.pr_off + tk.pair].x;
  }
  double v[3] = {q, q * fl + e * kf, q * sp};
  for (int c = 0; c < 3; ++c)
    for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < 3; ++c) red[c][threadIdx.x >> 5] = v[c];
  __syncthreads();
  if (threadIdx.x < 3) {
    double s = 0;
    for (int w = 0; w < 8; ++w) s += red[threadIdx.x][w];
    atomicAdd(&out[threadIdx.x], s);
  }
}

template <int C>
static void b2_eri_count_class(const B2PlanDev &P, double *d) {
  constexpr int TB = C == 5 ? 2 : (C == 2 || C == 4 ? 1 : 0), TK = C == 0 ? 0 : (C <= 2 ? 1 : 2);
  const long long n = P.su.n_task[C];
  if (n > 0) {
    k_eri_count<TB, TK><<<(unsigned)((n + 255) / 256), 256>>>(
        P.su.off + C * (P.h.nmol + 1ll), P.h.nmol, P.su.mol, P.su.pn, (double)B2_ERI_FLOPS[C],
        (double)B2_ERI_SPECIAL[C], (double)B2_ERI_KET_FLOPS[C], d);
    b2_count_launches(1);
  }
  if constexpr (C < 5) b2_eri_count_class<C + 1>(P, d);
}

int b2_launch_eri_count(B2PlanDev &P, double *host_out) {
  double *d = nullptr;
  B2_CUDA_TRY(b2_dmalloc_t(&d, 3 * sizeof(double)));
  B2_CUDA_TRY(cudaMemset(d, 0, 3 * sizeof(double)));
  b2_eri_count_class<0>(P, d);
  const int rc = cudaMemcpy(host_out, d, 3 * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess ? B2_OK : B2_ERR_CUDA;
  b2_dfree(d);
  return rc;
}
