// Device-resident SCF step (sm_100a), FP64, one CTA per molecule.
//
// Follows the reference iteration (nanoDFT.py:40-102, dft.py:789-882):
//   H = H_core + (J - hyb/2 K) + V_xc
//   DIIS (nanoDFT.py:338-364): err = S D H - (S D H)^T stored in a ring of 9, B-matrix
//     row/column head+1 <- <err_k, err>, masked until filled, c = pinv(B)[0,:]
//     (pinv as jnp.linalg.pinv: singular values below 10*max(m,n)*eps*s_max dropped),
//     H <- sum_k c[k+1] H_k
//   C = L^T eigvec(L H L^T) with L = inv(cholesky(S)) (nanoDFT.py:69, 239)
//   D = 2 C_occ C_occ^T (nanoDFT.py:72)
// The eigensolver is a parallel one-sided Jacobi method (round-robin pair ordering) on the
// matrix held in shared memory; the reference uses jnp.linalg.eigh or TessellateIPU's
// Jacobi ipu_eigh (nanoDFT.py:370-393).
#include <type_traits>
#include "device_plan.cuh"
#include "dmma.cuh"
#include "scf.cuh"

__device__ double b2_block_sum(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  double s = 0;
  for (int i = 0; i < nw; ++i) s += red[i];
  __syncthreads();
  return s;
}

__device__ double b2_block_max(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  double s = 0;
  for (int i = 0; i < nw; ++i) s = fmax(s, red[i]);
  __syncthreads();
  return s;
}

// ------------------------------------------------------------------ small dense products
// Both SCF kernels run one molecule per CTA with 64 Q threads (2 Q warps) for the orbital bucket
// N <= 16 Q.  acc += A B by float64 MMA (m16n8k8): warp w owns columns 8w..8w+7 and every 16-row
// tile, so a B fragment serves Q products.  fa(r, k) and fb(k, c) return zero outside N.  The
// inner products of the form before ran one output element per thread with two loads per FMA.
template <int Q, typename FA, typename FB>
__device__ __forceinline__ void b2_mm(double (&acc)[Q][4], int N, int K, FA fa, FB fb) {
  const int w = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
  for (int i = 0; i < Q; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0;
  if (8 * w >= N) return;
#pragma unroll 2
  for (int k0 = 0; k0 < K; k0 += 8) {
    const double b[2] = {fb(k0 + t, 8 * w + g), fb(k0 + t + 4, 8 * w + g)};
#pragma unroll
    for (int i = 0; i < Q; ++i)
      if (16 * i < N) {
        const int r = 16 * i + g;
        const double a[4] = {fa(r, k0 + t), fa(r + 8, k0 + t), fa(r, k0 + t + 4), fa(r + 8, k0 + t + 4)};
        b2_dmma(acc[i], a, b);
      }
  }
}
// f(r, c, value) for every element of the product with r, c < N
template <int Q, typename F>
__device__ __forceinline__ void b2_mm_out(const double (&acc)[Q][4], int N, F f) {
  const int w = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int r = 16 * i + g + 8 * (c >> 1), col = 8 * w + 2 * t + (c & 1);
      if (r < N && col < N) f(r, col, acc[i][c]);
    }
}

// CTAs per SM that the shared memory of the two kernels allows, kept within reach of the registers
// (many molecules at once; a single one has the SM to itself)
#define B2_SCF_CTAS(Q) ((Q) == 1 ? 10 : (Q) == 2 ? 6 : 7 - (Q))

// ------------------------------------------------------------------ eigensolver
// One-sided Jacobi (Hestenes) on the symmetric A: G = A / |A| + 2 I (|A| the largest row sum, so
// the spectrum of G lies in [1, 3]), columns rotated pairwise until they are orthogonal; then
// column i = g_i v_i with v_i the eigenvector and A's eigenvalue |A| (|g_i| - 2).  Rotating
// columns needs no eigenvector accumulation and no second (row) phase: a round-robin round is one
// dot product, one rotation and one barrier, 8 lanes per pair, every pair of the molecule at once.
// The two-sided form before (rotation phase on n/2 threads, then one pass over every 2 x 2 block
// and the eigenvectors, two barriers) took 2.2 us per round at 62 orbitals.
// The angle's tangent is taken in float32 (the rotation itself is exactly orthogonal: cosine and
// sine follow from that tangent in float64), which leaves 1e-7 of a coupling behind and shortens
// the round's serial chain.  A sweep is the last when its largest cosine was below 3e-9 and all its
// angles below 1e-6: what such rotations mix into pairs already treated is at rounding level.  A
// wide rotation may come from a cosine of any size where eigenvalues coincide, and carries the
// couplings of one column over to the other, so another sweep follows it.  Within such a block a
// cosine below 3e-15 is rounding (a dot product of 70 terms) and left alone, or its arbitrary angle
// would undo the sweep's work again and again.  |C^T S C - 1| over 20 warm-started iterations of
// CF4, cubane and neopentane: <= 2e-14, as the two-sided form had (3e-14); 7e-10 with the cosines
// alone as the criterion.  Other molecules take 0-2 sweeps more over those iterations.
// G: column-major, leading dimension LD = 16 Q + 8 (8 modulo 16 doubles: neighbouring groups on
// different banks), rows and columns beyond N zero.  ev[i] <- eigenvalues, nv[i] <- 1 / |g_i|.
template <int Q>
__device__ int b2_jacobi1(double *G, int N, double *nrm, double *ev, double *nv, double scale, int max_sweeps) {
  constexpr int LD = 16 * Q + 8, RP = 2 * Q;
  const int n = (N + 1) & ~1, half = n >> 1;
  const int grp = threadIdx.x >> 3, li = threadIdx.x & 7;
  const bool on = grp < half;
  const int k = on ? grp : 0;
  auto dot = [&](const double *a, const double *b) {
    double x = 0;
#pragma unroll
    for (int j = 0; j < RP; ++j) x += a[li + 8 * j] * b[li + 8 * j];
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x;
  };
  auto norms = [&]() {
    const double *c0 = G + k * LD, *c1 = G + (k + half) * LD;
    const double a = dot(c0, c0), b = dot(c1, c1);
    if (on && li == 0) { nrm[k] = a; nrm[k + half] = b; }
    __syncthreads();
  };
  int sweep = 0;
  bool more = true;
  for (; sweep < max_sweeps && more; ++sweep) {
    norms();
    bool big = false;
    for (int r = 0; r < n - 1; ++r) {
      // round-robin pairs: index 0 fixed, the others rotate by r (k - 1 + r < 2 (n - 1))
      int a = k - 1 + r, b = n - 2 - k + r;
      if (a >= n - 1) a -= n - 1;
      if (b >= n - 1) b -= n - 1;
      a = (k == 0) ? 0 : a + 1;
      b += 1;
      double *cp = G + min(a, b) * LD, *cq = G + max(a, b) * LD;
      const double app = on ? nrm[min(a, b)] : 0.0, aqq = on ? nrm[max(a, b)] : 0.0;
      double vp[RP], vq[RP], x = 0, x1 = 0;          // two chains
#pragma unroll
      for (int j = 0; j < RP; ++j) {
        vp[j] = on ? cp[li + 8 * j] : 0.0;
        vq[j] = on ? cq[li + 8 * j] : 0.0;
        if (j & 1) x1 += vp[j] * vq[j];
        else x += vp[j] * vq[j];
      }
      x += x1;
      x += __shfl_xor_sync(0xffffffffu, x, 4);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      const double x2 = x * x, pq = app * aqq;
      const bool act = on && x2 > 1e-31 * pq;
      double t = 0.0;
      if (act) {
        // sym.schur2 (Golub & Van Loan): t = sign(d b) |b| / (|d| + sqrt(d^2 + b^2)), d = aqq - app, b = 2 x
        const float d = (float)(aqq - app), bb = (float)(2.0 * x);
        const float q2 = d * d + bb * bb;
        const float tf = copysignf(1.0f, d * bb) * __fdividef(fabsf(bb), fabsf(d) + q2 * rsqrtf(q2));
        t = d == 0.0f ? (x > 0 ? 1.0 : -1.0) : (double)tf;
      }
      const bool wide = fabs(t) > 1e-6;
      if (act && (!wide || x2 > 1e-29 * pq)) {
        big = big || wide || x2 > 1e-17 * pq;
        // 1 / sqrt(1 + t^2): float seed (e = 1 - u y^2 near 1e-7), one third-order step (Householder)
        const double u = fma(t, t, 1.0), y = (double)rsqrtf((float)u), e = fma(-u * y, y, 1.0);
        const double c = fma(y * e, fma(0.375, e, 0.5), y), s = t * c;
#pragma unroll
        for (int j = 0; j < RP; ++j) {
          cp[li + 8 * j] = c * vp[j] - s * vq[j];
          cq[li + 8 * j] = s * vp[j] + c * vq[j];
        }
        if (li == 0) {
          // |g_p'|^2 = c^2 app - 2 c s x + s^2 aqq, the trace is kept
          const double np = c * c * app - 2.0 * c * s * x + s * s * aqq;
          nrm[min(a, b)] = np;
          nrm[max(a, b)] = app + aqq - np;
        }
      }
      __syncthreads();
    }
    more = __syncthreads_or(big);
  }
  norms();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double g = sqrt(nrm[i]);
    ev[i] = i < N ? (g - 2.0) * scale : 1e300;
    nv[i] = i < N ? 1.0 / g : 0.0;
  }
  __syncthreads();
  return sweep;
}

// Jacobi on the leading ne rows and columns of the 10 x 10 DIIS matrix A (shared memory, row-major;
// the border and the filled ring slots, rounded up to an even number; the others are zero, i.e.
// decoupled) run by one warp; V <- the eigenvectors.  Round-robin order: the ne / 2 rotations of a
// round act on disjoint pairs, so as many lanes compute them, and the pairs, and up to 25 lanes apply
// G_k A_kl G_l^T to the 2 x 2 blocks.  What bounds it is the chain of rounds.  k_fock_diis per call at
// 7 orbitals: 95 us in the serial order (45 dependent rotations per sweep), 61 us in rounds, 48 us with
// the tangent in float32, 41 us over the leading rows alone.  The float32 tangent is brought to float64
// by Newton's steps with a float32 slope (2 us per call): with it alone the iteration
// stops with 1e-14 of a coupling left, and the first coefficient came out 4e-15 to 9e-15 off where the
// serial order had 3e-16.
// Couplings below float32's range are far below the stopping norm (the border of B holds ones).
__device__ void b2_jacobi_small_warp(double *A, double *V, double *rot, int *prs, int ne) {
  constexpr int n = 10;
  const int l = threadIdx.x & 31, half = ne >> 1;
  const int bk = l / half, bl = l - bk * half;            // this lane's block of pairs
  const bool blk = l < half * half;
  for (int e = l; e < n * n; e += 32) V[e] = (e / n == e - (e / n) * n) ? 1.0 : 0.0;
  __syncwarp();
  for (int sweep = 0; sweep < 50; ++sweep) {
    double off = 0, tot = 0;
    for (int e = l; e < n * n; e += 32) {
      const double x = A[e] * A[e];
      tot += x;
      if (e / n != e - (e / n) * n) off += x;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    if (off <= 1e-28 * tot || off < 1e-300) break;
    for (int r = 0; r < ne - 1; ++r) {
      if (l < half) {
        // round-robin pairs: index 0 fixed, the others rotate by r
        int a = l - 1 + r, b = ne - 2 - l + r;
        if (a >= ne - 1) a -= ne - 1;
        if (b >= ne - 1) b -= ne - 1;
        a = (l == 0) ? 0 : a + 1;
        b += 1;
        const int p = min(a, b), q = max(a, b);
        double c = 1.0, s = 0.0;
        const double apq = A[p * n + q], app = A[p * n + p], aqq = A[q * n + q];
        if (fabs(apq) > 1e-36 && apq * apq > 1e-36 * fabs(app * aqq)) {
          // tau = (aqq - app) / (2 apq), t = sign(tau) / (|tau| + sqrt(1 + tau^2)) (sym.schur2)
          const double d = aqq - app;
          const float df = (float)d, bf = (float)(2.0 * apq), tau = fminf(fmaxf(df / bf, -1e18f), 1e18f);
          const float tf = copysignf(1.0f, tau) / (fabsf(tau) + sqrtf(1.0f + tau * tau));
          // two Newton steps on apq t^2 + d t - apq = 0 (slope from the float32 tangent)
          const double ri = (double)__fdividef(1.0f, fmaf(bf, tf, df));
          double t = (double)tf;
#pragma unroll
          for (int k = 0; k < 2; ++k) t = fma(-fma(apq * t, t, fma(d, t, -apq)), ri, t);
          c = rsqrt(1.0 + t * t);
          s = t * c;
        }
        rot[2 * l] = c;
        rot[2 * l + 1] = s;
        prs[2 * l] = p;
        prs[2 * l + 1] = q;
      }
      __syncwarp();
      if (blk) {
        const int p = prs[2 * bk] * n, q = prs[2 * bk + 1] * n, u = prs[2 * bl], v = prs[2 * bl + 1];
        const double ck = rot[2 * bk], sk = rot[2 * bk + 1], cl = rot[2 * bl], sl = rot[2 * bl + 1];
        const double a00 = A[p + u], a01 = A[p + v], a10 = A[q + u], a11 = A[q + v];
        double *v0 = V + 2 * bk * n, *v1 = v0 + n;         // V's rows 2 bk, 2 bk + 1, columns of pair bl
        const double x0 = v0[u], y0 = v0[v], x1 = v1[u], y1 = v1[v];
        const double b00 = ck * a00 - sk * a10, b10 = sk * a00 + ck * a10;
        const double b01 = ck * a01 - sk * a11, b11 = sk * a01 + ck * a11;
        A[p + u] = cl * b00 - sl * b01;
        A[p + v] = sl * b00 + cl * b01;
        A[q + u] = cl * b10 - sl * b11;
        A[q + v] = sl * b10 + cl * b11;
        v0[u] = cl * x0 - sl * y0;
        v0[v] = sl * x0 + cl * y0;
        v1[u] = cl * x1 - sl * y1;
        v1[v] = sl * x1 + cl * y1;
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------------ Fock + DIIS
// ring layout per molecule (offset mat_off * 9): errs[9][N*N], hams[9][N*N]; B: 100 doubles
// Bound by latency at one molecule per CTA; 62 orbitals, one molecule: 172 us per call before (two
// products with one output element per thread, serial 10 x 10 Jacobi), 139 us with element-wise
// ring passes, 95 us with several elements' loads in flight, 99 us with the tangents in float64.
template <int Q>
__global__ void __launch_bounds__(64 * Q, B2_SCF_CTAS(Q))
k_fock_diis(const B2MolDev *__restrict__ mols, const int *__restrict__ active,
            const int *__restrict__ iter, double hyb, int use_diis, const double *__restrict__ Hcore,
            const double *__restrict__ S, const double *__restrict__ D, const double *__restrict__ J,
            const double *__restrict__ K, const double *__restrict__ Vxc, double *__restrict__ H,
            double *__restrict__ diffJK, double *__restrict__ ring_err, double *__restrict__ ring_h,
            double *__restrict__ Bmat, double *__restrict__ diis_err, const int *__restrict__ map) {
  const int m = map ? map[blockIdx.x] : blockIdx.x;
  if (active && !active[m]) return;
  constexpr int LD = 16 * Q + 4;                   // 4 modulo 16 doubles: fragment loads without bank conflicts
  extern __shared__ double sm[];
  __shared__ double red[32];
  __shared__ double sc[10];
  __shared__ double stmp[9];
  __shared__ double sA[100], sV[100], sRot[10];
  __shared__ int sPrs[10];
  const B2MolDev md = mols[m];
  const int N = md.nao, NN = N * N;
  const long long mo = md.mat_off;
  double *sH = sm, *sT = sH + 16 * Q * LD;
  for (int e = threadIdx.x; e < 2 * 16 * Q * LD; e += blockDim.x) sm[e] = 0.0;   // padding stays zero
  __syncthreads();
#pragma unroll 4
  for (int e = threadIdx.x; e < NN; e += blockDim.x) {
    const double djk = J[mo + e] - 0.5 * hyb * K[mo + e];
    diffJK[mo + e] = djk;
    const double h = Hcore[mo + e] + djk + Vxc[mo + e];
    if (!use_diis) H[mo + e] = h;
    else sH[(e / N) * LD + e - (e / N) * N] = h;
  }
  if (!use_diis) return;
  const int it = iter[m];
  const int nd = 9, head = it % nd;
  double acc[Q][4];
  const double *gS = S + mo, *gD = D + mo;
  b2_mm<Q>(acc, N, N, [&](int r, int k) { return r < N && k < N ? gS[r * N + k] : 0.0; },
           [&](int k, int c) { return k < N && c < N ? gD[k * N + c] : 0.0; });      // S D
  b2_mm_out<Q>(acc, N, [&](int r, int c, double v) { sT[r * LD + c] = v; });
  __syncthreads();
  b2_mm<Q>(acc, N, N, [&](int r, int k) { return sT[r * LD + k]; }, [&](int k, int c) { return sH[k * LD + c]; });
  __syncthreads();
  b2_mm_out<Q>(acc, N, [&](int r, int c, double v) { sT[r * LD + c] = v; });          // S D H
  __syncthreads();
  double *er = ring_err + mo * nd, *hr = ring_h + mo * nd;
  const int nfill = min(it + 1, nd);
  double emax = 0, s9[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) s9[k] = 0.0;
  // the nine dot products <err_k, err_new> in the same pass; two elements' ring loads in flight
  for (int e0 = threadIdx.x; e0 < NN; e0 += 2 * blockDim.x) {
    double r[2][9];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = e0 + h * (int)blockDim.x;
#pragma unroll
      for (int k = 0; k < 9; ++k) r[h][k] = k < nfill && k != head && e < NN ? er[(long long)k * NN + e] : 0.0;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = e0 + h * (int)blockDim.x;
      if (e >= NN) break;
      const int a = e / N, b = e - (e / N) * N;
      const double v = sT[a * LD + b] - sT[b * LD + a];
      emax = fmax(emax, fabs(v));
      er[(long long)head * NN + e] = v;
      hr[(long long)head * NN + e] = sH[a * LD + b];
#pragma unroll
      for (int k = 0; k < 9; ++k)
        if (k < nfill) s9[k] += (k == head ? v : r[h][k]) * v;
    }
  }
  emax = b2_block_max(emax, red);
  {
    __shared__ double red9[9][10];                  // at most 320 threads: 10 warps
    const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      double v = s9[k];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if ((threadIdx.x & 31) == 0) red9[k][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < nd) {
      double sum = 0;
      for (int i = 0; i < nw; ++i) sum += red9[threadIdx.x][i];
      stmp[threadIdx.x] = (threadIdx.x < nfill) ? sum : 0.0;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int l = threadIdx.x;
    double *B = Bmat + (long long)m * 100;
    if (l < 10) {
      if (it == 0)
        for (int j = 0; j < 10; ++j) B[l * 10 + j] = (l == 0) == (j == 0) ? 0.0 : 1.0;
    }
    __syncwarp();
    if (l < nd) { B[(head + 1) * 10 + 1 + l] = stmp[l]; B[(1 + l) * 10 + head + 1] = stmp[l]; }
    __syncwarp();
    // masked copy: rows/columns of unfilled ring slots are zero
    for (int i = l; i < 100; i += 32) {
      const int r = i / 10, c = i - r * 10;
      const bool keep = (r == 0 || r - 1 < nfill) && (c == 0 || c - 1 < nfill);
      sA[i] = keep ? B[i] : 0.0;
    }
    __syncwarp();
    b2_jacobi_small_warp(sA, sV, sRot, sPrs, (nfill + 2) & ~1);
    __syncwarp();
    double smax = 0;
    for (int i = 0; i < 10; ++i) smax = fmax(smax, fabs(sA[i * 10 + i]));
    const double cut = 10.0 * 10.0 * 2.220446049250313e-16 * smax;
    if (l < 10) {
      double c = 0;
      for (int k = 0; k < 10; ++k) {
        const double lam = sA[k * 10 + k];
        if (fabs(lam) > cut) c += sV[0 * 10 + k] * sV[l * 10 + k] / lam;
      }
      sc[l] = c;
    }
    if (l == 0) diis_err[m] = emax;
  }
  __syncthreads();
#pragma unroll 4
  for (int e = threadIdx.x; e < NN; e += blockDim.x) {
    double s = 0;
#pragma unroll
    for (int k = 0; k < 9; ++k)                      // loads of the whole ring in flight at once
      if (k < nfill) s += sc[k + 1] * hr[(long long)k * NN + e];
    H[mo + e] = s;
  }
}

// ------------------------------------------------------------------ eigensolve + density
// F' = L H L^T; with a previous eigenvector basis W (ws, per molecule) and iter > 0 the Jacobi
// sweeps run on W^T F' W, which is nearly diagonal once the SCF settles (2-3 sweeps instead of
// 6-8); the eigenvectors are W V'.  The result is the same eigen-decomposition up to the sign
// and order of eigenvectors, which the density does not depend on.
// Products: M = L^T W, T = H M, A = M^T T, W' = W V', C = L^T W', D = 2 C_occ C_occ^T, all by
// float64 MMA; two matrices in shared memory (74 KB at 64 orbitals, 3 CTAs per SM).  62 orbitals,
// one molecule: 428 us per call before, 161 us with one sweep
// fewer where the cosines alone decided the last one (168 us with one dot-product chain and the
// library's reciprocal root), 171 us now.
template <int Q>
__global__ void __launch_bounds__(64 * Q, B2_SCF_CTAS(Q))
k_eigh_density(const B2MolDev *__restrict__ mols, const int *__restrict__ active,
               const int *__restrict__ iter, const double *__restrict__ H,
               const double *__restrict__ Linv, double *__restrict__ D, double *__restrict__ mo_energy,
               double *__restrict__ C, double *__restrict__ ws, int *__restrict__ sweeps,
               const int *__restrict__ map) {
  const int m = map ? map[blockIdx.x] : blockIdx.x;
  if (active && !active[m]) return;
  constexpr int LD = 16 * Q + 8, NM = 16 * Q;
  extern __shared__ double sm[];
  __shared__ double red[32], nrm[NM], evals[NM], nv[NM];
  __shared__ int order[NM];
  const B2MolDev md = mols[m];
  const int N = md.nao, NN = N * N;
  const int n = (N + 1) & ~1;                     // even size for the round-robin ordering
  const long long mo = md.mat_off;
  const bool warm = ws && iter && iter[m] > 0;
  double *s1 = sm, *s2 = sm + NM * LD;             // column-major, padding zero
  const double *gL = Linv + mo, *gH = H + mo, *gW = ws ? ws + mo : nullptr;
  for (int e = threadIdx.x; e < 2 * NM * LD; e += blockDim.x) sm[e] = 0.0;
  __syncthreads();
  double acc[Q][4];
  auto LT = [&](int r, int k) { return r < N && k < N ? gL[k * N + r] : 0.0; };
  if (warm) {                                                                    // M = L^T W
    b2_mm<Q>(acc, N, N, LT, [&](int k, int c) { return k < N && c < N ? gW[k * N + c] : 0.0; });
    b2_mm_out<Q>(acc, N, [&](int r, int c, double v) { s1[c * LD + r] = v; });
  } else {
    for (int e = threadIdx.x; e < NN; e += blockDim.x) s1[(e / N) * LD + e - (e / N) * N] = gL[e];
  }
  __syncthreads();
  b2_mm<Q>(acc, N, N, [&](int r, int k) { return r < N && k < N ? gH[r * N + k] : 0.0; },
           [&](int k, int c) { return s1[c * LD + k]; });                        // T = H M
  b2_mm_out<Q>(acc, N, [&](int r, int c, double v) { s2[c * LD + r] = v; });
  __syncthreads();
  b2_mm<Q>(acc, N, N, [&](int r, int k) { return s1[r * LD + k]; }, [&](int k, int c) { return s2[c * LD + k]; });
  __syncthreads();
  b2_mm_out<Q>(acc, N, [&](int r, int c, double v) { s1[c * LD + r] = v; });     // A = M^T T
  __syncthreads();
  // scale = largest column sum of |A|; G = A / scale + 2 I
  double rs = 0;
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    double x = 0;
    for (int r = 0; r < N; ++r) x += fabs(s1[c * LD + r]);
    rs = fmax(rs, x);
  }
  rs = b2_block_max(rs, red);
  const double scale = rs > 0.0 ? rs : 1.0, inv = 1.0 / scale;
  for (int e = threadIdx.x; e < NN; e += blockDim.x) {
    const int c = e / N, r = e - (e / N) * N;
    s1[c * LD + r] = s1[c * LD + r] * inv + (r == c ? 2.0 : 0.0);
  }
  __syncthreads();
  const int sw = b2_jacobi1<Q>(s1, N, nrm, evals, nv, scale, 30);
  // eigenvectors in the orthogonal basis, W' = W V' (warm) or V', into s2 and ws
  if (warm) {
    b2_mm<Q>(acc, N, N, [&](int r, int k) { return r < N && k < N ? gW[r * N + k] : 0.0; },
             [&](int k, int c) { return s1[c * LD + k]; });
    __syncthreads();                               // every warp has read W
    b2_mm_out<Q>(acc, N, [&](int r, int c, double v) {
      s2[c * LD + r] = v * nv[c];
      ws[mo + r * N + c] = v * nv[c];
    });
  } else {
    for (int e = threadIdx.x; e < NN; e += blockDim.x) {
      const int c = e / N, r = e - (e / N) * N;
      const double v = s1[c * LD + r] * nv[c];
      s2[c * LD + r] = v;
      if (ws) ws[mo + r * N + c] = v;
    }
  }
  // ascending order of eigenvalues: a total order (NaN sorts as +inf, ties by index), so the
  // ranks are a permutation of 0..n-1 whatever the values (every order[] slot is written)
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double li = evals[i] == evals[i] ? evals[i] : INFINITY;
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double lj = evals[j] == evals[j] ? evals[j] : INFINITY;
      rank += (lj < li) || (lj == li && j < i);
    }
    order[rank] = i;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < N; k += blockDim.x) mo_energy[(long long)m * B2_MAXNAO + k] = evals[order[k]];
  // C = L^T W' (columns unsorted), into s1
  b2_mm<Q>(acc, N, N, LT, [&](int k, int c) { return s2[c * LD + k]; });
  b2_mm_out<Q>(acc, N, [&](int r, int c, double v) { s1[c * LD + r] = v; });
  __syncthreads();
  const int nocc = md.nocc;
  auto occ = [&](int r, int k) { return k < nocc ? s1[order[k] * LD + r] : 0.0; };
  b2_mm<Q>(acc, N, nocc, occ, [&](int k, int c) { return occ(c, k); });
  b2_mm_out<Q>(acc, N, [&](int r, int c, double v) { D[mo + r * N + c] = 2.0 * v; });
  if (C)
    for (int e = threadIdx.x; e < NN; e += blockDim.x) C[mo + e] = s1[order[e - (e / N) * N] * LD + e / N];
  if (threadIdx.x == 0 && sweeps) sweeps[m] = sw;
}

// energies [E, E_core, E_J_K/2, E_xc, E_nuc] (nanoDFT.py:20-38)
__global__ void k_energy(const B2MolDev *__restrict__ mols, const int *__restrict__ active,
                         const double *__restrict__ D, const double *__restrict__ Hcore,
                         const double *__restrict__ diffJK, const double *__restrict__ exc,
                         const double *__restrict__ enuc, double *__restrict__ out) {
  const int m = blockIdx.x;
  if (active && !active[m]) return;
  __shared__ double red[32];
  const B2MolDev md = mols[m];
  const int NN = md.nao * md.nao;
  double ec = 0, ej = 0;
  for (int e = threadIdx.x; e < NN; e += blockDim.x) {
    const double d = D[md.mat_off + e];
    ec += d * Hcore[md.mat_off + e];
    ej += d * diffJK[md.mat_off + e];
  }
  ec = b2_block_sum(ec, red);
  ej = b2_block_sum(ej, red);
  if (threadIdx.x == 0) {
    double *o = out + (long long)m * 5;
    o[0] = ec + 0.5 * ej + exc[m] + enuc[m];
    o[1] = ec;
    o[2] = 0.5 * ej;
    o[3] = exc[m];
    o[4] = enuc[m];
  }
}

// end of one SCF iteration (nanoDFT.py:74-80): diff_JK = J - hyb/2 K of the new density
// (get_JK, nanoDFT.py:125-139), the five energy terms (nanoDFT.py:20-38) and the molecule's
// iteration counter advanced; with Vsym also V <- V + V^T of the XC kernels; inactive molecules are
// left untouched.  One launch fewer per iteration, and V + V^T runs where the matrices are read
// anyway; launches and dependent round trips are what a small molecule's iteration consists of.
__global__ void k_energy_jk(const B2MolDev *__restrict__ mols, const int *__restrict__ active,
                            const double *__restrict__ D, const double *__restrict__ Hcore,
                            const double *__restrict__ J, const double *__restrict__ K, double hyb,
                            const double *__restrict__ exc, const double *__restrict__ enuc,
                            double *__restrict__ diffJK, double *__restrict__ out, int *__restrict__ iter,
                            double *__restrict__ Vsym) {
  const int m = blockIdx.x;
  if (active && !active[m]) return;
  __shared__ double red[32];
  const B2MolDev md = mols[m];
  const int NN = md.nao * md.nao;
  double ec = 0, ej = 0;
#pragma unroll 4
  for (int e = threadIdx.x; e < NN; e += blockDim.x) {
    const long long a = md.mat_off + e;
    const double d = D[a];
    const double djk = J[a] - 0.5 * hyb * K[a];
    diffJK[a] = djk;
    ec += d * Hcore[a];
    ej += d * djk;
  }
  if (Vsym) {                                      // V <- V + V^T, four elements' loads in flight
    double *v = Vsym + md.mat_off;
    for (int e0 = threadIdx.x; e0 < NN; e0 += 4 * blockDim.x) {
      double x[4];
      int t[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int e = e0 + k * (int)blockDim.x, a = e / md.nao, b = e - (e / md.nao) * md.nao;
        t[k] = e < NN && a <= b ? b * md.nao + a : -1;
        x[k] = t[k] >= 0 ? v[e] + v[t[k]] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (t[k] >= 0) v[e0 + k * (int)blockDim.x] = v[t[k]] = x[k];
    }
  }
  ec = b2_block_sum(ec, red);
  ej = b2_block_sum(ej, red);
  if (threadIdx.x == 0) {
    double *o = out + (long long)m * 5;
    o[0] = ec + 0.5 * ej + exc[m] + enuc[m];
    o[1] = ec;
    o[2] = 0.5 * ej;
    o[3] = exc[m];
    o[4] = enuc[m];
    if (iter) iter[m] += 1;
  }
}

int b2_launch_energy_jk(const B2PlanDev &P, const int *active, const double *D, const double *Hcore,
                        const double *J, const double *K, double hyb, const double *exc,
                        const double *enuc, double *diffJK, double *out, int *iter, double *Vsym, cudaStream_t st) {
  k_energy_jk<<<P.h.nmol, 256, 0, st>>>(P.mols, active, D, Hcore, J, K, hyb, exc, enuc, diffJK, out, iter, Vsym);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

// L = inv(cholesky(S)) per molecule (FP64), one CTA per molecule (serial-ish, small N)
__global__ void k_chol_inv(const B2MolDev *__restrict__ mols, const double *__restrict__ S,
                           double *__restrict__ Linv, int *__restrict__ status) {
  const int m = blockIdx.x;
  extern __shared__ double sm[];
  const B2MolDev md = mols[m];
  const int N = md.nao, NN = N * N;
  double *sC = sm, *sI = sm + NN;
  for (int e = threadIdx.x; e < NN; e += blockDim.x) sC[e] = S[md.mat_off + e];
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  // right-looking Cholesky: lower triangle of sC
  for (int k = 0; k < N; ++k) {
    if (threadIdx.x == 0) {
      const double d = sC[k * N + k];
      if (!(d > 0)) bad = 1;
      sC[k * N + k] = sqrt(fmax(d, 1e-300));
    }
    __syncthreads();
    const double dk = sC[k * N + k];
    for (int i = k + 1 + threadIdx.x; i < N; i += blockDim.x) sC[i * N + k] /= dk;
    __syncthreads();
    for (int e = threadIdx.x; e < (N - k - 1) * (N - k - 1); e += blockDim.x) {
      const int i = k + 1 + e / (N - k - 1), j = k + 1 + e % (N - k - 1);
      if (j <= i) sC[i * N + j] -= sC[i * N + k] * sC[j * N + k];
    }
    __syncthreads();
  }
  // inverse of the lower-triangular factor, column by column (forward substitution)
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    for (int i = 0; i < N; ++i) {
      double s = (i == c) ? 1.0 : 0.0;
      for (int k = c; k < i; ++k) s -= sC[i * N + k] * sI[k * N + c];
      sI[i * N + c] = (i < c) ? 0.0 : s / sC[i * N + i];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < NN; e += blockDim.x) Linv[md.mat_off + e] = sI[e];
  if (threadIdx.x == 0 && status) status[m] = bad ? B2_ERR_NOT_PD : B2_OK;
}

static size_t b2_fock_smem(int Q) { return sizeof(double) * 2 * 16 * Q * (16 * Q + 4); }
static size_t b2_eigh_smem(int Q) { return sizeof(double) * 2 * 16 * Q * (16 * Q + 8); }

// One launch per orbital bucket (nao <= 16, 32, 48, 64, more) with shared memory sized for that
// bucket, so small molecules run several CTAs per SM.  The bucket launches go to the plan's
// bucket streams, forked from and joined back to the caller's stream with events, so they run
// concurrently (a serial sequence of launches would leave the GPU idle at each launch's tail).
template <typename F>
static int b2_per_bucket(const B2PlanDev &P, cudaStream_t st, F launch) {
  const bool sub = P.sub.n > 0;
  const std::vector<int> &off = sub ? P.sub.bkt_off_h : P.bkt_off_h;
  const int *map = sub ? P.sub.bkt_map : P.bkt_map;
  int used = 0;
  for (int b = 0; b < B2_NBKT; ++b) used += off[b + 1] > off[b];
  if (used > 1) B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[B2_NBKT], st));
  for (int b = B2_NBKT - 1; b >= 0; --b) {          // largest molecules first
    const int n = off[b + 1] - off[b];
    if (n <= 0) continue;
    const cudaStream_t s = used > 1 ? P.bkt_stream[b] : st;   // one bucket: the caller's stream itself
    if (used > 1) B2_CUDA_TRY(cudaStreamWaitEvent(s, P.bkt_ev[B2_NBKT], 0));
    B2_CUDA_TRY(launch(b + 1, n, map + off[b], s));
    b2_count_launches(1);
    B2_CUDA_TRY(cudaGetLastError());
    if (used > 1) {
      B2_CUDA_TRY(cudaEventRecord(P.bkt_ev[b], s));
      B2_CUDA_TRY(cudaStreamWaitEvent(st, P.bkt_ev[b], 0));
    }
  }
  return B2_OK;
}

// f(integral constant Q) for the bucket q = Q
template <typename F> static cudaError_t b2_by_bucket(int q, F f) {
  switch (q) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    default: return f(std::integral_constant<int, 5>{});
  }
}

int b2_launch_fock_diis(const B2PlanDev &P, const int *active, const int *iter, double hyb,
                        int use_diis, const double *Hcore, const double *S, const double *D,
                        const double *J, const double *K, const double *Vxc, double *H,
                        double *diffJK, double *ring_err, double *ring_h, double *Bmat,
                        double *diis_err, cudaStream_t st) {
  return b2_per_bucket(P, st, [&](int q, int n, const int *map, cudaStream_t s) {
    return b2_by_bucket(q, [&](auto Q) {
      cudaError_t e = cudaFuncSetAttribute(k_fock_diis<Q.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)b2_fock_smem(q));
      if (e == cudaSuccess)
        k_fock_diis<Q.value><<<n, 64 * q, b2_fock_smem(q), s>>>(P.mols, active, iter, hyb, use_diis, Hcore, S, D, J, K,
                                                                Vxc, H, diffJK, ring_err, ring_h, Bmat, diis_err, map);
      return e;
    });
  });
}

int b2_launch_eigh_density(const B2PlanDev &P, const int *active, const int *iter, const double *H,
                           const double *Linv, double *D, double *mo_energy, double *C, double *ws,
                           int *sweeps, cudaStream_t st) {
  return b2_per_bucket(P, st, [&](int q, int n, const int *map, cudaStream_t s) {
    return b2_by_bucket(q, [&](auto Q) {
      cudaError_t e = cudaFuncSetAttribute(k_eigh_density<Q.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)b2_eigh_smem(q));
      if (e == cudaSuccess)
        k_eigh_density<Q.value><<<n, 64 * q, b2_eigh_smem(q), s>>>(P.mols, active, iter, H, Linv, D, mo_energy, C, ws,
                                                                   sweeps, map);
      return e;
    });
  });
}

int b2_launch_energy(const B2PlanDev &P, const int *active, const double *D, const double *Hcore,
                     const double *diffJK, const double *exc, const double *enuc, double *out,
                     cudaStream_t st) {
  k_energy<<<P.h.nmol, 256, 0, st>>>(P.mols, active, D, Hcore, diffJK, exc, enuc, out);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

int b2_launch_chol_inv(const B2PlanDev &P, const double *S, double *Linv, int *status,
                       cudaStream_t st) {
  size_t sm = sizeof(double) * 2 * P.h.max_nao * P.h.max_nao;
  B2_CUDA_TRY(cudaFuncSetAttribute(k_chol_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  k_chol_inv<<<P.h.nmol, 128, sm, st>>>(P.mols, S, Linv, status);
  b2_count_launches(1);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}
