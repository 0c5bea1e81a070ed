// hkb_kdist.cu -- per-bin sort + Chebyshev k-distribution fit (sm_100a).
//
// One CTA per (state, bin) does the whole post-processing chain of
// heliosk.cu:2046-2193 on the bin's values while they sit in shared memory:
//   sort (total order on the FP64 bit patterns)          heliosk.cu:2046-2051
//   findCut                                              resample.h:362-388
//   rescale(+1), copyK2                                  resample.h:397-461
//   lnK                                                  resample.h:472-481
//   leastSquare (first nc-1 reflections, back-solve)     resample.h:243-353
//   optional expfx + rescale(-1) reconstruction          resample.h:497-524
// The Householder factorisation of the Chebyshev Vandermonde matrix is done
// once per (Nxb, nC) by qr_kernel (resample.h:14-37, 73-227), a single CTA.
// Bins above KD_MAX_NXB points run kdist_big_kernel on a global scratch slice.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cub/block/block_merge_sort.cuh>

#include "hkb_kernels.h"
#include "hkb_types.h"

namespace hkb {

constexpr int KD_THREADS = 1024;
constexpr int KD_MAX_NC = 100;  // def_NmaxSample, define.h:55

__device__ __forceinline__ uint64_t f2key(double v) {
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double key2f(uint64_t k) {
  const uint64_t b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

// block-wide maximum and sum; every thread gets the result
__device__ double block_max(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  double t = (lane < nw) ? red[lane] : 0.0;
  for (int o = 16; o > 0; o >>= 1) t = fmax(t, __shfl_xor_sync(0xffffffffu, t, o));
  return t;
}

// the sum with one barrier: red2 holds two 32-entry buffers used in turn by consecutive calls (a thread may start the next call's write while
// others still read this call's buffer, never the same buffer)
__device__ __forceinline__ double block_sum1(double v, double *red2, int parity) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  double *red = red2 + 32 * parity;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[w] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  double t = (lane < nw) ? red[lane] : 0.0;
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Vandermonde_kernel + QR_kernel (resample.h:14-37, 73-227), one CTA.
// V is column-major nxb x nc; on return it holds the Householder vectors
// below/on the diagonal and R above it; C, D as in the reference.
//
// moments = 1 (kdist_moments): the fit takes Q^T b from the bin's Chebyshev
// moments (fit_moments) and needs, of the reflections, only the row f = e_(nc-1)^T
// H_(nc-2) .. H_0 that gives the last element after nc - 1 of them, and the
// matrix M that takes (A^T b, f . b) to the coefficients (both substitutions
// with R).  f's first nc - 1 entries replace Cv[0 .. nc-2] and the others the
// last column from row nc - 1 on; M replaces R and the heads of the
// reflections, V[i + nxb j] for i, j < nc but for its last entry, 1 / D[nc-1].
// Dynamic shared memory: 2 nc^2 doubles with moments, else none.
// Latency of one CTA: two passes over a column (L2) and a barrier per pair of
// columns.  hk_kdist_noalloc, which factorises on each call, on 5 bins, without
// moments / with f and M formed by reflections of three barriers / so: 10000 x
// 20 1138 / 1195 / 1083 us, 2858 x 90 7960 / 8760 / 7730, 3000 x 30 1008 / 1046 /
// 889.
__global__ void __launch_bounds__(KD_THREADS)
qr_kernel(int nxb, int nc, int moments, double *__restrict__ V, double *__restrict__ Cv,
          double *__restrict__ D) {
  __shared__ double red[64], red_max[32], s_v0, s_head[KD_MAX_NC];
  for (int id = threadIdx.x; id < nxb; id += blockDim.x) {
    const double x = id * 2.0 / ((double)nxb - 1.0) - 1.0;
    V[id] = 1.0;
    if (nc > 1) V[id + (int64_t)nxb] = x;
    double t = x, t0 = 1.0;
    for (int i = 2; i < nc; ++i) {
      const double tt = t;
      t = __fma_rn(2.0 * x, t, -t0);
      t0 = tt;
      V[id + (int64_t)nxb * i] = t;
    }
  }
  __syncthreads();
  // Thread tid owns the rows k = tid + n blockDim in every column (nc <= blockDim),
  // so a sum's barrier is the only one a column needs.
  const int tid = threadIdx.x, nt = blockDim.x;
  int par = 0;  // block_sum1's buffer
  for (int i = 0; i < nc; ++i) {
    double *vi = V + (int64_t)nxb * i;
    const int k0 = tid >= i ? tid : tid + nt;  // the thread's first row at or below i
    double m = 0.0;
    for (int k = k0; k < nxb; k += nt) m = fmax(m, fabs(vi[k]));
    const double scale = block_max(m, red_max);
    double ss = 0.0;
    for (int k = k0; k < nxb; k += nt) {
      const double v = vi[k] / scale;
      vi[k] = v;
      ss = __fma_rn(v, v, ss);
    }
    if (tid == i) s_v0 = vi[i];
    ss = block_sum1(ss, red, par);  // (its barrier publishes s_v0)
    par ^= 1;
    const double s = sqrt(ss), v0 = s_v0;
    const double sigma = (v0 < 0.0) ? -s : s, c = sigma * (v0 + sigma);
    if (tid == i) {
      vi[i] = v0 + sigma;
      Cv[i] = c;
      D[i] = -scale * sigma;
    }
    for (int j = i + 1; j < nc; ++j) {
      double *vj = V + (int64_t)nxb * j;
      double dot = 0.0;
      for (int k = k0; k < nxb; k += nt) dot = __fma_rn(vi[k], vj[k], dot);
      dot = block_sum1(dot, red, par);
      par ^= 1;
      const double t = dot / c;
      for (int k = k0; k < nxb; k += nt) vj[k] = __fma_rn(-t, vi[k], vj[k]);
    }
  }
  if (!moments) return;
  // f = H_0 (H_1 ( .. H_(nc-2) e_(nc-1))), rows >= nc - 1 in the last column,
  // the first rows in s_head (every thread its own rows, as above)
  double *f = V + (int64_t)nxb * (nc - 1);
  for (int k = tid; k < nxb; k += nt) {
    if (k < nc - 1) s_head[k] = 0.0;
    else f[k] = k == nc - 1 ? 1.0 : 0.0;
  }
  for (int j = nc - 2; j >= 0; --j) {
    const double *vj = V + (int64_t)nxb * j;
    const int k0 = tid >= j ? tid : tid + nt;
    double dot = 0.0;
    for (int k = k0; k < nxb; k += nt) dot = __fma_rn(vj[k], k < nc - 1 ? s_head[k] : f[k], dot);
    dot = block_sum1(dot, red, par);
    par ^= 1;
    const double t = dot / Cv[j];
    for (int k = k0; k < nxb; k += nt) {
      double &w = k < nc - 1 ? s_head[k] : f[k];
      w = __fma_rn(-t, vj[k], w);
    }
  }
  __syncthreads();
  // column j of M: the unit vector j through the substitutions, thread j
  extern __shared__ double qr_dyn[];
  double *R = qr_dyn, *X = qr_dyn + nc * nc;  // X[i nc + j]: element i of column j
  for (int q = threadIdx.x; q < nc * nc; q += blockDim.x) {
    const int i = q / nc, j = q - i * nc;
    R[q] = j > i ? V[i + (int64_t)nxb * j] : (i == j ? D[i] : 0.0);
  }
  for (int k = threadIdx.x; k < nc - 1; k += blockDim.x) Cv[k] = s_head[k];
  __syncthreads();
  if (threadIdx.x < nc) {
    const int j = threadIdx.x;
    // R^T z = e_j on the first nc - 1 rows; the last element is f . b itself
    for (int i = 0; i < nc; ++i) {
      double t = i == j ? 1.0 : 0.0;
      if (i < nc - 1) {
        for (int k = 0; k < i; ++k) t = __fma_rn(-R[k * nc + i], X[k * nc + j], t);
        t /= R[i * nc + i];
      }
      X[i * nc + j] = t;
    }
    // R c = z (the reference's reduction keeps 64 partial sums)
    for (int i = nc - 1; i >= 0; --i) {
      double t = X[i * nc + j];
      for (int k = i + 1; k < nc && k < 64; ++k) t = __fma_rn(-R[i * nc + k], X[k * nc + j], t);
      t /= R[i * nc + i];
      X[i * nc + j] = t;
      if (i < nc - 1 || j < nc - 1) V[i + (int64_t)nxb * j] = t;
    }
  }
}

// Whether the fit of (nxb, nc) goes through the moments.  The Chebyshev basis on
// nxb equally spaced points degrades with nc^2 / nxb and, for few points, with
// nc / nxb: condition number 3.2 at 120 points x 20, 7.0 at 2858 x 100, 4.1 at
// 350 x 35 (6.1 at 10000 x 30) on this rule's edge, but 34 at 480 x 80 and 131 at
// 600 x 100 beyond it, and the moments square it.  Inside the rule the
// coefficients are nearer the exact fit than the reflections' (fit_moments).
// Below 4 coefficients the reflections do not spread a non-finite value to all
// of them, so those keep the reflections.
static __host__ __device__ inline bool kdist_moments(int nxb, int nc) {
  return nc >= 4 && 6 * nc <= nxb && 2 * nc * nc <= 7 * nxb;
}

// Threads that sum a bin in the fit, by its size alone: the narrowest CTA that
// holds it.  A wider CTA (few bins) lets as many of its threads sum in the same
// order, so a state keeps its coefficients in any batch and on any GPU.
static __host__ __device__ inline int kdist_sum_threads(int nxb) {
  return nxb > 6144 ? KD_THREADS : nxb > 3072 ? KD_THREADS / 2 : KD_THREADS / 4;
}

struct KdistArgs {
  const double *K;       // nstates x nx, unsorted
  int64_t k_stride;
  int nxb, nbins, nc, pow2;
  double kmin, unitScale;
  const double *V, *Cv, *D;
  double *coeff;         // nstates x nbins x nc
  int *nxmin;            // nstates x nbins
  double *sorted;        // optional nstates x nx
  double *recon;         // optional nstates x nx
  double *scratch;       // kdist_big_kernel's work
};

constexpr uint64_t KD_KEY_END = 0xffffffffffffffffull;  // after every key of a value

// 2 j / den - 1 with the quotient rounded as the division rounds it: a product
// with inv = 1 / den and one residual step (Markstein, IBM J. Res. Dev. 34, 1990).
// Equal to the division for every 0 <= j <= den <= 12300, and in 2e8 random
// pairs up to den = 2^31 (tests/test_fp64_helpers.py takes a part of them).
__device__ __forceinline__ double grid_pos(int j, double den, double inv) {
  const double t = 2.0 * j, q = t * inv;
  return __fma_rn(__fma_rn(-q, den, t), inv, q) - 1.0;
}

// findCut (resample.h:362-388) on the sorted bin: within a bin at most one
// index j has K[j] <= kmin < K[j+1]; the empty-bin rules follow it.  s_trans
// holds -1 and a barrier has passed.
__device__ __forceinline__ int find_cut(const double *work, int nxb, double kmin, bool last_bin,
                                        int *s_trans) {
  // transitions at local j <= nxb-2; for the bin's last index the reference's
  // "complete empty bin" rule gives the same Nxb (and the state's last index
  // is never visited: id < NL-1)
  for (int j = threadIdx.x; j < nxb - 1; j += blockDim.x)
    if (work[j] <= kmin && work[j + 1] > kmin) *s_trans = j;
  __syncthreads();
  const int jt = *s_trans;
  int nxmin = jt >= 0 ? jt + 1 : 0;
  if (!last_bin) {
    if (work[nxb - 1] <= kmin) nxmin = nxb;
  } else if (nxb >= 3 && work[nxb - 3] <= kmin) {
    // id == NL-3 rule; a transition at the later id NL-2 wins the race
    nxmin = (jt == nxb - 2) ? nxb - 1 : nxb;
  }
  return nxmin;
}

// rescale(+1) of one element
__device__ __forceinline__ double rescale_up(const double *work, int nxb, int nxmin, int j) {
  double ii = __fma_rn(1.0 - nxmin / ((double)(nxb - 1)), (double)j, (double)nxmin);
  if (ii >= nxb - 1) ii = 0.999999 * (nxb - 1);
  const int il = (int)(ii / ((double)nxb) * nxb);
  const double Kl = work[il], Kr = work[il + 1];
  return __fma_rn(Kr - Kl, ii - il, Kl);
}

// rescale(-1) of one element of the reconstruction
__device__ __forceinline__ double rescale_down(const double *work, int nxb, int nxmin, double kmin,
                                               int j) {
  if (nxmin <= 0) return work[j];
  if (j < nxmin) return kmin;
  double ii = (j - nxmin) / ((double)(nxb - nxmin - 1)) * (nxb - 1);
  if (ii >= nxb - 1) ii = 0.999999 * (nxb - 1);
  const int il = (int)(ii / ((double)nxb) * nxb);
  const double Kl = work[il], Kr = work[il + 1];
  return __fma_rn(Kr - Kl, ii - il, Kl);
}

// leastSquare_kernel with the reflections: Q^T b by the first nc-1 of them, the
// sums by kdist_sum_threads threads, each its elements k = tid + n vt (k >= j) in
// turn, then the back-substitution by one thread, whose result is s_c (and co).
// A CTA of that width needs one barrier per reflection, a wider one another for
// the elements that its other threads change.  red: 64 doubles.
__device__ void fit_reflections(const KdistArgs &a, double *work, const double *s_cv, const double *s_d,
                                double *red, double *s_c, double *__restrict__ co) {
  const int nxb = a.nxb, nc = a.nc, tid = threadIdx.x, nt = blockDim.x, vt = kdist_sum_threads(nxb);
  for (int j = 0; j < nc - 1; ++j) {
    const double *vj = a.V + (int64_t)nxb * j;
    double dot = 0.0;
    if (tid < vt)
      for (int k = tid; k < nxb; k += vt)
        if (k >= j) dot = __fma_rn(vj[k], work[k], dot);
    dot = block_sum1(dot, red, j & 1);
    const double t = dot / s_cv[j];
    for (int k = tid; k < nxb; k += nt)
      if (k >= j) work[k] = __fma_rn(-t, vj[k], work[k]);
    if (nt > vt) __syncthreads();
  }
  __syncthreads();
  if (tid == 0) {
    // the reference's reduction keeps 64 partial sums
    const int lim = nc < 64 ? nc : 64;
    double *bb = work;
    bb[nc - 1] /= s_d[nc - 1];
    for (int i = nc - 2; i >= 0; --i) {
      double sum = 0.0;
      for (int j = i + 1; j < lim; ++j) sum = __fma_rn(a.V[i + (int64_t)nxb * j], bb[j], sum);
      bb[i] = (bb[i] - sum) / s_d[i];
    }
    for (int i = 0; i < nc; ++i) {
      co[i] = bb[i];
      s_c[i] = bb[i];
    }
  }
  __syncthreads();
}

// The fit from the bin's Chebyshev moments m_j = sum_k T_j(x_k) b_k, j < nc-1:
// A^T b = R^T Q^T b, so a forward substitution with R gives the first nc - 1
// elements of Q^T b, and the last one, which the reference leaves with nc - 1
// reflections, is f . b; the coefficients are M (m, f . b) (qr_kernel).  The
// T_j come from their recurrence in registers, at x_k and -x_k together
// (T_j(-x) = (-1)^j T_j(x)): 10 DFMA per point for ten moments, where the
// reflections read 19 columns of V from L2 (1.5 MB per 10000-point bin) and
// closed each with a block-wide sum.  The moments go in groups of KD_MG, each
// running the recurrence up to its first.
//
// The moments are those of b - p, p the cubic through four of the sorted values
// (x = -1, -1/2, 1/2, 1; without its T_3 for nc = 4), and p's coefficients are
// added to the result: p lies in the span of T_0 .. T_(nc-2), which the fit gives
// back exactly (f is orthogonal to it), and what the sums and M round is then
// a small remainder, not b.  Largest coefficient error in 64 bits against
// extended precision, median over spectra (reflections / moments of b / of
// b - p): 10000 x 20 9.8e-16 / 2.8e-15 / 3.5e-16, 120 x 20 9.2e-16 / 3.2e-15 /
// 3.8e-16, 2858 x 100 9.2e-16 / 9.1e-15 / 6.1e-16.
// The sums are those of VT = kdist_sum_threads threads of NF elements or more; a
// wider CTA spreads their warps' groups over its own warps.
// buf: (groups * KD_MG + 1) * VT / 32 doubles, then M if it fits.
constexpr int KD_MG = 10;
template <int THREADS, int NF, int VT>
__device__ __forceinline__ void fit_moments(const KdistArgs &a, const double *b, const double *s_d,
                                            double *buf, int buf_doubles, double *s_z,
                                            double *s_c, double *__restrict__ co) {
  constexpr int WARPS = THREADS / 32;
  const int n = a.nxb, nc = a.nc, nm = nc - 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int groups = (nm + KD_MG - 1) / KD_MG;
  constexpr int VW = VT / 32;
  const bool sums = VT == THREADS || tid < VT;  // one of the VT threads
  double *Ms = buf + (groups * KD_MG + 1) * VW;
  const bool in_smem = (groups * KD_MG + 1) * VW + nc * nc <= buf_doubles;
  // M and f come from L2: their loads are issued before the moments' arithmetic
  double f[NF];
  const double *ft = a.V + (int64_t)n * nm;  // f, rows >= nc - 1
#pragma unroll
  for (int i = 0; i < NF; ++i) {
    const int k = tid + i * VT;
    f[i] = sums && k < n ? (k < nm ? a.Cv[k] : ft[k]) : 0.0;
  }
  if (in_smem)
    for (int q = tid; q < nc * nc; q += THREADS) {
      const int j = q / nc, i = q - j * nc;
      Ms[q] = q == nc * nc - 1 ? 1.0 / s_d[nm] : a.V[i + (int64_t)n * j];
    }
  double af = 0.0;
#pragma unroll
  for (int i = 0; i < NF; ++i) {
    const int k = tid + i * VT;
    if (sums && k < n) af = __fma_rn(f[i], b[k], af);
  }
  // (f is finite, but 0 x inf where b is not: the finite check below covers it)
  if (sums)
    for (int k = tid + NF * VT; k < n; k += VT) af = __fma_rn(ft[k], b[k], af);
  for (int o = 16; o > 0; o >>= 1) af += __shfl_xor_sync(0xffffffffu, af, o);
  if (lane == 0 && warp < VW) buf[groups * KD_MG * VW + warp] = af;
  // p = sum p_j T_j
  double p0, p1, p2, p3;
  {
    const int i1 = (n - 1) / 4, i2 = n - 1 - i1;
    const double ve = b[n - 1] + b[0], vi = b[i2] + b[i1], de = b[n - 1] - b[0], di = b[i2] - b[i1];
    p0 = (0.5 * ve + vi) * (1.0 / 3.0);
    p1 = (de + di) * (1.0 / 3.0);
    p2 = (ve - vi) * (1.0 / 3.0);
    p3 = nc > 4 ? (de - 2.0 * di) * (1.0 / 6.0) : 0.0;
  }
  const double den = (double)n - 1.0, inv = 1.0 / den;
  for (int u = warp; u < groups * VW; u += WARPS) {
    const int gq = u / VW, w = VT == THREADS ? warp : u - gq * VW;  // group, and warp of the VT threads
    double acc[KD_MG];
#pragma unroll
    for (int q = 0; q < KD_MG; ++q) acc[q] = 0.0;
    for (int k = w * 32 + lane; k < (n + 1) / 2; k += VT) {
      const int k2 = n - 1 - k;
      // (the middle point of an odd count has x = 0: odd T vanish)
      const bool two = k2 > k;
      const double bl = b[k], bh = two ? b[k2] : 0.0;
      const double x = grid_pos(k, den, inv), x2 = 2.0 * x, m2 = two ? -2.0 : -1.0;
      double ta = __fma_rn(x2, x, -1.0), tb = __fma_rn(x2, ta, -x);  // T_2, T_3
      // sum and difference of b - p at x and -x
      const double s = __fma_rn(m2, __fma_rn(p2, ta, p0), bl + bh);
      const double d = __fma_rn(m2, __fma_rn(p3, tb, p1 * x), bl - bh);
      if (gq == 0) {
        acc[0] += s;
        acc[1] = __fma_rn(x, d, acc[1]);
      } else {
        for (int i = 2; i < gq * KD_MG; i += 2) {
          ta = __fma_rn(x2, tb, -ta);
          tb = __fma_rn(x2, ta, -tb);
        }
        acc[0] = __fma_rn(ta, s, acc[0]);
        acc[1] = __fma_rn(tb, d, acc[1]);
        ta = __fma_rn(x2, tb, -ta);
        tb = __fma_rn(x2, ta, -tb);
      }
#pragma unroll
      for (int q = 2; q < KD_MG; q += 2) {
        acc[q] = __fma_rn(ta, s, acc[q]);
        acc[q + 1] = __fma_rn(tb, d, acc[q + 1]);
        ta = __fma_rn(x2, tb, -ta);
        tb = __fma_rn(x2, ta, -tb);
      }
    }
    // warp sums: the first level halves the values each lane carries
    const bool up = lane & 16;
#pragma unroll
    for (int q = 0; q < KD_MG / 2; ++q) {
      const double give = up ? acc[q] : acc[q + KD_MG / 2], keep = up ? acc[q + KD_MG / 2] : acc[q];
      acc[q] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < KD_MG / 2; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
    if ((lane & 15) == 0)
#pragma unroll
      for (int q = 0; q < KD_MG / 2; ++q) buf[(gq * KD_MG + q + (up ? KD_MG / 2 : 0)) * VW + w] = acc[q];
  }
  __syncthreads();
  // sums over the warps: value v to s_z[v], f . b to s_z[nc - 1]
  for (int v = warp; v < nc; v += WARPS) {
    const int src = v < nm ? v : groups * KD_MG;
    double t = lane < VW ? buf[src * VW + lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) s_z[v] = t;
  }
  __syncthreads();
  if (tid < nc) {
    double c = 0.0;
    if (in_smem) {
#pragma unroll 5
      for (int j = 0; j < nc; ++j) c = __fma_rn(Ms[j * nc + tid], s_z[j], c);
    } else {
      for (int j = 0; j < nc; ++j)
        c = __fma_rn(j == nm && tid == nm ? 1.0 / s_d[nm] : a.V[tid + (int64_t)n * j], s_z[j], c);
    }
    c += tid == 0 ? p0 : tid == 1 ? p1 : tid == 2 ? p2 : tid == 3 ? p3 : 0.0;
    // a non-finite b (m_0 sums b - p) leaves no coefficient finite
    if (!isfinite(s_z[0])) c = __longlong_as_double(0x7ff8000000000000ll);
    co[tid] = c;
    s_c[tid] = c;
  }
  __syncthreads();
}

// ------------------------------------------------- sort in shared memory
// the low 32 bits of (v - mn) >> sh
__device__ __forceinline__ unsigned prefix32(uint64_t v, uint64_t mn, int sh) {
  const uint64_t u = v - mn;
  const unsigned lo = (unsigned)u, hi = (unsigned)(u >> 32);
  return sh < 32 ? __funnelshift_r(lo, hi, sh) : hi >> (sh - 32);
}

// Sort by distribution of the keys v of the CTA (key e = warp 32 IPT + i 32 +
// lane in v[i], e < n), nfloor of which equal the smallest, floor, and the others
// lie at or above mn: they go to keys[nfloor ..] in the order of their
// prefixes (v - mn) >> sh, below KD_STEPS THREADS, each at its prefix's start
// plus the counter's atomic, and then each finds its place among those of its
// prefix by comparing with all of them.  False, with keys[] untouched, if more than
// KD_RUN keys share a prefix.
constexpr int KD_STEPS = 8, KD_RUN = 64;
template <int THREADS, int IPT>
__device__ __forceinline__ bool prefix_sort(const uint64_t (&v)[IPT], int n, uint64_t floor,
                                            int nfloor, uint64_t mn, int sh, uint64_t *keys,
                                            unsigned *cnt, int *s_scan, int *s_long) {
  constexpr int WARPS = THREADS / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint4 *c4 = reinterpret_cast<uint4 *>(cnt);
#pragma unroll
  for (int q = 0; q < KD_STEPS / 4; ++q) c4[tid + q * THREADS] = make_uint4(0, 0, 0, 0);
  if (tid == 0) *s_long = 0;
  __syncthreads();
  const int e0 = warp * 32 * IPT + lane;
  auto in = [&](int i) { return e0 + 32 * i < n && !(nfloor > 0 && v[i] == floor); };
  unsigned at_[IPT];
  // (the first key of every thread finds most crowded bins: the atomics of a
  // crowd are taken in turn.  480 bins of 10000 points in one crowd, sort alone:
  // 188 us without this look, 168 with it, 172 by the merge sort at once)
  at_[0] = in(0) ? atomicAdd(cnt + prefix32(v[0], mn, sh), 1u) : 0u;
  if (at_[0] >= KD_RUN) *s_long = 1;
  __syncthreads();
  if (*s_long) return false;
#pragma unroll
  for (int i = 1; i < IPT; ++i) at_[i] = in(i) ? atomicAdd(cnt + prefix32(v[i], mn, sh), 1u) : 0u;
  __syncthreads();
  uint4 c[KD_STEPS / 4];
  unsigned sum = 0, most = 0;
#pragma unroll
  for (int q = 0; q < KD_STEPS / 4; ++q) {
    c[q] = c4[(KD_STEPS / 4) * tid + q];
    sum += c[q].x + c[q].y + c[q].z + c[q].w;
    most = max(max(most, max(c[q].x, c[q].y)), max(c[q].z, c[q].w));
  }
  if (most > KD_RUN) *s_long = 1;
  unsigned incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) s_scan[warp] = (int)incl;
  __syncthreads();
  if (*s_long) return false;
  unsigned at = nfloor + incl - sum;
#pragma unroll
  for (int w = 0; w < WARPS; ++w)
    if (w < warp) at += s_scan[w];
#pragma unroll
  for (int q = 0; q < KD_STEPS / 4; ++q) {
    uint4 o;
    o.x = at;
    o.y = o.x + c[q].x;
    o.z = o.y + c[q].y;
    o.w = o.z + c[q].z;
    at = o.w + c[q].w;
    c4[(KD_STEPS / 4) * tid + q] = o;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < IPT; ++i)
    if (in(i)) {
      at_[i] += cnt[prefix32(v[i], mn, sh)];
      keys[at_[i]] = v[i];
    }
  for (int k = tid; k < nfloor; k += THREADS) keys[k] = floor;
  __syncthreads();
  if (sh == 0) return true;  // the prefix is the whole key
#pragma unroll
  for (int i = 0; i < IPT; ++i)
    if (in(i)) {
      const unsigned d = prefix32(v[i], mn, sh);
      const unsigned j0 = cnt[d], j1 = d + 1 < KD_STEPS * THREADS ? cnt[d + 1] : (unsigned)n;
      unsigned k = j0;
      for (unsigned j = j0; j < j1; ++j) {
        const uint64_t x = keys[j];
        k += x < v[i] || (x == v[i] && j < at_[i]);
      }
      at_[i] = k;
    }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < IPT; ++i)
    if (in(i)) keys[at_[i]] = v[i];
  __syncthreads();
  return true;
}

struct KeyLess {
  __device__ __forceinline__ bool operator()(uint64_t x, uint64_t y) const { return x < y; }
};

// The bin sorted into keys[] by a block merge sort in registers whose tile
// (THREADS IPT + 1 keys) uses tile; out of line, so that the usual path keeps
// its registers.
template <int THREADS, int IPT>
__device__ __noinline__ void merge_sort(const double *__restrict__ src, int n, void *tile, uint64_t *keys) {
  using Sorter = cub::BlockMergeSort<uint64_t, THREADS, IPT>;
  uint64_t v[IPT];
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const int e = threadIdx.x + i * THREADS;
    v[i] = e < n ? f2key(src[e]) : KD_KEY_END;
  }
  Sorter(*static_cast<typename Sorter::TempStorage *>(tile)).Sort(v, KeyLess());
  __syncthreads();  // the tile overlays keys[]
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const int k = threadIdx.x * IPT + i;
    if (k < n) keys[k] = v[i];
  }
  __syncthreads();
}

// One CTA per (state, bin), THREADS IPT >= nxb points, VT = kdist_sum_threads(nxb).
//
// Sort: the keys' span in the bin (largest - smallest, in the order of the
// FP64 bit patterns; points that no line reaches, at kmin, apart) is cut to
// KD_STEPS THREADS steps, about one per key, and prefix_sort orders the keys by
// step and within each step.  A bin whose values crowd into few steps takes a
// block merge sort in registers.
// Measured, 480 bins of 10000 points (block merge sort and reflections ->
// this): sort alone 173 -> 90 us (172 -> 168 for bins that fall back); with
// sorted values, fit of 20 coefficients and reconstruction written 482 -> 185.
// Bound: latency, one 1024-thread CTA per SM in phases between barriers (load
// 8 %, sort 35 %, ln 10 %, moments 25 %, reconstruction 16 % of a bin's time);
// its 115 MB of traffic would take 18 us.
template <int THREADS, int IPT, int VT>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
kdist_kernel(KdistArgs a) {
  constexpr int WARPS = THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[64];
  __shared__ uint64_t s_mm[2 * WARPS];
  __shared__ int s_trans, s_long, s_scan[WARPS];
  __shared__ double s_c[KD_MAX_NC], s_cv[KD_MAX_NC], s_d[KD_MAX_NC], s_z[KD_MAX_NC];
  const int b = blockIdx.x, s = blockIdx.y;
  const int nxb = a.nxb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned *cnt = reinterpret_cast<unsigned *>(smem_raw);  // KD_STEPS THREADS counters
  uint64_t *keys = reinterpret_cast<uint64_t *>(smem_raw + sizeof(unsigned) * KD_STEPS * THREADS);
  double *work = reinterpret_cast<double *>(keys);
  const double *src = a.K + (int64_t)s * a.k_stride + (int64_t)b * nxb;

  // the smallest key other than floor (kmin's) and the largest; how many are floor
  const uint64_t floor = f2key(a.kmin);
  uint64_t v[IPT], mn = KD_KEY_END, mx = 0;
  int nf = 0;
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const int e = warp * 32 * IPT + i * 32 + lane;
    v[i] = KD_KEY_END;
    if (e < nxb) {
      v[i] = f2key(src[e]);
      if (v[i] == floor) ++nf;
      else mn = v[i] < mn ? v[i] : mn;
      mx = v[i] > mx ? v[i] : mx;
    }
  }
  for (int i = tid; i < a.nc; i += THREADS) {
    s_cv[i] = a.Cv[i];
    s_d[i] = a.D[i];
  }
  if (tid == 0) s_trans = -1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint64_t u = __shfl_xor_sync(0xffffffffu, mn, o), w = __shfl_xor_sync(0xffffffffu, mx, o);
    mn = u < mn ? u : mn;
    mx = w > mx ? w : mx;
  }
  nf = __reduce_add_sync(0xffffffffu, nf);
  if (lane == 0) {
    s_mm[warp] = mn;
    s_mm[WARPS + warp] = mx;
    s_scan[warp] = nf;
  }
  __syncthreads();
  int nfloor = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    mn = s_mm[w] < mn ? s_mm[w] : mn;
    mx = s_mm[WARPS + w] > mx ? s_mm[WARPS + w] : mx;
    nfloor += s_scan[w];
  }
  if (nfloor == nxb) {
    mn = mx;
  } else if (nfloor > 0 && mn < floor) {
    nfloor = 0;  // floor is not the smallest key: no key apart
  }
  const int bits = 64 - __clzll((long long)(mx - mn));
  const int sh = max(0, bits - (31 - __clz(KD_STEPS * THREADS)));
  if (!prefix_sort<THREADS, IPT>(v, nxb, floor, nfloor, mn, sh, keys, cnt, s_scan, &s_long))
    merge_sort<THREADS, IPT>(src, nxb, smem_raw, keys);
  double *dst = a.sorted ? a.sorted + (int64_t)s * a.k_stride + (int64_t)b * nxb : nullptr;
  for (int i = tid; i < nxb; i += THREADS) {
    const double x = key2f(keys[i]);
    work[i] = x;
    if (dst) dst[i] = x;
  }
  if (a.coeff == nullptr) return;
  __syncthreads();
  const int nxmin = find_cut(work, nxb, a.kmin, b == a.nbins - 1, &s_trans);
  if (tid == 0) a.nxmin[(int64_t)s * a.nbins + b] = nxmin;
  if (nxmin > 0) {
    double t[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const int j = tid + i * THREADS;
      if (j < nxb) t[i] = rescale_up(work, nxb, nxmin, j);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const int j = tid + i * THREADS;
      if (j < nxb) work[j] = t[i];
    }
  }
  __syncthreads();
  for (int j = tid; j < nxb; j += THREADS) work[j] = log(work[j] * a.unitScale);
  __syncthreads();
  const int nc = a.nc;
  double *co = a.coeff + ((int64_t)s * a.nbins + b) * nc;
  if (kdist_moments(nxb, nc))
    fit_moments<THREADS, IPT * (THREADS / VT) < 12 ? IPT * (THREADS / VT) : 12, VT>(a, work, s_d, reinterpret_cast<double *>(cnt), KD_STEPS * THREADS / 2, s_z, s_c, co);
  else
    fit_reflections(a, work, s_cv, s_d, red, s_c, co);
  if (a.recon == nullptr) return;

  // expfx_kernel (x = -1 + 2 j / Nxb) then rescale(-1): the even and odd parts
  // of the series at x give the values at x and -x = x_(Nxb - j)
  const double inv = 1.0 / (double)nxb, iu = 1.0 / a.unitScale;
  for (int j = tid; j <= nxb / 2; j += THREADS) {
    const double x = grid_pos(j, (double)nxb, inv), x2 = 2.0 * x;
    double ta = __fma_rn(x2, x, -1.0), tb = __fma_rn(x2, ta, -x), ev = 0.0, od = 0.0;  // T_2, T_3
    int i = 2;
    for (; i + 1 < nc; i += 2) {
      ev = __fma_rn(ta, s_c[i], ev);
      od = __fma_rn(tb, s_c[i + 1], od);
      ta = __fma_rn(x2, tb, -ta);
      tb = __fma_rn(x2, ta, -tb);
    }
    if (i < nc) ev = __fma_rn(ta, s_c[i], ev);
    // the two largest terms last, so the others' roundings stay small (10000 x 20:
    // 0.7e-15 rms of the value, 1.3e-15 with them first, 0.9e-15 by Clenshaw's sum)
    ev += s_c[0];
    if (nc > 1) od = __fma_rn(x, s_c[1], od);
    work[j] = exp(ev + od) * iu;
    if (j > 0 && nxb - j > j) work[nxb - j] = exp(ev - od) * iu;
  }
  __syncthreads();
  double *rec = a.recon + (int64_t)s * a.k_stride + (int64_t)b * nxb;
  for (int j = tid; j < nxb; j += THREADS) rec[j] = rescale_down(work, nxb, nxmin, a.kmin, j);
}

// Bins above KD_MAX_NXB points: the same chain on a global scratch slice of
// next_pow2(nxb) + nxb words per bin, sorted by a bitonic network.
__global__ void __launch_bounds__(KD_THREADS)
kdist_big_kernel(KdistArgs a) {
  __shared__ double red[64];
  __shared__ int s_trans;
  __shared__ double s_c[KD_MAX_NC], s_cv[KD_MAX_NC], s_d[KD_MAX_NC], s_z[KD_MAX_NC];
  constexpr int BUF = 4096;  // (groups KD_MG + 1) 32 at nc = 100, and M up to nc = 29
  __shared__ double s_buf[BUF];
  const int b = blockIdx.x, s = blockIdx.y;
  const int nxb = a.nxb, P2 = a.pow2;
  const int tid = threadIdx.x, nt = blockDim.x;
  const size_t slot = ((size_t)s * a.nbins + b) * (size_t)(P2 + nxb);
  uint64_t *keys = reinterpret_cast<uint64_t *>(a.scratch + slot);
  double *work = a.scratch + slot + P2;
  const double *src = a.K + (int64_t)s * a.k_stride + (int64_t)b * nxb;
  for (int i = tid; i < P2; i += nt) keys[i] = (i < nxb) ? f2key(src[i]) : KD_KEY_END;
  for (int i = tid; i < a.nc; i += nt) {
    s_cv[i] = a.Cv[i];
    s_d[i] = a.D[i];
  }
  if (tid == 0) s_trans = -1;
  __syncthreads();
  for (int size = 2; size <= P2; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = tid; i < (P2 >> 1); i += nt) {
        const int pos = 2 * i - (i & (stride - 1));
        const int q = pos + stride;
        const uint64_t x = keys[pos], y = keys[q];
        const bool up = (pos & size) == 0;
        if ((x > y) == up) {
          keys[pos] = y;
          keys[q] = x;
        }
      }
      __syncthreads();
    }
  }
  for (int i = tid; i < nxb; i += nt) work[i] = key2f(keys[i]);
  __syncthreads();
  if (a.sorted) {
    double *dst = a.sorted + (int64_t)s * a.k_stride + (int64_t)b * nxb;
    for (int i = tid; i < nxb; i += nt) dst[i] = work[i];
  }
  if (a.coeff == nullptr) return;
  const int nxmin = find_cut(work, nxb, a.kmin, b == a.nbins - 1, &s_trans);
  if (tid == 0) a.nxmin[(int64_t)s * a.nbins + b] = nxmin;
  if (nxmin > 0) {
    double *tmp = reinterpret_cast<double *>(keys);
    for (int j = tid; j < nxb; j += nt) tmp[j] = rescale_up(work, nxb, nxmin, j);
    __syncthreads();
    for (int j = tid; j < nxb; j += nt) work[j] = tmp[j];
  }
  __syncthreads();
  for (int j = tid; j < nxb; j += nt) work[j] = log(work[j] * a.unitScale);
  __syncthreads();
  const int nc = a.nc;
  double *co = a.coeff + ((int64_t)s * a.nbins + b) * nc;
  if (kdist_moments(nxb, nc)) fit_moments<KD_THREADS, 8, KD_THREADS>(a, work, s_d, s_buf, BUF, s_z, s_c, co);
  else fit_reflections(a, work, s_cv, s_d, red, s_c, co);
  if (a.recon == nullptr) return;

  // expfx_kernel (x = -1 + 2 j / Nxb) then rescale(-1)
  for (int j = tid; j < nxb; j += nt) {
    const double x = -1.0 + j * 2.0 / ((double)nxb);
    double d1 = 0.0, d2 = 0.0;
    for (int i = nc - 1; i >= 1; --i) {
      const double t = d1;
      d1 = __fma_rn(2.0 * x, d1, -d2) + s_c[i];
      d2 = t;
    }
    const double f = __fma_rn(x, d1, -d2) + 0.5 * s_c[0] + 0.5 * s_c[0];
    work[j] = exp(f) / a.unitScale;
  }
  __syncthreads();
  double *dst = a.recon + (int64_t)s * a.k_stride + (int64_t)b * nxb;
  for (int j = tid; j < nxb; j += nt) dst[j] = rescale_down(work, nxb, nxmin, a.kmin, j);
}

__global__ void grid_pos_kernel(int64_t n, const double *__restrict__ j, const double *__restrict__ den,
                                double *__restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = grid_pos((int)j[i], den[i], 1.0 / den[i]);
}

cudaError_t launch_grid_pos(int64_t n, const double *j_d, const double *den_d, double *out_d, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  grid_pos_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(n, j_d, den_d, out_d);
  return cudaGetLastError();
}

static int next_pow2(int v) {
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}

size_t kdist_scratch_doubles(int nxb, int nbins, int nstates) {
  if (nxb <= KD_MAX_NXB) return 0;
  return (size_t)nstates * nbins * (size_t)(next_pow2(nxb) + nxb);
}

cudaError_t launch_qr(int nxb, int nc, double *V_d, double *C_d, double *D_d,
                      cudaStream_t stream) {
  const bool moments = kdist_moments(nxb, nc);
  const size_t dyn = moments ? 2 * sizeof(double) * (size_t)nc * nc : 0;
  if (dyn > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(qr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
  }
  qr_kernel<<<1, KD_THREADS, dyn, stream>>>(nxb, nc, moments, V_d, C_d, D_d);
  return cudaGetLastError();
}

cudaError_t launch_kdist(const double *K_d, int64_t k_stride, int nstates,
                         int nxb, int nbins, int nc, double kmin,
                         double unitScale, const double *V_d, const double *C_d,
                         const double *D_d, double *coeff_d, int *nxmin_d,
                         double *sorted_d, double *recon_d, double *scratch_d,
                         cudaStream_t stream) {
  if (nstates <= 0 || nbins <= 0) return cudaSuccess;
  KdistArgs a;
  a.K = K_d;
  a.k_stride = k_stride;
  a.nxb = nxb;
  a.nbins = nbins;
  a.nc = nc;
  a.pow2 = next_pow2(nxb);
  a.kmin = kmin;
  a.unitScale = unitScale;
  a.V = V_d;
  a.Cv = C_d;
  a.D = D_d;
  a.coeff = coeff_d;
  a.nxmin = nxmin_d;
  a.sorted = sorted_d;
  a.recon = recon_d;
  a.scratch = scratch_d;
  const dim3 grid(nbins, nstates);
  if (nxb > KD_MAX_NXB) {
    if (scratch_d == nullptr) return cudaErrorInvalidValue;
    kdist_big_kernel<<<grid, KD_THREADS, 0, stream>>>(a);
    return cudaGetLastError();
  }
  auto run = [&](auto kfn, int threads, int keys) -> cudaError_t {
    // counters and keys; the merge sort's tile overlays them
    const size_t dyn = std::max(sizeof(unsigned) * KD_STEPS * threads + (size_t)nxb * 8,
                                ((size_t)threads * keys + 2) * 8);
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    kfn<<<grid, threads, dyn, stream>>>(a);
    return cudaGetLastError();
  };
  // 1024 threads share an SM: the smallest CTA that holds the bin at 12 keys a
  // thread lets the barriers of one bin hide behind another's work (20
  // coefficients, 3000 points: 3000 bins 191 us in 256 threads, 241 in 512, 346
  // in 1024; 6000 points 395 in 512, 498 in 1024); with fewer bins than SMs a
  // wider CTA finishes its bin sooner (30 bins of 3000 points 25 us in 1024
  // threads, 31 in 256; 6000 points 33 in 1024, 37 in 512).  The coefficients
  // are the same to the bit (kdist_sum_threads).
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int64_t ctas = (int64_t)nbins * nstates;
  const int thr = (nxb > 6144 || ctas <= nsm) ? 1024 : (nxb > 3072 || ctas <= 2 * nsm) ? 512 : 256;
  const int ipt = (nxb + thr - 1) / thr, vt = kdist_sum_threads(nxb);
#define KD_CASE(T, I, V) \
  if (thr == T && ipt <= I && vt == V) return run(kdist_kernel<T, I, V>, T, I);
  KD_CASE(1024, 8, 1024)
  KD_CASE(1024, 10, 1024)
  KD_CASE(1024, 12, 1024)
  KD_CASE(1024, 4, 512)
  KD_CASE(1024, 6, 512)
  KD_CASE(1024, 2, 256)
  KD_CASE(1024, 4, 256)
  KD_CASE(512, 8, 512)
  KD_CASE(512, 10, 512)
  KD_CASE(512, 12, 512)
  KD_CASE(512, 4, 256)
  KD_CASE(512, 8, 256)
  KD_CASE(256, 4, 256)
  KD_CASE(256, 8, 256)
  KD_CASE(256, 12, 256)
#undef KD_CASE
  return cudaErrorInvalidValue;
}

}  // namespace hkb
