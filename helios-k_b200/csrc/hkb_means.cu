// hkb_means.cu -- Planck / Rosseland mean opacities and the transmission
// function of the binned opacity (sm_100a), FP64.
//
// Means (resample.h:635-773, Mean_kernel + IntegrateMean_kernel, equal
// spacing): per state, over the grid,
//   S0 = sum B K,  S1 = sum (dB/dT) / K (K != 0),  S2 = sum B,  S3 = sum dB/dT,
// plus the reference's end weights; Planck mean = S0 / S2, Rosseland mean =
// S3 / S1.  B and dB/dT are formed per point inside the reduction (the
// reference writes them to two Nx arrays first), so one pass reads K once:
// means_partial_kernel sums grid chunks, means_final_kernel adds the chunks
// in a fixed order and the end weights (deterministic).
//
// Transmission (resample.h:541-608, Integrate_kernel): per (state, bin) and
// m_j = exp((j - nTr/2) dTr),
//   Tr_j = (sum_k exp(-K_k m_j) + end weights) / (Nxb - 1) (Nxb - Nxmin) / Nxb
//          + exp(-kmin m_j) Nxmin / Nxb.
// One CTA per (state, bin) stages the bin in shared memory once; each warp
// takes values j (no block barrier per j, where the reference reduces 512
// threads per j).  Blocks of TR_B consecutive values whose spread times m_j is
// small -- most blocks of a sorted bin, at most m_j -- are one exponential and
// a polynomial; the others are summed value by value.
#include <cuda_runtime.h>

#include <algorithm>

#include "hkb_device.cuh"
#include "hkb_kernels.h"

namespace hkb {

// resample.h:611-619: index idy gets w[idy], index n-1-idy gets w[2-idy]
__constant__ double c_wS[3] = {-5.0 / 8.0, 1.0 / 6.0, -1.0 / 24.0};

// Mean_kernel's Planck function and its T derivative, same operations
__device__ __forceinline__ void planck_bd(double nu, double T, double &B, double &R) {
  if (nu == 0.0) {
    B = 0.0;
    R = 0.0;
    return;
  }
  const double nu3 = __dmul_rn(__dmul_rn(nu, nu), nu);
  const double t1 = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(2.0, HK_H), nu3), HK_C), HK_C);
  const double t2 = __ddiv_rn(__dmul_rn(__dmul_rn(HK_H, nu), HK_C), __dmul_rn(HK_KB, T));
  const double e = exp(t2);
  B = __ddiv_rn(t1, __dsub_rn(e, 1.0));
  R = __ddiv_rn(__dmul_rn(t1, t2), __dmul_rn(T, __dadd_rn(__dsub_rn(e, 2.0), __ddiv_rn(1.0, e))));
}

constexpr int MN_THREADS = 256;

__global__ void __launch_bounds__(MN_THREADS)
means_partial_kernel(const double *__restrict__ K, int64_t k_stride, GridDev g,
                     const double *__restrict__ T, int nchunk, double *__restrict__ part) {
  const int s = blockIdx.y, c = blockIdx.x;
  const double Ts = T[s];
  const double *Ks = K + (int64_t)s * k_stride;
  const int64_t per = (g.nx + nchunk - 1) / nchunk;
  const int64_t i0 = (int64_t)c * per, i1 = min(i0 + per, g.nx);
  double a[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t i = i0 + threadIdx.x; i < i1; i += MN_THREADS) {
    double B, R;
    planck_bd(grid_x(g, i), Ts, B, R);
    const double k = Ks[i];
    a[0] = __fma_rn(B, k, a[0]);
    if (k != 0.0) a[1] = __dadd_rn(a[1], __ddiv_rn(R, k));
    a[2] = __dadd_rn(a[2], B);
    a[3] = __dadd_rn(a[3], R);
  }
  __shared__ double red[4][MN_THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    double v = a[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[q][w] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    for (int k = 0; k < MN_THREADS / 32; ++k) v += red[threadIdx.x][k];
    part[((int64_t)s * nchunk + c) * 4 + threadIdx.x] = v;
  }
}

__global__ void means_final_kernel(const double *__restrict__ K, int64_t k_stride, GridDev g,
                                   const double *__restrict__ T, int nchunk,
                                   const double *__restrict__ part, double *__restrict__ out) {
  // warp q adds the chunks of sum q: lane-strided, then a shuffle tree
  const int s = blockIdx.x, q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v = 0.0;
  for (int c = lane; c < nchunk; c += 32) v += part[((int64_t)s * nchunk + c) * 4 + q];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane != 0) return;
  const double *Ks = K + (int64_t)s * k_stride;
  const int64_t n = g.nx;
  for (int idy = 0; idy < 3 && n >= 3; ++idy) {
    const int64_t ia[2] = {idy, n - 1 - idy};
    const double wt[2] = {c_wS[idy], c_wS[2 - idy]};
    for (int e = 0; e < 2; ++e) {
      double B, R;
      planck_bd(grid_x(g, ia[e]), T[s], B, R);
      const double k = Ks[ia[e]];
      if (q == 0) v = __dadd_rn(v, __dmul_rn(wt[e], __dmul_rn(B, k)));
      if (q == 1 && k != 0.0) v = __dadd_rn(v, __dmul_rn(wt[e], __ddiv_rn(R, k)));
      if (q == 2) v = __dadd_rn(v, __dmul_rn(wt[e], B));
      if (q == 3) v = __dadd_rn(v, __dmul_rn(wt[e], R));
    }
  }
  out[(int64_t)s * 4 + q] = v;
}

size_t means_scratch_doubles(int nstates, int64_t nx) {
  const int nchunk = (int)std::min<int64_t>(592, std::max<int64_t>(1, nx / 4096));
  return (size_t)nstates * nchunk * 4;
}

cudaError_t launch_means(const double *K_d, int64_t k_stride, const GridDev &g, const double *T_d,
                         int nstates, double *scratch_d, double *out_d, cudaStream_t stream) {
  if (nstates <= 0 || g.nx <= 0) return cudaSuccess;
  const int nchunk = (int)std::min<int64_t>(592, std::max<int64_t>(1, g.nx / 4096));
  dim3 grid(nchunk, nstates);
  means_partial_kernel<<<grid, MN_THREADS, 0, stream>>>(K_d, k_stride, g, T_d, nchunk, scratch_d);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  means_final_kernel<<<nstates, 128, 0, stream>>>(K_d, k_stride, g, T_d, nchunk, scratch_d, out_d);
  return cudaGetLastError();
}

// ------------------------------------------------------------ transmission
constexpr int TR_THREADS = 1024;
constexpr int TR_SMEM_MAX = 200 * 1024;  // values that do not fit stay in global memory (L2)
// Sum over a block of exp(-K_k m) = exp(-c m) sum_k exp(-(K_k - c) m), c the middle
// of the block's values and h their half spread: for d = h m <= 1 its Taylor
// series to degree TR_P leaves d^19 / 19! < 1e-17, with the block's power
// sums sum_k ((K_k - c) / h)^p / p! formed once per bin.
constexpr int TR_B = 32, TR_P = 18;

// Bins below this many points, or this many exponentials, are summed value by
// value: forming the power sums takes each block's thread a few us (300 bins,
// with / without them: 300 points and 10 m_j 58 / 42 us, 1000 m_j 572 / 598; 1000
// points and 10 m_j 67 / 54, 100 m_j 132 / 147, 1000 m_j 631 / 997).
constexpr int TR_MIN_NXB = 512, TR_MIN_EXPS = 30000;

// doubles of shared memory per block: c, h, the smallest value, TR_P + 1 sums
constexpr int TR_W = TR_P + 4;
static size_t tr_words(int nxb) { return (size_t)((nxb + TR_B - 1) / TR_B) * TR_W * sizeof(double); }

// 180 bins of 10000 values x 1000 m_j: 4.58 ms with an exponential per value
// (1.8e9 of them), 0.58 ms so (about 40 of 313 blocks per m_j still value by
// value).  Bound: instruction issue (74 % of slots; FP64 pipe 43 %).  Unsorted
// values of 13 decades, whose blocks are all too wide: 300 bins of 10000 x 100 m_j
// 824 us value by value, 1098 with power sums that no m_j can use, 813 without.
__global__ void __launch_bounds__(TR_THREADS)
transmission_kernel(const double *__restrict__ K, int64_t k_stride, int nxb, int nbins,
                    const int *__restrict__ nxmin, double kmin, int nTr, double dTr, int use_smem,
                    int poly_ok, double *__restrict__ Tr) {
  extern __shared__ __align__(16) double kb_s[];
  const int b = blockIdx.x, s = blockIdx.y;
  const double *src = K + (int64_t)s * k_stride + (int64_t)b * nxb;
  const double *kb = src;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nblk = (nxb + TR_B - 1) / TR_B;
  // block q's words at w[word nblk + q]
  double *w = use_smem ? kb_s + nxb : kb_s;
  if (use_smem) {
    for (int k = threadIdx.x; k < nxb; k += TR_THREADS) kb_s[k] = src[k];
    __syncthreads();
    kb = kb_s;
  }
  if (poly_ok) {
    // the third smallest m_j
    const double m3 = exp(fmin(-(nTr / 2) * dTr, (nTr - 1 - nTr / 2) * dTr) + 2.0 * fabs(dTr));
    for (int q = threadIdx.x; q < nblk; q += TR_THREADS) {
      // (each lane starts at another value of its block: no bank conflicts)
      const int k0 = q * TR_B, nk = min(TR_B, nxb - k0);
      double lo = kb[k0], hi = lo;
      bool finite = true;
      for (int i = 0; i < TR_B; ++i) {
        const int k = (i + lane) & (TR_B - 1);
        if (k >= nk) continue;
        const double v = kb[k0 + k];
        lo = fmin(lo, v);
        hi = fmax(hi, v);
        finite = finite && isfinite(v);
      }
      const double c = 0.5 * lo + 0.5 * hi, h = 0.5 * hi - 0.5 * lo, ih = h > 0.0 ? 1.0 / h : 0.0;
      // (a spread too small to divide by, or a value that is not finite: value by
      // value; so a spread too wide for all but the two smallest m_j, whose power
      // sums would cost more than they save)
      const bool ok = finite && (h == 0.0 || isfinite(ih)) && h * m3 <= 1.0;
      double a[TR_P + 1];
#pragma unroll
      for (int p = 0; p <= TR_P; ++p) a[p] = 0.0;
      for (int i = 0; i < TR_B && ok; ++i) {
        const int k = (i + lane) & (TR_B - 1);
        if (k >= nk) continue;
        const double t = (kb[k0 + k] - c) * ih;
        double tp = 1.0;
#pragma unroll
        for (int p = 0; p <= TR_P; ++p) {
          a[p] += tp;
          tp *= t;
        }
      }
      w[q] = c;
      w[nblk + q] = ok ? h : CUDART_INF;
      w[2 * nblk + q] = finite ? lo : -CUDART_INF;
      double f = 1.0;
#pragma unroll
      for (int p = 0; p <= TR_P; ++p) {
        w[(3 + p) * nblk + q] = a[p] * f;
        f *= -1.0 / (p + 1.0);  // (-1)^p / p!
      }
    }
    __syncthreads();
  }
  const int nm = nxmin ? nxmin[(int64_t)s * nbins + b] : 0;
  double *out = Tr + ((int64_t)s * nbins + b) * nTr;
  // this CTA's share of the m_j (gridDim.z of them per bin)
  for (int j = blockIdx.z * (TR_THREADS / 32) + warp; j < nTr; j += gridDim.z * (TR_THREADS / 32)) {
    const double m = exp((double)(j - nTr / 2) * dTr);
    double a = 0.0;
    if (poly_ok) {
      for (int q0 = 0; q0 < nblk; q0 += 32) {
        const int q = q0 + lane;
        const double d = q < nblk ? w[nblk + q] * m : 0.0;
        // (beyond 700 the factor exp(-c m) would be subnormal)
        const bool poly = q < nblk && d <= 1.0 && w[q] * m < 700.0;
        // exp(-x) is 0 beyond x = 745.2
        bool each = q < nblk && !poly && !(w[2 * nblk + q] * m > 746.0);
        if (poly) {
          double t = w[(3 + TR_P) * nblk + q];
#pragma unroll
          for (int p = TR_P - 1; p >= 0; --p) t = __fma_rn(t, d, w[(3 + p) * nblk + q]);
          a = __fma_rn(exp(-w[q] * m), t, a);
        }
        unsigned e = __ballot_sync(0xffffffffu, each);
        if (e == __ballot_sync(0xffffffffu, q < nblk)) {
          // every block of the group (unsorted values): one loop over them
          const int end = min(nxb, (q0 + 32) * TR_B);
#pragma unroll 4
          for (int k = q0 * TR_B + lane; k < end; k += 32) a += exp(-kb[k] * m);
          e = 0u;
        }
        for (; e; e &= e - 1) {
          const int k = (q0 + __ffs(e) - 1) * TR_B + lane;
          if (k < nxb) a += exp(-kb[k] * m);
        }
      }
    } else {
      for (int k = lane; k < nxb; k += 32) a += exp(-kb[k] * m);
    }
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) {
      for (int idy = 0; idy < 3 && nxb >= 3; ++idy) {
        a = __dadd_rn(a, __dmul_rn(c_wS[idy], exp(-kb[idy] * m)));
        a = __dadd_rn(a, __dmul_rn(c_wS[2 - idy], exp(-kb[nxb - 1 - idy] * m)));
      }
      const double t0 = __ddiv_rn(__dmul_rn(__ddiv_rn(a, (double)(nxb - 1)), (double)(nxb - nm)),
                                  (double)nxb);
      const double t1 = __ddiv_rn(__dmul_rn(exp(-kmin * m), (double)nm), (double)nxb);
      out[j] = __dadd_rn(t0, t1);
    }
  }
}

cudaError_t launch_transmission(const double *K_d, int64_t k_stride, int nstates, int nxb,
                                int nbins, const int *nxmin_d, double kmin, int nTr, double dTr,
                                double *Tr_d, cudaStream_t stream) {
  if (nstates <= 0 || nbins <= 0 || nTr <= 0) return cudaSuccess;
  const size_t words = tr_words(nxb), vals = (size_t)nxb * sizeof(double);
  const int poly_ok = words <= (size_t)TR_SMEM_MAX && nxb >= TR_MIN_NXB && (int64_t)nxb * nTr >= TR_MIN_EXPS;
  const int use_smem = vals + (poly_ok ? words : 0) <= (size_t)TR_SMEM_MAX;
  const size_t smem = (use_smem ? vals : 0) + (poly_ok ? words : 0);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(transmission_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  // One CTA per SM (registers): the m_j of a bin are shared by as many CTAs as
  // waste the least of the last wave; staging a bin and its power sums again
  // costs about 2 % of its 1000 sums.
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int64_t bins = (int64_t)nbins * nstates;
  int share = 1;
  double best = 0.0;
  for (int z = 1; z <= 8 && z * TR_THREADS / 32 <= std::max(nTr, TR_THREADS / 32); ++z) {
    const double cost = (double)((bins * z + nsm - 1) / nsm) * (1.0 / z + 0.02 * 1000.0 / nTr);
    if (z == 1 || cost < best) {
      best = cost;
      share = z;
    }
  }
  dim3 grid(nbins, nstates, share);
  transmission_kernel<<<grid, TR_THREADS, smem, stream>>>(
      K_d, k_stride, nxb, nbins, nxmin_d, kmin, nTr, dTr, use_smem, poly_ok, Tr_d);
  return cudaGetLastError();
}

}  // namespace hkb
