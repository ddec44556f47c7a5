/*
 * ncg_prepare.cu -- device side of NcmStatsDistKDE / NcmStatsDistVKDE prepare.
 *
 *  global_cov       Welford covariance of all centres
 *  global_chol      its upper Cholesky
 *                   (numcosmo/ncm/stats/ncm_stats_dist_kde.c:379-450,
 *                    numcosmo/ncm/stats/ncm_stats_vec.c:511-565,2376-2398)
 *  whiten           invUsample = X U^{-1}  (ncm_stats_dist_kde.c:477-480)
 *  knn              exact k nearest neighbours in the whitened space, ordered
 *                   by (squared distance, index) as the reference kd-tree
 *                   (numcosmo/external/misc/kdtree.c:28-38,193-320,
 *                    numcosmo/external/misc/rb_knn_list.c:32-40)
 *  local_cov_chol   per-kernel Welford covariance of the neighbours (in that
 *                   order) + Cholesky (ncm_stats_dist_vkde.c:426-488)
 *  nearpd           Higham nearPD / diagonal fallback for the factors that
 *                   failed (ncm_stats_dist_vkde.c:338-360,
 *                   numcosmo/ncm/algebra/ncm_matrix.c:1248-1344)
 *  vkde_finish      lnnorm_i (ncm_stats_dist_kernel_{gauss,st}.c get_lnnorm)
 *                   and the eval operand U_i^{-T}/h
 *
 * The covariance, Cholesky, whitening and distance arithmetic use explicitly
 * rounded operations (no FMA contraction) in the reference's operation order,
 * so the factors and the kNN sets are bit-identical to a CPU evaluation of
 * the same formulas compiled without contraction.
 */
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "ncg_internal.h"

#include <mutex>

/* Raise a kernel's dynamic shared-memory limit on the current device to at
 * least `bytes`, never lowering it: host threads that launch the same kernel
 * with different sizes at the same time (several handles prepared at once)
 * cannot then launch under a smaller limit another thread set in between.
 * limit[dev] remembers what was set, under one lock for all kernels. */
static std::mutex g_smem_mu;

extern "C" cudaError_t
ncg_raise_smem_limit (const void *fn, size_t bytes, int *limit)
{
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);

  if (e != cudaSuccess)
    return e;

  if (dev < 0 || dev >= NCG_MAX_DEVICES)
    return cudaErrorInvalidDevice;

  std::lock_guard<std::mutex> lock (g_smem_mu);

  if ((size_t) limit[dev] >= bytes)
    return cudaSuccess;

  e = cudaFuncSetAttribute (fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bytes);

  if (e == cudaSuccess)
    limit[dev] = (int) bytes;

  return e;
}

#define PREP_THREADS 128

/* ------------------------------------------------------------------------ */
/* Welford covariance (ncm_stats_vec.c:511-565, get_cov_matrix :2376-2398),   */
/* bit for bit in the reference's order.  With weight t (rows so far) and     */
/* mean m, row x does                                                        */
/*   delta = x - m;  R = delta / (t + 1);  m += R;  var += (t delta) R;        */
/*   C_rc += (x_r - m_r) delta_c      (m_r updated, delta_c from before).      */
/*                                                                          */
/* What bounds it: the running mean is one dependent chain per coordinate,    */
/* and a dependent FP64 instruction takes 64 cycles here, a division 561      */
/* (measured).  The divisor t + 1 is known in advance, so the quotient is      */
/* taken as R = fma (delta, yh, delta * yl) with yh = fl(1 / (t + 1)) and       */
/* yl = fl((1 - (t + 1) yh) yh): before its one rounding the sum is within      */
/* 2^-104 of delta / (t + 1), and a quotient by an integer below 2^31 lies at   */
/* least 2^-32 ulp from the middle of two doubles (and never on it), so this   */
/* is the correctly rounded quotient.  Deltas outside 2^-895 .. 2^1004 (where   */
/* yl's product may lose bits) take the division itself.  A row then costs     */
/* 4 dependent instructions instead of a division and 3.                       */
/* ------------------------------------------------------------------------ */

__device__ __forceinline__ void
_recip_pair (double w, double *yh, double *yl)
{
  *yh = __ddiv_rn (1.0, w);
  *yl = __dmul_rn (__fma_rn (-w, *yh, 1.0), *yh);
}

/* delta in the range of the product form (or zero) */
__device__ __forceinline__ bool
_quot_ok (double delta)
{
  const uint32_t hi = (uint32_t) __double2hiint (delta) & 0x7fffffffu;

  return ((hi >> 20) - 128u < 1900u) | ((hi | (uint32_t) __double2loint (delta)) == 0u);
}

__device__ __forceinline__ double
_quot (double delta, double yh, double yl)
{
  return __fma_rn (delta, yh, __dmul_rn (delta, yl));
}

/* (r, c), r < c, of the e-th strictly-upper element, row by row */
__device__ __forceinline__ void
_upper_rc (int e, int d, int *r, int *c)
{
  int rr = 0, rem = e;

  while (rem >= d - 1 - rr)
  {
    rem -= d - 1 - rr;
    rr++;
  }

  *r = rr;
  *c = rr + 1 + rem;
}

/* The running means of all n rows: one CTA, warp 0 walks the chain (lane =
 * coordinate, alone on its SM sub-partition's FP64 pipe), warp 1 adds the
 * rows up in order beside it (the mixed form's anchor mu), warps 2 and 3 stage
 * the next rows and reciprocals.  mean[t] (after row t) and R[t] go out for
 * _welford_acc_kernel.  256 cycles a row: n = 8192, d = 16 takes 1.1 ms; one
 * CTA with divisions, the covariance sums in the same pipes and a kernel of
 * its own for mu took 7.2 ms. */
#define WM_ROWS 64

__global__ void __launch_bounds__ (PREP_THREADS)
_welford_mean_kernel (const double *__restrict__ X, int n, int d, double *__restrict__ mean,
                      double *__restrict__ Rq, double *__restrict__ mu)
{
  __shared__ double xs[2][WM_ROWS][NCG_DMAX];
  __shared__ double yh[2][WM_ROWS], yl[2][WM_ROWS];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nch = (n + WM_ROWS - 1) / WM_ROWS;
  double m = 0.0, sum = 0.0;

  for (int ch = -1; ch < nch; ch++)
  {
    if (w >= 2 && ch + 1 < nch)
    {
      const int t0 = (ch + 1) * WM_ROWS, tn = min (WM_ROWS, n - t0), buf = (ch + 1) & 1;

      for (int t = w - 2; t < tn; t += 2)
        if (lane < d)
          xs[buf][t][lane] = X[(size_t) (t0 + t) * d + lane];

      if (tid - 64 < tn)
        _recip_pair ((double) (t0 + tid - 64) + 1.0, &yh[buf][tid - 64], &yl[buf][tid - 64]);
    }
    else if (w < 2 && ch >= 0 && lane < d)
    {
      const int t0 = ch * WM_ROWS, tn = min (WM_ROWS, n - t0), buf = ch & 1;

      if (w == 0)
      {
        const double m0 = m;
        int ok          = 1;
        double *mo = mean + (size_t) t0 * d + lane, *ro = Rq + (size_t) t0 * d + lane;

#pragma unroll 8
        for (int t = 0; t < tn; t++)
        {
          const double delta = __dsub_rn (xs[buf][t][lane], m);
          const double R     = _quot (delta, yh[buf][t], yl[buf][t]);

          ok &= (int) _quot_ok (delta);
          m   = __dadd_rn (m, R);
          mo[(size_t) t * d] = m;
          ro[(size_t) t * d] = R;
        }

        if (!ok)
        {
          m = m0;

          for (int t = 0; t < tn; t++)
          {
            const double delta = __dsub_rn (xs[buf][t][lane], m);
            const double R     = __ddiv_rn (delta, (double) (t0 + t) + 1.0);

            m = __dadd_rn (m, R);
            mo[(size_t) t * d] = m;
            ro[(size_t) t * d] = R;
          }
        }
      }
      else
      {
#pragma unroll 8
        for (int t = 0; t < tn; t++)
          sum = __dadd_rn (sum, xs[buf][t][lane]);
      }
    }

    __syncthreads ();
  }

  if (w == 1 && lane < d)
    mu[lane] = __ddiv_rn (sum, (double) n);
}

/* The covariance sums from the running means: a CTA takes 32 off-diagonal
 * elements (row by row), the last one the variances.  The products of
 * different rows are independent; only the additions are a chain, so warp 0
 * adds (64 cycles a row, alone on its sub-partition but for warp 4, which only
 * writes the row numbers) what the other six warps multiply one chunk of rows
 * ahead, at three FP64 instructions a row the same 64 cycles on their three
 * sub-partitions.  Each of them holds its rows of the next chunk in registers
 * (the loads waited for in place took 1.0 ms at n = 8192, d = 16; 0.4 ms so). */
#define WA_PER 11
#define WA_ROWS (6 * WA_PER)
#define WA_TH 256

__global__ void __launch_bounds__ (WA_TH)
_welford_acc_kernel (const double *__restrict__ X, const double *__restrict__ mean, const double *__restrict__ Rq,
                     int n, int d, double *__restrict__ cov)
{
  __shared__ double prod[2][WA_ROWS][32];
  __shared__ double wt[2][WA_ROWS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int E    = d * (d - 1) / 2;
  const bool var = blockIdx.x == gridDim.x - 1;
  const int e    = var ? lane : blockIdx.x * 32 + lane;
  const bool in  = e < (var ? d : E);
  const int pw   = (w < 4) ? w - 1 : w - 2;     /* producers: warps 1-3, 5-7 */
  const int nch  = (n + WA_ROWS - 1) / WA_ROWS;
  int r = 0, c = 0;
  double acc = 0.0;
  double xc[WA_PER], mc[WA_PER], xr[WA_PER], mr[WA_PER];

  if (in && !var)
    _upper_rc (e, d, &r, &c);
  else if (in)
    r = c = e;

  /* step ch: loads of chunk ch + 2, products of chunk ch + 1, sum of chunk ch */
  for (int ch = -2; ch < nch; ch++)
  {
    if (w == 0)
    {
      if (ch >= 0)
      {
        const int tn = min (WA_ROWS, n - ch * WA_ROWS);

#pragma unroll 11
        for (int t = 0; t < tn; t++)
          acc = __dadd_rn (acc, prod[ch & 1][t][lane]);
      }
    }
    else if (w == 4)
    {
      for (int t = lane; t < WA_ROWS; t += 32)
        wt[ch & 1][t] = (double) ((ch + 2) * WA_ROWS + t);
    }
    else
    {
      if (ch >= -1 && ch + 1 < nch)
      {
        /* off-diagonal: (x_r - m_r)(x_c - m'_c), m' the mean before the row;
         * variance: (t (x_c - m'_c)) R */
#pragma unroll
        for (int q = 0; q < WA_PER; q++)
        {
          const double delta = __dsub_rn (xc[q], mc[q]);
          const double left  = var ? __dmul_rn (wt[(ch + 1) & 1][pw + 6 * q], delta) : __dsub_rn (xr[q], mr[q]);

          prod[(ch + 1) & 1][pw + 6 * q][lane] = __dmul_rn (left, var ? mr[q] : delta);
        }
      }

      if (ch + 2 < nch)
      {
#pragma unroll
        for (int q = 0; q < WA_PER; q++)
        {
          const int t      = min ((ch + 2) * WA_ROWS + pw + 6 * q, n - 1);
          const size_t row = (size_t) t * d;

          xc[q] = X[row + c];
          mc[q] = (t > 0) ? mean[row - d + c] : 0.0;
          xr[q] = X[row + r];
          mr[q] = var ? Rq[row + c] : mean[row + r];
        }
      }
    }

    __syncthreads ();
  }

  if (w == 0 && in)
  {
    const double W    = (double) n;
    const double bias = __ddiv_rn (1.0, __dsub_rn (W, __ddiv_rn (W, W)));
    const double v    = __dmul_rn (acc, bias);

    cov[r * d + c] = v;
    cov[c * d + r] = v;
  }
}

/* In-place upper Cholesky of sm.A (Sigma = U^T U), column by column in the
 * order of orc_cholesky_upper.  Returns LAPACK-style info in all threads. */
__device__ int
_chol_block (double *A, int d, int *info)
{
  const int tid = threadIdx.x, nth = blockDim.x;

  if (tid == 0)
    *info = 0;

  __syncthreads ();

  for (int j = 0; j < d; j++)
  {
    if (tid == 0)
    {
      double ajj = A[j * d + j];

      for (int k = 0; k < j; k++)
        ajj = __dsub_rn (ajj, __dmul_rn (A[k * d + j], A[k * d + j]));

      if (!(ajj > 0.0))
      {
        A[j * d + j] = ajj;
        *info        = j + 1;
      }
      else
      {
        A[j * d + j] = __dsqrt_rn (ajj);
      }
    }

    __syncthreads ();

    if (*info != 0)
      return *info;

    {
      const double ajj = A[j * d + j];

      for (int i = j + 1 + tid; i < d; i += nth)
      {
        double aji = A[j * d + i];

        for (int k = 0; k < j; k++)
          aji = __dsub_rn (aji, __dmul_rn (A[k * d + j], A[k * d + i]));

        A[j * d + i] = __ddiv_rn (aji, ajj);
      }
    }

    __syncthreads ();
  }

  return 0;
}

struct CholSmem
{
  double A[NCG_DMAX * NCG_DMAX];
  int    info;
};

/* frexp-guarded 2 ln det (ncm_matrix.c:1158-1186) */
__device__ double
_chol_lndet (const double *U, int d, int ld)
{
  const double lb = 1.0e-200, ub = 1.0e+200;
  double detL     = 1.0;
  long exponent   = 0;

  for (int i = 0; i < d; i++)
  {
    const double Lii   = fabs (U[i * ld + i]);
    const double ndetL = detL * Lii;

    if ((ndetL < lb) || (ndetL > ub))
    {
      int e = 0;

      detL      = frexp (ndetL, &e);
      exponent += e;
    }
    else
    {
      detL = ndetL;
    }
  }

  return 2.0 * (log (detL) + exponent * 0.69314718055994530941723212145818);
}

/* kernel lnnorm: ncm_stats_dist_kernel_gauss.c:201-207, ncm_stats_dist_kernel_st.c:240-252;
 * _lnnorm0 is the Student-t form's part without the determinant (two
 * lgammas), the same for every kernel of a launch */
__device__ double
_lnnorm0 (int kernel, double nu, int d)
{
  if (kernel == NCG_KERNEL_GAUSS)
    return 0.0;

  return (lgamma (nu / 2.0) - lgamma ((nu + d) / 2.0)) + (d / 2.0) * (NCG_LNPI + log (nu));
}

__device__ __forceinline__ double
_lnnorm_of (int kernel, int d, double ln0, double lndet)
{
  if (kernel == NCG_KERNEL_GAUSS)
    return 0.5 * (d * NCG_LN2PI + lndet);

  return ln0 + 0.5 * lndet;
}

/* ------------------------------------------------------------------------ */

/* upper Cholesky of the global covariance */
__global__ void __launch_bounds__ (PREP_THREADS)
_global_chol_kernel (const double *__restrict__ cov, int d, double *U, int32_t *flag, ncg_prep_status_t *st)
{
  __shared__ CholSmem sm;
  const int tid = threadIdx.x;

  for (int i = tid; i < d * d; i += blockDim.x)
    sm.A[i] = cov[i];

  __syncthreads ();

  if (_chol_block (sm.A, d, &sm.info) != 0)
  {
    /* leave the covariance in U for the nearPD pass */
    for (int i = tid; i < d * d; i += blockDim.x)
      U[i] = cov[i];

    if (tid == 0)
    {
      flag[0] = 1;
      atomicAdd (&st->n_flagged, 1);
    }

    return;
  }

  for (int i = tid; i < d * d; i += blockDim.x)
  {
    const int r = i / d, c = i - r * d;

    U[i] = (c >= r) ? sm.A[i] : 0.0;
  }

  if (tid == 0)
    flag[0] = 0;
}

extern "C" cudaError_t
ncg_launch_global_chol (const double *cov, int d, double *U, int32_t *flag, ncg_prep_status_t *st, cudaStream_t s)
{
  _global_chol_kernel<<<1, PREP_THREADS, 0, s>>> (cov, d, U, flag, st);

  return cudaGetLastError ();
}

/* the sample covariance of n rows and their mean; mean and Rq: n x d work each */
extern "C" cudaError_t
ncg_launch_global_cov (const double *X, int n, int d, double *cov, double *mu, double *mean, double *Rq,
                       cudaStream_t s)
{
  _welford_mean_kernel<<<1, PREP_THREADS, 0, s>>> (X, n, d, mean, Rq, mu);
  _welford_acc_kernel<<<(d * (d - 1) / 2 + 31) / 32 + 1, WA_TH, 0, s>>> (X, mean, Rq, n, d, cov);

  return cudaGetLastError ();
}

__global__ void
_global_lnnorm_kernel (const double *U, int d, int kernel, double nu, ncg_prep_status_t *st)
{
  if (threadIdx.x == 0 && blockIdx.x == 0)
  {
    st->ln0           = _lnnorm0 (kernel, nu, d);
    st->kernel_lnnorm = _lnnorm_of (kernel, d, st->ln0, _chol_lndet (U, d, d));
  }
}

extern "C" cudaError_t
ncg_launch_global_lnnorm (const double *U, int d, int kernel, double nu, ncg_prep_status_t *st,
                          cudaStream_t s)
{
  _global_lnnorm_kernel<<<1, 32, 0, s>>> (U, d, kernel, nu, st);

  return cudaGetLastError ();
}

/* ------------------------------------------------------------------------ */

/* Y = X U^{-1} row by row (dtrsm Right/Upper/NoTrans, kde.c:477-480) */
__global__ void
_whiten_kernel (const double *__restrict__ X, const double *__restrict__ U, int n, int d,
                double *__restrict__ Y)
{
  __shared__ double sU[NCG_DMAX * NCG_DMAX];

  for (int i = threadIdx.x; i < d * d; i += blockDim.x)
    sU[i] = U[i];

  __syncthreads ();

  const int row = blockIdx.x * blockDim.x + threadIdx.x;

  if (row >= n)
    return;

  double y[NCG_DMAX];
  const double *x = X + (size_t) row * d;

  for (int j = 0; j < d; j++)
  {
    double s = x[j];

    for (int k = 0; k < j; k++)
      s = __dsub_rn (s, __dmul_rn (y[k], sU[k * d + j]));

    y[j] = __ddiv_rn (s, sU[j * d + j]);
  }

  for (int j = 0; j < d; j++)
    Y[(size_t) row * d + j] = y[j];
}

extern "C" cudaError_t
ncg_launch_whiten (const double *X, const double *U, int n, int d, double *Y, cudaStream_t s)
{
  const int th = 128;

  _whiten_kernel<<<(n + th - 1) / th, th, 0, s>>> (X, U, n, d, Y);

  return cudaGetLastError ();
}

/* ------------------------------------------------------------------------ */
/* Exact kNN, ordered by (FP64 squared distance, index).                      */
/*                                                                          */
/* FP64 distances to every point would cost 3 d n FP64 operations a query     */
/* (5.1 of the 6.2 ms at n = 8192, d = 16), so _knn32_kernel screens the       */
/* points on FP32 distances within a proven error and takes FP64 distances    */
/* only of the ones that can be among the k nearest.  With v = Y - anchor      */
/* and N = max |v|, the FP32 coordinates are off by 2^-24 |v| each, so the      */
/* FP32 difference vector is off by e <= 2^-22 N (conversion of both ends and  */
/* the subtraction), and the sum of its squares by a relative (d + 1) 2^-24   */
/* <= g = 2^-18.  If k points have FP32 sums <= T, the k-th FP64 distance is  */
/* at most sqrt (T (1 + g)) + e, and every point that near has an FP32 sum of  */
/* at most (sqrt (T (1 + g)) + 2 e)^2 / (1 - g); the code uses 2 e and 2 g,    */
/* which also covers the FP64 roundings.  T comes from a bisection on counts, */
/* stopped once the list fits its room, so k plus a few FP64 distances are   */
/* taken.  A query whose list overflows (many equal or nearly equal            */
/* distances) or whose coordinates leave the FP32 range goes to _knn_kernel.  */
/* ------------------------------------------------------------------------ */

#define KNN_THREADS 512
#define KNN_SMEM_NMAX 16384

static inline int
_pow2_ceil (int k)
{
  int p = 1;

  while (p < k)
    p <<= 1;

  return p;
}

/* All squared distances of one query in FP64, into shared memory (or a
 * per-CTA global slice for large n), MSB-first radix select of the k-th
 * (distance, index) key, ordered compaction of ties, bitonic sort.  The queries
 * are list[0 .. *count), or all nq (list NULL). */
__global__ void __launch_bounds__ (KNN_THREADS)
_knn_kernel (const double *__restrict__ Y, int n, int nq, int d, int k, int kp2, int32_t *__restrict__ out,
             uint64_t *__restrict__ gkeys, const int32_t *__restrict__ list, const int32_t *__restrict__ count)
{
  extern __shared__ __align__ (16) unsigned char knn_smem[];
  __shared__ double yq[NCG_DMAX];
  __shared__ unsigned int hist[256];
  __shared__ unsigned long long s_prefix;
  __shared__ int s_need, s_cnt_lt, s_eq_base;
  __shared__ int warp_tot[KNN_THREADS / 32];

  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, wid = tid >> 5;
  uint64_t *selk = (uint64_t *) knn_smem;
  int32_t *seli  = (int32_t *) (selk + kp2);
  uint64_t *keys = gkeys ? gkeys + (size_t) blockIdx.x * n : (uint64_t *) (seli + kp2 + (kp2 & 1));

  const int nlist = list ? *count : nq;

  for (int iq = blockIdx.x; iq < nlist; iq += gridDim.x)
  {
    const int q = list ? list[iq] : iq;

    __syncthreads ();

    if (tid < d)
      yq[tid] = Y[(size_t) q * d + tid];

    __syncthreads ();

    /* squared distances summed in coordinate order, candidate minus query */
    for (int j = tid; j < n; j += nth)
    {
      const double *p = Y + (size_t) j * d;
      double dist     = 0.0;

      for (int c = 0; c < d; c++)
      {
        const double df = __dsub_rn (p[c], yq[c]);

        dist = __dadd_rn (dist, __dmul_rn (df, df));
      }

      keys[j] = (uint64_t) __double_as_longlong (dist);
    }

    if (tid == 0)
    {
      s_prefix = 0ULL;
      s_need   = k;
      s_cnt_lt = 0;
    }

    __syncthreads ();

    /* radix select of the k-th smallest key */
    unsigned long long mask = 0ULL;

    for (int pass = 7; pass >= 0; pass--)
    {
      const int sh = 8 * pass;

      for (int b = tid; b < 256; b += nth)
        hist[b] = 0;

      __syncthreads ();

      const unsigned long long prefix = s_prefix;

      for (int j = tid; j < n; j += nth)
      {
        const unsigned long long key = keys[j];

        if ((key & mask) == prefix)
          atomicAdd (&hist[(key >> sh) & 255ULL], 1U);
      }

      __syncthreads ();

      if (tid == 0)
      {
        int need = s_need;
        int b    = 0;

        for (b = 0; b < 256; b++)
        {
          if ((int) hist[b] >= need)
            break;

          need -= hist[b];
        }

        if (b > 255)
          b = 255;

        s_need   = need;
        s_prefix = prefix | ((unsigned long long) b << sh);
      }

      mask |= (255ULL << sh);
      __syncthreads ();
    }

    const unsigned long long T = s_prefix;
    const int need_eq          = s_need;   /* how many keys equal to T are kept */

    if (tid == 0)
      s_eq_base = 0;

    __syncthreads ();

    /* compaction: keys < T anywhere (sorted later), keys == T by index order */
    for (int base = 0; base < n; base += nth)
    {
      const int j      = base + tid;
      const bool valid = j < n;
      const unsigned long long key = valid ? keys[j] : ~0ULL;
      const bool lt    = valid && key < T;
      const bool eq    = valid && key == T;

      if (lt)
      {
        const int pos = atomicAdd (&s_cnt_lt, 1);

        if (pos < k - need_eq)
        {
          selk[pos] = key;
          seli[pos] = j;
        }
      }

      const unsigned int bal = __ballot_sync (0xffffffffu, eq);

      if (lane == 0)
        warp_tot[wid] = __popc (bal);

      __syncthreads ();

      if (eq)
      {
        int rank = s_eq_base + __popc (bal & ((1u << lane) - 1u));

        for (int w = 0; w < wid; w++)
          rank += warp_tot[w];

        if (rank < need_eq)
        {
          selk[(k - need_eq) + rank] = key;
          seli[(k - need_eq) + rank] = j;
        }
      }

      __syncthreads ();

      if (tid == 0)
      {
        int tot = 0;

        for (int w = 0; w < nth / 32; w++)
          tot += warp_tot[w];

        s_eq_base += tot;
      }

      __syncthreads ();
    }

    for (int t = k + tid; t < kp2; t += nth)
    {
      selk[t] = ~0ULL;
      seli[t] = 0x7fffffff;
    }

    __syncthreads ();

    /* bitonic sort of (key, index) ascending */
    for (int size = 2; size <= kp2; size <<= 1)
    {
      for (int stride = size >> 1; stride > 0; stride >>= 1)
      {
        for (int t = tid; t < kp2; t += nth)
        {
          const int u = t ^ stride;

          if (u > t)
          {
            const bool up = ((t & size) == 0);
            const uint64_t ka = selk[t], kb = selk[u];
            const int32_t ia = seli[t], ib = seli[u];
            const bool gt = (ka > kb) || (ka == kb && ia > ib);

            if (gt == up)
            {
              selk[t] = kb;
              selk[u] = ka;
              seli[t] = ib;
              seli[u] = ia;
            }
          }
        }

        __syncthreads ();
      }
    }

    for (int t = tid; t < k; t += nth)
      out[(size_t) q * k + t] = seli[t];
  }
}

/* The FP32 coordinates of the screen, Yt[c][j] = fl32 (Y[j][c] - anchor[c]) for
 * j < npad (0 past n), the anchor being the mean of 32 spread rows, and
 * nmax2 = the float bits of (an upper bound of) the largest |Y - anchor|^2. */
#define Y32_TH 256

__global__ void __launch_bounds__ (Y32_TH)
_y32_kernel (const double *__restrict__ Y, int n, int npad, int d, float *__restrict__ Yt,
             int32_t *__restrict__ nmax2)
{
  __shared__ double an[NCG_DMAX];
  __shared__ float red[Y32_TH / 32];
  const int tid = threadIdx.x;

  if (tid < d)
  {
    double s = 0.0;

    for (int i = 0; i < 32; i++)
      s += Y[(size_t) ((int64_t) i * n / 32) * d + tid];

    an[tid] = s * (1.0 / 32.0);
  }

  __syncthreads ();

  const int j = blockIdx.x * Y32_TH + tid;
  float s2    = 0.0f;

  if (j < npad)
    for (int c = 0; c < d; c++)
    {
      const float v = (j < n) ? __double2float_rn (Y[(size_t) j * d + c] - an[c]) : 0.0f;

      s2 = fmaf (v, v, s2);
      Yt[(size_t) c * npad + j] = v;
    }

  s2 *= 1.0f + 0x1p-17f;

#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    s2 = fmaxf (s2, __shfl_xor_sync (0xffffffffu, s2, o));

  if ((tid & 31) == 0)
    red[tid >> 5] = s2;

  __syncthreads ();

  if (tid == 0)
  {
    for (int w = 1; w < Y32_TH / 32; w++)
      s2 = fmaxf (s2, red[w]);

    atomicMax (nmax2, __float_as_int (s2));
  }
}

__device__ __forceinline__ void
_bar_group (int id, int threads)
{
  asm volatile ("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

/* QT queries per CTA: their FP32 sums together (each coordinate row is read
 * once for the QT), then KNN_THREADS / QT threads per query select, measure
 * and sort. */
template <int QT>
__global__ void __launch_bounds__ (KNN_THREADS)
_knn32_kernel (const double *__restrict__ Y, const float *__restrict__ Yt, int n, int npad, int nq, int d, int k,
               int cap, const int32_t *__restrict__ nmax2, int32_t *__restrict__ out, int32_t *__restrict__ count,
               int32_t *__restrict__ list)
{
  extern __shared__ __align__ (16) unsigned char knn_smem[];
  __shared__ float yq[NCG_DMAX][QT];
  __shared__ int red[2][QT][KNN_THREADS / QT / 32];
  __shared__ int s_cnt[QT];
  constexpr int GT = KNN_THREADS / QT, GW = GT / 32;
  const int tid = threadIdx.x, g = tid / GT, gt = tid - g * GT, gw = gt >> 5, lane = tid & 31;
  float *keys    = (float *) knn_smem;                                  /* [QT][npad] */
  uint64_t *selk = (uint64_t *) (keys + (size_t) QT * npad) + (size_t) g * cap;
  int32_t *seli  = (int32_t *) ((uint64_t *) (keys + (size_t) QT * npad) + (size_t) QT * cap) + (size_t) g * cap;

  const int q0 = blockIdx.x * QT;

  for (int e = tid; e < d * QT; e += KNN_THREADS)
    yq[e / QT][e % QT] = (q0 + e % QT < nq) ? Yt[(size_t) (e / QT) * npad + q0 + e % QT] : 0.0f;

  if (gt == 0)
    s_cnt[g] = 0;

  __syncthreads ();

  for (int j = tid * 4; j < npad; j += KNN_THREADS * 4)
  {
    float s[QT][4];

#pragma unroll
    for (int q = 0; q < QT; q++)
#pragma unroll
      for (int e = 0; e < 4; e++)
        s[q][e] = 0.0f;

#pragma unroll 4
    for (int c = 0; c < d; c++)
    {
      const float4 v = *(const float4 *) (Yt + (size_t) c * npad + j);

#pragma unroll
      for (int q = 0; q < QT; q++)
      {
        const float y = yq[c][q];
        const float t0 = v.x - y, t1 = v.y - y, t2 = v.z - y, t3 = v.w - y;

        s[q][0] = fmaf (t0, t0, s[q][0]);
        s[q][1] = fmaf (t1, t1, s[q][1]);
        s[q][2] = fmaf (t2, t2, s[q][2]);
        s[q][3] = fmaf (t3, t3, s[q][3]);
      }
    }

#pragma unroll
    for (int q = 0; q < QT; q++)
    {
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (j + e >= n)
          s[q][e] = CUDART_INF_F;

      *(float4 *) (keys + (size_t) q * npad + j) = make_float4 (s[q][0], s[q][1], s[q][2], s[q][3]);
    }
  }

  __syncthreads ();

  const int q = q0 + g;

  if (q >= nq)
    return;

  const float *kg = keys + (size_t) g * npad;
  const float nm  = __int_as_float (*nmax2);
  const double e2 = 2.0 * 0x1p-22 * sqrt ((double) nm), g2 = 2.0 * 0x1p-18;
  const int slack = (cap - k) / 2;
  uint32_t lo = 0, hi = 0x7f7fffffu;      /* count (T = lo) < k unless lo = 0; count (hi) >= k once checked */
  bool have = false;

  /* count of sums <= the float of bits `mid` */
  for (int it = 0; it < 40 && (lo < hi || !have); it++)
  {
    const uint32_t mid = have ? lo + (hi - lo) / 2 : hi;
    const float T      = __uint_as_float (mid);
    int cnt            = 0;

    for (int j = gt * 4; j < npad; j += GT * 4)
    {
      const float4 v = *(const float4 *) (kg + j);

      cnt += (v.x <= T) + (v.y <= T) + (v.z <= T) + (v.w <= T);
    }

    cnt = __reduce_add_sync (0xffffffffu, cnt);

    if (lane == 0)
      red[it & 1][g][gw] = cnt;

    _bar_group (1 + g, GT);
    cnt = 0;

#pragma unroll
    for (int w = 0; w < GW; w++)
      cnt += red[it & 1][g][w];

    if (cnt >= k)
    {
      hi   = mid;
      have = true;

      if (cnt <= k + slack)
        break;
    }
    else if (!have)
      break;      /* fewer than k finite sums */
    else
      lo = mid + 1;
  }

  /* the bounds hold while no square can leave FP32's normal range unnoticed */
  bool ok = have && nm >= 0x1p-60f && nm <= 0x1p+100f;

  if (ok)
  {
    const double r    = sqrt ((double) __uint_as_float (hi) * (1.0 + g2)) + 2.0 * e2;
    const double cut  = r * r / (1.0 - g2);
    const float cutf  = __double2float_ru (cut);

    for (int j = gt; j < n; j += GT)
      if (kg[j] <= cutf)
      {
        const int pos = atomicAdd (&s_cnt[g], 1);

        if (pos < cap)
          seli[pos] = j;
      }

    _bar_group (1 + g, GT);
    ok = s_cnt[g] <= cap;
  }

  if (!ok)
  {
    if (gt == 0)
      list[atomicAdd (count, 1)] = q;

    return;
  }

  const int nc = s_cnt[g];

  /* FP64 squared distances summed in coordinate order, candidate minus query */
  for (int t = gt; t < cap; t += GT)
  {
    uint64_t key = ~0ULL;

    if (t < nc)
    {
      const double *p = Y + (size_t) seli[t] * d, *yd = Y + (size_t) q * d;
      double dist     = 0.0;

#pragma unroll 4
      for (int c = 0; c < d; c++)
      {
        const double df = __dsub_rn (p[c], yd[c]);

        dist = __dadd_rn (dist, __dmul_rn (df, df));
      }

      key = (uint64_t) __double_as_longlong (dist);
    }
    else
      seli[t] = 0x7fffffff;

    selk[t] = key;
  }

  _bar_group (1 + g, GT);

  /* bitonic sort of (key, index) ascending */
  for (int size = 2; size <= cap; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1)
    {
      for (int h = gt; h < cap / 2; h += GT)
      {
        const int t = 2 * h - (h & (stride - 1)), u = t + stride;
        const uint64_t ka = selk[t], kb = selk[u];
        const int32_t ia = seli[t], ib = seli[u];
        const bool gt_ = (ka > kb) || (ka == kb && ia > ib);

        if (gt_ == ((t & size) == 0))
        {
          selk[t] = kb;
          selk[u] = ka;
          seli[t] = ib;
          seli[u] = ia;
        }
      }

      _bar_group (1 + g, GT);
    }

  for (int t = gt; t < k; t += GT)
    out[(size_t) q * k + t] = seli[t];
}

static inline int
_knn_npad (int n)
{
  return (n + 3) / 4 * 4;
}

/* room of the screened list: the next power of two with an eighth (32 at
 * least) to spare */
static inline int
_knn_cap (int k)
{
  return _pow2_ceil (k + (k / 8 > 32 ? k / 8 : 32));
}

#define KNN32_SMEM (200 * 1024)

static inline size_t
_knn32_smem (int qt, int n, int k)
{
  return (size_t) qt * ((size_t) _knn_npad (n) * sizeof (float) + (size_t) _knn_cap (k) * 12);
}

/* [Yt: d npad floats | nmax2, count | list: n ints | pad to 256 | FP64 keys of the large-n form] */
static inline size_t
_knn_screen_bytes (int n, int d)
{
  return (((size_t) d * _knn_npad (n) + 4 + (size_t) n) * 4 + 255) / 256 * 256;
}

extern "C" size_t
ncg_knn_scratch_bytes (int n, int d, int k)
{
  (void) k;

  return _knn_screen_bytes (n, d) + (n <= KNN_SMEM_NMAX ? 0 : (size_t) 4 * 152 * (size_t) n * sizeof (uint64_t));
}

template <int QT>
static cudaError_t
_run_knn32 (const double *Y, const float *Yt, int n, int nq, int d, int k, const int32_t *meta, int32_t *knn,
            int32_t *count, int32_t *list, cudaStream_t s)
{
  static int limit[NCG_MAX_DEVICES];
  const size_t smem = _knn32_smem (QT, n, k);
  cudaError_t e     = ncg_raise_smem_limit ((const void *) _knn32_kernel<QT>, smem, limit);

  if (e != cudaSuccess)
    return e;

  _knn32_kernel<QT><<<(nq + QT - 1) / QT, KNN_THREADS, smem, s>>> (Y, Yt, n, _knn_npad (n), nq, d, k, _knn_cap (k),
                                                                  meta, knn, count, list);

  return cudaGetLastError ();
}

/* the k nearest of the n points Y to each of the first nq of them (the
 * kernels; with a split cross-validation the other observations only enter
 * as neighbours); scratch of ncg_knn_scratch_bytes */
extern "C" cudaError_t
ncg_launch_knn (const double *Y, int n, int nq, int d, int k, int32_t *knn, uint64_t *scratch, cudaStream_t s)
{
  const int kp2      = _pow2_ceil (k);
  const bool in_smem = (n <= KNN_SMEM_NMAX);
  size_t smem        = (size_t) kp2 * (sizeof (uint64_t) + sizeof (int32_t)) + 8;
  int grid           = nq;
  cudaError_t e;

  if (k > NCG_KNN_KMAX || k > n || nq > n || nq <= 0 || scratch == NULL)
    return cudaErrorInvalidValue;

  float *Yt       = (float *) scratch;
  int32_t *meta   = (int32_t *) (Yt + (size_t) d * _knn_npad (n)), *list = meta + 4;
  uint64_t *gkeys = (uint64_t *) ((char *) scratch + _knn_screen_bytes (n, d));
  /* the screen while one query's sums fit an SM (n <= 46000 or so); four
   * queries share a pass over the coordinates where four fit */
  const bool screen = _knn32_smem (1, n, k) <= KNN32_SMEM;

  if (screen)
  {
    if ((e = cudaMemsetAsync (meta, 0, 4 * sizeof (int32_t), s)) != cudaSuccess)
      return e;

    _y32_kernel<<<(_knn_npad (n) + Y32_TH - 1) / Y32_TH, Y32_TH, 0, s>>> (Y, n, _knn_npad (n), d, Yt, meta);

    if ((e = cudaGetLastError ()) != cudaSuccess)
      return e;

    if (_knn32_smem (4, n, k) <= KNN32_SMEM)
      e = _run_knn32<4> (Y, Yt, n, nq, d, k, meta, knn, meta + 1, list, s);
    else if (_knn32_smem (2, n, k) <= KNN32_SMEM)
      e = _run_knn32<2> (Y, Yt, n, nq, d, k, meta, knn, meta + 1, list, s);
    else
      e = _run_knn32<1> (Y, Yt, n, nq, d, k, meta, knn, meta + 1, list, s);

    if (e != cudaSuccess)
      return e;
  }

  if (in_smem)
    smem += (size_t) n * sizeof (uint64_t);

  if ((!in_smem || screen) && grid > 4 * 152)
    grid = 4 * 152;

  /* raised whatever the size: the kernel's static arrays count against the
   * 48 KiB default too */
  static int limit[NCG_MAX_DEVICES];

  e = ncg_raise_smem_limit ((const void *) _knn_kernel, smem, limit);

  if (e != cudaSuccess)
    return e;

  _knn_kernel<<<grid, KNN_THREADS, smem, s>>> (Y, n, nq, d, k, kp2, knn, in_smem ? NULL : gkeys,
                                               screen ? list : NULL, screen ? meta + 1 : NULL);

  return cudaGetLastError ();
}

/* ------------------------------------------------------------------------ */

/* Local covariances and factors, 4 kpw kernels per CTA.  Rows are staged 16
 * at a time for all of them; a warp walks the mean chains of kpw kernels (lane
 * = kernel x coordinate: a warp instruction costs the same however few lanes
 * work, so d = 16 takes two kernels per warp), then the CTA's threads add
 * the off-diagonal products, each thread Q elements of the 4 kpw d (d - 1) / 2
 * in registers, and each warp factors its kernels, lane = column.  Counted in
 * FP64 warp instructions per kernel and row at d = 16: 4 for the chain and 7.5
 * for the products, where one CTA per kernel with divisions took 30; the rate
 * of the FP64 pipes bounds it (n = 8192, k = 409: 7.3 ms before, 2.4 ms now). */
#define LC_ROWS 16

template <int Q>
__global__ void __launch_bounds__ (PREP_THREADS)
_local_cov_chol_kernel (const double *__restrict__ X, const int32_t *__restrict__ knn, int n, int nq, int d, int k,
                        int kpw, double *__restrict__ Ui, int32_t *__restrict__ flag, ncg_prep_status_t *st)
{
  __shared__ double buf[2 * 4 * 32 * LC_ROWS];      /* 4 kpw d <= 128 columns of xs and of delta */
  __shared__ double yh[LC_ROWS], yl[LC_ROWS], wt[LC_ROWS];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int kb = 4 * kpw, E = d * (d - 1) / 2, kd = LC_ROWS * d;
  const int i0 = blockIdx.x * kb;
  double *xs = buf, *dl = buf + kb * kd;

  /* chain lane: kernel gk of the CTA, coordinate gc */
  const bool chain = lane < kpw * d && i0 + w * kpw + lane / d < nq;
  const int gk = chain ? w * kpw + lane / d : 0, gc = chain ? lane % d : 0;
  double m = 0.0, var = 0.0;

  /* product elements */
  double acc[Q];
  int oa[Q], ob[Q];

#pragma unroll
  for (int q = 0; q < Q; q++)
  {
    const int e = tid + q * PREP_THREADS;

    acc[q] = 0.0;
    oa[q]  = 0;
    ob[q]  = 0;

    if (e < kb * E)
    {
      int r, c;

      _upper_rc (e % E, d, &r, &c);
      oa[q] = (e / E) * kd + r;
      ob[q] = (e / E) * kd + c;
    }
  }

  for (int t0 = 0; t0 < k; t0 += LC_ROWS)
  {
    const int tn = min (LC_ROWS, k - t0);

    __syncthreads ();

    for (int idx = tid; idx < kb * kd; idx += PREP_THREADS)
    {
      const int kk = idx / kd, rem = idx - kk * kd, t = rem / d, c = rem - t * d;
      double x = 0.0;

      if (t < tn && i0 + kk < nq)
      {
        int r = knn[(size_t) (i0 + kk) * k + t0 + t];

        if (r < 0 || r >= n)
        {
          if (c == 0)
            atomicAdd (&st->n_badindex, 1);

          r = 0;
        }

        x = X[(size_t) r * d + c];
      }

      xs[idx] = x;
    }

    if (tid < tn)
    {
      wt[tid] = (double) (t0 + tid);
      _recip_pair (wt[tid] + 1.0, &yh[tid], &yl[tid]);
    }

    __syncthreads ();

    if (chain)
    {
      double *px = xs + gk * kd + gc, *pd = dl + gk * kd + gc;

#pragma unroll 4
      for (int t = 0; t < tn; t++)
      {
        const double x     = px[t * d];
        const double delta = __dsub_rn (x, m);
        double R           = _quot (delta, yh[t], yl[t]);

        if (!_quot_ok (delta))
          R = __ddiv_rn (delta, wt[t] + 1.0);

        m         = __dadd_rn (m, R);
        var       = __dadd_rn (var, __dmul_rn (__dmul_rn (wt[t], delta), R));
        px[t * d] = __dsub_rn (x, m);
        pd[t * d] = delta;
      }
    }

    __syncthreads ();

#pragma unroll 2
    for (int t = 0; t < tn; t++)
    {
#pragma unroll
      for (int q = 0; q < Q; q++)
        acc[q] = __dadd_rn (acc[q], __dmul_rn (xs[oa[q] + t * d], dl[ob[q] + t * d]));
    }
  }

  /* the covariances, d x d per kernel, over the staging buffer */
  const double W    = (double) k;
  const double bias = __ddiv_rn (1.0, __dsub_rn (W, __ddiv_rn (W, W)));
  double *cov       = buf;

  __syncthreads ();

#pragma unroll
  for (int q = 0; q < Q; q++)
  {
    const int e = tid + q * PREP_THREADS;

    if (e < kb * E)
    {
      const int kk   = e / E, r = oa[q] - kk * kd, c = ob[q] - kk * kd;
      const double v = __dmul_rn (acc[q], bias);

      cov[kk * d * d + r * d + c] = v;
      cov[kk * d * d + c * d + r] = v;
    }
  }

  if (chain)
    cov[gk * d * d + gc * d + gc] = __dmul_rn (var, bias);

  __syncthreads ();

  /* the covariance stays in the output slot unless the factor succeeds */
  for (int idx = tid; idx < kb * d * d; idx += PREP_THREADS)
    if (i0 + idx / (d * d) < nq)
      Ui[(size_t) i0 * d * d + idx] = cov[idx];

  __syncthreads ();

  /* upper Cholesky in the order of _chol_block, row j of every kernel of the
   * warp at once (idle lanes follow with kernel 0's row) */
  double *A   = cov + gk * d * d;
  const int g = (lane / d) * d;     /* first lane of this kernel */
  bool ok     = true;

  for (int j = 0; j < d; j++)
  {
    const bool mine = chain && gc >= j;
    double v        = mine ? A[j * d + gc] : 1.0;

    if (mine)
      for (int q = 0; q < j; q++)
        v = __dsub_rn (v, __dmul_rn (A[q * d + j], A[q * d + gc]));

    const double piv = __shfl_sync (0xffffffffu, v, (g + j) & 31);

    ok = ok && piv > 0.0;

    if (mine && ok)
    {
      const double u = __dsqrt_rn (piv);

      A[j * d + gc] = (gc == j) ? u : __ddiv_rn (v, u);
    }

    __syncwarp ();
  }

  if (chain)
  {
    const int i = i0 + gk;

    if (ok)
    {
      double *Uo = Ui + (size_t) i * d * d;

      for (int r = 0; r < d; r++)
        Uo[r * d + gc] = (gc >= r) ? A[r * d + gc] : 0.0;
    }

    if (gc == 0)
    {
      flag[i] = ok ? 0 : 1;

      if (!ok)
        atomicAdd (&st->n_flagged, 1);
    }
  }
}

/* the nq kernels' local covariances from their neighbour lists (indices
 * into the n observations) and their upper Cholesky factors */
extern "C" cudaError_t
ncg_launch_local_cov_chol (const double *X, const int32_t *knn, int n, int nq, int d, int k, double *Ui,
                           int32_t *flag, ncg_prep_status_t *st, cudaStream_t s)
{
  int kpw = (d >= 4) ? 32 / d : 8;

  /* fewer kernels per warp while the CTAs would not give every SM two */
  while (kpw > 1 && (nq + 4 * kpw - 1) / (4 * kpw) < 2 * 152)
    kpw = (kpw + 1) / 2;

  const int grid = (nq + 4 * kpw - 1) / (4 * kpw);
  const int q    = (4 * kpw * (d * (d - 1) / 2) + PREP_THREADS - 1) / PREP_THREADS;

#define LC_RUN(Q) _local_cov_chol_kernel<Q><<<grid, PREP_THREADS, 0, s>>> (X, knn, n, nq, d, k, kpw, Ui, flag, st)

  if (q <= 2)
    LC_RUN (2);
  else if (q <= 4)
    LC_RUN (4);
  else if (q <= 6)
    LC_RUN (6);
  else if (q <= 8)
    LC_RUN (8);
  else if (q <= 12)
    LC_RUN (12);
  else
    LC_RUN (16);

  return cudaGetLastError ();
}

/* upper Cholesky of the covariance each slot of Ui holds (the robust types
 * compute it elsewhere); flags as _local_cov_chol_kernel */
__global__ void __launch_bounds__ (PREP_THREADS)
_chol_slots_kernel (double *__restrict__ Ui, int n, int d, int32_t *__restrict__ flag, ncg_prep_status_t *st)
{
  __shared__ CholSmem sm;
  const int tid = threadIdx.x;

  for (int i = blockIdx.x; i < n; i += gridDim.x)
  {
    double *Uo = Ui + (size_t) i * d * d;

    for (int e = tid; e < d * d; e += blockDim.x)
      sm.A[e] = Uo[e];

    __syncthreads ();

    const int info = _chol_block (sm.A, d, &sm.info);

    if (info != 0)
    {
      if (tid == 0)
      {
        flag[i] = 1;
        atomicAdd (&st->n_flagged, 1);
      }
    }
    else
    {
      for (int e = tid; e < d * d; e += blockDim.x)
      {
        const int r = e / d, c = e - r * d;

        Uo[e] = (c >= r) ? sm.A[e] : 0.0;
      }

      if (tid == 0)
        flag[i] = 0;
    }

    __syncthreads ();
  }
}

extern "C" cudaError_t
ncg_launch_chol_slots (double *Ui, int n, int d, int32_t *flag, ncg_prep_status_t *st, cudaStream_t s)
{
  const int grid = (n < 152 * 16) ? n : 152 * 16;

  _chol_slots_kernel<<<grid, PREP_THREADS, 0, s>>> (Ui, n, d, flag, st);

  return cudaGetLastError ();
}

/* ------------------------------------------------------------------------ */
/* nearPD fallback: one CTA per failed factor, all state in shared memory.    */
/*                                                                          */
/* Restates ncm_matrix_nearPD (numcosmo/ncm/algebra/ncm_matrix.c:1248-1344)   */
/* with cholesky_decomp = TRUE, as the oracle does: Higham's alternating      */
/* projections with the unit diagonal restored, negative eigenvalues raised  */
/* to min_pos_ev * DBL_EPSILON, until the Cholesky of the iterate succeeds or */
/* maxiter is passed; then the diagonal fallback of _cholesky_decomp.         */
/* The eigen-decomposition (dsyevr in the reference) is a cyclic Jacobi with */
/* the round-robin pair order: each round rotates d/2 disjoint pairs at once */
/* (the rotations of disjoint pairs commute), d-1 rounds a sweep, the        */
/* oracle's stopping rule (off-diagonal mass <= 1e-30 of the diagonal's).    */
/* The Cholesky test is right-looking over the threads with the same         */
/* operations in the same order as the serial one (bit-identical).           */
/* ------------------------------------------------------------------------ */

#include "ncg_jacobi.cuh"

/* upper Cholesky of S in place, right-looking over the threads; returns
 * 0 or the failing column + 1 (same value in every thread) */
__device__ int
_npd_chol (double (*S)[NPD_LD], int d)
{
  const int tid = threadIdx.x;

  for (int j = 0; j < d; j++)
  {
    const double ajj = S[j][j];

    if (!(ajj > 0.0))
    {
      __syncthreads ();

      return j + 1;
    }

    const double ujj = __dsqrt_rn (ajj);

    for (int i = j + 1 + tid; i < d; i += NPD_THREADS)
      S[j][i] = __ddiv_rn (S[j][i], ujj);

    __syncthreads ();

    if (tid == 0)
      S[j][j] = ujj;

    const int w = d - j - 1;

    for (int e = tid; e < w * w; e += NPD_THREADS)
    {
      const int r = j + 1 + e / w, c = j + 1 + e % w;

      if (c >= r)
        S[r][c] = __dsub_rn (S[r][c], __dmul_rn (S[j][r], S[j][c]));
    }

    __syncthreads ();
  }

  return 0;
}

__global__ void __launch_bounds__ (NPD_THREADS)
_nearpd_kernel (double *M, int count, const int32_t *ids, int d, int maxiter, int32_t *flag,
                ncg_prep_status_t *st)
{
  __shared__ double Y[NCG_DMAX][NPD_LD];    /* the iterate                  */
  __shared__ double R[NCG_DMAX][NPD_LD];    /* its copy / Cholesky work     */
  __shared__ double DS[NCG_DMAX][NPD_LD];   /* Dykstra correction           */
  __shared__ double V[NCG_DMAX][NPD_LD];    /* eigenvectors (columns)       */
  __shared__ double diag[NCG_DMAX], eva[NCG_DMAX], red[NPD_THREADS / 32];
  __shared__ double2 cs[NCG_DMAX / 2];
  __shared__ int perm[NCG_DMAX];
  __shared__ double s_minpos;

  const int t   = blockIdx.x;
  const int tid = threadIdx.x;

  if (t >= count)
    return;

  const int i = ids ? ids[t] : t;
  double *A   = M + (size_t) i * d * d;   /* covariance in, factor out */
  int ret     = 0;

  for (int e = tid; e < d * d; e += NPD_THREADS)
  {
    Y[e / d][e % d]  = A[e];
    DS[e / d][e % d] = 0.0;
  }

  __syncthreads ();

  if (tid < d)
    diag[tid] = Y[tid][tid];

  for (int iter = 0;; iter++)
  {
    /* Y -= D_S and R = Y (kept for D_S); Y is then taken apart by Jacobi */
    for (int e = tid; e < d * d; e += NPD_THREADS)
    {
      const int r = e / d, c = e % d;
      const double y = Y[r][c] - DS[r][c];

      Y[r][c] = y;
      R[r][c] = y;
    }

    __syncthreads ();

    _npd_jacobi (Y, V, d, eva, cs, red);

    /* eigenvalues ascending (the oracle's insertion sort), floor of the
     * negative ones at min_pos_ev * DBL_EPSILON */
    if (tid == 0)
    {
      double mp = CUDART_INF;

      for (int k = 0; k < d; k++)
      {
        perm[k] = k;

        if (eva[k] > 0.0)
          mp = fmin (eva[k], mp);
      }

      for (int p = 1; p < d; p++)
      {
        const int cur = perm[p];
        int q         = p - 1;

        while (q >= 0 && eva[perm[q]] > eva[cur])
        {
          perm[q + 1] = perm[q];
          q--;
        }

        perm[q + 1] = cur;
      }

      s_minpos = mp;
    }

    __syncthreads ();

    if (tid < d)
    {
      const double ev = eva[tid];

      eva[tid] = sqrt ((ev < 0.0) ? s_minpos * 2.220446049250313080847e-16 : ev);
    }

    __syncthreads ();

    /* Y = sum_k (s_k v_k)(s_k v_k)^T in ascending eigenvalue order, then
     * D_S = Y - R and the diagonal restored */
    for (int e = tid; e < d * d; e += NPD_THREADS)
    {
      const int r = e / d, c = e % d;

      if (c < r)
        continue;

      double sum = 0.0;

      for (int k = 0; k < d; k++)
      {
        const int pk  = perm[k];
        const double sk = eva[pk];

        sum += (V[r][pk] * sk) * (V[c][pk] * sk);
      }

      DS[r][c] = sum - R[r][c];
      DS[c][r] = sum - R[c][r];
      Y[r][c]  = (r == c) ? diag[r] : sum;
      Y[c][r]  = (r == c) ? diag[r] : sum;
    }

    __syncthreads ();

    for (int e = tid; e < d * d; e += NPD_THREADS)
      R[e / d][e % d] = Y[e / d][e % d];

    __syncthreads ();

    if ((ret = _npd_chol (R, d)) == 0)
      break;

    if (iter > maxiter)
      break;
  }

  if (ret != 0)
  {
    /* diagonal fallback */
    for (int e = tid; e < d * d; e += NPD_THREADS)
      R[e / d][e % d] = (e / d == e % d) ? diag[e / d] : 0.0;

    __syncthreads ();

    if (_npd_chol (R, d) != 0 && tid == 0)
    {
      atomicAdd (&st->n_fail, 1);
      flag[i] = 2;
    }
  }

  __syncthreads ();

  for (int e = tid; e < d * d; e += NPD_THREADS)
  {
    const int r = e / d, c = e % d;

    A[e] = (c >= r) ? R[r][c] : 0.0;
  }

  if (tid == 0)
  {
    atomicAdd (&st->n_fallback, 1);

    if (flag[i] != 2)
      flag[i] = 0;
  }
}

extern "C" cudaError_t
ncg_launch_nearpd (double *cov_then_U, int count, const int32_t *ids, int d, int maxiter, int32_t *flag,
                   ncg_prep_status_t *st, cudaStream_t s)
{
  if (count <= 0)
    return cudaSuccess;

  if (d > NCG_DMAX)
    return cudaErrorInvalidValue;

  _nearpd_kernel<<<count, NPD_THREADS, 0, s>>> (cov_then_U, count, ids, d, maxiter, flag, st);

  return cudaGetLastError ();
}

/* ids of the flagged factors (order irrelevant) */
__global__ void
_compact_flags_kernel (const int32_t *flag, int n, int32_t *ids, int32_t *count)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;

  if (i < n && flag[i] == 1)
    ids[atomicAdd (count, 1)] = i;
}

extern "C" cudaError_t
ncg_launch_compact_flags (const int32_t *flag, int n, int32_t *ids, int32_t *count, cudaStream_t s)
{
  _compact_flags_kernel<<<(n + 255) / 256, 256, 0, s>>> (flag, n, ids, count);

  return cudaGetLastError ();
}

/* ------------------------------------------------------------------------ */
/* lnnorm_i and the FP64 eval operand: centre (dp) + U_i^{-T}/h packed lower  */
/* by rows (dp(dp+1)/2), zero padded past d.  One warp per kernel; lane c    */
/* computes column c of W = (U_i^T)^{-1}.                                    */
/* ------------------------------------------------------------------------ */

#define FIN_WARPS 2

__global__ void __launch_bounds__ (FIN_WARPS * 32)
_vkde_finish_kernel (const double *__restrict__ X, const double *__restrict__ Ui, const int32_t *flag,
                     int n, int d, int kernel, const double *__restrict__ ln0p, double inv_href,
                     double *__restrict__ lnnorm, double *__restrict__ pack)
{
  __shared__ double sU[FIN_WARPS][NCG_DMAX * NCG_DMAX];
  __shared__ double sW[FIN_WARPS][NCG_DMAX * NCG_DMAX];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int dp   = ncg_pad_dim (d);
  const int P    = dp * (dp + 1) / 2;
  const int S    = dp + P;
  const double ln0 = *ln0p;

  for (int i = blockIdx.x * FIN_WARPS + w; i < n; i += gridDim.x * FIN_WARPS)
  {
    const double *U = Ui + (size_t) i * d * d;
    double *pk      = pack + (size_t) i * S;

    for (int e = lane; e < d * d; e += 32)
      sU[w][e] = U[e];

    __syncwarp ();

    if (lane < d)
    {
      const int c = lane;

      sW[w][c * d + c] = 1.0 / sU[w][c * d + c];

      for (int r = c + 1; r < d; r++)
      {
        double s = 0.0;

        for (int m = c; m < r; m++)
          s += sU[w][m * d + r] * sW[w][m * d + c];

        sW[w][r * d + c] = -s / sU[w][r * d + r];
      }
    }

    __syncwarp ();

    for (int e = lane; e < dp; e += 32)
      pk[e] = (e < d) ? X[(size_t) i * d + e] : 0.0;

    for (int r = 0; r < dp; r++)
      if (lane <= r)
        pk[dp + r * (r + 1) / 2 + lane] = (r < d && lane < d) ? sW[w][r * d + lane] * inv_href : 0.0;

    if (lane == 0)
      lnnorm[i] = _lnnorm_of (kernel, d, ln0, _chol_lndet (sU[w], d, d));

    __syncwarp ();
  }
}

extern "C" cudaError_t
ncg_launch_vkde_finish (const double *X, double *Ui, const int32_t *flag, int n, int d, int kernel,
                        const ncg_prep_status_t *st, double href, double *lnnorm, double *pack64, cudaStream_t s)
{
  int grid = (n + FIN_WARPS - 1) / FIN_WARPS;

  if (grid > 152 * 32)
    grid = 152 * 32;

  _vkde_finish_kernel<<<grid, FIN_WARPS * 32, 0, s>>> (X, Ui, flag, n, d, kernel, &st->ln0, 1.0 / href, lnnorm,
                                                        pack64);

  return cudaGetLastError ();
}

/* KDE operand: whitened centres / h (dp), and Vg = U^{-T}/h packed lower for
 * whitening the evaluation points. */
/* Vg = scale U^{-T}, packed lower by rows with dp padding, by one warp: lane c
 * computes column c of W = U^{-T}, so the d(d+1)/2 products and the divisions
 * of a serial inverse (97 us at d = 16, one lane) run d at a time; W: d x d
 * shared work */
__device__ __forceinline__ void
_vg_warp (const double *__restrict__ U, int d, double scale, double *__restrict__ Vg, double *W)
{
  const int lane = threadIdx.x & 31, dp = ncg_pad_dim (d);

  if (lane < d)
  {
    const int c = lane;

    W[c * d + c] = 1.0 / U[c * d + c];

    for (int r = c + 1; r < d; r++)
    {
      double s = 0.0;

      for (int m = c; m < r; m++)
        s += U[m * d + r] * W[m * d + c];

      W[r * d + c] = -s / U[r * d + r];
    }
  }

  __syncwarp ();

  for (int r = 0; r < dp; r++)
    if (lane <= r)
      Vg[r * (r + 1) / 2 + lane] = (r < d && lane < d) ? W[r * d + lane] * scale : 0.0;
}

__global__ void __launch_bounds__ (128)
_kde_finish_kernel (const double *__restrict__ Y, const double *__restrict__ U, int n, int d,
                    double inv_href, double *__restrict__ pack, double *__restrict__ Vg)
{
  __shared__ double W[NCG_DMAX * NCG_DMAX];
  const int dp = ncg_pad_dim (d);
  const int i  = blockIdx.x * blockDim.x + threadIdx.x;

  if (i < n)
    for (int e = 0; e < dp; e++)
      pack[(size_t) i * dp + e] = (e < d) ? Y[(size_t) i * d + e] * inv_href : 0.0;

  if (blockIdx.x == 0 && threadIdx.x < 32)
    _vg_warp (U, d, inv_href, Vg, W);
}

extern "C" cudaError_t
ncg_launch_kde_finish (const double *Y, const double *U, int n, int d, double href, double *pack64,
                       double *Vg, cudaStream_t s)
{
  _kde_finish_kernel<<<(n + 127) / 128, 128, 0, s>>> (Y, U, n, d, 1.0 / href, pack64, Vg);

  return cudaGetLastError ();
}

/* mean of the centres in row order, lane = coordinate (the anchor of the mixed
 * form where no sample covariance is taken); the other warps stage the rows */
__global__ void __launch_bounds__ (PREP_THREADS)
_mean_kernel (const double *__restrict__ X, int n, int d, double *__restrict__ mu)
{
  __shared__ double xs[2][WM_ROWS][NCG_DMAX];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nch  = (n + WM_ROWS - 1) / WM_ROWS;
  double sum     = 0.0;

  for (int ch = -1; ch < nch; ch++)
  {
    if (w > 0 && ch + 1 < nch && lane < d)
    {
      const int t0 = (ch + 1) * WM_ROWS, tn = min (WM_ROWS, n - t0);

      for (int t = w - 1; t < tn; t += 3)
        xs[(ch + 1) & 1][t][lane] = X[(size_t) (t0 + t) * d + lane];
    }
    else if (w == 0 && ch >= 0 && lane < d)
    {
      const int tn = min (WM_ROWS, n - ch * WM_ROWS);

#pragma unroll 8
      for (int t = 0; t < tn; t++)
        sum = __dadd_rn (sum, xs[ch & 1][t][lane]);
    }

    __syncthreads ();
  }

  if (w == 0 && lane < d)
    mu[lane] = __ddiv_rn (sum, (double) n);
}

extern "C" cudaError_t
ncg_launch_mean (const double *X, int n, int d, double *mu, cudaStream_t s)
{
  _mean_kernel<<<1, PREP_THREADS, 0, s>>> (X, n, d, mu);

  return cudaGetLastError ();
}

/* Vg = scale * U^{-T} (the global whitening of the evaluation points) */
__global__ void __launch_bounds__ (32)
_global_vg_kernel (const double *__restrict__ U, int d, double scale, double *__restrict__ Vg)
{
  __shared__ double W[NCG_DMAX * NCG_DMAX];

  _vg_warp (U, d, scale, Vg, W);
}

extern "C" cudaError_t
ncg_launch_global_vg (const double *U, int d, double scale, double *Vg, cudaStream_t s)
{
  _global_vg_kernel<<<1, 32, 0, s>>> (U, d, scale, Vg);

  return cudaGetLastError ();
}

/* c_i = ln w_i - lnnorm_i (VKDE) or ln w_i (KDE); marks wcum stale */
__global__ void
_weights_c_kernel (const double *w, const double *lnnorm, int n, int kind, double *c)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;

  if (i < n)
    c[i] = (kind == NCG_VKDE) ? log (w[i]) - lnnorm[i] : log (w[i]);
}

extern "C" cudaError_t
ncg_launch_weights_c (const double *w, const double *lnnorm, int n, int kind, double *c,
                      double *wcum_dirty, cudaStream_t s)
{
  (void) wcum_dirty;
  _weights_c_kernel<<<(n + 255) / 256, 256, 0, s>>> (w, lnnorm, n, kind, c);

  return cudaGetLastError ();
}

__global__ void
_fill_kernel (double *p, double v, int64_t n)
{
  for (int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x)
    p[i] = v;
}

extern "C" cudaError_t
ncg_launch_fill (double *p, double v, int64_t n, cudaStream_t s)
{
  int64_t g = (n + 255) / 256;

  if (g > 152 * 8)
    g = 152 * 8;

  if (g < 1)
    g = 1;

  _fill_kernel<<<(int) g, 256, 0, s>>> (p, v, n);

  return cudaGetLastError ();
}
