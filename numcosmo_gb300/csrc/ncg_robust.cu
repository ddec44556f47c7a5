/*
 * ncg_robust.cu -- the robust covariance types of NcmStatsDistKDE/VKDE
 * (cov-type ROBUST_DIAG and ROBUST): ncm_stats_vec_compute_cov_robust_diag
 * and ncm_stats_vec_compute_cov_robust_ogk
 * (numcosmo/ncm/stats/ncm_stats_vec.c:1833-1884, 1898-2077), used for the
 * global covariance (ncm_stats_dist_kde.c:423-440) and for each VKDE kernel's
 * neighbourhood (ncm_stats_dist_vkde.c:467-472).
 *
 * Both rest on the Qn scale estimator (GSL gsl_stats_Qn_from_sorted_data;
 * Rousseeuw & Croux 1993, Croux & Rousseeuw 1992):
 *   Qn = 2.21914 d_m {|x_a - x_b|; a < b}_(k),  k = C(h, 2),  h = floor(m/2) + 1,
 * d_m the small-sample factor (tabulated for m <= 9, m/(m+1.4) for odd and
 * m/(m+3.8) for even m above).  One CTA (large sets) or one warp (the VKDE
 * neighbourhoods) computes one Qn: a bitonic sort of the m values in shared
 * memory on order-preserving integer keys, then the k-th smallest pairwise
 * difference found exactly: bisection over the bit patterns of non-negative
 * doubles (their order is the integer order) with
 * count(t) = #{a < b : x_b - x_a <= t} until the bracket holds few differences,
 * and those ranked by value.  The smallest t with count(t) >= k is the order
 * statistic itself (a difference of two sample values, computed as the
 * reference computes it).
 *
 * Each test fl64(x_b - x_a) <= t of the count is first decided on FP32
 * copies of the sorted values less their median c (FP64 runs at 1/64 of the
 * FP32 rate on this part): with y = fl32(x - c), b = y_a, tf = fl32(t) and
 * e = 2^-19 (|b| + tf) + 2^-100, y_b <= b + tf - e proves the test true and
 * y_b > b + tf + e proves it false (the shift, the conversions, the float
 * sums and the FP64 rounding of the difference stay below
 * 2^-21.4 (|b| + tf) + 10 2^-126 for sets with every |x - c| < 2^100); the
 * band between, and every test of a set with larger values, is decided in
 * FP64.  The decisions, and so the selected difference, are those of the
 * FP64 count.
 *
 * Sets.  A set is m rows of the sample X (n x d): the whole sample (global
 * covariance) or the k nearest neighbours of one kernel (rows from the kNN
 * list).  The OGK estimate of a set runs in five launches over all sets:
 *   1. sigma_i = Qn(x_i) per coordinate (ROBUST_DIAG ends here: cov = diag sigma^2);
 *   2. per pair i < j with y = x / sigma (times the reciprocal, as the
 *      reference scales its columns): C_ij = (Qn(y_i + y_j)^2 - Qn(y_i - y_j)^2) / 4,
 *      C_ii = 1;
 *   3. eigenvectors E of C (cyclic Jacobi in place of dsyevr), ascending;
 *   4. sigma_z_i = Qn(z_i), z_i = E_i . y (the projections on eigenvector i);
 *   5. cov = sum_i (sigma_z_i E_i o sigma)(sigma_z_i E_i o sigma)^T.
 * The covariance goes where the sample covariance would (the VKDE factor
 * slot, or the global covariance) and is factorised there.
 */
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "ncg_internal.h"
#include "ncg_jacobi.cuh"

#define RQ_TH 256        /* CTAs of a warp per Qn, at most */
#define RQ_CTA_TH 1024   /* the CTA per Qn: 32 warps, one sum per lane in _rq_block_sum */

/* ------------------------------------------------------------ the estimator */

/* (host: a division per Qn would be a tenth of its FP64 work) */
static double
_qn_dn (int m)
{
  /* small-sample factors for m = 2..9, Croux & Rousseeuw (1992) */
  switch (m)
  {
    case 2: return 0.399;
    case 3: return 0.994;
    case 4: return 0.512;
    case 5: return 0.844;
    case 6: return 0.611;
    case 7: return 0.857;
    case 8: return 0.669;
    case 9: return 0.872;
    default: break;
  }

  return (m & 1) ? m / (m + 1.4) : m / (m + 3.8);
}

/* sum over the CTA of RQ_CTA_TH threads (red: RQ_CTA_TH / 32 values) */
__device__ __forceinline__ int
_rq_block_sum (int v, int *red)
{
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;

  v = __reduce_add_sync (0xffffffffu, v);
  __syncthreads ();

  if (lane == 0)
    red[wid] = v;

  __syncthreads ();

  return __reduce_add_sync (0xffffffffu, red[lane]);
}

/* order-preserving map of a double's bits to a signed integer (its own
 * inverse): non-negative values keep their bits, negative ones flip all
 * but the sign; the orders agree for every non-NaN value (-0 < +0 only
 * separates equal values) */
__device__ __forceinline__ long long
_qn_key (long long b)
{
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

/* sort v[0..mpad) ascending (slots from m on padded with +inf) by a bitonic
 * network on the keys, by nt threads t = 0..nt-1 synchronised by sync; then
 * f[a] = fl32(v[a] - v[m/2]) (the median taken out, so that the FP32 copies
 * keep the spread of a set far from zero) */
template <typename Sync>
__device__ __forceinline__ void
_qn_sort (double *v, float *f, int m, int mpad, int t0, int nt, Sync sync)
{
  long long *kv = (long long *) v;

  for (int t = t0; t < mpad; t += nt)
    kv[t] = (t < m) ? _qn_key (kv[t]) : __double_as_longlong (CUDART_INF);

  sync ();

  for (int k = 2; k <= mpad; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1)
    {
      /* the stage's pairs, one per thread */
      for (int p = t0; p < mpad / 2; p += nt)
      {
        const int t       = 2 * p - (p & (j - 1)), u = t + j;
        const long long a = kv[t], b = kv[u];

        if ((a > b) == ((t & k) == 0))
        {
          kv[t] = b;
          kv[u] = a;
        }
      }

      sync ();
    }

  for (int t = t0; t < mpad; t += nt)
    kv[t] = _qn_key (kv[t]);

  sync ();

  const double c = v[m >> 1];

  for (int t = t0; t < mpad; t += nt)
    f[t] = __double2float_rn (v[t] - c);

  sync ();
}

/* the row x_a of a count and its FP32 decision band (NaN bounds: every
 * test goes to FP64) */
struct QnRow
{
  double x;
  float lo, hi;
};

__device__ __forceinline__ QnRow
_qn_row (const double *v, const float *f, int a, float tf, bool fast)
{
  QnRow r;

  r.x = v[a];

  if (fast)
  {
    const float b = f[a], c = b + tf, e = 0x1p-19f * (fabsf (b) + tf) + 0x1p-100f;

    r.lo = c - e;
    r.hi = c + e;
  }
  else
  {
    r.lo = CUDART_NAN_F;
    r.hi = CUDART_NAN_F;
  }

  return r;
}

/* fl64(y - x) <= t, as a call: inlined, the two FP64 instructions are predicated
 * and go through their pipe (64 cycles each) for every test, also where no lane
 * needs them.  They were what bound the counts: 75 % of the pipe's cycles */
__device__ __noinline__ bool
_qn_le64 (double y, double x, double t)
{
  return y - x <= t;
}

/* fl64(v[j] - r.x) <= t, for j past the row (v[j] >= r.x) */
__device__ __forceinline__ bool
_qn_le (const double *v, const float *f, int j, const QnRow &r, double t)
{
  const float y = f[j];

  if (y <= r.lo)
    return true;

  if (y > r.hi)
    return false;

  return _qn_le64 (v[j], r.x, t);
}

/* the FP32 band holds for the set: every |v - v[m/2]| < 2^100 (v sorted) */
__device__ __forceinline__ bool
_qn_fast (const double *v, int m)
{
  const double c = v[m >> 1];

  return fabs (v[0] - c) < 0x1p100 && fabs (v[m - 1] - c) < 0x1p100;
}

/* The k-th smallest difference is bracketed by bisection, and the bracket's last
 * few differences are ranked.  A count over threshold t moves lo or hi (bit
 * patterns of non-negative doubles); cL and cH, the counts below lo and up to
 * hi, say how many differences the bracket still holds, and the steps end when
 * those fit the ranking.  While nothing is known to lie below, the threshold
 * steps down from hi by octaves (3, 6, 12, ...): a scale estimate is within a few of
 * the range, where halving the patterns of [0, hi] spends its first steps near
 * 1e-154 and takes ten to reach the right octave.  Bisecting all 62 bits took 62
 * counts; now about 9 for 100 values and 16 for 2000: with the FP64 tests off the
 * counts (_qn_le64) the pairs of 2048 sets of 102 rows, d = 8, took 2550 -> 950 us
 * and those of one set of 2048 rows 860 -> 150 us. */
struct QnBracket
{
  unsigned long long lo, hi;
  int cL, cH, kk;
  unsigned long long down;

  __device__ QnBracket (const double *v, int m)
  {
    const int h       = m / 2 + 1;
    const double span = v[m - 1] - v[0];

    lo   = 0ull;
    hi   = (unsigned long long) __double_as_longlong (span > 0.0 ? span : 0.0);
    cL   = 0;
    cH   = m * (m - 1) / 2;
    kk   = h * (h - 1) / 2;
    down = 3ull << 52;
  }

  __device__ bool open (int cap) const
  {
    return lo < hi && cH - cL > cap;
  }

  __device__ unsigned long long mid ()
  {
    if (lo == 0ull && hi > down)
    {
      const unsigned long long t = hi - down;

      down *= 2;

      return t;
    }

    return lo + ((hi - lo) >> 1);
  }

  /* count c at threshold t; true when the bracket's upper end moved */
  __device__ bool take (unsigned long long t, int c)
  {
    if (c >= kk)
    {
      hi = t;
      cH = c;

      return true;
    }

    lo = t + 1;
    cL = c;

    return false;
  }

  /* the difference's ranking key; one that is no number sorts at the bracket's end */
  __device__ unsigned long long key (double dif) const
  {
    const unsigned long long b = (unsigned long long) __double_as_longlong (dif);

    return b < hi ? b : hi;
  }
};

/* how many differences are ranked: one per lane, one per thread of 8 warps */
#define QN_WARP_CAP 32
#define QN_CTA_CAP 256

/* largest j in [i, m) with fl64(v[j] - v[i]) <= t (monotone in j) */
__device__ __forceinline__ int
_qn_reach (const double *v, const float *f, int i, int m, double t, float tf, bool fast)
{
  const QnRow r = _qn_row (v, f, i, tf, fast);
  int a = i, b = m - 1;

  while (a < b)
  {
    const int md = (a + b + 1) >> 1;

    if (_qn_le (v, f, md, r, t))
      a = md;
    else
      b = md - 1;
  }

  return a;
}

/* Qn of v[0..m) (v holds mpad >= m slots, mpad a power of two; sorted on
 * return; f holds mpad floats); every thread gets the value.  The row searches
 * are dependent shared-memory trips, so the CTA is as wide as it can be: one
 * global estimate has 8 to 28 of them for d = 8, on 152 SMs */
__device__ double
_qn_cta (double *v, float *f, int m, int mpad, double cq, int *red)
{
  __shared__ unsigned long long cand[QN_CTA_CAP];
  __shared__ unsigned long long sel;
  __shared__ int ncand;
  const int tid = threadIdx.x;

  _qn_sort (v, f, m, mpad, tid, RQ_CTA_TH, [] () { __syncthreads (); });

  const bool fast = _qn_fast (v, m);
  QnBracket q (v, m);

  while (q.open (QN_CTA_CAP))
  {
    const unsigned long long mid = q.mid ();
    const double t = __longlong_as_double ((long long) mid);
    const float tf = __double2float_rn (t);
    int c          = 0;

    for (int i = tid; i < m - 1; i += RQ_CTA_TH)
      c += _qn_reach (v, f, i, m, t, tf, fast) - i;

    q.take (mid, _rq_block_sum (c, red));
  }

  if (q.lo < q.hi)
  {
    const int nc     = q.cH - q.cL;
    const double th  = __longlong_as_double ((long long) q.hi);
    const double tl  = __longlong_as_double ((long long) (q.lo > 0ull ? q.lo - 1 : 0ull));
    const float thf  = __double2float_rn (th), tlf = __double2float_rn (tl);
    const bool below = q.lo > 0ull;

    if (tid < QN_CTA_CAP)
      cand[tid] = q.hi;

    if (tid == 0)
    {
      ncand = 0;
      sel   = q.hi;
    }

    __syncthreads ();

    for (int i = tid; i < m - 1; i += RQ_CTA_TH)
    {
      const int H = _qn_reach (v, f, i, m, th, thf, fast);
      const int L = below ? _qn_reach (v, f, i, m, tl, tlf, fast) : i;

      if (H > L)
      {
        const int o = atomicAdd (&ncand, H - L);

        for (int j = L + 1; j <= H; j++)
          if (o + j - L - 1 < QN_CTA_CAP)
            cand[o + j - L - 1] = q.key (v[j] - v[i]);
      }
    }

    __syncthreads ();

    if (tid < nc)
    {
      const unsigned long long own = cand[tid];
      int rank = 0;

      for (int k = 0; k < nc; k++)
        rank += cand[k] < own || (cand[k] == own && k < tid);

      if (rank == q.kk - q.cL - 1)
        sel = own;
    }

    __syncthreads ();
    q.lo = sel;
    __syncthreads ();
  }

  return cq * __longlong_as_double ((long long) q.lo);
}

/* row a of set s; an index outside [0, n) is counted in *bad and replaced by 0 */
__device__ __forceinline__ int
_rq_row (const int32_t *idx, int s, int m, int a, int n, int32_t *bad)
{
  if (idx == NULL)
    return a;

  const int r = idx[(size_t) s * m + a];

  if (r < 0 || r >= n)
  {
    atomicAdd (bad, 1);

    return 0;
  }

  return r;
}

/* Qn of v[0..m) by one warp (sets of at most RQ_WARP_MPAD values): the
 * same sort and bisection as _qn_cta, each lane counting a contiguous run of
 * rows; a row's pointer a_i(t) = max{j : fl(v[j] - v[i]) <= t} is bounded by
 * its values at the bracket's ends, kept per row in bnd (L = a_i below lo,
 * H = a_i(hi), and a_i at the last step, 10 bits each), and by the previous
 * row's pointer (a_i >= a_{i-1}); a row whose bounds meet costs no test, so
 * once the bracket holds few differences a count is nearly free */
#define RQ_WARP_MPAD 1024

__device__ double
_qn_warp (double *v, float *f, uint32_t *bnd, int m, int mpad, double cq)
{
  const int lane = threadIdx.x & 31;

  _qn_sort (v, f, m, mpad, lane, 32, [] () { __syncwarp (); });

  const bool fast = _qn_fast (v, m);
  const int chunk = (m - 1 + 31) / 32, r0 = lane * chunk, r1 = min (m - 1, r0 + chunk);
  QnBracket q (v, m);
  int pend = 0;   /* the last step's verdict, applied as each row is read: 1 L := a, 2 H := a */

  for (int i = r0; i < r1; i++)
    bnd[i] = (uint32_t) i | ((uint32_t) (m - 1) << 10);

  while (q.open (QN_WARP_CAP))
  {
    const unsigned long long mid = q.mid ();
    const double t = __longlong_as_double ((long long) mid);
    const float tf = __double2float_rn (t);
    int c = 0, a = -1;

    for (int i = r0; i < r1; i++)
    {
      const uint32_t wd = bnd[i];
      int L = (int) (wd & 1023u), H = (int) ((wd >> 10) & 1023u);

      if (pend == 1)
        L = (int) (wd >> 20);
      else if (pend == 2)
        H = (int) (wd >> 20);

      int l = (a > L) ? a : L;

      if (l < H)
      {
        const QnRow r = _qn_row (v, f, i, tf, fast);

        if (i == r0)
        {
          int b = H;

          while (l < b)
          {
            const int md = (l + b + 1) >> 1;

            if (_qn_le (v, f, md, r, t))
              l = md;
            else
              b = md - 1;
          }
        }
        else
          while (l < H && _qn_le (v, f, l + 1, r, t))
            l++;
      }

      a = l;
      c += a - i;
      bnd[i] = (uint32_t) L | ((uint32_t) H << 10) | ((uint32_t) a << 20);
    }

    pend = q.take (mid, __reduce_add_sync (0xffffffffu, c)) ? 2 : 1;
  }

  if (q.lo < q.hi)
  {
    /* the bracket's differences, one per lane, through the copies' room */
    unsigned long long *cand = (unsigned long long *) f;
    const int nc             = q.cH - q.cL;
    int cnt = 0, o;

    for (int i = r0; i < r1; i++)
    {
      const uint32_t wd = bnd[i];
      const int L       = (int) ((pend == 1) ? wd >> 20 : wd & 1023u);
      const int H       = (int) ((pend == 2) ? wd >> 20 : (wd >> 10) & 1023u);

      cnt += max (H - L, 0);
    }

    o = cnt;

#pragma unroll
    for (int k = 1; k < 32; k <<= 1)
    {
      const int t = __shfl_up_sync (0xffffffffu, o, k);

      if (lane >= k)
        o += t;
    }

    o -= cnt;
    __syncwarp ();
    cand[lane] = q.hi;
    __syncwarp ();

    for (int i = r0; i < r1; i++)
    {
      const uint32_t wd = bnd[i];
      const int L       = (int) ((pend == 1) ? wd >> 20 : wd & 1023u);
      const int H       = (int) ((pend == 2) ? wd >> 20 : (wd >> 10) & 1023u);

      for (int j = L + 1; j <= H; j++, o++)
        if (o < QN_WARP_CAP)
          cand[o] = q.key (v[j] - v[i]);
    }

    __syncwarp ();

    const unsigned long long own = cand[lane];
    int rank = 0;

    for (int k = 0; k < nc; k++)
      rank += cand[k] < own || (cand[k] == own && k < lane);

    const unsigned w = __ballot_sync (0xffffffffu, lane < nc && rank == q.kk - q.cL - 1);

    q.lo = w ? __shfl_sync (0xffffffffu, own, __ffs (w) - 1) : q.hi;
  }

  return cq * __longlong_as_double ((long long) q.lo);
}

/* ------------------------------------------------------------------ stages */

/* A worker computes one Qn task: the whole CTA (W = false, large sets) or
 * one warp with its own slice of the shared values (W = true; CTAs of 2 to
 * RQ_WPB such warps, as many as keep the most warps resident). */
#define RQ_WPB (RQ_TH / 32)

/* floats of a worker's copies: room for the ranked differences of a small set */
__host__ __device__ __forceinline__ int
_rq_fpad (int mpad)
{
  return mpad < 2 * QN_WARP_CAP ? 2 * QN_WARP_CAP : mpad;
}

template <bool W>
struct RqWorker
{
  int id, t, nt;
  double *v;      /* the set's values (mpad slots) */
  float *f;       /* their FP32 copies, after every worker's values */
  uint32_t *bnd;  /* W: the rows' pointer bounds, after every worker's copies */

  __device__ RqWorker (double *smem, int mpad)
  {
    const int warp = threadIdx.x >> 5, wpb = W ? (int) (blockDim.x >> 5) : 1, fpad = _rq_fpad (mpad);

    id  = W ? blockIdx.x * wpb + warp : blockIdx.x;
    t   = W ? (threadIdx.x & 31) : threadIdx.x;
    nt  = W ? 32 : RQ_CTA_TH;
    v   = W ? smem + (size_t) warp * mpad : smem;
    f   = (float *) (smem + (size_t) mpad * wpb) + (W ? (size_t) warp * fpad : 0);
    bnd = W ? (uint32_t *) ((float *) (smem + (size_t) mpad * wpb) + (size_t) fpad * wpb) + (size_t) warp * mpad
            : NULL;
  }

  __device__ void sync () const
  {
    if (W)
      __syncwarp ();
    else
      __syncthreads ();
  }

  __device__ double qn (int m, int mpad, double cq, int *red) const
  {
    return W ? _qn_warp (v, f, bnd, m, mpad, cq) : _qn_cta (v, f, m, mpad, cq, red);
  }
};

/* 1. sigma[s][i] = Qn of coordinate i over the set; with diag the covariance
 * row i is written (sigma^2 on the diagonal), else C's row i (1 on the
 * diagonal) */
template <bool W>
__global__ void __launch_bounds__ (W ? RQ_TH : RQ_CTA_TH)
_rq_sigma_kernel (const double *__restrict__ X, int n, int d, int32_t *__restrict__ bad,
                  const int32_t *__restrict__ idx, int m, int mpad, double cq, int ntasks, double *__restrict__ sig,
                  double *__restrict__ out, int diag)
{
  extern __shared__ double rq_v[];
  __shared__ int red[RQ_CTA_TH / 32];
  const RqWorker<W> w (rq_v, mpad);

  if (w.id >= ntasks)   /* whole warps (W) or the whole CTA leave together */
    return;

  const int s = w.id / d, i = w.id % d;

  for (int a = w.t; a < m; a += w.nt)
    w.v[a] = X[(size_t) _rq_row (idx, s, m, a, n, bad) * d + i];

  w.sync ();

  const double q = w.qn (m, mpad, cq, red);

  if (w.t == 0)
    sig[(size_t) s * d + i] = q;

  if (w.t < d)
    out[(size_t) s * d * d + i * d + w.t] = (w.t == i) ? (diag ? q * q : 1.0) : 0.0;
}

/* 2. C[s][i][j] = C[s][j][i] = (Qn(y_i + y_j)^2 - Qn(y_i - y_j)^2) / 4 */
template <bool W>
__global__ void __launch_bounds__ (W ? RQ_TH : RQ_CTA_TH)
_rq_pair_kernel (const double *__restrict__ X, int n, int d, int32_t *__restrict__ bad,
                 const int32_t *__restrict__ idx, int m, int mpad, double cq, int ntasks, const double *__restrict__ sig,
                 double *__restrict__ C)
{
  extern __shared__ double rq_v[];
  __shared__ int red[RQ_CTA_TH / 32];
  const RqWorker<W> w (rq_v, mpad);

  if (w.id >= ntasks)
    return;

  const int np = d * (d - 1) / 2;
  const int s  = w.id / np;
  int p = w.id % np, i = 0;

  while (p >= d - 1 - i)
  {
    p -= d - 1 - i;
    i++;
  }

  const int j = i + 1 + p;
  /* both reciprocals in one division */
  const double rl = 1.0 / sig[(size_t) s * d + ((threadIdx.x & 1) ? j : i)];
  const double ri = __shfl_sync (0xffffffffu, rl, 0), rj = __shfl_sync (0xffffffffu, rl, 1);
  double sq0 = 0.0, sq1 = 0.0;

  for (int pass = 0; pass < 2; pass++)
  {
    for (int a = w.t; a < m; a += w.nt)
    {
      const double *x = X + (size_t) _rq_row (idx, s, m, a, n, bad) * d;
      const double yi = x[i] * ri, yj = x[j] * rj;

      w.v[a] = pass ? yi - yj : yi + yj;
    }

    w.sync ();

    const double q = w.qn (m, mpad, cq, red);

    if (pass)
      sq1 = q * q;
    else
      sq0 = q * q;

    w.sync ();
  }

  if (w.t == 0)
  {
    const double c = 0.25 * (sq0 - sq1);

    C[(size_t) s * d * d + i * d + j] = c;
    C[(size_t) s * d * d + j * d + i] = c;
  }
}

#define EIG_TH 256
#define EIG_SETS 8

/* 3. E[s] rows = eigenvectors of C[s], eigenvalues ascending: cyclic Jacobi as
 * _npd_jacobi does it, for several sets at once.  A round's angles (two square
 * roots and three divisions, some 50 FP64 instructions of 64 cycles) cost the
 * same for the d / 2 rotations of one set as for a warp full of them: 2048 sets of
 * 8 x 8 with a CTA each took 466 us, 8 sets to a CTA 206 us (one set 145, now 120).
 * A set that has converged is left as it is while the others of its CTA go on.
 * G: sets per CTA, a power of two. */
__global__ void __launch_bounds__ (EIG_TH)
_rq_eig_kernel (const double *__restrict__ C, int d, int nsets, int G, double *__restrict__ E)
{
  extern __shared__ double rq_wv[];   /* per set W, then V: d rows of ld */
  __shared__ double2 cs[32], part[EIG_TH / 32];
  __shared__ int live[EIG_SETS], perm[EIG_SETS][NCG_DMAX];
  const int tps = EIG_TH / G, ld = d | 1, m = d + (d & 1), np = m / 2;
  const int tid = threadIdx.x, s0 = blockIdx.x * G, ng = min (G, nsets - s0);
  const int mat = d * ld;
  /* divisions by d (of e < 2^12) and np (of at most 32) as products */
  const int dinv = (1 << 20) / d + 1, npinv = (1 << 16) / np + 1;

  for (int e = tid; e < G * d * d; e += EIG_TH)
  {
    const int g = e / (d * d), r = e / d % d, c = e % d;
    double *W   = rq_wv + 2 * g * mat;

    W[r * ld + c]       = (g < ng) ? C[(size_t) (s0 + g) * d * d + r * d + c] : 0.0;
    W[mat + r * ld + c] = (r == c) ? 1.0 : 0.0;
  }

  __syncthreads ();

  for (int sweep = 0; sweep < 100; sweep++)
  {
    {
      const double *W = rq_wv + 2 * (tid / tps) * mat;
      double off = 0.0, dg = 0.0;

      for (int e = tid % tps; e < d * d; e += tps)
      {
        const int r = e / d, c = e % d;
        const double v = W[r * ld + c];

        if (c > r)
          off += v * v;
        else if (c == r)
          dg += v * v;
      }

#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
      {
        off += __shfl_xor_sync (0xffffffffu, off, o);
        dg  += __shfl_xor_sync (0xffffffffu, dg, o);
      }

      /* tps is a multiple of 32 */
      if ((tid & 31) == 0)
        part[tid >> 5] = make_double2 (off, dg);
    }

    __syncthreads ();

    int on = 0;

    if (tid < G)
    {
      double off = 0.0, dg = 0.0;

      for (int t = 0; t < tps / 32; t++)
      {
        off += part[tid * (tps / 32) + t].x;
        dg  += part[tid * (tps / 32) + t].y;
      }

      on        = tid < ng && !(off <= 1.0e-30 * dg || off == 0.0);
      live[tid] = on;
    }

    if (!__syncthreads_or (on))
      break;

    for (int r = 0; r < m - 1; r++)
    {
      if (tid < G * np)
      {
        const int g     = tid / np, k = tid % np;
        const double *W = rq_wv + 2 * g * mat;
        const int x = _rr_seat (k, r, m), y = _rr_seat (m - 1 - k, r, m), p = min (x, y), q = max (x, y);
        double c = 1.0, sn = 0.0;

        if (q < d && live[g])
        {
          const double apq = W[p * ld + q];

          if (apq != 0.0)
          {
            const double theta = (W[q * ld + q] - W[p * ld + p]) / (2.0 * apq);
            const double t     = (theta >= 0.0 ? 1.0 : -1.0) / (fabs (theta) + sqrt (theta * theta + 1.0));

            c  = 1.0 / sqrt (t * t + 1.0);
            sn = t * c;
          }
        }

        cs[tid] = make_double2 (c, sn);
      }

      __syncthreads ();

      /* W J and V J: columns p, q of every row (V's rows follow W's) */
      for (int e = tid; e < G * np * 2 * d; e += EIG_TH)
      {
        const int gk = (e * dinv) >> 21, row = e - gk * 2 * d;
        const int s = (gk * npinv) >> 16, k = gk - s * np;
        const int x = _rr_seat (k, r, m), y = _rr_seat (m - 1 - k, r, m), p = min (x, y), q = max (x, y);
        const double2 g = cs[gk];

        if (q >= d || g.y == 0.0)
          continue;

        double *Z       = rq_wv + 2 * s * mat + row * ld;
        const double zp = Z[p], zq = Z[q];

        Z[p] = g.x * zp - g.y * zq;
        Z[q] = g.y * zp + g.x * zq;
      }

      __syncthreads ();

      /* J^T (W J): rows p, q of every column */
      for (int e = tid; e < G * np * d; e += EIG_TH)
      {
        const int gk = (e * dinv) >> 20, col = e - gk * d;
        const int s = (gk * npinv) >> 16, k = gk - s * np;
        const int x = _rr_seat (k, r, m), y = _rr_seat (m - 1 - k, r, m), p = min (x, y), q = max (x, y);
        const double2 g = cs[gk];

        if (q >= d || g.y == 0.0)
          continue;

        double *W       = rq_wv + 2 * s * mat + col;
        const double wp = W[p * ld], wq = W[q * ld];

        W[p * ld] = g.x * wp - g.y * wq;
        W[q * ld] = g.y * wp + g.x * wq;
      }

      __syncthreads ();
    }
  }

  if (tid < ng)
  {
    const double *W = rq_wv + 2 * tid * mat;
    int *pm         = perm[tid];

    for (int a = 0; a < d; a++)
      pm[a] = a;

    /* ascending eigenvalues (ties keep their index order) */
    for (int a = 1; a < d; a++)
    {
      const int pa = pm[a];
      int b        = a - 1;

      while (b >= 0 && W[pm[b] * (ld + 1)] > W[pa * (ld + 1)])
      {
        pm[b + 1] = pm[b];
        b--;
      }

      pm[b + 1] = pa;
    }
  }

  __syncthreads ();

  for (int e = tid; e < ng * d * d; e += EIG_TH)
  {
    const int g = e / (d * d), r = e / d % d, c = e % d;

    E[(size_t) s0 * d * d + e] = rq_wv[(2 * g + 1) * mat + c * ld + perm[g][r]];
  }
}

/* 4. sigz[s][i] = Qn of z_i = E_i . y over the set */
template <bool W>
__global__ void __launch_bounds__ (W ? RQ_TH : RQ_CTA_TH)
_rq_z_kernel (const double *__restrict__ X, int n, int d, int32_t *__restrict__ bad,
              const int32_t *__restrict__ idx, int m, int mpad, double cq, int ntasks, const double *__restrict__ sig,
              const double *__restrict__ E, double *__restrict__ sigz)
{
  extern __shared__ double rq_v[];
  __shared__ int red[RQ_CTA_TH / 32];
  __shared__ double eis[RQ_WPB][NCG_DMAX], rss[RQ_WPB][NCG_DMAX];
  const RqWorker<W> w (rq_v, mpad);

  if (w.id >= ntasks)
    return;

  const int s = w.id / d, i = w.id % d, slot = W ? (threadIdx.x >> 5) : 0;
  double *ei = eis[slot], *rs = rss[slot];

  if (w.t < d)
  {
    ei[w.t] = E[(size_t) s * d * d + i * d + w.t];
    rs[w.t] = 1.0 / sig[(size_t) s * d + w.t];
  }

  w.sync ();

  for (int a = w.t; a < m; a += w.nt)
  {
    const double *x = X + (size_t) _rq_row (idx, s, m, a, n, bad) * d;
    double z        = 0.0;

    for (int r = 0; r < d; r++)
      z += ei[r] * (x[r] * rs[r]);

    w.v[a] = z;
  }

  w.sync ();

  const double q = w.qn (m, mpad, cq, red);

  if (w.t == 0)
    sigz[(size_t) s * d + i] = q;
}

/* 5. cov[s] = V^T V with V_ij = sigz_i E_ij sig_j, full symmetric storage */
__global__ void
_rq_final_kernel (const double *__restrict__ E, int d, const double *__restrict__ sig,
                  const double *__restrict__ sigz, double *__restrict__ out)
{
  const int s = blockIdx.x;
  const double *Es = E + (size_t) s * d * d, *sg = sig + (size_t) s * d, *sz = sigz + (size_t) s * d;

  for (int e = threadIdx.x; e < d * d; e += blockDim.x)
  {
    const int p = e / d, q = e % d;
    const int a = (p <= q) ? p : q, b = (p <= q) ? q : p;
    double c = 0.0;

    for (int i = 0; i < d; i++)
      c += (sz[i] * Es[i * d + a] * sg[a]) * (sz[i] * Es[i * d + b] * sg[b]);

    out[(size_t) s * d * d + e] = c;
  }
}

/* ------------------------------------------------------------------- host */

static int
_pow2_at_least (int m)
{
  int p = 1;

  while (p < m)
    p <<= 1;

  return p;
}

extern "C" size_t
ncg_robust_work_doubles (int nsets, int d)
{
  return (size_t) nsets * (2 * (size_t) d + 2 * (size_t) d * d);
}

/* warps per CTA of a warp-per-Qn kernel: of RQ_WPB, RQ_WPB/2, .., 2 the one
 * with the most warps resident per SM under its shared memory (ties: the
 * larger CTA) */
static int
_rq_wpb (const void *fn, size_t per_warp)
{
  int best = RQ_WPB, best_warps = -1;

  for (int w = RQ_WPB; w >= 2; w >>= 1)
  {
    int nb = 0;

    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor (&nb, fn, 32 * w, per_warp * w) != cudaSuccess)
    {
      (void) cudaGetLastError ();
      continue;
    }

    if (nb * w > best_warps)
    {
      best_warps = nb * w;
      best       = w;
    }
  }

  return best;
}

template <bool W>
static cudaError_t
_robust_launch (const double *X, int n, int d, const int32_t *idx, int m, int nsets, int ogk, double *sig,
                double *sigz, double *C, double *E, double *out, int32_t *bad, cudaStream_t s)
{
  const int mpad        = _pow2_at_least (m);
  const size_t per_warp = (W ? sizeof (double) + sizeof (uint32_t) : sizeof (double)) * (size_t) mpad +
                          sizeof (float) * (size_t) _rq_fpad (mpad);
  const size_t smax     = per_warp * (W ? RQ_WPB : 1);
  const int t1 = nsets * d, t2 = nsets * (d * (d - 1) / 2);
  const double cq = 2.21914 * _qn_dn (m);
  cudaError_t e;
  /* sets per CTA of the eigenvectors: as many as fill a warp with angles, but
   * not fewer CTAs than SMs */
  int G = d <= 8 ? EIG_SETS : (d <= 16 ? EIG_SETS / 2 : EIG_SETS / 4);

  while (G > 1 && nsets < 152 * G)
    G /= 2;

  /* raised whatever the size: the kernels' static arrays (up to 4 KiB) count
   * against the 48 KiB default too */
  static int lim_sigma[NCG_MAX_DEVICES], lim_pair[NCG_MAX_DEVICES], lim_z[NCG_MAX_DEVICES];

  if ((e = ncg_raise_smem_limit ((const void *) _rq_sigma_kernel<W>, smax, lim_sigma)) != cudaSuccess ||
      (e = ncg_raise_smem_limit ((const void *) _rq_pair_kernel<W>, smax, lim_pair)) != cudaSuccess ||
      (e = ncg_raise_smem_limit ((const void *) _rq_z_kernel<W>, smax, lim_z)) != cudaSuccess)
    return e;

  const int w1 = W ? _rq_wpb ((const void *) _rq_sigma_kernel<W>, per_warp) : 1;
  const int w2 = W ? _rq_wpb ((const void *) _rq_pair_kernel<W>, per_warp) : 1;
  const int w3 = W ? _rq_wpb ((const void *) _rq_z_kernel<W>, per_warp) : 1;

  _rq_sigma_kernel<W><<<(t1 + w1 - 1) / w1, W ? 32 * w1 : RQ_CTA_TH, per_warp * w1, s>>> (X, n, d, bad, idx, m, mpad, cq,
                                                                                          t1, sig, ogk ? C : out, !ogk);

  if (ogk)
  {
    if (d > 1)
      _rq_pair_kernel<W><<<(t2 + w2 - 1) / w2, W ? 32 * w2 : RQ_CTA_TH, per_warp * w2, s>>> (X, n, d, bad, idx, m, mpad,
                                                                                             cq, t2, sig, C);

    _rq_eig_kernel<<<(nsets + G - 1) / G, EIG_TH, sizeof (double) * 2 * G * d * (d | 1), s>>> (C, d, nsets, G, E);
    _rq_z_kernel<W><<<(t1 + w3 - 1) / w3, W ? 32 * w3 : RQ_CTA_TH, per_warp * w3, s>>> (X, n, d, bad, idx, m, mpad, cq, t1,
                                                                                    sig, E, sigz);
    _rq_final_kernel<<<nsets, 128, 0, s>>> (E, d, sig, sigz, out);
  }

  return cudaGetLastError ();
}

extern "C" cudaError_t
ncg_launch_robust_cov (const double *X, int n, int d, const int32_t *idx, int m, int nsets, int ogk,
                       double *work, double *out, int32_t *bad, cudaStream_t s)
{
  if (nsets <= 0 || m < 4 || m > NCG_ROBUST_MAX_ROWS || d < 1 || d > NCG_DMAX)
    return cudaErrorInvalidValue;

  double *sig  = work;
  double *sigz = sig + (size_t) nsets * d;
  double *C    = sigz + (size_t) nsets * d;
  double *E    = C + (size_t) nsets * d * d;

  /* a warp per Qn for small sets (the VKDE neighbourhoods), the CTA for large ones */
  if (_pow2_at_least (m) <= RQ_WARP_MPAD)
    return _robust_launch<true> (X, n, d, idx, m, nsets, ogk, sig, sigz, C, E, out, bad, s);

  return _robust_launch<false> (X, n, d, idx, m, nsets, ogk, sig, sigz, C, E, out, bad, s);
}
