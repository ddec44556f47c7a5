/*
 * ncg_eval_q64.cu -- the FP64 VKDE eval_m2lnp with chi^2 from the tensor cores.
 *
 * Restates _ncm_stats_dist_vkde_eval_weights_m2lnp
 * (numcosmo/ncm/stats/ncm_stats_dist_vkde.c:682-723) for many points.  The
 * whitening y = W_i (x - theta_i) of a pair takes d(d+5)/2 + d FP64
 * instructions of 64 cycles each (168 at d = 16) against 20 for the rest of
 * the pair, so FP64 arithmetic on the FP64 pipes bounds the plain kernel.
 * Here chi^2_ij comes out of an integer product on the tensor cores, exact
 * but for the rounding of its operands, and the FP64 pipes do the log and
 * the exponential only.
 *
 * The product.  With global coordinates x' = V (x - mu), V = U_g^{-T}, and
 * W'_i = W_i V^{-1}, P = W'_i^T W'_i,
 *   chi^2 = sum_{a<=b} z_a z_b Q_ab,   z = (x', s) 2^-e,  s = 4,
 * Q holding P_aa, 2 P_ab, -2 (P theta')_a / s and theta'^T P theta' / s^2: one
 * dot product of length K = (d+1)(d+2)/2 per pair, one output per pair.
 * (Forming the d coordinates of y instead would need fewer bits, but d times
 * the accumulators; the epilogue, not the products, is what has to be short.)
 * z_a z_b is at most 1 by the point's power of two 2^e, Q at most 1 by the
 * kernel's 2^f.  Both are rounded to fixed point of NS = 10 balanced digits of
 * B bits (Ozaki et al., Numer. Algorithms 59, 2012: products of short slices
 * are exact), each digit an FP16 integer of magnitude <= 2^(B-1); the digit
 * products d_i e_j of one order o = i + j are summed over K and i by
 * tcgen05.mma.kind::f16 into one FP32 accumulator per order, where integers
 * below 2^24 are exact: (o + 1) K 2^(2B-2) stays below that for the orders that
 * matter with B = 8 up to d = 16 (K <= 153: o <= 5) and B = 7 above (K <= 561:
 * o <= 6); sums of higher orders would have to align hundreds of extreme
 * digits to round, by a unit of 2^-61 or less.  Orders above 9 are dropped.
 * The fixed point is absolute: chi^2 is off by about sqrt(K) 2^(2e + f - 10 B),
 * against roughly 2^-52 chi^2 |W| |x| / |y| of the plain form's own roundings.
 * So a point with 2e + f above 10 B - 52, f the largest of the kernels (q_range:
 * points far outside the sample, or any in the presence of very narrow kernels), is
 * left to the merge, which evaluates it in the plain form; and where the largest f is above
 * q_fmax, which leaves no room for points, these kernels do nothing and the caller's plain
 * form serves the call.  x', W', P and theta' are formed in
 * double-double, so nothing else enters.
 *
 * Kernel.  Tiles of 128 points x 48 kernels.  Per 16 features (a K step) the
 * 10 slices of the points (A, 40 KB) and of the kernels (B, 15 KB) come in by
 * bulk copy; slice i of A multiplies the stacked slices 0..9-i of B in one or
 * two MMAs (N <= 240) whose output columns are the orders i..9, so the slices of
 * A are read once each: 15 MMAs for 55 slice products.  The accumulators take
 * 480 of the 512 TMEM columns.  Sixteen epilogue warps (four per
 * sub-partition, each 32 points and a quarter of the kernels) first turn the ten
 * orders of their 12 kernels into 12 doubles with integer instructions, give
 * the TMEM back, and then run the FP64 part while the tensor cores work on the
 * next tile.  At d = 16 a tile takes
 * about 6 thousand cycles of MMA and 70 thousand of FP64: the FP64 pipes are
 * the bound again, at 20 instructions a pair (Student-t) instead of 188.
 *
 * Every mbarrier wait is bounded; on timeout the CTA records an error flag,
 * drains its copies, waits for its MMAs and frees TMEM.
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "ncg_internal.h"
#include "ncg_eval_tiles.cuh"
#include "ncg_fastmath.cuh"
#include "ncg_tc_ptx.cuh"

#define Q_M 128                       /* points per tile                    */
#define Q_NK 48                       /* kernels per tile                   */
#define Q_NS 10                       /* slices (and orders)                */
#define Q_ROWS (Q_NK * Q_NS)          /* 480 stacked rows of B              */
#define Q_A_LBO (Q_M * 16)            /* one 8-wide K chunk of a slice of A */
#define Q_A_SLICE (2 * Q_A_LBO)
#define Q_A_STEP (Q_NS * Q_A_SLICE)   /* 40960 */
#define Q_B_LBO (Q_ROWS * 16)
#define Q_B_STEP (2 * Q_B_LBO)        /* 15360 */
#define Q_STAGES 4
#define Q_N1 (5 * Q_NK)               /* columns of the first MMA of a slice */
#define Q_EPI_WARP0 2
#define Q_EPI_WARPS 16
#define Q_THREADS ((Q_EPI_WARP0 + Q_EPI_WARPS) * 32)
#define Q_WG (Q_EPI_WARPS / 4)        /* epilogue warps per 32 points       */
#define Q_KPW (Q_NK / Q_WG)           /* kernels per epilogue warp          */
#define Q_S 4.0                       /* the homogeneous coordinate         */
#define Q_CHUNK 8192                  /* points per launch (scratch)        */
#define Q_FAR 0x7fffffff              /* exponent of a point that takes the plain form */
#define Q_BAD_F 0x3fffffff            /* f of a kernel whose operand is not finite */

__host__ __device__ static inline int
q_bits (int d)
{
  return d <= 16 ? 8 : 7;
}

/* largest 2e + f: the rounding of chi^2 stays within sqrt (K) 2^-52 (3e-15 at d = 16,
 * 5e-15 at d = 32) */
__host__ __device__ static inline int
q_range (int d)
{
  return 10 * q_bits (d) - 52;
}

/* largest f, for points inside the sample (2e = 6 or 8) */
__host__ __device__ static inline int
q_fmax (int d)
{
  return d <= 16 ? 20 : 12;
}

__host__ __device__ static inline int
q_features (int d)
{
  return (d + 1) * (d + 2) / 2;
}

__host__ __device__ static inline int
q_steps (int d)
{
  return (q_features (d) + 15) / 16;
}

/* ------------------------------------------------------------ double-double */

struct dd
{
  double h, l;
};

__device__ __forceinline__ dd
_two_sum (double a, double b)
{
  const double s = __dadd_rn (a, b), t = __dsub_rn (s, a);

  return { s, __dadd_rn (__dsub_rn (a, __dsub_rn (s, t)), __dsub_rn (b, t)) };
}

/* acc += a b, the product exact */
__device__ __forceinline__ void
_dd_mac (dd &acc, double a, double b)
{
  const double p = __dmul_rn (a, b);
  const dd s     = _two_sum (acc.h, p);

  acc.h = s.h;
  acc.l = __dadd_rn (acc.l, __dadd_rn (s.l, __fma_rn (a, b, -p)));
}

/* acc += (ah + al)(bh + bl) to 2^-104 */
__device__ __forceinline__ void
_dd_mac2 (dd &acc, dd a, dd b)
{
  _dd_mac (acc, a.h, b.h);
  acc.l = __fma_rn (a.h, b.l, __fma_rn (a.l, b.h, acc.l));
}

/* renormalised */
__device__ __forceinline__ dd
_dd_norm (dd a)
{
  return _two_sum (a.h, a.l);
}

/* floor(log2 |x|) + 1 of a finite nonzero normal x: |x| < 2^that */
__device__ __forceinline__ int
_exp_above (double x)
{
  return (int) (((uint32_t) __double2hiint (x) >> 20) & 0x7ffu) - 1022;
}

/* inf or NaN */
__device__ __forceinline__ bool
_not_finite (double x)
{
  return ((uint32_t) __double2hiint (x) >> 20 & 0x7ffu) == 0x7ffu;
}

/* 2^e, e clamped to the normal range */
__device__ __forceinline__ double
_pow2 (int e)
{
  e = e < -1022 ? -1022 : (e > 1023 ? 1023 : e);

  return __hiloint2double ((1023 + e) << 20, 0);
}

/* the NS digits of v 2^-e (|v| <= 2^e), v = h + l, as FP16 integers
 * dig[slice * ld] */
__device__ __forceinline__ void
_digits (dd v, double scale, int bits, uint16_t *dig, int ld)
{
  /* scale = 2^-e; A = rint (v 2^31), B = rint of the rest times 2^(10 bits - 1) */
  const double h  = v.h * scale, l = v.l * scale;
  const double za = fma (h, 0x1p31, 0x1.8p52);
  const double r  = fma (za - 0x1.8p52, -0x1p-31, h) + l;
  const double zb = fma (r, _pow2 (10 * bits - 1), 0x1.8p52);
  /* 1.5 2^52 + n has the bits of 1.5 2^52 plus n */
  const long long A = __double_as_longlong (za) - 0x4338000000000000LL;
  const long long B = __double_as_longlong (zb) - 0x4338000000000000LL;
  const int half  = 1 << (bits - 1);
  unsigned __int128 V    = ((unsigned __int128) (__int128) A << (10 * bits - 32)) + (unsigned __int128) (__int128) B;
  unsigned __int128 bias = 0;

#pragma unroll
  for (int i = 0; i < Q_NS; i++)
    bias = (bias << bits) + half;

  V += bias;

#pragma unroll
  for (int i = Q_NS - 1; i >= 0; i--)
  {
    const int u = (i > 0) ? (int) ((uint32_t) V & (uint32_t) (2 * half - 1)) : (int) (uint32_t) V;

    dig[i * ld] = __half_as_ushort (__hsub (__ushort_as_half ((uint16_t) (0x6400 + u)),
                                            __ushort_as_half ((uint16_t) (0x6400 + half))));
    V >>= bits;
  }
}

/* (a, b), a <= b, of feature e over D coordinates, row by row */
__device__ __forceinline__ void
_feature (int e, int D, int *a, int *b)
{
  int r = 0;

  while (e >= D - r)
  {
    e -= D - r;
    r++;
  }

  *a = r;
  *b = r + e;
}

/* the digits of one operand row from shared memory to its 16-byte units:
 * base + step * step_bytes + slice * slice_bytes + chunk * lbo */
__device__ __forceinline__ void
_store_row (const uint16_t *dig, int ld, int steps, uint8_t *base, size_t step_bytes, int slice_bytes, int lbo,
            int lane)
{
  for (int u = lane; u < steps * 2 * Q_NS; u += 32)
  {
    const int sl = u / (2 * steps), k8 = u - sl * 2 * steps;

    *(uint4 *) (base + (size_t) (k8 >> 1) * step_bytes + (size_t) sl * slice_bytes + (size_t) (k8 & 1) * lbo) =
      *(const uint4 *) (dig + sl * ld + k8 * 8);
  }
}

/* ------------------------------------------------------------------- operands */

/* Zl = the correction of V^{-1} = U^T + Zl to double-double accuracy: with
 * E = I - V U^T, V^{-1} = U^T (I - E)^{-1} = U^T + U^T E to second order.
 * Lower triangular, d x d. */
__global__ void __launch_bounds__ (1024)
_q_global_kernel (const double *__restrict__ U, const double *__restrict__ Vg, int d, double *__restrict__ Zl)
{
  __shared__ double E[NCG_DMAX][NCG_DMAX];
  const int r = threadIdx.x / d, c = threadIdx.x % d;
  const bool in = r < d && c <= r;

  if (in)
  {
    dd acc = { (r == c) ? -1.0 : 0.0, 0.0 };

    for (int m = c; m <= r; m++)
      _dd_mac (acc, Vg[r * (r + 1) / 2 + m], U[c * d + m]);

    E[r][c] = -(acc.h + acc.l);
  }

  __syncthreads ();

  if (r < d)
  {
    double s = 0.0;

    if (in)
      for (int m = c; m <= r; m++)
        s = fma (U[m * d + r], E[m][c], s);

    Zl[r * d + c] = s;
  }
}

#define QB_WARPS 2

/* shared memory of the kernel operand's builder: per warp W | W' h, l | P h, l |
 * theta' h, l | delta h, l | digits */
__host__ __device__ static inline size_t
q_build_b_warp (int d)
{
  const size_t T = (size_t) d * (d + 1) / 2;

  return (5 * T + 4 * (size_t) d) * 8 / 16 * 16 + 16 + (size_t) Q_NS * q_steps (d) * 16 * 2;
}

/* one warp per kernel */
__global__ void __launch_bounds__ (QB_WARPS * 32)
_q_build_B_kernel (const double *__restrict__ X, const double *__restrict__ pack, int S64, int dp, int n, int d,
                   const double *__restrict__ U, const double *__restrict__ Vg, const double *__restrict__ Zl,
                   const double *__restrict__ mu, double fac, uint8_t *__restrict__ B, double *__restrict__ sck,
                   int32_t *__restrict__ fmax_)
{
  extern __shared__ __align__ (16) uint8_t q_smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int T = d * (d + 1) / 2, K = q_features (d), steps = q_steps (d), Kp = steps * 16, bits = q_bits (d);
  double *Ws  = (double *) (q_smem + w * q_build_b_warp (d));
  double *Wh = Ws + T, *Wl = Wh + T, *Ph = Wl + T, *Pl = Ph + T, *th = Pl + T, *tl = th + d, *eh = tl + d, *el = eh + d;
  uint16_t *dig = (uint16_t *) (q_smem + w * q_build_b_warp (d) + (5 * (size_t) T + 4 * (size_t) d) * 8 / 16 * 16 + 16);
  const int i   = blockIdx.x * QB_WARPS + w;
  const int npad = (n + Q_NK - 1) / Q_NK * Q_NK;

  if (i >= npad)
    return;

  uint8_t *row = B + (size_t) (i / Q_NK) * steps * Q_B_STEP + (size_t) (i % Q_NK / 8) * 128 + (size_t) (i % 8) * 16;

  if (i >= n)
  {
    for (int e = lane; e < Q_NS * Kp; e += 32)
      dig[e] = 0;

    __syncwarp ();
    _store_row (dig, Kp, steps, row, Q_B_STEP, Q_NK * 16, Q_B_LBO, lane);

    if (lane == 0)
      sck[i] = 0.0;

    return;
  }

  const double *pk = pack + (size_t) i * S64 + dp;

  for (int e = lane; e < T; e += 32)
    Ws[e] = pk[e];

  if (lane < d)
  {
    const dd t = _two_sum (X[(size_t) i * d + lane], -mu[lane]);

    eh[lane] = t.h;
    el[lane] = t.l;
  }

  __syncwarp ();

  /* theta' = V (theta - mu) */
  if (lane < d)
  {
    dd acc = { 0.0, 0.0 };

    for (int c = 0; c <= lane; c++)
    {
      const double v = Vg[lane * (lane + 1) / 2 + c];

      _dd_mac (acc, v, eh[c]);
      acc.l = __fma_rn (v, el[c], acc.l);
    }

    acc      = _dd_norm (acc);
    th[lane] = acc.h;
    tl[lane] = acc.l;
  }

  /* W' = W (U^T + Zl), lower triangular, packed by rows; taken diagonal by
   * diagonal, so that the lanes' sums have about the same length */
  for (int t = lane; t < T; t += 32)
  {
    int q = (int) ((sqrtf (8.0f * t + 1.0f) - 1.0f) * 0.5f);

    while (q * (q + 1) / 2 > t)
      q--;

    while ((q + 1) * (q + 2) / 2 <= t)
      q++;

    const int c = t - q * (q + 1) / 2, r = c + d - 1 - q, e = r * (r + 1) / 2 + c;
    dd acc      = { 0.0, 0.0 };

    for (int m = c; m <= r; m++)
    {
      const double v = Ws[r * (r + 1) / 2 + m];

      _dd_mac (acc, v, U[c * d + m]);
      acc.l = __fma_rn (v, Zl[m * d + c], acc.l);
    }

    acc   = _dd_norm (acc);
    Wh[e] = acc.h;
    Wl[e] = acc.l;
  }

  __syncwarp ();

  /* P = W'^T W', packed as its lower triangle (b, a), a <= b; a maximum leaves
   * a NaN out, so what is not finite is noted beside it */
  double mx = 0.0;
  bool bad  = false;

  for (int e = lane; e < T; e += 32)
  {
    int b = (int) ((sqrtf (8.0f * e + 1.0f) - 1.0f) * 0.5f);

    while (b * (b + 1) / 2 > e)
      b--;

    while ((b + 1) * (b + 2) / 2 <= e)
      b++;

    const int a = e - b * (b + 1) / 2;
    dd acc      = { 0.0, 0.0 };

    for (int r = b; r < d; r++)
      _dd_mac2 (acc, { Wh[r * (r + 1) / 2 + a], Wl[r * (r + 1) / 2 + a] },
                { Wh[r * (r + 1) / 2 + b], Wl[r * (r + 1) / 2 + b] });

    acc   = _dd_norm (acc);
    Ph[e] = acc.h;
    Pl[e] = acc.l;
    mx    = fmax (mx, (a == b) ? acc.h : 2.0 * fabs (acc.h));
    bad   = bad || _not_finite (acc.h);
  }

  __syncwarp ();

  /* lin_a = -2 (P theta')_a / s (lane a), cst = -sum_a lin_a theta'_a / (2 s) */
  dd lin = { 0.0, 0.0 }, cst = { 0.0, 0.0 };

  if (lane < d)
  {
    for (int b = 0; b < d; b++)
    {
      const int e = (lane <= b) ? b * (b + 1) / 2 + lane : lane * (lane + 1) / 2 + b;

      _dd_mac2 (lin, { Ph[e], Pl[e] }, { th[b], tl[b] });
    }

    lin   = _dd_norm (lin);
    lin.h *= -2.0 / Q_S;
    lin.l *= -2.0 / Q_S;
    _dd_mac2 (cst, lin, { th[lane], tl[lane] });
  }

#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    const dd s = _two_sum (cst.h, __shfl_xor_sync (0xffffffffu, cst.h, o));

    cst.l = cst.l + __shfl_xor_sync (0xffffffffu, cst.l, o) + s.l;
    cst.h = s.h;
  }

  cst    = _dd_norm (cst);
  cst.h *= -0.5 / Q_S;
  cst.l *= -0.5 / Q_S;
  mx     = fmax (fmax (mx, fabs (lin.h)), fabs (cst.h));
  bad    = __any_sync (0xffffffffu, bad || _not_finite (lin.h) || _not_finite (cst.h) || _not_finite (mx));

#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    mx = fmax (mx, __shfl_xor_sync (0xffffffffu, mx, o));

  const int f    = _exp_above (mx);
  const double sc = _pow2 (-f);

  /* an operand that is not finite or far out of range is not used: its digits
   * do not matter */
  if (lane == 0)
  {
    sck[i] = fac * _pow2 (f - 2 * (bits - 1) - 9 * bits);
    atomicMax (fmax_, bad ? Q_BAD_F : f);
  }

  /* lin and cst beside theta' (which is done with) */
  __syncwarp ();

  if (lane < d)
  {
    th[lane] = lin.h;
    tl[lane] = lin.l;
  }

  __syncwarp ();

  for (int e = lane; e < Kp; e += 32)
  {
    dd v = { 0.0, 0.0 };

    if (e < K)
    {
      int a, b;

      _feature (e, d + 1, &a, &b);

      if (b < d)
      {
        const double two = (a == b) ? 1.0 : 2.0;

        v = { two * Ph[b * (b + 1) / 2 + a], two * Pl[b * (b + 1) / 2 + a] };
      }
      else if (a < d)
        v = { th[a], tl[a] };
      else
        v = cst;
    }

    _digits (v, sc, bits, dig + e, Kp);
  }

  __syncwarp ();
  _store_row (dig, Kp, steps, row, Q_B_STEP, Q_NK * 16, Q_B_LBO, lane);
}

__global__ void
_q_tell_kernel (const int32_t *f, int fmax_, uint32_t epoch, unsigned long long *word)
{
  *(volatile unsigned long long *) word = (unsigned long long) epoch << 32 | (*f <= fmax_ ? 1u : 0u);
}

#define QA_WARPS 4

__host__ __device__ static inline size_t
q_build_a_warp (int d)
{
  return (size_t) (4 * NCG_DMAX + 4) * 8 + (size_t) Q_NS * q_steps (d) * 16 * 2;
}

/* one warp per point; rows past m are zero, and those of points past q_range.  Also
 * clears the error word. */
__global__ void __launch_bounds__ (QA_WARPS * 32)
_q_build_A_kernel (const double *__restrict__ Xq, int64_t m, int d, const double *__restrict__ Vg,
                   const double *__restrict__ mu, const int32_t *__restrict__ fmax_, uint8_t *__restrict__ A,
                   int32_t *__restrict__ pe2, int *err)
{
  extern __shared__ __align__ (16) uint8_t q_smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int K = q_features (d), steps = q_steps (d), Kp = steps * 16, bits = q_bits (d);
  double *zh    = (double *) (q_smem + w * q_build_a_warp (d));
  double *zl = zh + NCG_DMAX + 1, *eh = zl + NCG_DMAX + 1, *el = eh + NCG_DMAX;
  uint16_t *dig = (uint16_t *) (q_smem + w * q_build_a_warp (d) + (4 * NCG_DMAX + 4) * 8);
  const int64_t j = (int64_t) blockIdx.x * QA_WARPS + w;

  if (blockIdx.x == 0 && threadIdx.x == 0)
    *err = 0;

  uint8_t *row = A + (size_t) (j / Q_M) * steps * Q_A_STEP + (size_t) (j % Q_M / 8) * 128 + (size_t) (j % 8) * 16;
  dd x         = { 0.0, 0.0 };
  bool finite  = true;

  if (j < m && lane < d)
  {
    const double v = Xq[j * d + lane];
    const dd t     = _two_sum (v, -mu[lane]);

    finite   = isfinite (v) && isfinite (t.h);
    eh[lane] = t.h;
    el[lane] = t.l;
  }

  finite = __all_sync (0xffffffffu, finite) && j < m;

  if (finite && lane < d)
  {
    for (int c = 0; c <= lane; c++)
    {
      const double v = Vg[lane * (lane + 1) / 2 + c];

      _dd_mac (x, v, eh[c]);
      x.l = __fma_rn (v, el[c], x.l);
    }

    x = _dd_norm (x);
  }

  double mx = fabs (x.h);

#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    mx = fmax (mx, __shfl_xor_sync (0xffffffffu, mx, o));

  /* past 2^510 chi^2 leaves FP64 (or the coordinates did, NaN included) */
  finite = finite && mx < 0x1p510;

  const int f = *fmax_, e = finite ? _exp_above (fmax (mx, Q_S)) : 0;

  finite = finite && f <= q_fmax (d) && 2 * e + f <= q_range (d);

  const double sc  = finite ? _pow2 (-e) : 0.0;

  if (lane < d)
  {
    zh[lane] = finite ? x.h * sc : 0.0;
    zl[lane] = finite ? x.l * sc : 0.0;
  }

  if (lane == 0)
  {
    zh[d]  = finite ? Q_S * sc : 0.0;
    zl[d]  = 0.0;
    pe2[j] = finite ? 2 * e : Q_FAR;
  }

  __syncwarp ();

  for (int q = lane; q < Kp; q += 32)
  {
    dd v = { 0.0, 0.0 };

    if (q < K && finite)
    {
      int a, b;

      _feature (q, d + 1, &a, &b);
      _dd_mac2 (v, { zh[a], zl[a] }, { zh[b], zl[b] });
    }

    _digits (v, 1.0, bits, dig + q, Kp);
  }

  __syncwarp ();
  _store_row (dig, Kp, steps, row, Q_A_STEP, Q_A_SLICE, Q_A_LBO, lane);
}

/* ------------------------------------------------------------------ the kernel */

struct QParams
{
  const uint8_t *A, *B;
  const int32_t *pe2, *f;
  const double *sck, *c;
  double2 *part;          /* [Q_WG nslices][m] */
  int *err, *flag_host;
  int64_t m;
  int n, steps, npt, nkt, nslices, tps, fmax_;
  double kappa;
  int fault;
};

struct QSmem
{
  uint8_t st[Q_STAGES][Q_A_STEP + Q_B_STEP];
  uint64_t full[Q_STAGES], empty[Q_STAGES], t_full, t_empty, done;
  uint32_t tmem_base;
  int err;
};

#define Q_SMEM_BYTES (sizeof (QSmem) + 1024)

/* D(f32)[128 x N] (+)= A(f16, 128 x 16) . B(f16, N x 16)^T */
__device__ __forceinline__ void
_q_mma (uint32_t dtmem, uint64_t adesc, uint64_t bdesc, int N, uint32_t accumulate)
{
  const uint32_t idesc = (1u << 4) | ((uint32_t) (N >> 3) << 17) | ((uint32_t) (Q_M >> 4) << 24);

  asm volatile ("{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                ::"r"(dtmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                : "memory");
}

__device__ __forceinline__ void
_tmem_ld4_async (uint32_t t, uint32_t *r)
{
  asm volatile ("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                : "r"(t)
                : "memory");
}

/* tie r[0..3] to the wait before it: no use may be scheduled ahead of it */
__device__ __forceinline__ void
_tie4 (uint32_t *r)
{
  asm volatile ("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]) : : "memory");
}

/* the ten orders of a pair as hi 2^(5 BITS) + lo, rounded to a double (0 if
 * negative: a chi^2 of nothing but rounding), in integer instructions: two
 * conversions and an FMA would hold the FP64 pipe for 192 cycles */
template <int BITS>
__device__ __forceinline__ double
_orders_to_double (const uint32_t (*r)[4], int k)
{
  long long hi = 0, lo = 0;

#pragma unroll
  for (int o = 0; o < 5; o++)
  {
    hi = hi * (1 << BITS) + __float2int_rn (__uint_as_float (r[o][k]));
    lo = lo * (1 << BITS) + __float2int_rn (__uint_as_float (r[o + 5][k]));
  }

  constexpr int SH = 5 * BITS;
  const unsigned long long a = (unsigned long long) hi << SH;
  const unsigned long long t0 = a + (unsigned long long) lo;
  const long long t1 = (hi >> (64 - SH)) + (lo >> 63) + (long long) (t0 < a);

  if (t1 < 0 || (t1 == 0 && t0 == 0))
    return 0.0;

  /* the leading 64 bits, normalised; n leading zeros of the 128 */
  const int n = t1 ? __clzll (t1) : 64 + __clzll ((long long) t0);
  const unsigned long long top = t1 ? (((unsigned long long) t1 << n) | (n ? t0 >> (64 - n) : 0ull)) : t0 << (n - 64);

  return __longlong_as_double (((long long) (1023 + 127 - n - 1) << 52) + (long long) (top >> 11) +
                               (long long) ((top >> 10) & 1));
}

template <int KERN, int BITS>
__global__ void __launch_bounds__ (Q_THREADS, 1)
_eval_q64_kernel (const QParams p)
{
  extern __shared__ __align__ (16) uint8_t q_smem[];
  QSmem &sm = *(QSmem *) (((uintptr_t) q_smem + 1023) & ~(uintptr_t) 1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nunits = p.npt * p.nslices;
  volatile int *err = &sm.err;

  /* the plain form serves the call */
  if (*p.f > p.fmax_)
    return;

  if (threadIdx.x == 0)
  {
    sm.err = 0;

    for (int s = 0; s < Q_STAGES; s++)
    {
      _mbar_init (&sm.full[s], 1);
      _mbar_init (&sm.empty[s], 1);
    }

    _mbar_init (&sm.t_full, 1);
    _mbar_init (&sm.t_empty, Q_EPI_WARPS);
    _mbar_init (&sm.done, 1);
    asm volatile ("fence.mbarrier_init.release.cluster;" ::: "memory");
  }

  if (warp == 1)
  {
    asm volatile ("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                  ::"r"(_smem_u32 (&sm.tmem_base)), "r"(512)
                  : "memory");
    asm volatile ("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  _tc_fence_before ();
  __syncthreads ();
  _tc_fence_after ();

  const uint32_t tmem = sm.tmem_base;

  if (warp == 0)
  {
    /* ---------------- producer ---------------- */
    if (lane == 0 && !p.fault)
    {
      int stage = 0;
      uint32_t phase = 0;
      int armed[Q_STAGES];

      for (int s = 0; s < Q_STAGES; s++)
        armed[s] = -1;

      for (int u = blockIdx.x; u < nunits && !*err; u += gridDim.x)
      {
        const int pt = u % p.npt, sl = u / p.npt;
        const int t1 = min (p.nkt, (sl + 1) * p.tps);

        for (int t = sl * p.tps; t < t1 && !*err; t++)
          for (int k = 0; k < p.steps; k++)
          {
            if (!_mbar_wait (&sm.empty[stage], phase ^ 1, err))
              break;

            _mbar_arrive_tx (&sm.full[stage], Q_A_STEP + Q_B_STEP);
            _bulk_g2s (sm.st[stage], p.A + ((size_t) pt * p.steps + k) * Q_A_STEP, Q_A_STEP, &sm.full[stage]);
            _bulk_g2s (sm.st[stage] + Q_A_STEP, p.B + ((size_t) t * p.steps + k) * Q_B_STEP, Q_B_STEP,
                       &sm.full[stage]);
            armed[stage] = (int) phase;

            if (++stage == Q_STAGES)
            {
              stage = 0;
              phase ^= 1;
            }
          }
      }

      for (int s = 0; s < Q_STAGES; s++)
        if (armed[s] >= 0)
          _mbar_wait (&sm.full[s], (uint32_t) armed[s], err, false);
    }
  }
  else if (warp == 1)
  {
    /* ---------------- MMA issuer ---------------- */
    if (lane == 0)
    {
      int stage = 0, tc = 0;
      uint32_t phase = 0;
      bool ok = true;

      for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x)
      {
        const int sl = u / p.npt, t1 = min (p.nkt, (sl + 1) * p.tps);

        for (int t = sl * p.tps; t < t1 && ok; t++, tc++)
        {
          ok = _mbar_wait (&sm.t_empty, (tc & 1) ^ 1, err);

          for (int k = 0; k < p.steps && ok; k++)
          {
            if (!(ok = _mbar_wait (&sm.full[stage], phase, err)))
              break;

            _tc_fence_after ();

            const uint8_t *As = sm.st[stage], *Bs = As + Q_A_STEP;

#pragma unroll
            for (int i = 0; i < Q_NS; i++)
            {
              const int N       = Q_ROWS - Q_NK * i, n1 = N < Q_N1 ? N : Q_N1;
              const uint32_t d  = tmem + (uint32_t) (Q_NK * i);
              const uint64_t ad = _sdesc (As + i * Q_A_SLICE, Q_A_LBO);
              const uint32_t ac = (i > 0 || k > 0) ? 1u : 0u;

              _q_mma (d, ad, _sdesc (Bs, Q_B_LBO), n1, ac);

              if (N > Q_N1)
                _q_mma (d + Q_N1, ad, _sdesc (Bs + Q_N1 * 16, Q_B_LBO), N - Q_N1, ac);
            }

            _mma_commit (&sm.empty[stage]);

            if (++stage == Q_STAGES)
            {
              stage = 0;
              phase ^= 1;
            }
          }

          if (ok)
            _mma_commit (&sm.t_full);
        }
      }

      /* every MMA this thread issued completes before TMEM is freed */
      _mma_commit (&sm.done);
      _mbar_wait (&sm.done, 0, err, false);
    }
  }
  else
  {
    /* ---------------- epilogue ---------------- */
    const int wg = (warp - Q_EPI_WARP0) >> 2;     /* which Q_KPW kernels of a tile */
    const int q  = warp & 3;                      /* TMEM lane quarter (hardware: warp id mod 4) */
    const uint32_t base = tmem + ((uint32_t) (q * 32) << 16) + (uint32_t) (wg * Q_KPW);
    int tc = 0;

    for (int u = blockIdx.x; u < nunits; u += gridDim.x)
    {
      const int pt = u % p.npt, sl = u / p.npt, t1 = min (p.nkt, (sl + 1) * p.tps);
      const int64_t j = (int64_t) pt * Q_M + q * 32 + lane;
      const int e2    = p.pe2[j];
      double g = NCG_LSE_EMPTY, s = 0.0;
      bool ok = true;

      for (int t = sl * p.tps; t < t1; t++, tc++)
      {
        /* the TMEM loads below are warp-collective: agree before issuing them */
        if (!__all_sync (0xffffffffu, _mbar_wait (&sm.t_full, tc & 1, err)))
        {
          ok = false;
          break;
        }

        _tc_fence_after ();

        double x[Q_KPW];

#pragma unroll
        for (int b = 0; b < Q_KPW / 4; b++)
        {
          uint32_t r[Q_NS][4];

#pragma unroll
          for (int o = 0; o < Q_NS; o++)
            _tmem_ld4_async (base + (uint32_t) (o * Q_NK + b * 4), r[o]);

          asm volatile ("tcgen05.wait::ld.sync.aligned;" ::: "memory");

#pragma unroll
          for (int o = 0; o < Q_NS; o++)
            _tie4 (r[o]);

#pragma unroll
          for (int k = 0; k < 4; k++)
            x[b * 4 + k] = _orders_to_double<BITS> (r, k);
        }

        _tc_fence_before ();
        __syncwarp ();

        if (lane == 0)
          _mbar_arrive (&sm.t_empty);

        const int i0 = t * Q_NK + wg * Q_KPW;

#pragma unroll
        for (int k = 0; k < Q_KPW; k++)
        {
          if (i0 + k >= p.n)
            break;

          /* the kernel's scale times 2^(2e), on the exponent (NaN for a point of the
           * merge's: its terms are left out) */
          const double sk = __ldg (p.sck + i0 + k), c = __ldg (p.c + i0 + k);
          const int hs    = __double2hiint (sk), ex = ((hs >> 20) & 0x7ff) + e2;
          const double sc = (e2 == Q_FAR)   ? CUDART_NAN
                            : (ex > 0x7fe)  ? __hiloint2double ((hs & 0x80000000) | 0x7ff00000, 0)
                                            : __hiloint2double ((hs & 0x800fffff) | (ex << 20), __double2loint (sk));

          ncg_lse_add ((KERN == NCG_KERNEL_GAUSS)     ? fma (x[k], sc, c)
                       : (KERN == NCG_KERNEL_ST_WIDE) ? ncg_lnt_wide (x[k] * sc, p.kappa, c)
                                                      : fma (p.kappa, ncg_log_ge1 (fma (x[k], sc, 1.0)), c), g, s);
        }
      }

      if (!ok)
        break;

      if (j < p.m)
        p.part[(size_t) (Q_WG * sl + wg) * p.m + j] = make_double2 (g, s);
    }
  }

  _tc_fence_before ();
  __syncthreads ();

  if (warp == 1)
  {
    _tc_fence_after ();
    asm volatile ("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }

  if (threadIdx.x == 0 && sm.err)
  {
    atomicExch (p.err, 1);

    if (p.flag_host != NULL)
      *(volatile int *) p.flag_host = 1;
  }
}

/* --------------------------------------------------------------------- merge */

#define QM_TH 256

struct QMerge
{
  const double2 *part;
  const int32_t *pe2, *f;
  const double *Xq, *pack, *c;
  double *out;
  int64_t m;
  int nparts, n, d, dp, linear, fmax_;
  double kappa, inv_nu, shift, d_ln_href;
};

/* this thread's kernels against the point xs, by the plain form (a kernel per
 * thread; the whitened difference in local memory, since d is not a constant here) */
template <int KERN>
__device__ __noinline__ double2
_q_plain (const QMerge &p, const double *xs)
{
  const int S = ncg_pack64_stride (NCG_VKDE, p.dp);
  double dl[NCG_DMAX];
  double g = NCG_LSE_EMPTY, s = 0.0;

  for (int i = threadIdx.x; i < p.n; i += QM_TH)
  {
    const double *pk = p.pack + (size_t) i * S, *W = pk + p.dp;
    double chi2      = 0.0;

    for (int c = 0; c < p.d; c++)
      dl[c] = xs[c] - pk[c];

    for (int r = 0; r < p.d; r++)
    {
      double y = 0.0;

      for (int c = 0; c <= r; c++)
        y = fma (*W++, dl[c], y);

      chi2 = fma (y, y, chi2);
    }

    ncg_lse_add (ncg_lnt_64<KERN> (chi2, p.c[i], p.kappa, p.inv_nu, false), g, s);
  }

  return make_double2 (g, s);
}

/* The slices of 32 points, as the merge of the plain form (ncg_eval.cu) combines
 * them; then, one after the other, those of the points that take the plain form,
 * the CTA's threads sharing the kernels.  Nothing is left to do there in a call on points
 * like the sample's. */
template <int KERN>
__global__ void __launch_bounds__ (QM_TH)
_q_merge_kernel (const QMerge p)
{
  __shared__ double red[QM_TH / 32][33];
  __shared__ double xs[NCG_DMAX];
  __shared__ double2 ex[QM_TH / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t j = (int64_t) blockIdx.x * 32 + lane;
  const bool far_ = j < p.m && p.pe2[j] == Q_FAR, in = j < p.m && !far_;
  double G = NCG_LSE_EMPTY, S = 0.0;

  if (*p.f > p.fmax_)
    return;

  if (in)
    for (int s = w; s < p.nparts; s += QM_TH / 32)
      G = fmax (G, p.part[(size_t) s * p.m + j].x);

  red[w][lane] = G;
  __syncthreads ();

#pragma unroll
  for (int q = 0; q < QM_TH / 32; q++)
    G = fmax (G, red[q][lane]);

  __syncthreads ();

  if (in)
    for (int s = w; s < p.nparts; s += QM_TH / 32)
    {
      const double2 q = p.part[(size_t) s * p.m + j];

      S = fma (q.y, ncg_exp (q.x - G), S);
    }

  red[w][lane] = S;
  __syncthreads ();

  if (w == 0 && in)
  {
#pragma unroll
    for (int q = 1; q < QM_TH / 32; q++)
      S += red[q][lane];

    const double lnp = ncg_lse_lnp (G, S, p.shift, NULL, p.d_ln_href);

    p.out[j] = p.linear ? exp (lnp) : -2.0 * lnp;
  }

  /* the same 32 points in every warp */
  for (uint32_t mask = __ballot_sync (0xffffffffu, far_); mask; mask &= mask - 1)
  {
    const int64_t jf = (int64_t) blockIdx.x * 32 + __ffs (mask) - 1;

    __syncthreads ();

    if (tid < p.d)
      xs[tid] = p.Xq[jf * p.d + tid];

    __syncthreads ();

    const double2 q = _q_plain<KERN> (p, xs);
    double M = q.x, T = q.y;

#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      M = fmax (M, __shfl_xor_sync (0xffffffffu, M, o));

    T *= ncg_exp (q.x - M);

#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      T += __shfl_xor_sync (0xffffffffu, T, o);

    if (lane == 0)
      ex[w] = make_double2 (M, T);

    __syncthreads ();

    if (tid == 0)
    {
      for (int k = 1; k < QM_TH / 32; k++)
      {
        const double N = fmax (M, ex[k].x);

        T = T * ncg_exp (M - N) + ex[k].y * ncg_exp (ex[k].x - N);
        M = N;
      }

      const double lnp = ncg_lse_lnp (M, T, p.shift, NULL, p.d_ln_href);

      p.out[jf] = p.linear ? exp (lnp) : -2.0 * lnp;
    }
  }
}

/* ------------------------------------------------------------------- host side */

#define Q_ALIGN(x) (((x) + 255) / 256 * 256)

/* The calls that take this form: VKDE from d = 5 (below, the plain form's
 * whitening is no longer than the rest of the pair), with enough points that
 * even the first call on a new fit, which builds the kernels' operand, is not
 * slower than the plain form (its cost equals that of 480 to 600 points from
 * d = 5 to 32, n = 1000 to 8192), and enough kernels for a few tiles. */
extern "C" int
ncg_q64_wanted (const ncg_eval_args_t *a)
{
  return a->kind == NCG_VKDE && a->d >= 5 && a->m >= 640 && a->n >= 384 && a->n <= (1 << 24);
}

extern "C" int
ncg_q64_fmax (int d)
{
  return q_fmax (d);
}

/* operand of n kernels: digits | scales (n padded) | Zl | largest f */
typedef struct { size_t sck, zl, fmax, total; } q_operand_t;

static q_operand_t
_q_operand (int n, int d)
{
  const size_t nkt = (size_t) (n + Q_NK - 1) / Q_NK;
  q_operand_t o;

  o.sck   = Q_ALIGN (nkt * q_steps (d) * Q_B_STEP);
  o.zl    = o.sck + Q_ALIGN (nkt * Q_NK * sizeof (double));
  o.fmax  = o.zl + Q_ALIGN ((size_t) d * d * sizeof (double));
  o.total = o.fmax + 256;

  return o;
}

extern "C" size_t
ncg_q64_operand_bytes (int n, int d)
{
  return _q_operand (n, d).total;
}

/* device address of the largest f of the operand */
extern "C" const int32_t *
ncg_q64_operand_fmax (const uint8_t *op, int n, int d)
{
  return (const int32_t *) (op + _q_operand (n, d).fmax);
}

/* the operand of a's kernels; *word (mapped host memory) gets `epoch` in its upper half and
 * whether their range leaves room for points in bit 0 */
extern "C" cudaError_t
ncg_launch_q64_operand (const ncg_eval_args_t *a, const double *X, const double *pack64, const double *U,
                        const double *Vg, const double *mu, uint8_t *op, unsigned long long *word, uint32_t epoch,
                        cudaStream_t s)
{
  static int limit[NCG_MAX_DEVICES];
  const q_operand_t o = _q_operand (a->n, a->d);
  const size_t smem   = QB_WARPS * q_build_b_warp (a->d);
  const int npad      = (a->n + Q_NK - 1) / Q_NK * Q_NK;
  cudaError_t e;

  if ((e = cudaMemsetAsync (op + o.fmax, 0x80, sizeof (int32_t), s)) != cudaSuccess)
    return e;

  if ((e = ncg_raise_smem_limit ((const void *) _q_build_B_kernel, smem, limit)) != cudaSuccess)
    return e;

  _q_global_kernel<<<1, 1024, 0, s>>> (U, Vg, a->d, (double *) (op + o.zl));
  _q_build_B_kernel<<<npad / QB_WARPS, QB_WARPS * 32, smem, s>>> (
    X, pack64, ncg_pack64_stride (NCG_VKDE, a->dp), a->dp, a->n, a->d, U, Vg, (const double *) (op + o.zl), mu,
    (a->kernel == NCG_KERNEL_ST) ? 1.0 / a->nu : -0.5, op, (double *) (op + o.sck), (int32_t *) (op + o.fmax));
  _q_tell_kernel<<<1, 1, 0, s>>> ((const int32_t *) (op + o.fmax), q_fmax (a->d), epoch, word);

  return cudaGetLastError ();
}

/* scratch of a call: digits of up to Q_CHUNK points | their exponents | pairs of
 * all points | error word */
typedef struct { size_t pe2, part, err, total; int npt, nkt, ns, tps; } q_scratch_t;

static q_scratch_t
_q_scratch (const ncg_eval_args_t *a)
{
  const int64_t mc = a->m < Q_CHUNK ? a->m : Q_CHUNK;
  q_scratch_t o;
  long best = -1;

  o.npt = (int) ((mc + Q_M - 1) / Q_M);
  o.nkt = (a->n + Q_NK - 1) / Q_NK;
  o.ns  = 1;

  /* slices of the kernel tiles with the shortest schedule of whole tiles */
  for (int sl = 1; sl <= o.nkt && sl <= 64; sl++)
  {
    const long tp = (o.nkt + sl - 1) / sl, cost = ((long) o.npt * sl + 151) / 152 * tp;

    if (best < 0 || cost < best)
    {
      best = cost;
      o.ns = sl;
    }
  }

  o.tps   = (o.nkt + o.ns - 1) / o.ns;
  o.ns    = (o.nkt + o.tps - 1) / o.tps;
  o.pe2   = Q_ALIGN ((size_t) o.npt * q_steps (a->d) * Q_A_STEP);
  o.part  = o.pe2 + Q_ALIGN ((size_t) o.npt * Q_M * sizeof (int32_t));
  o.err   = o.part + Q_ALIGN (Q_WG * (size_t) o.ns * (size_t) mc * sizeof (double2));
  o.total = o.err + 256;

  return o;
}

extern "C" size_t
ncg_q64_scratch_bytes (const ncg_eval_args_t *a)
{
  return _q_scratch (a).total;
}

template <int KERN, int BITS>
static cudaError_t
_run_q64 (const QParams &p, int grid, cudaStream_t s)
{
  static int limit[NCG_MAX_DEVICES];
  const cudaError_t e = ncg_raise_smem_limit ((const void *) _eval_q64_kernel<KERN, BITS>, Q_SMEM_BYTES, limit);

  if (e != cudaSuccess)
    return e;

  _eval_q64_kernel<KERN, BITS><<<grid, Q_THREADS, Q_SMEM_BYTES, s>>> (p);

  return cudaGetLastError ();
}

template <int KERN>
static cudaError_t
_run_q64_bits (const QParams &p, const QMerge &q, int d, int grid, cudaStream_t s)
{
  const cudaError_t e = (d <= 16) ? _run_q64<KERN, 8> (p, grid, s) : _run_q64<KERN, 7> (p, grid, s);

  if (e != cudaSuccess)
    return e;

  _q_merge_kernel<KERN><<<(unsigned) ((q.m + 31) / 32), QM_TH, 0, s>>> (q);

  return cudaGetLastError ();
}

extern "C" cudaError_t
ncg_launch_eval_q64 (const ncg_eval_args_t *a, const double *Xq, const uint8_t *op, const double *pack64,
                     const double *c, const double *mu, const double *Vg, double *out, void *scratch, int linear,
                     int *flag_host, cudaStream_t s)
{
  static int limit[NCG_MAX_DEVICES];
  const q_scratch_t o = _q_scratch (a);
  const q_operand_t b = _q_operand (a->n, a->d);
  const size_t smem   = QA_WARPS * q_build_a_warp (a->d);
  cudaError_t e;
  int dev, nsm;

  if (a->m <= 0 || a->n <= 0 || a->kind != NCG_VKDE)
    return cudaErrorInvalidValue;

  if ((e = cudaGetDevice (&dev)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute (&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
      (e = ncg_raise_smem_limit ((const void *) _q_build_A_kernel, smem, limit)) != cudaSuccess)
    return e;

  QParams p;

  p.A         = (const uint8_t *) scratch;
  p.B         = op;
  p.pe2       = (const int32_t *) ((uint8_t *) scratch + o.pe2);
  p.f         = (const int32_t *) (op + b.fmax);
  p.fmax_     = q_fmax (a->d);
  p.sck       = (const double *) (op + b.sck);
  p.c         = c;
  p.part      = (double2 *) ((uint8_t *) scratch + o.part);
  p.err       = (int *) ((uint8_t *) scratch + o.err);
  p.flag_host = flag_host;
  p.n         = a->n;
  p.steps     = q_steps (a->d);
  p.nkt       = o.nkt;
  p.nslices   = o.ns;
  p.tps       = o.tps;
  p.kappa     = a->kappa;
  p.fault     = ncg_fault_take (NCG_FAULT_EVAL_TC_WAIT);

  for (int64_t j0 = 0; j0 < a->m; j0 += Q_CHUNK)
  {
    const int64_t mc = (a->m - j0 < Q_CHUNK) ? a->m - j0 : Q_CHUNK;

    p.m   = mc;
    p.npt = (int) ((mc + Q_M - 1) / Q_M);

    _q_build_A_kernel<<<p.npt * (Q_M / QA_WARPS), QA_WARPS * 32, smem, s>>> (
      Xq + j0 * a->d, mc, a->d, Vg, mu, p.f, (uint8_t *) scratch, (int32_t *) p.pe2, p.err);

    if ((e = cudaGetLastError ()) != cudaSuccess)
      return e;

    const int units = p.npt * p.nslices, grid = units < nsm ? units : nsm;

    const QMerge q = { p.part, p.pe2, p.f, Xq + j0 * a->d, pack64, c, out + j0, mc, Q_WG * o.ns, a->n, a->d, a->dp,
                       linear, p.fmax_, a->kappa, 1.0 / a->nu, a->final_shift, a->d_ln_href };

    e = (a->kernel == NCG_KERNEL_GAUSS)  ? _run_q64_bits<NCG_KERNEL_GAUSS> (p, q, a->d, grid, s)
        : ncg_nu_wide (a->nu, a->d)      ? _run_q64_bits<NCG_KERNEL_ST_WIDE> (p, q, a->d, grid, s)
                                         : _run_q64_bits<NCG_KERNEL_ST> (p, q, a->d, grid, s);

    if (e != cudaSuccess)
      return e;
  }

  return cudaSuccess;
}
