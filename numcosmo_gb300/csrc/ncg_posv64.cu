/*
 * ncg_posv64.cu -- the FP64 normal equations of the NNLS on the tensor cores:
 * M = A^T A (ncm_matrix_square_to_sym, numcosmo/ncm/algebra/ncm_matrix.c:1548-1572)
 * and the solve of M x = b by Cholesky (dposv, ncm_nnls.c:640-652).
 *
 * What bounds it: a dense FP64 factorisation is n^3 / 3 operations on pipes that
 * issue a warp instruction per 64 cycles and sub-partition (1.26 TFLOP/s), while
 * the FP16 tensor cores multiply exact integers 1500 times as fast.  So the
 * symmetric products C (-)= P^T P run as sliced integer products (Ozaki et al.,
 * Numer. Algorithms 59, 2012): each column is scaled by its own power of two
 * (largest entry below 2^ex) and held as 63-bit fixed point, 7 balanced digits of
 * 9 bits in FP16; digit products of one order o = i + j are summed by
 * tcgen05.mma.kind::f16 over 32 rows into an FP32 accumulator, exactly ((o + 1)
 * 32 2^16 < 2^24 for all seven orders kept); the epilogue adds the orders of all
 * chunks in 128 bits and rounds once.  The dropped orders are below 2^-60 of
 * the two columns' largest entries, so the error is that of one rounding of
 * the sum, where an FMA chain rounds every term.
 *
 * Factorisation.  Right-looking in panels of 32 rows, two launches a panel:
 * _posv_panel_kernel eliminates and scales the panel's columns to the right by
 * the multipliers of its diagonal block and packs them as digits;
 * _syrk64_kernel takes the panel off the trailing block, and its CTA 0, done with
 * the first tile, factors the next diagonal block while the others update.  The
 * right-hand side rides along as one more column, which leaves U^{-T} b at the
 * end; _posv_back_kernel solves U x = U^{-T} b in one launch.
 * Measured at n = 1700 (n = 4096): panel 10 us (12), update 23 us with the
 * diagonal block's 27 beside it (78 us), U x = y 175 us (413 us); the whole solve
 * 1.76 ms (5.9 ms), the starts of its launches behind their predecessors.  The
 * plain form took 90 (diagonal) + 120 (panel) + 110 us (update) per 64 rows at
 * n = 1700 and 33 us per 64 rows for each triangle, 10 ms.  Left: the chain of 32
 * pivots (the bound below n = 1900), the epilogue of the update above.
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "ncg_internal.h"
#include "ncg_pdl.cuh"
#include "ncg_tc_ptx.cuh"

#define P_NS 7                        /* slices and orders                   */
#define P_BITS 9
#define P_FIX 62                      /* |v| < 2^ex is held as v 2^(62 - ex) */
#define P_K 32                        /* rows of a chunk (and of a panel)    */
#define P_SLAB (1 << 13)              /* chunks of a launch at most: the orders' sums stay below 2^62 */
#define P_T 128                       /* columns of a pack tile (MMA M)      */
#define P_N 32                        /* output columns of a tile            */
#define P_UNIT (P_T * 16)             /* 8 rows of one slice of a tile       */
#define P_LBO (P_NS * P_UNIT)         /* the next 8 rows                     */
#define P_CHUNK (4 * P_LBO)           /* 57344: 32 rows x 128 columns        */
#define P_BAD 0x3fffffff              /* column exponent: a non-finite entry */
#define P_ZERO (-1061109568)          /* column exponent: all zero (0xc0 bytes) */

/* ---------------------------------------------------------------- digits */

/* ex with |v| < 2^ex */
__device__ __forceinline__ int
_above (double v)
{
  const int e = (int) (((uint32_t) __double2hiint (v) >> 20) & 0x7ffu);

  return (e == 0x7ff) ? P_BAD : (v == 0.0) ? P_ZERO : (e > 0 ? e : 1) - 1022;
}

/* the digits of v 2^(62 - ex), dig[slice * ld], in integer instructions */
__device__ __forceinline__ void
_digits63 (double v, int ex, uint16_t *dig, int ld)
{
  const long long bits = __double_as_longlong (v);
  const int ef         = (int) ((bits >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long) bits & 0xfffffffffffffull;

  if (ef > 0)
    m |= 1ull << 52;

  /* m counts 2^(e - 53) with e = max (ef, 1) - 1022 */
  const int s = P_FIX - 53 - (ex - ((ef > 0 ? ef : 1) - 1022));
  long long V = 0;

  if (ex < P_BAD && ex > P_ZERO && s > -62)
    V = (long long) ((s >= 0) ? m << s : (m + (1ull << (-s - 1))) >> -s);

  if (bits < 0)
    V = -V;

  unsigned long long u = (unsigned long long) V, bias = 0;

#pragma unroll
  for (int i = 0; i < P_NS; i++)
    bias = (bias << P_BITS) + (1ull << (P_BITS - 1));

  u += bias;

#pragma unroll
  for (int i = P_NS - 1; i >= 0; i--)
  {
    const uint32_t d = (i > 0) ? (uint32_t) u & ((1u << P_BITS) - 1) : (uint32_t) u;

    /* 1024 + d less 1024 + 256 in FP16: exact */
    dig[i * ld] = __half_as_ushort (__hsub (__ushort_as_half ((uint16_t) (0x6400 + d)),
                                            __ushort_as_half ((uint16_t) (0x6400 + (1 << (P_BITS - 1))))));
    u >>= P_BITS;
  }
}

/* ------------------------------------------------------------------ A^T A */

/* ex[c] of the columns of A (nrows x ncols, row-major), over a block of rows;
 * ex starts at P_ZERO */
#define CE_ROWS 128

__global__ void __launch_bounds__ (128)
_col_exp_kernel (const double *__restrict__ A, int nrows, int ncols, int32_t *__restrict__ ex)
{
  const int c = blockIdx.x * 128 + threadIdx.x, r0 = blockIdx.y * CE_ROWS, r1 = min (nrows, r0 + CE_ROWS);
  int e       = P_ZERO;

  if (c >= ncols)
    return;

#pragma unroll 8
  for (int r = r0; r < r1; r++)
    e = max (e, _above (A[(size_t) r * ncols + c]));

  atomicMax (ex + c, e);
}

/* digits of rows [r0, r1) in 32-row chunks: block (t * nch + chunk) of the pack */
__global__ void __launch_bounds__ (256)
_pack63_kernel (const double *__restrict__ A, int r0, int r1, int ncols, int nch, const int32_t *__restrict__ ex,
                uint8_t *__restrict__ pk)
{
  __shared__ __align__ (16) uint16_t dig[P_NS][64][8];
  const int t = blockIdx.x / nch, ch = blockIdx.x % nch;
  uint8_t *blk = pk + (size_t) blockIdx.x * P_CHUNK;
  const int lc = threadIdx.x & 63, lr = threadIdx.x >> 6;

  for (int h = 0; h < 2; h++)
    for (int q = 0; q < 4; q++)
    {
      const int c = t * P_T + h * 64 + lc;

#pragma unroll
      for (int e = 0; e < 2; e++)
      {
        const int k = lr + 4 * e, r = r0 + ch * P_K + q * 8 + k;
        const bool in = c < ncols && r < r1;

        _digits63 (in ? A[(size_t) r * ncols + c] : 0.0, in ? ex[c] : 0, &dig[0][lc][k], 64 * 8);
      }

      __syncthreads ();

      for (int u = threadIdx.x; u < P_NS * 64; u += 256)
      {
        const int sl = u / 64, row = h * 64 + u % 64;

        *(uint4 *) (blk + (size_t) q * P_LBO + (size_t) sl * P_UNIT + (row >> 3) * 128 + (row & 7) * 16) =
          *(const uint4 *) &dig[sl][u % 64][0];
      }

      __syncthreads ();
    }
}

/* ---------------------------------------------------------- diagonal blocks */

/* The 32 x 32 diagonal block of a panel, factored by 16 warps, lane = column.
 * Warp 0 walks the chain of pivots: with row j finished it publishes the row and
 * the multipliers t_r = s_jr / s_jj, and takes t_(j+1) times it off row j + 1.  Ten
 * others, on the SM's other three sub-partitions so that their FP64 instructions
 * do not hold up the chain's, keep three rows each and take every step off them;
 * row r goes back to the chain after step r - 2.  So the chain is a reciprocal and 4
 * FP64 instructions (of 64 cycles each) per pivot, and the updates run beside it.
 * The quotient comes from the pivot's reciprocal in FP32 and one correction by its
 * remainder, so it is rounded like a division (the pivot of a repeated column is
 * then exactly zero); the moves between FP32 and FP64 are integer instructions
 * (conversions, divisions and square roots hold the FP64 pipe).  The rows are
 * scaled by 1 / sqrt (s_jj) at the end.  16 us from the first tile's end to the
 * stores (19 with four warps that each took their share of every step before the
 * next pivot). */
#define DG_WARPS 16

struct DiagSmem
{
  double S[P_K][P_K + 1];           /* the block; row j as it is handed back, then final */
  double T[P_K][P_K];               /* the multipliers of row j */
  double root[P_K], rinv[P_K];
  uint64_t full[P_K], next[P_K];    /* row j final, with its multipliers; row j taken through step j - 2 */
  int stop;                         /* not positive, or a wait that gave up */
};

/* by at least 64 threads, before the CTA's next barrier */
__device__ __forceinline__ void
_diag_init (DiagSmem &d, int tid)
{
  if (tid < 2 * P_K)
    _mbar_init (tid < P_K ? &d.full[tid] : &d.next[tid - P_K], 1);

  if (tid == 0)
    d.stop = 0;
}

__device__ __forceinline__ void
_bar_named (int id, int threads)
{
  asm volatile ("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

/* 1 / x to 2^-43 for a positive x, in FP32 and integer instructions: the FP32
 * reciprocal r0 of the mantissa's leading 24 bits, its residual with the next 23
 * taken in, and r1 = r0 (1 - f r0) added to r0 in units of its binade as a double
 * (1 / f stays in [1/2, 1], so the sum leaves that binade by the error only).  A
 * Newton step in FP64 gave as much for two more instructions of 64 cycles on the
 * pivots' chain. */
__device__ __forceinline__ double
_recip44 (double x)
{
  const int hi = __double2hiint (x), lo = __double2loint (x), ef = (hi >> 20) & 0x7ff;

  if (ef < 64 || ef > 1980)
    return 1.0 / x;

  /* mantissa in [1, 2): f + g, f its leading 24 bits */
  const float f = __int_as_float (0x3f800000 | ((hi & 0xfffff) << 3) | (int) ((uint32_t) lo >> 29));
  const float g = (__int_as_float (0x3f800000 | ((lo >> 6) & 0x7fffff)) - 1.0f) * 0x1p-23f;
  float r0;

  asm ("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(f));
  r0 = fminf (r0, 0x1.fffffep-1f);

  const float r1 = r0 * fmaf (-g, r0, fmaf (-f, r0, 1.0f));
  const int rb   = __float_as_int (r0);

  return __longlong_as_double (__double_as_longlong (__hiloint2double (((2045 - ef) << 20) | ((rb & 0x7fffff) >> 3), rb << 29)) +
                               __float2int_rn (r1 * 0x1p+53f));
}

/* a / u from ri near 1 / u, its remainder put right once: rounded like a division */
__device__ __forceinline__ double
_scaled (double a, double u, double ri)
{
  const double x = a * ri;

  return fma (fma (-x, u, a), ri, x);
}

/* d.S in, the factor (nb x nb, at A with leading dimension ld) out; Lt[j][r] =
 * s_jr / s_jj for r > j, root and rd (1 / root) for the panel's other columns.
 * DG_WARPS warps w with named barrier `bar`; d set up by _diag_init. */
__device__ __forceinline__ void
_diag_factor (DiagSmem &d, int w, int lane, int bar, int nb, double *__restrict__ A, int ld, double *__restrict__ Lt,
              double *__restrict__ root, double *__restrict__ rd, int col0, int32_t *__restrict__ info)
{
  volatile int *stop = &d.stop;
  const int b        = (w >> 2) * 3 + (w & 3) - 1;
  int fail = 0;

  /* the identity past nb */
  auto in = [&] (int r) -> double {
    return (r < nb && lane < nb) ? ((lane >= r) ? d.S[r][lane] : 0.0) : (r == lane ? 1.0 : 0.0);
  };

  if (w == 0)
  {
    double row = in (0);

#pragma unroll 1
    for (int j = 0; j < P_K; j++)
    {
      const double pv = __shfl_sync (0xffffffffu, row, j);
      const int ph    = __double2hiint (pv);

      /* not positive, inf or NaN, by the high word (an FP64 compare is 64 cycles) */
      if ((uint32_t) (ph - 1) >= 0x7fefffffu && !(ph == 0 && __double2loint (pv) != 0))
      {
        fail  = j + 1;
        *stop = 1;
        __syncwarp ();

        /* nobody waits for what does not come */
        if (lane >= j)
          _mbar_arrive (&d.full[lane]);

        break;
      }

      const double y0 = _recip44 (pv), q = row * y0, t = fma (fma (-q, pv, row), y0, q);
      double nx       = 0.0;

      /* only here: row j + 1 comes back a step's update after row j - 1 went out,
       * while this step's quotient is worked out */
      if (j == 0)
        nx = in (1);
      else if (j < P_K - 1)
      {
        if (!__all_sync (0xffffffffu, _mbar_wait (&d.next[j + 1], 0, stop)))
          break;

        nx = d.S[j + 1][lane];
      }

      const double rn = fma (-__shfl_sync (0xffffffffu, t, (j + 1) & 31), row, nx);

      d.S[j][lane] = row;
      d.T[j][lane] = t;
      __syncwarp ();

      if (lane == 0)
        _mbar_arrive (&d.full[j]);

      Lt[j * P_K + lane] = t;
      row                = rn;
    }
  }
  else if ((w & 3) != 0 && b < 10)
  {
    const int ra = 2 + b, rb = 21 - b, rc = 22 + b;
    double sa = in (ra), sb = in (rb), sc = in (rc), dj = 0.0;
    int j   = 0;
    bool go = true;

    auto wait = [&] () {
      go = __all_sync (0xffffffffu, _mbar_wait (&d.full[j], 0, stop) && !*stop);
      dj = d.S[j][lane];
    };

    auto back = [&] (int r, double v) {
      d.S[r][lane] = v;
      __syncwarp ();

      if (lane == 0)
        _mbar_arrive (&d.next[r]);
    };

#pragma unroll 1
    for (; j <= ra - 2 && go; j++)
    {
      wait ();
      sa = fma (-d.T[j][ra], dj, sa);

      if (j == ra - 2)
        back (ra, sa);

      sb = fma (-d.T[j][rb], dj, sb);
      sc = fma (-d.T[j][rc], dj, sc);
    }

#pragma unroll 1
    for (; j <= rb - 2 && go; j++)
    {
      wait ();
      sb = fma (-d.T[j][rb], dj, sb);

      if (j == rb - 2)
        back (rb, sb);

      sc = fma (-d.T[j][rc], dj, sc);
    }

#pragma unroll 1
    for (; j <= rc - 2 && go; j++)
    {
      wait ();
      sc = fma (-d.T[j][rc], dj, sc);
    }

    if (go)
      back (rc, sc);
  }

  _bar_named (bar, DG_WARPS * 32);

  if (*stop)
  {
    if (w == 0 && lane == 0)
    {
      if (fail)
        atomicCAS (info, 0, col0 + fail);
      else
        atomicExch (info, -1);
    }

    return;
  }

  ncg_pdl_next ();

  if (w == 0)
  {
    const double u = sqrt (d.S[lane][lane]), ri = 1.0 / u;

    d.root[lane] = u;
    d.rinv[lane] = ri;
    root[lane]   = u;

    if (lane < nb)
      rd[lane] = ri;
  }

  _bar_named (bar, DG_WARPS * 32);

#pragma unroll
  for (int r = w; r < P_K; r += DG_WARPS)
    if (r < nb && lane < nb && lane >= r)
      A[(size_t) r * ld + lane] = (lane == r) ? d.root[r] : _scaled (d.S[r][lane], d.root[r], d.rinv[r]);
}

/* ----------------------------------------------------- the symmetric product */

#define S_STAGES 2
#define S_A_BYTES P_CHUNK
#define S_B_UNIT (P_N * 16)                  /* 8 rows of one slice of the tile's columns */
#define S_B_LBO (P_NS * S_B_UNIT)
#define S_B_BYTES (4 * S_B_LBO)
#define S_EPI_WARP0 2
#define S_EPI_WARPS 16                       /* DG_WARPS of them factor the diagonal block */
#define S_THREADS ((S_EPI_WARP0 + S_EPI_WARPS) * 32)
#define S_TMEM (P_NS * P_N)                  /* 224 columns, two accumulators */

struct S64Params
{
  const uint8_t *pk;
  const int32_t *ex;
  double *C;              /* nn x nn block, leading dimension ldc */
  double *b;              /* column nn of the update (NULL: none) */
  double *Lt, *root, *rd; /* Lt not NULL: CTA 0 goes on to factor the leading 32 x 32 block of the result */
  int32_t *err;
  int nn, ldc, nch, mode; /* mode: 0 C = P^T P, 1 C -= P^T P, 2 C += P^T P */
  int col0;               /* the result's first column in the factorisation */
};

struct S64Smem
{
  uint8_t st[S_STAGES][S_A_BYTES + S_B_BYTES];
  uint64_t full[S_STAGES], empty[S_STAGES], t_full[2], t_empty[2], done;
  DiagSmem diag;
  uint32_t tmem_base;
  int err, skip, ndiag; /* skip: nothing to do; ndiag: epilogue warps that stored tile 0 */
};

#define S64_SMEM_BYTES (sizeof (S64Smem) + 1024)

/* D(f32)[128 x N] (+)= A(f16, 128 x 16) . B(f16, N x 16)^T */
__device__ __forceinline__ void
_s_mma (uint32_t dtmem, uint64_t adesc, uint64_t bdesc, int N, uint32_t accumulate)
{
  const uint32_t idesc = (1u << 4) | ((uint32_t) (N >> 3) << 17) | ((uint32_t) (P_T >> 4) << 24);

  asm volatile ("{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                ::"r"(dtmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                : "memory");
}

/* 16 lanes x 8 columns: thread t gets (row t / 4, columns 2 (t % 4) and + 1),
 * then the same of row t / 4 + 8, so that four neighbouring threads hold 64
 * contiguous bytes of a row of C (a row per lane would touch 32 lines per
 * access of C) */
__device__ __forceinline__ void
_s_ld (uint32_t t, uint32_t *r)
{
  asm volatile ("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                : "r"(t)
                : "memory");
}

/* output tile u: 128-column row tile ti, 32-column tile tj with a column at or
 * right of the tile's first row; ncol counts the columns (nn, or nn + 1) */
__device__ __forceinline__ bool
_s_tile (int u, int T_, int ncol, int *ti, int *tj)
{
  const int Tn = (ncol + P_N - 1) / P_N;

  for (int i = 0; i < T_; i++)
  {
    const int w = Tn - P_T / P_N * i;

    if (u < w)
    {
      *ti = i;
      *tj = P_T / P_N * i + u;

      return true;
    }

    u -= w;
  }

  return false;
}

/* hi 2^27 + lo rounded once (|hi| < 2^62, |lo| < 2^62: a chunk adds up to 2^48.1 to hi and
 * 2^42.4 to lo, and P_SLAB bounds their number), in integer instructions: two FP64
 * additions on biased mantissas did the same at 128 cycles of the FP64 pipe, which the
 * update then waited for */
__device__ __forceinline__ double
_join (long long hi, long long lo)
{
  const uint32_t mask = (1u << 27) - 1;
  const long long h   = hi + (lo >> 27);
  const uint32_t l    = (uint32_t) lo & mask;
  const bool neg      = h < 0;
  const unsigned long long a = (unsigned long long) (neg ? ~h + (l == 0) : h);
  const uint32_t b           = neg ? (0u - l) & mask : l;

  if (a == 0)
    return (double) (neg ? -(float) b : (float) b);   /* b < 2^24 or a rounding far below the sum's own */

  /* the leading 64 bits of a 2^27 + b, normalised */
  const int n = __clzll ((long long) a);
  const unsigned long long top = (a << n) | ((n >= 27) ? (unsigned long long) b << (n - 27) : (unsigned long long) (b >> (27 - n)));
  const long long v = ((long long) (1023 + 63 - n + 27 - 1) << 52) + (long long) (top >> 11) + (long long) ((top >> 10) & 1);

  return __longlong_as_double (v | ((long long) neg << 63));
}

/* 2^e; 0 below the normal range, inf above */
__device__ __forceinline__ double
_scale2 (int e)
{
  return __hiloint2double ((e < -1022) ? 0 : (min (e, 1024) + 1023) << 20, 0);
}

__global__ void __launch_bounds__ (S_THREADS, 1)
_syrk64_kernel (const S64Params p)
{
  extern __shared__ __align__ (16) uint8_t s64_raw[];
  S64Smem &sm = *(S64Smem *) (((uintptr_t) s64_raw + 1023) & ~(uintptr_t) 1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ncol = p.nn + (p.b != NULL), T_ = (p.nn + P_T - 1) / P_T;
  /* tiles blockIdx.x, blockIdx.x + ustep, ...; where CTA 0 has the diagonal
   * block to factor it takes tile 0 only */
  const bool lone = p.Lt != NULL && gridDim.x > 1;
  const int ustep = !lone ? (int) gridDim.x : (blockIdx.x == 0 ? (1 << 28) : (int) gridDim.x - 1);
  volatile int *err = &sm.err;

  if (threadIdx.x == 0)
  {
    sm.ndiag = 0;

    for (int s = 0; s < S_STAGES; s++)
    {
      _mbar_init (&sm.full[s], 1);
      _mbar_init (&sm.empty[s], 1);
    }

    for (int b = 0; b < 2; b++)
    {
      _mbar_init (&sm.t_full[b], 1);
      _mbar_init (&sm.t_empty[b], S_EPI_WARPS);
    }

    _mbar_init (&sm.done, 1);
  }

  if (p.Lt != NULL && blockIdx.x == 0 && warp >= S_EPI_WARP0)
    _diag_init (sm.diag, threadIdx.x - S_EPI_WARP0 * 32);

  if (warp != 1)
    asm volatile ("fence.mbarrier_init.release.cluster;" ::: "memory");

  if (warp == 1)
  {
    asm volatile ("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                  ::"r"(_smem_u32 (&sm.tmem_base)), "r"(512)
                  : "memory");
    asm volatile ("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  (void) ncg_pdl_wait ();

  /* a factorisation that already failed (or timed out) needs no more updates */
  const bool skip = *(volatile int32_t *) p.err != 0;

  if (threadIdx.x == 0)
    sm.err = sm.skip = skip ? 1 : 0;

  _tc_fence_before ();
  __syncthreads ();
  _tc_fence_after ();

  const uint32_t tmem = sm.tmem_base;
  int ti, tj;

  if (warp == 0)
  {
    /* ---------------- producer ---------------- */
    if (lane == 0)
    {
      int stage = 0;
      uint32_t phase = 0;
      int armed[S_STAGES];

      for (int s = 0; s < S_STAGES; s++)
        armed[s] = -1;

      for (int u = blockIdx.x; !*err && _s_tile (u, T_, ncol, &ti, &tj); u += ustep)
        for (int c = 0; c < p.nch; c++)
        {
          if (!_mbar_wait (&sm.empty[stage], phase ^ 1, err))
            break;

          const uint8_t *a = p.pk + ((size_t) ti * p.nch + c) * P_CHUNK;
          const uint8_t *b = p.pk + ((size_t) (tj / (P_T / P_N)) * p.nch + c) * P_CHUNK + (tj % (P_T / P_N)) * S_B_UNIT;

          _mbar_arrive_tx (&sm.full[stage], S_A_BYTES + S_B_BYTES);
          _bulk_g2s (sm.st[stage], a, S_A_BYTES, &sm.full[stage]);

          /* the 32 columns' part of each (8 rows, slice) unit */
          for (int q = 0; q < 4 * P_NS; q++)
            _bulk_g2s (sm.st[stage] + S_A_BYTES + q * S_B_UNIT, b + (size_t) q * P_UNIT, S_B_UNIT, &sm.full[stage]);

          armed[stage] = (int) phase;

          if (++stage == S_STAGES)
          {
            stage = 0;
            phase ^= 1;
          }
        }

      for (int s = 0; s < S_STAGES; s++)
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
      bool ok = !*err;

      for (int u = blockIdx.x; ok && _s_tile (u, T_, ncol, &ti, &tj); u += ustep)
        for (int c = 0; c < p.nch && ok; c++, tc++)
        {
          const int tb = tc & 1;

          ok = _mbar_wait (&sm.t_empty[tb], ((tc >> 1) & 1) ^ 1, err) && _mbar_wait (&sm.full[stage], phase, err);

          if (!ok)
            break;

          _tc_fence_after ();

          const uint8_t *As = sm.st[stage], *Bs = As + S_A_BYTES;

          /* two 16-row steps; slice i meets the stacked slices 0..6-i of B, its
           * output columns being the orders i..6 */
#pragma unroll
          for (int ks = 0; ks < 2; ks++)
#pragma unroll
            for (int i = 0; i < P_NS; i++)
              _s_mma (tmem + (uint32_t) (tb * S_TMEM + i * P_N), _sdesc (As + 2 * ks * P_LBO + i * P_UNIT, P_LBO),
                      _sdesc (Bs + 2 * ks * S_B_LBO, S_B_LBO), P_N * (P_NS - i), (ks > 0 || i > 0) ? 1u : 0u);

          _mma_commit (&sm.empty[stage]);
          _mma_commit (&sm.t_full[tb]);

          if (++stage == S_STAGES)
          {
            stage = 0;
            phase ^= 1;
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
    const int wg = (warp - S_EPI_WARP0) >> 2;     /* which 8 columns */
    const int q  = warp & 3;                      /* TMEM lane quarter (hardware: warp id mod 4) */
    const uint32_t base = tmem + ((uint32_t) (q * 32) << 16) + (uint32_t) (wg * 8);
    int tc = 0;
    /* the same answer in every warp (the error flag may go up before the last of them
     * looks): all of them come to tile 0's barrier, or none */
    bool ok = !sm.skip;

    for (int u = blockIdx.x; ok && _s_tile (u, T_, ncol, &ti, &tj); u += ustep)
    {
      /* element k = 4 half + 2 h + c: row ib + 16 half + 8 h, column jb + c */
      const int ib = ti * P_T + q * 32 + (lane >> 2), jb = tj * P_N + wg * 8 + 2 * (lane & 3);
      long long hi[8], lo[8];
      double cv[8];
      int er[4], ec[2];

#pragma unroll
      for (int k = 0; k < 8; k++)
      {
        const int i = ib + 8 * (k >> 1), j = jb + (k & 1);

        hi[k] = lo[k] = 0;
        /* C on its way while the product is made */
        cv[k] = (p.mode != 0 && i < p.nn && j >= i && j < ncol)
                ? ((j < p.nn) ? p.C[(size_t) i * p.ldc + j] : p.b[i]) : 0.0;
      }

#pragma unroll
      for (int k = 0; k < 4; k++)
        er[k] = (ib + 8 * k < p.nn) ? p.ex[ib + 8 * k] : P_ZERO;

#pragma unroll
      for (int k = 0; k < 2; k++)
        ec[k] = (jb + k < ncol) ? p.ex[jb + k] : P_ZERO;

      for (int c = 0; c < p.nch; c++, tc++)
      {
        const int tb = tc & 1;

        if (!__all_sync (0xffffffffu, _mbar_wait (&sm.t_full[tb], (tc >> 1) & 1, err)))
        {
          ok = false;
          break;
        }

        _tc_fence_after ();

#pragma unroll
        for (int h = 0; h < 2; h++)
        {
          uint32_t r[P_NS][4];

#pragma unroll
          for (int o = 0; o < P_NS; o++)
            _s_ld (base + ((uint32_t) (h * 16) << 16) + (uint32_t) (tb * S_TMEM + o * P_N), r[o]);

          asm volatile ("tcgen05.wait::ld.sync.aligned;" ::: "memory");

#pragma unroll
          for (int o = 0; o < P_NS; o++)
            asm volatile ("" : "+r"(r[o][0]), "+r"(r[o][1]), "+r"(r[o][2]), "+r"(r[o][3]) : : "memory");

          if (h == 1)
          {
            _tc_fence_before ();
            __syncwarp ();

            if (lane == 0)
              _mbar_arrive (&sm.t_empty[tb]);
          }

#pragma unroll
          for (int k = 0; k < 4; k++)
          {
            int g[P_NS];

#pragma unroll
            for (int o = 0; o < P_NS; o++)
              g[o] = __float2int_rn (__uint_as_float (r[o][k]));

            /* |g[0]| <= 2^21, |g[1]| <= 2^22: their join stays in 32 bits */
            hi[4 * h + k] += (long long) (g[0] * (1 << P_BITS) + g[1]) * (1 << 2 * P_BITS) +
                             ((long long) g[2] * (1 << P_BITS) + g[3]);
            lo[4 * h + k] += (long long) g[4] * (1 << 2 * P_BITS) + ((long long) g[5] * (1 << P_BITS) + g[6]);
          }
        }
      }

      if (!ok)
      {
        /* a warp that gave up does not hold the others at tile 0's barrier */
        if (p.Lt != NULL && u == 0)
          _bar_named (1, S_EPI_WARPS * 32);

        break;
      }

#pragma unroll
      for (int k = 0; k < 8; k++)
      {
        const int i = ib + 8 * (k >> 1), j = jb + (k & 1);

        if (i >= p.nn || j < i || j >= ncol)
          continue;

        /* order 6 counts 2^(ei + ej - 70) */
        const int ei = er[k >> 1], ej = ec[k & 1];
        double sc    = (ei == P_ZERO || ej == P_ZERO) ? 0.0 : _scale2 (ei + ej - 70);

        if (ei == P_BAD || ej == P_BAD)
          sc = CUDART_NAN;

        const double v = fma (_join (hi[k], lo[k]), (p.mode == 1) ? -sc : sc, cv[k]);

        if (j < p.nn)
          p.C[(size_t) i * p.ldc + j] = v;
        else
          p.b[i] = v;

        if (p.Lt != NULL && u == 0 && i < P_K && j < P_K)
          sm.diag.S[i][j] = v;
      }

      __syncwarp ();

      if (p.Lt != NULL && u == 0)
      {
        /* the next panel's diagonal block, while the other CTAs update; not
         * if any warp gave up (the same answer in every warp) */
        if (lane == 0)
          atomicAdd (&sm.ndiag, 1);

        _bar_named (1, S_EPI_WARPS * 32);

        if (*(volatile int *) &sm.ndiag == S_EPI_WARPS)
          _diag_factor (sm.diag, warp - S_EPI_WARP0, lane, 2, min (p.nn, P_K), p.C, p.ldc, p.Lt, p.root, p.rd, p.col0,
                        p.err);
      }
    }
  }

  _tc_fence_before ();
  __syncthreads ();

  if (warp == 1)
  {
    _tc_fence_after ();
    asm volatile ("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }

  if (threadIdx.x == 0 && sm.err && !skip)
    atomicExch (p.err, -1);
}

/* ------------------------------------------------------------------ panels */

/* One panel: rows kb .. kb + nb of the columns right of its diagonal block
 * (and of b, column n), from the block's multipliers Lt.  16 columns per CTA: a
 * lane has column lane mod 16 and the rows 2w + lane / 16 mod 8, so that an FP64
 * instruction takes two rows and the columns spread over twice as many SMs (32
 * columns with a row per instruction: 13 us, now 10 us at n = 1700).  Step j
 * publishes the finished row j and the rows below take it off.  Then the rows are
 * scaled, written and packed as digits with their columns' exponents. */
#define PP_TH 128
#define PP_C 16

__global__ void __launch_bounds__ (PP_TH)
_posv_panel_kernel (double *__restrict__ A, int n, double *__restrict__ b, int kb, int nb,
                    const double *__restrict__ Lt, const double *__restrict__ root, uint8_t *__restrict__ pk,
                    int32_t *__restrict__ ex, const int32_t *__restrict__ info)
{
  __shared__ double L[P_K][P_K], row[2][PP_C];
  __shared__ int exm[8][PP_C];
  __shared__ __align__ (16) uint16_t dig[P_NS][PP_C][P_K + 8];
  const int tid = threadIdx.x, lane = tid & 31, c = tid & (PP_C - 1), r0 = tid / PP_C;
  const int rel = blockIdx.x * PP_C + c, col = kb + nb + rel;
  double a[4];

  const size_t pdl0 = ncg_pdl_wait ();

  Lt   += pdl0;
  root += pdl0;
  A += pdl0;
  b += pdl0;
  pk += pdl0;
  ex += pdl0;
  info += pdl0;

  if (*(volatile const int32_t *) info)
    return;

#pragma unroll
  for (int p = 0; p < 4; p++)
  {
    const int r = r0 + 8 * p;

    a[p] = (r < nb && col <= n) ? ((col < n) ? A[(size_t) (kb + r) * n + col] : b[kb + r]) : 0.0;
  }

#pragma unroll
  for (int p = 0; p < 8; p++)
    L[(tid >> 5) + 4 * p][lane] = Lt[((tid >> 5) + 4 * p) * P_K + lane];

#pragma unroll
  for (int p0 = 0; p0 < 4; p0++)
#pragma unroll
    for (int jj = 0; jj < 8; jj++)
    {
      const int j = 8 * p0 + jj;

      if (r0 == jj)
        row[j & 1][c] = a[p0];

      __syncthreads ();

      const double aj = row[j & 1][c];

      /* the warp's two rows may lie on either side of row j */
      if ((r0 | 1) > jj)
      {
        const double v = fma (-L[j][r0 + 8 * p0], aj, a[p0]);

        a[p0] = (r0 > jj) ? v : a[p0];
      }

#pragma unroll
      for (int p = p0 + 1; p < 4; p++)
        a[p] = fma (-L[j][r0 + 8 * p], aj, a[p]);
    }

  ncg_pdl_next ();

  /* row r = lane's root and near its reciprocal */
  const double ur = root[lane], rr = _recip44 (ur);
  int e = P_ZERO;

#pragma unroll
  for (int p = 0; p < 4; p++)
  {
    const int r = r0 + 8 * p;

    a[p] = _scaled (a[p], __shfl_sync (0xffffffffu, ur, r), __shfl_sync (0xffffffffu, rr, r));
    e    = max (e, _above (a[p]));

    if (r < nb && col <= n)
    {
      if (col < n)
        A[(size_t) (kb + r) * n + col] = a[p];
      else
        b[kb + r] = a[p];
    }
  }

  /* the columns' digits */
  exm[r0][c] = e;
  __syncthreads ();

#pragma unroll
  for (int q = 0; q < 8; q++)
    e = max (e, exm[q][c]);

  if (r0 == 0 && col <= n)
    ex[rel] = e;

#pragma unroll
  for (int p = 0; p < 4; p++)
    _digits63 (a[p], e, &dig[0][c][r0 + 8 * p], PP_C * (P_K + 8));

  __syncthreads ();

  uint8_t *blk = pk + (size_t) (blockIdx.x / (P_T / PP_C)) * P_CHUNK;

  for (int u = tid; u < 4 * P_NS * PP_C; u += PP_TH)
  {
    const int cc = u % PP_C, qs = u / PP_C, sl = qs % P_NS, q = qs / P_NS;
    const int r  = (blockIdx.x % (P_T / PP_C)) * PP_C + cc;

    *(uint4 *) (blk + (size_t) q * P_LBO + (size_t) sl * P_UNIT + (r >> 3) * 128 + (r & 7) * 16) =
      *(const uint4 *) &dig[sl][cc][q * 8];
  }
}

/* the first diagonal block; info = 0 */
__global__ void __launch_bounds__ (DG_WARPS * 32)
_posv_begin_kernel (double *__restrict__ A, int n, double *__restrict__ Lt, double *__restrict__ root,
                    double *__restrict__ rd, int32_t *info)
{
  __shared__ DiagSmem d;
  const int tid = threadIdx.x, nb = min (n, P_K);

  _diag_init (d, tid);
  asm volatile ("fence.mbarrier_init.release.cluster;" ::: "memory");

  for (int e = tid; e < P_K * P_K; e += DG_WARPS * 32)
  {
    const int r = e / P_K, c = e % P_K;

    d.S[r][c] = (r < nb && c < nb && c >= r) ? A[(size_t) r * n + c] : 0.0;
  }

  if (tid == 0)
    *info = 0;

  __syncthreads ();
  _diag_factor (d, tid >> 5, tid & 31, 1, nb, A, n, Lt, root, rd, 0, info);
}

/* ------------------------------------------------------- U x = y, one launch */

/* Blocks of 32 rows from the last, each CTA taking the next by ticket, so
 * it only waits for blocks of CTAs that already run.  A finished block
 * publishes each value as two words that carry their own validity (half of
 * the bits and a mark), which the readers poll (one memory round trip, no flag
 * and no fence); all words are zeroed by the host before the launch.  A wait
 * gives up after PB_SPIN polls, sets *info = -1 and the launch goes on with
 * what it has, so it always ends. */
#define PB_TH 128
#define PB_SPIN (1 << 21)
#define PB_MARK 0x5a5a5a5au

__device__ __forceinline__ void
_pb_put (unsigned long long *w, double v)
{
  const unsigned long long h = ((unsigned long long) PB_MARK << 32) | (uint32_t) __double2hiint (v);
  const unsigned long long l = ((unsigned long long) PB_MARK << 32) | (uint32_t) __double2loint (v);

  asm volatile ("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(w), "l"(h), "l"(l) : "memory");
}

__device__ __forceinline__ double
_pb_get (const unsigned long long *w, int32_t *info)
{
  unsigned long long h, l;

  for (int k = 0;; k++)
  {
    asm volatile ("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(h), "=l"(l) : "l"(w) : "memory");

    if ((uint32_t) (h >> 32) == PB_MARK && (uint32_t) (l >> 32) == PB_MARK)
      break;

    if (k > PB_SPIN || ((k & 255) == 255 && *(volatile int32_t *) info < 0))
    {
      atomicExch (info, -1);
      break;
    }
  }

  return __hiloint2double ((int) (uint32_t) h, (int) (uint32_t) l);
}

__global__ void __launch_bounds__ (PB_TH)
_posv_back_kernel (const double *__restrict__ U, int n, const double *__restrict__ rd, double *__restrict__ b,
                   unsigned long long *__restrict__ words, int32_t *__restrict__ ticket, int32_t *__restrict__ info)
{
  __shared__ double S[P_K][P_K + 1];
  __shared__ double sv[P_K];
  __shared__ int blk;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nbk = (n + P_K - 1) / P_K;

  if (*(volatile int32_t *) info)
    return;

  if (tid == 0)
    blk = nbk - 1 - atomicAdd (ticket, 1);

  __syncthreads ();

  const int i = blk, kb = i * P_K, nb = min (P_K, n - kb);
  double acc[8];

  for (int e = tid; e < P_K * P_K; e += PB_TH)
  {
    const int r = e / P_K, c = e % P_K;

    /* columns over their diagonal: the substitution then runs on the unscaled
     * values, a shuffle and an FMA a row */
    S[r][c] = (r < nb && c < nb && c > r) ? U[(size_t) (kb + r) * n + kb + c] * rd[kb + c] : 0.0;
  }

#pragma unroll
  for (int p = 0; p < 8; p++)
    acc[p] = 0.0;

  /* rows 8w .. 8w + 7 of the block, lane = column of block j */
  for (int j = nbk - 1; j > i; j--)
  {
    const int c = j * P_K + lane;
    double u[8];

#pragma unroll
    for (int p = 0; p < 8; p++)
      u[p] = (c < n && 8 * w + p < nb) ? U[(size_t) (kb + 8 * w + p) * n + c] : 0.0;

    const double x = (c < n) ? _pb_get (words + 2 * (size_t) c, info) : 0.0;

#pragma unroll
    for (int p = 0; p < 8; p++)
      acc[p] = fma (u[p], x, acc[p]);
  }

  /* sums over the lanes: halve the values a lane keeps, then plain steps */
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
  {
    const bool up = (lane & (4 * o)) != 0;

#pragma unroll
    for (int p = 0; p < o; p++)
    {
      const double send = up ? acc[p] : acc[p + o], keep = up ? acc[p + o] : acc[p];

      acc[p] = keep + __shfl_xor_sync (0xffffffffu, send, 4 * o);
    }
  }

  acc[0] += __shfl_xor_sync (0xffffffffu, acc[0], 2);
  acc[0] += __shfl_xor_sync (0xffffffffu, acc[0], 1);

  if ((lane & 3) == 0)
  {
    const int r = 8 * w + (lane >> 2);

    sv[r] = (r < nb) ? b[kb + r] - acc[0] : 0.0;
  }

  __syncthreads ();

  if (w == 0)
  {
    double y        = sv[lane];
    const double ri = (lane < nb) ? rd[kb + lane] : 0.0;

    for (int r = nb - 1; r > 0; r--)
    {
      const double x = __shfl_sync (0xffffffffu, y, r);

      if (lane < r)
        y = fma (-S[lane][r], x, y);
    }

    y *= ri;

    if (lane < nb)
    {
      _pb_put (words + 2 * (size_t) (kb + lane), y);
      b[kb + lane] = y;
    }
  }
}

/* ------------------------------------------------------------------- host side */

/* SM count of the current device, and the kernel's shared-memory opt-in there */
static cudaError_t
_syrk64_sms (int *nsm)
{
  static int limit[NCG_MAX_DEVICES];
  int dev = 0;
  cudaError_t e = cudaGetDevice (&dev);

  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute (nsm, cudaDevAttrMultiProcessorCount, dev);

  if (e == cudaSuccess)
    e = ncg_raise_smem_limit ((const void *) _syrk64_kernel, S64_SMEM_BYTES, limit);

  return e;
}

static cudaError_t
_run_syrk64 (const S64Params &p, int nsm, cudaStream_t s)
{
  const int Tn = (p.nn + (p.b != NULL) + P_N - 1) / P_N;
  int tiles    = 0;

  for (int i = 0; i < (p.nn + P_T - 1) / P_T && tiles < nsm; i++)
    tiles += Tn - P_T / P_N * i;

  ncg_pdl_launch (_syrk64_kernel, tiles < nsm ? tiles : nsm, S_THREADS, S64_SMEM_BYTES, s, p);

  return cudaGetLastError ();
}

#define P_ALIGN(x) (((x) + 255) / 256 * 256)

/* work of posv on up to n unknowns: panel digits | column exponents | rd | Lt,
 * root | words | ticket */
typedef struct { size_t ex, rd, lt, words, ticket, total; } posv_work_t;

static posv_work_t
_posv_work (int n)
{
  posv_work_t o;

  o.ex     = P_ALIGN ((size_t) (n / P_T + 2) * P_CHUNK);
  o.rd     = o.ex + P_ALIGN (((size_t) n + 64) * sizeof (int32_t));
  o.lt     = o.rd + P_ALIGN ((size_t) n * sizeof (double));
  o.words  = o.lt + P_ALIGN ((P_K * P_K + P_K) * sizeof (double));
  o.ticket = o.words + P_ALIGN ((size_t) n * 16);
  o.total  = o.ticket + 256;

  return o;
}

extern "C" size_t
ncg_posv_work_bytes (int n)
{
  return _posv_work (n).total;
}

/* A x = b for the upper-stored symmetric A (n x n, overwritten by its factor)
 * and b (overwritten by x); *info = 0, the failing column + 1, or -1 when a
 * bounded device wait gave up */
extern "C" cudaError_t
ncg_launch_posv (double *A, int n, double *b, int32_t *info, void *work, cudaStream_t s)
{
  const posv_work_t o = _posv_work (n);
  uint8_t *pk         = (uint8_t *) work;
  int32_t *ex         = (int32_t *) (pk + o.ex), *ticket = (int32_t *) (pk + o.ticket);
  double *rd          = (double *) (pk + o.rd), *Lt = (double *) (pk + o.lt), *root = Lt + P_K * P_K;
  cudaError_t e;

  int nsm;

  if (n <= 0)
    return cudaSuccess;

  if ((e = _syrk64_sms (&nsm)) != cudaSuccess)
    return e;

  /* words and ticket */
  if ((e = cudaMemsetAsync (pk + o.words, 0, o.total - o.words, s)) != cudaSuccess)
    return e;

  _posv_begin_kernel<<<1, DG_WARPS * 32, 0, s>>> (A, n, Lt, root, rd, info);

  for (int kb = 0; kb < n; kb += P_K)
  {
    const int nb = (n - kb < P_K) ? n - kb : P_K, rest = n - kb - nb;

    ncg_pdl_launch (_posv_panel_kernel, (rest + 1 + PP_C - 1) / PP_C, PP_TH, 0, s, A, n, b, kb, nb, Lt, root, pk, ex, info);

    if ((e = cudaGetLastError ()) != cudaSuccess)
      return e;

    if (rest > 0)
    {
      S64Params p;

      p.pk   = pk;
      p.ex   = ex;
      p.C    = A + (size_t) (kb + nb) * n + kb + nb;
      p.b    = b + kb + nb;
      p.Lt   = Lt;
      p.root = root;
      p.rd   = rd + kb + nb;
      p.col0 = kb + nb;
      p.err  = info;
      p.nn   = rest;
      p.ldc  = n;
      p.nch  = 1;
      p.mode = 1;

      if ((e = _run_syrk64 (p, nsm, s)) != cudaSuccess)
        return e;
    }
  }

  _posv_back_kernel<<<(n + P_K - 1) / P_K, PB_TH, 0, s>>> (A, n, rd, b, (unsigned long long *) (pk + o.words), ticket,
                                                         info);

  return cudaGetLastError ();
}

/* M = A^T A over the upper triangle (A nrows x ncols, row-major), digits in
 * slabs of rows that fit the scratch of `cap` bytes; ex: ncols column exponents;
 * *err = -1 when a bounded device wait gave up (0 before the call) */
extern "C" cudaError_t
ncg_launch_syrk_upper64 (const double *A, int nrows, int ncols, double *M, void *scratch, size_t cap, int32_t *ex,
                         int32_t *err, cudaStream_t s)
{
  const int T_ = (ncols + P_T - 1) / P_T;
  int slab     = (int) (cap / ((size_t) T_ * P_CHUNK) < (size_t) P_SLAB ? cap / ((size_t) T_ * P_CHUNK) : P_SLAB);
  cudaError_t e;
  int nsm;

  if (slab <= 0)
    return cudaErrorInvalidValue;

  if ((e = _syrk64_sms (&nsm)) != cudaSuccess)
    return e;

  /* P_ZERO in every word */
  if ((e = cudaMemsetAsync (ex, 0xc0, sizeof (int32_t) * ncols, s)) != cudaSuccess)
    return e;

  _col_exp_kernel<<<dim3 ((ncols + 127) / 128, (nrows + CE_ROWS - 1) / CE_ROWS), 128, 0, s>>> (A, nrows, ncols, ex);

  for (int r0 = 0; r0 < nrows; r0 += slab * P_K)
  {
    const int r1 = (nrows - r0 > slab * P_K) ? r0 + slab * P_K : nrows, nch = (r1 - r0 + P_K - 1) / P_K;
    S64Params p;

    _pack63_kernel<<<T_ * nch, 256, 0, s>>> (A, r0, r1, ncols, nch, ex, (uint8_t *) scratch);

    p.pk   = (const uint8_t *) scratch;
    p.ex   = ex;
    p.C    = M;
    p.b    = NULL;
    p.Lt   = NULL;
    p.root = NULL;
    p.rd   = NULL;
    p.col0 = 0;
    p.err  = err;
    p.nn   = ncols;
    p.ldc  = ncols;
    p.nch  = nch;
    p.mode = (r0 == 0) ? 0 : 2;

    if ((e = _run_syrk64 (p, nsm, s)) != cudaSuccess)
      return e;
  }

  return cudaGetLastError ();
}
