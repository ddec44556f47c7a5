/*
 * ncg_linalg.cu -- dense kernels behind prepare_interp's NNLS
 * (ncm_nnls_solve, numcosmo/ncm/algebra/ncm_nnls.c:767-871, NORMAL umethod):
 *
 *   syrk_upper_f32  M = A^T A, upper triangle (ncm_matrix_square_to_sym,
 *                   numcosmo/ncm/algebra/ncm_matrix.c:1548-1572) in FP32 for the
 *                   mixed solver's preconditioner (FP64: ncg_posv64.cu)
 *   gemv            y = alpha op(A) x + beta y, deterministic reductions
 *   gather_sub      M[P,P], b[P] for an active set P (ncm_iset_get_submatrix)
 *   potrf_f32       blocked right-looking Cholesky, upper, row-major (the FP64
 *                   solve: ncg_posv64.cu)
 *   residual_norm   res = f - A x and |res|^2 (ncm_nnls.c:700-711)
 *   pcg_*           the FP64 conjugate-gradient refinement of the mixed solver
 *
 * Every reduction has a fixed order, so two runs give identical bits.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "ncg_internal.h"
#include "ncg_pdl.cuh"
#include "ncg_syrk_tc.cuh"

/* FP32 products (the mixed solver's A^T A below 256 columns):
 * 128 x 128 upper tiles, 256 threads of 8 x 8 outputs (rows ty*4 + {0..3} and
 * 64 + ty*4 + {0..3}, columns likewise by tx), contraction rows staged 8 at a
 * time in double-buffered shared memory (the next chunk is loaded into
 * registers while the current one is used).  Each output is still one FMA
 * chain over the rows in ascending order. */
#define SY_T 128
#define SY_KB 8

template <typename TI>
__global__ void __launch_bounds__ (256)
_syrk128_f32_kernel (const TI *__restrict__ A, int lda, int r0, int r1, int off, int nn, float *__restrict__ C,
                     int ldc)
{
  __shared__ __align__ (16) float As[2][SY_KB][SY_T];
  __shared__ __align__ (16) float Bs[2][SY_KB][SY_T];

  const int T_ = (nn + SY_T - 1) / SY_T;
  int b = blockIdx.x, ti = 0;

  while (b >= T_ - ti)
  {
    b -= T_ - ti;
    ti++;
  }

  const int tj  = ti + b;
  const int i0  = off + ti * SY_T, j0 = off + tj * SY_T, end = off + nn;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int lr  = tid >> 5, lc = (tid & 31) * 4;      /* loader: row of the chunk, 4 columns */
  float acc[8][8];
  float ra[4], rb[4];

#pragma unroll
  for (int p = 0; p < 8; p++)
#pragma unroll
    for (int q = 0; q < 8; q++)
      acc[p][q] = 0.0f;

  /* chunk rows [rb0, rb0 + 8): this thread's row lr, columns lc..lc+3 */
#define SY_LOAD(rb0)                                                                          \
  do {                                                                                        \
    const int r_ = (rb0) + lr;                                                                \
    _Pragma ("unroll") for (int q = 0; q < 4; q++)                                            \
    {                                                                                         \
      ra[q] = (r_ < r1 && i0 + lc + q < end) ? (float) A[(size_t) r_ * lda + i0 + lc + q] : 0.0f; \
      rb[q] = (r_ < r1 && j0 + lc + q < end) ? (float) A[(size_t) r_ * lda + j0 + lc + q] : 0.0f; \
    }                                                                                         \
  } while (0)

  int buf = 0;

  SY_LOAD (r0);
  *(float4 *) &As[0][lr][lc] = make_float4 (ra[0], ra[1], ra[2], ra[3]);
  *(float4 *) &Bs[0][lr][lc] = make_float4 (rb[0], rb[1], rb[2], rb[3]);
  __syncthreads ();

  for (int rb0 = r0; rb0 < r1; rb0 += SY_KB)
  {
    const bool more = rb0 + SY_KB < r1;

    if (more)
      SY_LOAD (rb0 + SY_KB);

#pragma unroll
    for (int k = 0; k < SY_KB; k++)
    {
      const float4 a0 = *(const float4 *) &As[buf][k][ty * 4], a1 = *(const float4 *) &As[buf][k][64 + ty * 4];
      const float4 b0 = *(const float4 *) &Bs[buf][k][tx * 4], b1 = *(const float4 *) &Bs[buf][k][64 + tx * 4];
      const float a[8]  = { a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w };
      const float bb[8] = { b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w };

#pragma unroll
      for (int p = 0; p < 8; p++)
#pragma unroll
        for (int q = 0; q < 8; q++)
          acc[p][q] = fmaf (a[p], bb[q], acc[p][q]);
    }

    if (more)
    {
      *(float4 *) &As[buf ^ 1][lr][lc] = make_float4 (ra[0], ra[1], ra[2], ra[3]);
      *(float4 *) &Bs[buf ^ 1][lr][lc] = make_float4 (rb[0], rb[1], rb[2], rb[3]);
    }

    __syncthreads ();
    buf ^= 1;
  }

#undef SY_LOAD

#pragma unroll
  for (int p = 0; p < 8; p++)
  {
    const int i = i0 + ((p < 4) ? ty * 4 + p : 64 + ty * 4 + p - 4);

#pragma unroll
    for (int q = 0; q < 8; q++)
    {
      const int j = j0 + ((q < 4) ? tx * 4 + q : 64 + tx * 4 + q - 4);

      if (i < end && j < end && j >= i)
      {
        C[(size_t) i * ldc + j] = acc[p][q];
      }
    }
  }
}

template <typename TI>
static cudaError_t
_syrk128 (const TI *A, int lda, int r0, int r1, int off, int nn, float *C, int ldc, cudaStream_t s)
{
  if (nn <= 0 || r1 <= r0)
    return cudaSuccess;

  const int T_ = (nn + SY_T - 1) / SY_T;

  _syrk128_f32_kernel<TI><<<T_ * (T_ + 1) / 2, 256, 0, s>>> (A, lda, r0, r1, off, nn, C, ldc);

  return cudaGetLastError ();
}

extern "C" cudaError_t
ncg_launch_syrk_upper_f32 (const double *A, int nrows, int ncols, float *M, cudaStream_t s)
{
  return _syrk128<double> (A, ncols, 0, nrows, 0, ncols, M, ncols, s);
}

/* ---- gemv ---------------------------------------------------------------
 * Bound by the FP64 pipes from n = 2000 or so (n^2 FMAs, 27 us at n = 4096;
 * HBM would take 20), by latency below; the products of the refinement run on the
 * columns P of the active set alone. */

/* y[r] = alpha sum_a A[r][P[a]] x[a] + beta y[r] (P NULL: a itself); one warp per row */
__global__ void __launch_bounds__ (256)
_gemv_n_kernel (const double *__restrict__ A, int nrows, int lda, const int32_t *__restrict__ P, int np, double alpha,
                const double *__restrict__ x, double beta, double *__restrict__ y)
{
  const size_t pdl0 = ncg_pdl_enter ();

  A += pdl0;
  P += pdl0;
  x += pdl0;
  y += pdl0;

  const int lane = threadIdx.x & 31;
  const int r    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;

  if (r >= nrows)
    return;

  const double *row = A + (size_t) r * lda;
  double s          = 0.0;

#pragma unroll 8
  for (int a = lane; a < np; a += 32)
    s = fma (row[P ? P[a] : a], x[a], s);

#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    s += __shfl_xor_sync (0xffffffffu, s, o);

  if (lane == 0)
    y[r] = (beta == 0.0) ? alpha * s : fma (beta, y[r], alpha * s);
}

/* rows of a block of the transposed product: at most 64 blocks, so that their
 * sums are short, and at least 16 rows (256 rows whatever the size left 8 CTAs
 * waiting for memory one row after another at n = 512: 62 us, 6 us now) */
static inline int
_gt_rows (int nrows)
{
  const int r = (nrows + 63) / 64;

  return r < 16 ? 16 : r;
}

/* part[rb][a] = sum over rows of block rb of A[r][P[a]] x[r], or of
 * A[r][P[a]]^2 (x NULL) */
__global__ void __launch_bounds__ (128)
_gemv_t_partial_kernel (const double *__restrict__ A, int nrows, int lda, const int32_t *__restrict__ P, int np,
                        const double *__restrict__ x, int rows, double *__restrict__ part)
{
  const size_t pdl0 = ncg_pdl_enter ();

  A += pdl0;
  P += pdl0;
  x += pdl0;
  part += pdl0;

  const int a  = blockIdx.x * blockDim.x + threadIdx.x;
  const int rb = blockIdx.y;

  if (a >= np)
    return;

  const int r0 = rb * rows, r1 = min (nrows, r0 + rows);
  const double *col = A + (P ? P[a] : a);
  double s          = 0.0;

#pragma unroll 8
  for (int r = r0; r < r1; r++)
  {
    const double v = col[(size_t) r * lda];

    s = fma (v, x ? x[r] : v, s);
  }

  part[(size_t) rb * np + a] = s;
}

/* y[a] = the blocks' sum, or b[a] less it (b not NULL) */
__global__ void __launch_bounds__ (128)
_gemv_t_final_kernel (const double *__restrict__ part, int nrb, int np, const double *__restrict__ b,
                      double *__restrict__ y)
{
  const size_t pdl0 = ncg_pdl_enter ();

  part += pdl0;
  b += pdl0;
  y += pdl0;

  const int a = blockIdx.x * blockDim.x + threadIdx.x;

  if (a >= np)
    return;

  double s = 0.0;

#pragma unroll 8
  for (int rb = 0; rb < nrb; rb++)
    s += part[(size_t) rb * np + a];

  y[a] = b ? b[a] - s : s;
}

extern "C" size_t
ncg_gemv_t_scratch (int nrows, int ncols)
{
  const int rows = _gt_rows (nrows);

  return (size_t) ((nrows + rows - 1) / rows) * (size_t) ncols * sizeof (double);
}

/* y = (A[:, P])^T x, or b less it */
static cudaError_t
_gemv_t (const double *A, int nrows, int lda, const int32_t *P, int np, const double *x, const double *b, double *y,
         double *part, cudaStream_t s)
{
  const int rows = _gt_rows (nrows), nrb = (nrows + rows - 1) / rows;

  ncg_pdl_launch (_gemv_t_partial_kernel, dim3 ((np + 127) / 128, nrb), 128, 0, s, A, nrows, lda, P, np, x, rows, part);
  ncg_pdl_launch (_gemv_t_final_kernel, (np + 127) / 128, 128, 0, s, part, nrb, np, b, y);

  return cudaGetLastError ();
}

static cudaError_t
_gemv_n (const double *A, int nrows, int lda, const int32_t *P, int np, double alpha, const double *x, double beta,
         double *y, cudaStream_t s)
{
  ncg_pdl_launch (_gemv_n_kernel, (unsigned) (((size_t) nrows * 32 + 255) / 256), 256, 0, s, A, nrows, lda, P, np,
                  alpha, x, beta, y);

  return cudaGetLastError ();
}

/* y = A^T x */
extern "C" cudaError_t
ncg_launch_gemv_t (const double *A, int nrows, int ncols, const double *x, double *y, double *part, cudaStream_t s)
{
  return _gemv_t (A, nrows, ncols, NULL, ncols, x, NULL, y, part, s);
}

/* diagM[c] = sum_r A[r][c]^2, the FP64 diagonal of A^T A */
extern "C" cudaError_t
ncg_launch_colsumsq (const double *A, int nrows, int ncols, double *out, double *part, cudaStream_t s)
{
  return _gemv_t (A, nrows, ncols, NULL, ncols, NULL, NULL, out, part, s);
}

/* ---- active-set gather / scatter ----------------------------------------- */

__global__ void
_gather_kernel (const double *__restrict__ M, int n, const int32_t *__restrict__ P, int np,
                double *__restrict__ Msub, const double *__restrict__ b, double *__restrict__ bsub)
{
  const int a = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;

  if (a >= np)
    return;

  const size_t ra = (size_t) P[a] * n;

  for (int bb = c; bb < np; bb += gridDim.x * blockDim.x)
    Msub[(size_t) a * np + bb] = (bb >= a) ? M[ra + P[bb]] : 0.0;

  if (c == 0)
    bsub[a] = b[P[a]];
}

extern "C" cudaError_t
ncg_launch_gather_sub (const double *M, int n, const int32_t *P, int np, double *Msub, const double *b,
                       double *bsub, cudaStream_t s)
{
  if (np <= 0)
    return cudaSuccess;

  dim3 g ((np + 255) / 256 < 8 ? (np + 255) / 256 : 8, np);

  _gather_kernel<<<g, 256, 0, s>>> (M, n, P, np, Msub, b, bsub);

  return cudaGetLastError ();
}

/* The mixed solver's preconditioner operand, in two launches: Dsub[a] =
 * 1/sqrt(diagM[P_a]) (Jacobi scaling, FP64) and bsub[a] = b[P_a]; then
 * Msub[a][b] = D_a M32[P_a][P_b] D_b in FP32, upper triangle only, with the
 * unit diagonal raised by `shift`; its leading 64 x 64 block in dg as well, where
 * the factorisation reads it. */
__global__ void
_scale_vec_kernel (const int32_t *__restrict__ P, int np, const double *__restrict__ diagM,
                   double *__restrict__ Dsub, const double *__restrict__ b, double *__restrict__ bsub)
{
  const size_t pdl0 = ncg_pdl_enter ();

  P += pdl0;
  diagM += pdl0;
  b += pdl0;
  Dsub += pdl0;
  bsub += pdl0;

  const int a = blockIdx.x * blockDim.x + threadIdx.x;

  if (a < np)
  {
    const int pa = P[a];

    Dsub[a] = 1.0 / sqrt (diagM[pa]);
    bsub[a] = b[pa];
  }
}

__global__ void
_gather_scaled_kernel (const float *__restrict__ M32, int n, const int32_t *__restrict__ P, int np,
                       const double *__restrict__ Dsub, float shift, float *__restrict__ Msub,
                       float *__restrict__ dg)
{
  const size_t pdl0 = ncg_pdl_enter ();

  M32 += pdl0;
  P += pdl0;
  Dsub += pdl0;
  Msub += pdl0;
  dg += pdl0;

  const int a = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;

  if (a >= np)
    return;

  const float *row = M32 + (size_t) P[a] * n;
  const float Da   = (float) Dsub[a];

  for (int bb = c; bb < np; bb += gridDim.x * blockDim.x)
  {
    float v = 0.0f;

    if (bb > a)
      v = (Da * row[P[bb]]) * (float) Dsub[bb];
    else if (bb == a)
      v = (Da * row[P[bb]]) * Da * (1.0f + shift);

    Msub[(size_t) a * np + bb] = v;

    if (a < 64 && bb < 64)
      dg[a * 64 + bb] = v;
  }
}

extern "C" cudaError_t
ncg_launch_gather_scaled_f32 (const float *M32, int n, const int32_t *P, int np, const double *diagM, double shift,
                              float *Msub, float *dg, double *Dsub, const double *b, double *bsub, cudaStream_t s)
{
  if (np <= 0)
    return cudaSuccess;

  dim3 g ((np + 255) / 256 < 8 ? (np + 255) / 256 : 8, np);

  ncg_pdl_launch (_scale_vec_kernel, (np + 255) / 256, 256, 0, s, P, np, diagM, Dsub, b, bsub);
  ncg_pdl_launch (_gather_scaled_kernel, g, 256, 0, s, M32, n, P, np, Dsub, (float) shift, Msub, dg);

  return cudaGetLastError ();
}

__global__ void
_scatter_kernel (const double *__restrict__ xsub, const int32_t *__restrict__ P, int np, int n, double *__restrict__ x)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;

  if (i < n)
    x[i] = 0.0;
}

__global__ void
_scatter2_kernel (const double *__restrict__ xsub, const int32_t *__restrict__ P, int np, double *__restrict__ x)
{
  const int a = blockIdx.x * blockDim.x + threadIdx.x;

  if (a < np)
    x[P[a]] = xsub[a];
}

extern "C" cudaError_t
ncg_launch_scatter_x (const double *xsub, const int32_t *P, int np, int n, double *x, cudaStream_t s)
{
  _scatter_kernel<<<(n + 255) / 256, 256, 0, s>>> (xsub, P, np, n, x);

  if (np > 0)
    _scatter2_kernel<<<(np + 255) / 256, 256, 0, s>>> (xsub, P, np, x);

  return cudaGetLastError ();
}

/* ---- blocked Cholesky ------------------------------------------------------ */

#define PB 64

/* S[r][c] = A[(r0 + r) ld + c0 + c] for r, c < nb (zero elsewhere), B x B
 * block, NT threads; the loads go out in batches of up to 32 per thread so
 * that they overlap instead of waiting for one another */
template <typename T, int NT, int B>
__device__ __forceinline__ void
_stage_block (T (*S)[B + 1], const T *__restrict__ A, int ld, int r0, int c0, int nb, int tid)
{
  constexpr int PER = (B * B + NT - 1) / NT;
  constexpr int CH  = (PER < 32) ? PER : 32;

#pragma unroll
  for (int k0 = 0; k0 < PER; k0 += CH)
  {
    T v[CH];

#pragma unroll
    for (int k = 0; k < CH; k++)
    {
      const int e = tid + (k0 + k) * NT;
      const int r = e / B, c = e % B;

      v[k] = (e < B * B && r < nb && c < nb) ? A[(size_t) (r0 + r) * ld + c0 + c] : (T) 0;
    }

#pragma unroll
    for (int k = 0; k < CH; k++)
    {
      const int e = tid + (k0 + k) * NT;

      if (e < B * B)
        S[e / B][e % B] = v[k];
    }
  }
}

/* ---- the FP32 preconditioner's panels ---- */

/* One panel: the diagonal block (raw in dg, 64 x 64) and 64 of the columns to
 * its right per CTA, eliminated in the same steps.  Both live in registers,
 * 4 x 4 elements each per thread (element (ty + 16p, tx + 16q)); a step
 * publishes two raw rows j, j + 1 of both through shared memory, one barrier, and
 * every thread works out row j + 1 as row j leaves it where it needs it, then takes
 * s_jr s_jc / a_jj of both rows off its elements; the square roots and the rows'
 * scaling wait for the end, where all rows take them at once.  CTA 0 writes the
 * factored block.  It is bound by the chain of 32 steps (a barrier, two
 * shared-memory trips and two reciprocals each), which every CTA walks for itself:
 * as two launches, the factor and then the columns against it, a panel took
 * 10 + 11 us (24 + 27 with the row scaled on the chain and a pack through FP64),
 * row by row in one 14.7 us; 10.8 us so (mean over the panels at n = 3000).  pk
 * (may be NULL): the panel as the tensor-core update's operand. */
/* 1 / x of a pivot, the hardware's value (1 ulp) with one correction by its residual: within
 * 2^-24 (1 + 2^-20), as good as a correctly rounded one at two instructions on the chain */
__device__ __forceinline__ float
_rcp_pivot (float x)
{
  float r;

  asm ("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));

  return fmaf (r, fmaf (-x, r, 1.0f), r);
}

__global__ void __launch_bounds__ (256)
_potrf_panel_f32_kernel (float *A, int ld, int kb, int nb, int n, const float *__restrict__ dg, int32_t *info,
                         float *pk)
{
  const size_t pdl0 = ncg_pdl_enter ();

  dg += pdl0;

  __shared__ float row[2][2][2 * PB];
  __shared__ float X[PB][PB + 1];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int c0  = kb + nb + blockIdx.x * PB;
  float s[4][4], a[4][4], piv[4];
  int fail = 0;

  /* agreed on by the CTA: CTA 0 may be writing it */
  if (__syncthreads_or (*(volatile int32_t *) info))
    return;

  /* the identity past nb */
#pragma unroll
  for (int p = 0; p < 4; p++)
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      const int r = ty + 16 * p, c = tx + 16 * q;

      s[p][q] = (r < nb && c < nb) ? ((c >= r) ? dg[r * PB + c] : 0.0f) : (r == c ? 1.0f : 0.0f);
      a[p][q] = (r < nb && c0 + c < n) ? A[(size_t) (kb + r) * ld + c0 + c] : 0.0f;
      piv[p]  = 1.0f;
    }

#pragma unroll
  for (int p = 0; p < 4; p++)
    for (int jj = 0; jj < 16; jj += 2)
    {
      const int j = 16 * p + jj;
      float *r0 = row[(jj >> 1) & 1][0], *r1 = row[(jj >> 1) & 1][1];

      if (fail)
        break;

      if ((ty & ~1) == jj)
      {
        float *rb = (ty & 1) ? r1 : r0;

#pragma unroll
        for (int q = 0; q < 4; q++)
        {
          if (q >= p)
            rb[tx + 16 * q] = s[p][q];

          rb[PB + tx + 16 * q] = a[p][q];
        }
      }

      __syncthreads ();

      const float a0 = r0[j], b0 = r0[j + 1], i0 = -_rcp_pivot (a0), l = b0 * i0, a1 = fmaf (l, b0, r1[j + 1]);

      if (!(a0 > 0.0f) || !(a1 > 0.0f))
      {
        fail = (a0 > 0.0f) ? j + 2 : j + 1;
        break;
      }

      const float i1 = -_rcp_pivot (a1);
      float c0v[4], c1v[4], d0v[4], d1v[4];

      if ((ty & ~1) == jj)
        piv[p] = (ty & 1) ? a1 : a0;

#pragma unroll
      for (int q = 0; q < 4; q++)
      {
        c0v[q] = (q >= p) ? r0[tx + 16 * q] : 0.0f;
        c1v[q] = (q >= p) ? fmaf (l, c0v[q], r1[tx + 16 * q]) : 0.0f;
        d0v[q] = r0[PB + tx + 16 * q];
        d1v[q] = fmaf (l, d0v[q], r1[PB + tx + 16 * q]);
      }

#pragma unroll
      for (int pp = p; pp < 4; pp++)
      {
        const int r    = ty + 16 * pp;
        const float v0 = r0[r], v1 = fmaf (l, v0, r1[r]);
        const float t0 = (r > j) ? v0 * i0 : 0.0f, t1 = (r > j + 1) ? v1 * i1 : 0.0f;

#pragma unroll
        for (int q = pp; q < 4; q++)
          s[pp][q] = fmaf (t1, c1v[q], fmaf (t0, c0v[q], s[pp][q]));

#pragma unroll
        for (int q = 0; q < 4; q++)
          a[pp][q] = fmaf (t1, d1v[q], fmaf (t0, d0v[q], a[pp][q]));
      }
    }

  if (fail)
  {
    /* every CTA finds the same step */
    if (tid == 0 && blockIdx.x == 0)
      atomicCAS (info, 0, kb + fail);

    return;
  }

#pragma unroll
  for (int p = 0; p < 4; p++)
  {
    const int r   = ty + 16 * p;
    const float u = __fsqrt_rn (piv[p]), ri = __frcp_rn (u);

#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      const int c = tx + 16 * q;

      a[p][q] *= ri;
      X[r][c]  = a[p][q];

      if (r < nb && c0 + c < n)
        A[(size_t) (kb + r) * ld + c0 + c] = a[p][q];

      if (blockIdx.x == 0 && r < nb && c < nb && c >= r)
        A[(size_t) (kb + r) * ld + kb + c] = (c == r) ? u : s[p][q] * ri;
    }
  }

  if (pk == NULL)
    return;

  __syncthreads ();

  /* units of four rows of a column */
  float *blk = pk + (size_t) (blockIdx.x / 2) * 2 * (SK_BLOCK / 4);

  for (int e = tid; e < PB * 16; e += 256)
  {
    const int c = e & 63, k = (e >> 6) * 4;

    _put_split4f (blk + (size_t) (k / SK_KC) * (SK_BLOCK / 4), (blockIdx.x & 1) * PB + c, k % SK_KC, X[k][c], X[k + 1][c],
                  X[k + 2][c], X[k + 3][c]);
  }
}

/* C -= P^T P on the upper tiles of the nn x nn trailing block for a panel of
 * nb <= 64 rows: 64 x 64 tiles, the whole panel slice of both sides staged at
 * once, 4 x 4 outputs per thread, C loaded while the panel arrives.  One FMA
 * chain per output over the rows in ascending order.  The leading tile also
 * goes to dg, the next panel's raw diagonal block.  11 us on average below
 * 2560 columns, where the general tile kernel (16 rows a stage) took 18 and the
 * tensor-core update 13: there its set-up and the traffic of C decide, not the
 * products. */
__global__ void __launch_bounds__ (256)
_potrf_update_f32_kernel (float *A, int ld, int kb, int nb, int off, int nn, float *__restrict__ dg,
                          const int32_t *info)
{
  const size_t pdl0 = ncg_pdl_wait ();

  dg += pdl0;

  __shared__ __align__ (16) float As[PB][PB];
  __shared__ __align__ (16) float Bs[PB][PB];
  const int T_ = (nn + PB - 1) / PB;
  int b = blockIdx.x, ti = 0;

  if (*info)
    return;

  while (b >= T_ - ti)
  {
    b -= T_ - ti;
    ti++;
  }

  const int tj  = ti + b, i0 = off + ti * PB, j0 = off + tj * PB, end = off + nn;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int lc  = tid & 63, lr = tid >> 6;
  float va[16], vb[16], acc[4][4];

#pragma unroll
  for (int q = 0; q < 16; q++)
  {
    const int r = lr + 4 * q;

    va[q] = (r < nb && i0 + lc < end) ? A[(size_t) (kb + r) * ld + i0 + lc] : 0.0f;
    vb[q] = (r < nb && j0 + lc < end) ? A[(size_t) (kb + r) * ld + j0 + lc] : 0.0f;
  }

#pragma unroll
  for (int p = 0; p < 4; p++)
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      const int i = i0 + ty * 4 + p, j = j0 + tx * 4 + q;

      acc[p][q] = (i < end && j < end && j >= i) ? A[(size_t) i * ld + j] : 0.0f;
    }

#pragma unroll
  for (int q = 0; q < 16; q++)
  {
    As[lr + 4 * q][lc] = -va[q];
    Bs[lr + 4 * q][lc] = vb[q];
  }

  __syncthreads ();

#pragma unroll 16
  for (int k = 0; k < PB; k++)
  {
    const float4 x = *(const float4 *) &As[k][ty * 4], y = *(const float4 *) &Bs[k][tx * 4];
    const float xv[4] = { x.x, x.y, x.z, x.w }, yv[4] = { y.x, y.y, y.z, y.w };

#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
      for (int q = 0; q < 4; q++)
        acc[p][q] = fmaf (xv[p], yv[q], acc[p][q]);
  }

  ncg_pdl_next ();

#pragma unroll
  for (int p = 0; p < 4; p++)
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      const int i = i0 + ty * 4 + p, j = j0 + tx * 4 + q;

      if (i < end && j < end && j >= i)
        A[(size_t) i * ld + j] = acc[p][q];

      if (blockIdx.x == 0)
        dg[(ty * 4 + p) * PB + tx * 4 + q] = acc[p][q];
    }
}

__global__ void
_zero_int_kernel (int32_t *p)
{
  *p = 0;
}

/* trailing blocks at least this wide take the tensor-core update */
#define POTRF_TC_MIN 2560

/* work of potrf_f32 on n columns: the panel's tensor-core operand, then the raw
 * diagonal block */
extern "C" size_t
ncg_potrf_f32_work_bytes (int n)
{
  return ncg_syrk_tc_pack_bytes (n, PB) + sizeof (float) * PB * PB;
}

extern "C" float *
ncg_potrf_f32_dg (float *work, int n)
{
  return work + ncg_syrk_tc_pack_bytes (n, PB) / sizeof (float);
}

/* upper Cholesky of A (n x n, in place); work's diagonal block holds the leading
 * 64 x 64 of A already (ncg_launch_gather_scaled_f32 leaves it there) */
extern "C" cudaError_t
ncg_launch_potrf_f32 (float *A, int n, int32_t *info, float *work, int cap, cudaStream_t s)
{
  float *dg = ncg_potrf_f32_dg (work, cap);

  _zero_int_kernel<<<1, 1, 0, s>>> (info);

  for (int kb = 0; kb < n; kb += PB)
  {
    const int nb  = (n - kb < PB) ? n - kb : PB, rest = n - kb - nb;
    const bool tc = rest >= POTRF_TC_MIN;

    ncg_pdl_launch (_potrf_panel_f32_kernel, rest > 0 ? (rest + PB - 1) / PB : 1, 256, 0, s, A, n, kb, nb, n, dg, info,
                    tc ? work : NULL);

    if (tc)
    {
      const cudaError_t e = ncg_launch_syrk_tc (work, nb, rest, A + (size_t) (kb + nb) * n + kb + nb, n, 1, dg, info, s);

      if (e != cudaSuccess)
        return e;
    }
    else if (rest > 0)
    {
      const int T_ = (rest + PB - 1) / PB;

      ncg_pdl_launch (_potrf_update_f32_kernel, T_ * (T_ + 1) / 2, 256, 0, s, A, n, kb, nb, kb + nb, rest, dg, info);
    }
  }

  return cudaGetLastError ();
}

/* ---- residuals --------------------------------------------------------- */

__global__ void
_sumsq_kernel (const double *__restrict__ v, int n, double *__restrict__ out)
{
  __shared__ double red[1024];
  double s = 0.0;

  for (int i = threadIdx.x; i < n; i += blockDim.x)
    s = fma (v[i], v[i], s);

  red[threadIdx.x] = s;
  __syncthreads ();

  for (int st = blockDim.x / 2; st > 0; st >>= 1)
  {
    if (threadIdx.x < st)
      red[threadIdx.x] += red[threadIdx.x + st];

    __syncthreads ();
  }

  if (threadIdx.x == 0)
    *out = red[0];
}

extern "C" cudaError_t
ncg_launch_residual_norm (const double *A, int nrows, int ncols, const double *x, const double *f, double *res,
                          double *rnorm2, cudaStream_t s)
{
  cudaError_t e = cudaMemcpyAsync (res, f, sizeof (double) * nrows, cudaMemcpyDeviceToDevice, s);

  if (e != cudaSuccess)
    return e;

  e = _gemv_n (A, nrows, ncols, NULL, ncols, -1.0, x, 1.0, res, s);

  if (e != cudaSuccess)
    return e;

  _sumsq_kernel<<<1, 1024, 0, s>>> (res, nrows, rnorm2);

  return cudaGetLastError ();
}

/* ---- weight normalisation (ncm_stats_dist.c:1086-1093) ------------------- */

/* one CTA; the total as a tree (one thread's chain of n additions took 243 us at
 * n = 4096) */
__global__ void __launch_bounds__ (1024)
_normalize_weights_kernel (double *w, int n, double shrink, int32_t *bad)
{
  __shared__ double red[32];
  const int tid = threadIdx.x, lane = tid & 31;
  double t      = 0.0;

  for (int i = tid; i < n; i += 1024)
    t += w[i];

#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    t += __shfl_xor_sync (0xffffffffu, t, o);

  if (lane == 0)
    red[tid >> 5] = t;

  __syncthreads ();
  t = red[lane];

#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    t += __shfl_xor_sync (0xffffffffu, t, o);

  const double sc = (1.0 - shrink) / t, ad = shrink / n;

  if (tid == 0)
    *bad = !(t > 0.0);

  for (int i = tid; i < n; i += 1024)
    w[i] = __dadd_rn (__dmul_rn (w[i], sc), ad);
}

extern "C" cudaError_t
ncg_launch_normalize_weights (double *w, int n, double shrink, int32_t *bad, cudaStream_t s)
{
  _normalize_weights_kernel<<<1, 1024, 0, s>>> (w, n, shrink, bad);

  return cudaGetLastError ();
}

/* ---- mixed solver: FP32 preconditioned FP64 conjugate gradients ----------
 *
 * Solves the active-set normal equations A_P^T A_P x = A_P^T 1 with the
 * products taken from A in FP64 (so the residual is an FP64 residual of the
 * reference's own system) and the preconditioner D R^{-1} R^{-T} D from the
 * FP32 Cholesky factor R of the Jacobi-scaled D (A^T A)_P D.  The conjugate
 * direction uses the flexible (Polak-Ribiere) beta, which stays robust when
 * the FP32 preconditioner is not exactly linear.  The scalars live on the
 * device (sc[]), so an iteration needs no host round trip; the host reads
 * sc[PCG_RR] to decide when to stop.
 */

#define DOT_TH 256
#define DOT_CTAS 64

/* K sums over all threads of the grid (part: 3 DOT_CTAS, count: zero): the CTAs
 * leave partial sums and the last one to finish (a counter, cleared again) adds
 * them up in CTA order.  True in one thread of the grid, which then has them in s */
template <int K>
__device__ bool
_dots_sum (double (&s)[3], double *part, int32_t *count)
{
  __shared__ double red[3][DOT_TH / 32];
  __shared__ int last;
  const int tid = threadIdx.x, lane = tid & 31;

#pragma unroll
  for (int k = 0; k < K; k++)
  {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      s[k] += __shfl_xor_sync (0xffffffffu, s[k], o);

    if (lane == 0)
      red[k][tid >> 5] = s[k];
  }

  __syncthreads ();

  if (tid < K)
  {
    double t = red[tid][0];

    for (int k = 1; k < DOT_TH / 32; k++)
      t += red[tid][k];

    part[tid * DOT_CTAS + blockIdx.x] = t;
    __threadfence ();
  }

  __syncthreads ();

  if (tid == 0)
    last = atomicAdd (count, 1) == (int) gridDim.x - 1;

  __syncthreads ();

  if (!last || tid >= 32)
    return false;

  __threadfence ();

  double t = 0.0;

  if (tid < K)
    for (int k = 0; k < (int) gridDim.x; k++)
      t += __ldcg (part + tid * DOT_CTAS + k);

#pragma unroll
  for (int k = 0; k < K; k++)
    s[k] = __shfl_sync (0xffffffffu, t, k);

  if (tid == 0)
    *count = 0;

  return tid == 0;
}

/* The scalars of one point of the iteration, as many dot products as it needs
 * in one launch (one CTA of 1024 threads per product took 8 to 10 us each).
 *  MODE 0 (start): RZ = <r, z>, BB = |D b|^2, RR = |D r|^2, and p = z
 *  MODE 1: PQ = <p, q>
 *  MODE 2: RZ' = <r, z>, <z, r_prev>; BE = (RZ' - <z, r_prev>) / RZ
 *          (Polak-Ribiere), then RZ = RZ'
 *  MODE 3: RR = |D r|^2 */
template <int MODE>
__global__ void __launch_bounds__ (DOT_TH)
_pcg_dots_kernel (const double *__restrict__ u, const double *__restrict__ v, const double *__restrict__ w,
                  const double *__restrict__ D, double *__restrict__ p, int n, double *__restrict__ sc,
                  double *__restrict__ part, int32_t *__restrict__ count)
{
  const size_t pdl0 = ncg_pdl_enter ();

  u += pdl0;
  v += pdl0;
  w += pdl0;
  D += pdl0;
  p += pdl0;
  sc += pdl0;
  part += pdl0;
  count += pdl0;

  double s[3] = { 0.0, 0.0, 0.0 };

  for (int i = blockIdx.x * DOT_TH + threadIdx.x; i < n; i += gridDim.x * DOT_TH)
  {
    const double ui = u[i];

    if (MODE == 3)
    {
      const double di = D[i] * ui;

      s[0] = fma (di, di, s[0]);
      continue;
    }

    const double vi = v[i];

    s[0] = fma (ui, vi, s[0]);

    if (MODE == 0)
    {
      const double di = D[i] * ui, b = D[i] * w[i];

      s[1] = fma (b, b, s[1]);
      s[2] = fma (di, di, s[2]);
      p[i] = vi;
    }
    else if (MODE == 2)
      s[1] = fma (vi, w[i], s[1]);
  }

  if (!_dots_sum<(MODE == 0) ? 3 : (MODE == 2) ? 2 : 1> (s, part, count))
    return;

  if (MODE == 0)
  {
    sc[NCG_PCG_RZ] = s[0];
    sc[NCG_PCG_BB] = s[1];
    sc[NCG_PCG_RR] = s[2];
  }
  else if (MODE == 1)
    sc[NCG_PCG_PQ] = s[0];
  else if (MODE == 2)
  {
    sc[NCG_PCG_BE] = (s[0] - s[1]) / sc[NCG_PCG_RZ];
    sc[NCG_PCG_RZ] = s[0];
  }
  else
    sc[NCG_PCG_RR] = s[0];
}

/* x += alpha p, r_prev = r, r -= alpha q with alpha = sc[RZ] / sc[PQ], and RR =
 * |D r|^2 of the new r, so that the host can stop before the next
 * preconditioning (two triangular solves, 160 us at n = 3000, per solve).  A
 * direction with RZ not above zero is not taken: the host stops at RZ */
__global__ void __launch_bounds__ (DOT_TH)
_pcg_step_kernel (double *__restrict__ x, double *__restrict__ r, double *__restrict__ rprev,
                  const double *__restrict__ p, const double *__restrict__ q, const double *__restrict__ D, int n,
                  double *__restrict__ sc, double *__restrict__ part, int32_t *__restrict__ count)
{
  const size_t pdl0 = ncg_pdl_enter ();

  p += pdl0;
  q += pdl0;
  D += pdl0;
  x += pdl0;
  r += pdl0;
  rprev += pdl0;
  sc += pdl0;
  part += pdl0;
  count += pdl0;

  const double rz = sc[NCG_PCG_RZ], al = (rz > 0.0) ? rz / sc[NCG_PCG_PQ] : 0.0;
  double s[3] = { 0.0, 0.0, 0.0 };

  for (int i = blockIdx.x * DOT_TH + threadIdx.x; i < n; i += gridDim.x * DOT_TH)
  {
    const double ri = r[i], rn = fma (-al, q[i], ri), di = D[i] * rn;

    x[i]     = fma (al, p[i], x[i]);
    rprev[i] = ri;
    r[i]     = rn;
    s[0]     = fma (di, di, s[0]);
  }

  if (_dots_sum<1> (s, part, count))
    sc[NCG_PCG_RR] = s[0];
}

/* p = z + BE p */
__global__ void
_pcg_dir_kernel (double *__restrict__ p, const double *__restrict__ z, int n, const double *sc)
{
  const size_t pdl0 = ncg_pdl_enter ();

  z += pdl0;
  p += pdl0;

  const int i = blockIdx.x * blockDim.x + threadIdx.x;

  if (i < n)
    p[i] = fma (sc[NCG_PCG_BE], p[i], z[i]);
}

/* q = A_P^T (A_P v) for a compact v on the set P (np entries), or b less it; A
 * nrows x n; yf: nrows-long work, part the transposed product's scratch */
extern "C" cudaError_t
ncg_launch_pcg_matvec (const double *A, int nrows, int n, const int32_t *P, int np, const double *v, const double *b,
                       double *yf, double *part, double *q, cudaStream_t s)
{
  const cudaError_t e = _gemv_n (A, nrows, n, P, np, 1.0, v, 0.0, yf, s);

  return (e == cudaSuccess) ? _gemv_t (A, nrows, n, P, np, yf, b, q, part, s) : e;
}

/* ---- chained triangular solves of the FP32 preconditioner ----------------
 *
 * z = D (R^T R)^{-1} D r, one launch per triangular solve instead of one per
 * block of SB rows.  Each CTA takes the next block from a ticket counter, so every
 * block it waits for belongs to a CTA that is already running and the launch
 * cannot deadlock whatever the residency.  While the blocks before its own
 * finish, a CTA streams its off-diagonal SB x SB tiles of R (the loads do not
 * depend on the waits), then applies the inverse of its diagonal block
 * (ncg_launch_trinv_diag_f32, once per factorisation).  A block publishes
 * each of its values as one 64-bit word (value, epoch): a single-copy
 * atomic store that carries its own validity, so a reader polls the value
 * itself (one memory round trip, no flag and no fence).  The epoch is unique
 * to the launch (the host counts launches; the words are zeroed when the
 * buffer is set up, and epochs start at 1).  Every block's arithmetic runs in
 * a fixed order, so results do not depend on timing.
 *
 * sync: [0] ticket, [1] finished CTAs, [2] timeout seen; zero between
 * launches (the last CTA to finish clears them).  A wait gives up after
 * CS_SPIN polls, sets *err = 1 and sync[2], and the launch goes on with what
 * it has, so it always ends; a later wait that sees sync[2] does not spin. */
/* The block of the solves.  A step is a memory round trip and two small products
 * whatever the block: with 64 rows, 71 and 87 us at n = 3000 (17 and 18 at 512),
 * with 128 and the half rows of the inverse in registers 40 and 44 us (10 and
 * 10); the inverses then take 16 instead of 9 us, once per factorisation. */
#define SB 128
#define CS_TH 256
#define CS_SPIN (1 << 21)

__device__ __forceinline__ unsigned long long
_ld_relaxed64 (const unsigned long long *p)
{
  unsigned long long v;

  asm volatile ("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");

  return v;
}

__device__ __forceinline__ int
_ld_relaxed32 (const int32_t *p)
{
  int v;

  asm volatile ("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");

  return v;
}

/* publish value v of this launch */
__device__ __forceinline__ void
_cs_put (unsigned long long *w, float v, uint32_t epoch)
{
  const unsigned long long x = ((unsigned long long) epoch << 32) | __float_as_uint (v);

  asm volatile ("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(w), "l"(x) : "memory");
}

/* the value of word w once this launch has published it */
__device__ __forceinline__ float
_cs_get (const unsigned long long *w, uint32_t epoch, int32_t *sync, double *err)
{
  unsigned long long x = _ld_relaxed64 (w);
  int k = 0;

  while ((uint32_t) (x >> 32) != epoch)
  {
    if (++k > CS_SPIN || ((k & 255) == 0 && _ld_relaxed32 (sync + 2) != 0))
    {
      atomicExch (sync + 2, 1);
      *err = 1.0;
      break;
    }

    x = _ld_relaxed64 (w);
  }

  return __uint_as_float ((uint32_t) x);
}

/* the values of words w[0], w[32], w[64] and w[96] below w[n], polled together: one
 * after the other each costs a memory round trip */
__device__ __forceinline__ void
_cs_get4 (const unsigned long long *w, int n, float (&v)[4], uint32_t epoch, int32_t *sync, double *err)
{
  unsigned long long x[4];
  int k = 0;

  for (;;)
  {
    bool all = true;

#pragma unroll
    for (int q = 0; q < 4; q++)
      x[q] = (32 * q < n) ? _ld_relaxed64 (w + 32 * q) : (unsigned long long) epoch << 32;

#pragma unroll
    for (int q = 0; q < 4; q++)
      all = all && (uint32_t) (x[q] >> 32) == epoch;

    if (all)
      break;

    if (++k > CS_SPIN || ((k & 255) == 0 && _ld_relaxed32 (sync + 2) != 0))
    {
      atomicExch (sync + 2, 1);
      *err = 1.0;
      break;
    }
  }

#pragma unroll
  for (int q = 0; q < 4; q++)
    v[q] = __uint_as_float ((uint32_t) x[q]);
}

/* count the CTA as finished; the last one clears the ticket and the counters */
__device__ __forceinline__ void
_cs_finish (int32_t *sync, int tid)
{
  __syncthreads ();

  if (tid == 0 && atomicAdd (sync + 1, 1) == (int) gridDim.x - 1)
  {
    sync[0] = 0;
    sync[1] = 0;
    sync[2] = 0;
  }
}

/* V_i = (U_ii^T)^{-1}, lower triangular, for each SB x SB diagonal block of the
 * upper factor U (zero outside the nb x nb triangle of a partial last block).
 * With U_ii = [U11 U12; 0 U22]: V11 and V22 by substitution, thread c column c
 * in registers as the panel solve does it (36 us with the column in shared
 * memory and a division per row), then V21 = -V22 (U12^T V11), two 64 x 64
 * products of 4 x 4 outputs a thread. */
#define TI 64

__global__ void __launch_bounds__ (256)
_trinv_diag_kernel (const float *__restrict__ U, int n, float *__restrict__ V)
{
  const size_t pdl0 = ncg_pdl_enter ();

  U += pdl0;
  V += pdl0;

  __shared__ __align__ (16) float S[2][TI][TI];   /* U11, U22, then V11, V22^T */
  __shared__ __align__ (16) float T[TI][TI];      /* 1 / diagonal, then U12, then U12^T V11 */
  const int i = blockIdx.x, kb = i * SB, nb = (n - kb < SB) ? n - kb : SB, tid = threadIdx.x;
  float *Vi   = V + (size_t) i * SB * SB;

#pragma unroll 16
  for (int e = tid; e < 2 * TI * TI; e += 256)
  {
    const int h = e / (TI * TI), r = (e / TI) % TI, c = e % TI;

    S[h][r][c] = (h * TI + c < nb && c >= r) ? U[(size_t) (kb + h * TI + r) * n + kb + h * TI + c] : 0.0f;
  }

  __syncthreads ();

  if (tid < SB)
    T[0][tid] = (tid < nb) ? __frcp_rn (S[tid / TI][tid % TI][tid % TI]) : 0.0f;

  __syncthreads ();

  const int h = (tid / TI) & 1, c = tid % TI;
  float x[TI];

  if (tid < SB)
  {
#pragma unroll
    for (int r = 0; r < TI; r++)
      x[r] = (r == c) ? 1.0f : 0.0f;

#pragma unroll
    for (int r = 0; r < TI; r++)
    {
      x[r] *= T[0][h * TI + r];

      const float t = -x[r];

#pragma unroll
      for (int m = (r + 1) / 4 * 4; m < TI; m += 4)
      {
        const float4 v = *(const float4 *) &S[h][r][m];

        if (m + 0 > r)
          x[m + 0] = fmaf (v.x, t, x[m + 0]);
        if (m + 1 > r)
          x[m + 1] = fmaf (v.y, t, x[m + 1]);
        if (m + 2 > r)
          x[m + 2] = fmaf (v.z, t, x[m + 2]);
        if (m + 3 > r)
          x[m + 3] = fmaf (v.w, t, x[m + 3]);
      }
    }
  }

  __syncthreads ();

  if (tid < SB)
  {
#pragma unroll
    for (int r = 0; r < TI; r++)
    {
      Vi[(size_t) (h * TI + r) * SB + h * TI + c] = x[r];

      if (h == 0)
        S[0][r][c] = x[r];
    }

    /* V22 by columns, for the product's reads along a row */
    if (h == 1)
#pragma unroll
      for (int r = 0; r < TI; r += 4)
        *(float4 *) &S[1][c][r] = make_float4 (x[r], x[r + 1], x[r + 2], x[r + 3]);
  }

#pragma unroll
  for (int e = tid; e < TI * TI; e += 256)
  {
    const int r = e / TI, cc = e % TI;

    T[r][cc]                            = (TI + cc < nb) ? U[(size_t) (kb + r) * n + kb + TI + cc] : 0.0f;
    Vi[(size_t) r * SB + TI + cc]       = 0.0f;
  }

  __syncthreads ();

  /* rows 4 ty.., columns 4 tx..: first T = U12^T V11, then V21 = -V22 T */
  const int tx = tid & 15, ty = tid >> 4;
  float acc[4][4];

  for (int pass = 0; pass < 2; pass++)
  {
    const float (*L)[TI] = pass ? S[1] : T, (*R)[TI] = pass ? T : S[0];

#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
      for (int q = 0; q < 4; q++)
        acc[p][q] = 0.0f;

#pragma unroll 8
    for (int k = 0; k < TI; k++)
    {
      const float4 l = *(const float4 *) &L[k][4 * ty], r = *(const float4 *) &R[k][4 * tx];
      const float lv[4] = { l.x, l.y, l.z, l.w }, rv[4] = { r.x, r.y, r.z, r.w };

#pragma unroll
      for (int p = 0; p < 4; p++)
#pragma unroll
        for (int q = 0; q < 4; q++)
          acc[p][q] = fmaf (lv[p], rv[q], acc[p][q]);
    }

    __syncthreads ();

#pragma unroll
    for (int p = 0; p < 4; p++)
    {
      if (pass == 0)
        *(float4 *) &T[4 * ty + p][4 * tx] = make_float4 (acc[p][0], acc[p][1], acc[p][2], acc[p][3]);
      else
        *(float4 *) &Vi[(size_t) (TI + 4 * ty + p) * SB + 4 * tx] =
          make_float4 (-acc[p][0], -acc[p][1], -acc[p][2], -acc[p][3]);
    }

    __syncthreads ();
  }
}

/* sv . Vr over 64 entries, four chains */
__device__ __forceinline__ float
_cs_dot (const float (&Vr)[SB / 2], const float *sv)
{
  float acc[4] = { 0.0f, 0.0f, 0.0f, 0.0f };

#pragma unroll
  for (int c = 0; c < SB / 2; c += 4)
  {
    const float4 b = *(const float4 *) (sv + c);

    acc[0] = fmaf (Vr[c + 0], b.x, acc[0]);
    acc[1] = fmaf (Vr[c + 1], b.y, acc[1]);
    acc[2] = fmaf (Vr[c + 2], b.z, acc[2]);
    acc[3] = fmaf (Vr[c + 3], b.w, acc[3]);
  }

  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

/* U^T y = (float) (D r): block i, y_i = V_i ((D r)_i - sum_{j<i} U_ji^T y_j);
 * warp w owns rows 16w..16w+15 of each tile, lanes four of its columns; thread
 * (row, half) holds its half row of V_i in registers before its turn comes */
__global__ void __launch_bounds__ (CS_TH)
_fsolve_chain_kernel (const float *__restrict__ U, const float *__restrict__ V, const double *__restrict__ D,
                      const double *__restrict__ r, int n, unsigned long long *__restrict__ y, uint32_t epoch,
                      uint32_t pepoch, int32_t *__restrict__ sync, double *__restrict__ err)
{
  const size_t pdl0 = ncg_pdl_enter ();

  U += pdl0;
  V += pdl0;
  D += pdl0;
  r += pdl0;
  y += pdl0;
  sync += pdl0;
  err += pdl0;

  __shared__ float part[CS_TH / 32][SB];
  __shared__ __align__ (16) float sv[SB];
  __shared__ int blk;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;

  if (tid == 0)
    blk = atomicAdd (sync, 1);

  __syncthreads ();

  const int i = blk, kb = i * SB, nb = (n - kb < SB) ? n - kb : SB, vrow = tid >> 1, vh = (tid & 1) * (SB / 2);
  float Vr[SB / 2];

#pragma unroll
  for (int c = 0; c < SB / 2; c += 4)
  {
    const float4 v = *(const float4 *) (V + (size_t) i * SB * SB + vrow * SB + vh + c);

    Vr[c + 0] = v.x;
    Vr[c + 1] = v.y;
    Vr[c + 2] = v.z;
    Vr[c + 3] = v.w;
  }

  const double bd = (tid < nb) ? D[kb + tid] * r[kb + tid] : 0.0;
  float a[4]      = { 0.0f, 0.0f, 0.0f, 0.0f };

  for (int j = 0; j < i; j++)
  {
    const float *row = U + (size_t) (j * SB + wid * 16) * n + kb + lane;
    float u[4][16];

#pragma unroll
    for (int rr = 0; rr < 16; rr++)
#pragma unroll
      for (int q = 0; q < 4; q++)
        u[q][rr] = (lane + 32 * q < nb) ? row[(size_t) rr * n + 32 * q] : 0.0f;

    /* y_j of this warp's 16 rows: lane rr waits for row rr, then shares it */
    const float ym = (lane < 16) ? _cs_get (y + j * SB + wid * 16 + lane, epoch, sync, err) : 0.0f;

#pragma unroll
    for (int rr = 0; rr < 16; rr++)
    {
      const float yv = __shfl_sync (0xffffffffu, ym, rr);

#pragma unroll
      for (int q = 0; q < 4; q++)
        a[q] = fmaf (u[q][rr], yv, a[q]);
    }
  }

#pragma unroll
  for (int q = 0; q < 4; q++)
    part[wid][lane + 32 * q] = a[q];

  __syncthreads ();

  if (tid < SB)
  {
    float b = (float) bd;

    if (tid < nb)
    {
      float t = 0.0f;

#pragma unroll
      for (int w = 0; w < CS_TH / 32; w++)
        t += part[w][tid];

      b -= t;
    }

    sv[tid] = b;
  }

  __syncthreads ();

  float acc = _cs_dot (Vr, sv + vh);

  acc += __shfl_xor_sync (0xffffffffu, acc, 1);

  if (vh == 0 && vrow < nb)
    _cs_put (y + kb + vrow, acc, pepoch);

  _cs_finish (sync, tid);
}

/* U x = y, z = D x: block i (from the last), x_i = V_i^T (y_i - sum_{j>i} U_ij x_j) */
__global__ void __launch_bounds__ (CS_TH)
_bsolve_chain_kernel (const float *__restrict__ U, const float *__restrict__ V, const double *__restrict__ D,
                      const unsigned long long *__restrict__ y, int n, unsigned long long *__restrict__ x,
                      uint32_t epoch, uint32_t pepoch, double *__restrict__ z, int32_t *__restrict__ sync,
                      double *__restrict__ err)
{
  const size_t pdl0 = ncg_pdl_enter ();

  U += pdl0;
  V += pdl0;
  D += pdl0;
  y += pdl0;
  x += pdl0;
  z += pdl0;
  sync += pdl0;
  err += pdl0;

  __shared__ __align__ (16) float sv[SB];
  __shared__ float half[SB];
  __shared__ int blk;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nbk = (n + SB - 1) / SB;

  if (tid == 0)
    blk = nbk - 1 - atomicAdd (sync, 1);

  __syncthreads ();

  /* column vrow of V_i, entries vh.. (the halves in warps of their own, so that
   * the loads of V run along its rows) */
  const int i = blk, kb = i * SB, nb = (n - kb < SB) ? n - kb : SB, r0 = wid * 16;
  const int vrow = tid & (SB - 1), vh = (tid / SB) * (SB / 2);
  float Vr[SB / 2], p[16];

#pragma unroll
  for (int c = 0; c < SB / 2; c++)
    Vr[c] = V[(size_t) i * SB * SB + (vh + c) * SB + vrow];

#pragma unroll
  for (int rr = 0; rr < 16; rr++)
    p[rr] = 0.0f;

  const double dz = (vrow < nb) ? D[kb + vrow] : 0.0;

  for (int j = nbk - 1; j > i; j--)
  {
    const int jb = j * SB, nbj = (n - jb < SB) ? n - jb : SB;
    const float *row = U + (size_t) (kb + r0) * n + jb + lane;
    float u[4][16], xv[4];

#pragma unroll
    for (int rr = 0; rr < 16; rr++)
    {
#pragma unroll
      for (int q = 0; q < 4; q++)
        u[q][rr] = (r0 + rr < nb && lane + 32 * q < nbj) ? row[32 * q] : 0.0f;

      row += n;
    }

    _cs_get4 (x + jb + lane, nbj - lane, xv, epoch, sync, err);

#pragma unroll
    for (int rr = 0; rr < 16; rr++)
#pragma unroll
      for (int q = 0; q < 4; q++)
        p[rr] = fmaf (u[q][rr], xv[q], p[rr]);
  }

  /* sums over the lanes of 16 values: at each halving a lane keeps the half of
   * its values that its bit selects and gets their other halves (15 + 1
   * shuffles; the block waits for this on the chain) */
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
  {
    const bool up = (lane & (2 * o)) != 0;

#pragma unroll
    for (int q = 0; q < o; q++)
    {
      const float send = up ? p[q] : p[q + o], keep = up ? p[q + o] : p[q];

      p[q] = keep + __shfl_xor_sync (0xffffffffu, send, 2 * o);
    }
  }

  p[0] += __shfl_xor_sync (0xffffffffu, p[0], 1);

  if ((lane & 1) == 0)
  {
    const int r = r0 + (lane >> 1);

    sv[r] = (r < nb) ? __uint_as_float ((uint32_t) y[kb + r]) - p[0] : 0.0f;
  }

  __syncthreads ();

  float acc = _cs_dot (Vr, sv + vh);

  if (vh != 0)
    half[vrow] = acc;

  __syncthreads ();

  if (vh == 0 && vrow < nb)
  {
    acc += half[vrow];
    _cs_put (x + kb + vrow, acc, pepoch);
    z[kb + vrow] = dz * (double) acc;
  }

  _cs_finish (sync, tid);
}

extern "C" size_t
ncg_pcg_trinv_bytes (int n)
{
  return sizeof (float) * SB * SB * (size_t) ((n + SB - 1) / SB);
}

extern "C" size_t
ncg_pcg_sync_bytes (int n)
{
  (void) n;

  return sizeof (int32_t) * 4;
}

extern "C" size_t
ncg_pcg_chain_bytes (int n)
{
  return sizeof (unsigned long long) * 2 * (size_t) n;
}

extern "C" cudaError_t
ncg_launch_trinv_diag_f32 (const float *U, int n, float *V, cudaStream_t s)
{
  if (n <= 0)
    return cudaSuccess;

  ncg_pdl_launch (_trinv_diag_kernel, (n + SB - 1) / SB, 256, 0, s, U, n, V);

  return cudaGetLastError ();
}

extern "C" cudaError_t
ncg_launch_pcg_precond (const float *R, const float *V, const double *D, int np, const double *r, void *chain,
                        uint32_t *epoch, double *z, int32_t *sync, double *err, cudaStream_t s)
{
  if (np <= 0)
    return cudaSuccess;

  const int nbk = (np + SB - 1) / SB;
  unsigned long long *y = (unsigned long long *) chain, *x = y + np;
  const uint32_t ey = ++*epoch, ex = ++*epoch;
  /* values are published under the launch's own epoch; the wait-fault test
   * hook publishes the forward solve's under one that no reader waits for,
   * so its first dependent wait runs out (CS_SPIN polls) and reports */
  const uint32_t py = ncg_fault_take (NCG_FAULT_CHAIN_WAIT) ? ey ^ 0x80000000u : ey;

  ncg_pdl_launch (_fsolve_chain_kernel, nbk, CS_TH, 0, s, R, V, D, r, np, y, ey, py, sync, err);
  ncg_pdl_launch (_bsolve_chain_kernel, nbk, CS_TH, 0, s, R, V, D, y, np, x, ex, ex, z, sync, err);

  return cudaGetLastError ();
}

extern "C" size_t
ncg_pcg_sc_bytes (void)
{
  return sizeof (double) * (NCG_PCG_NSC + 3 * DOT_CTAS + 1);
}

/* CTAs of a launch that sums over n entries */
static int
_dots_grid (int n)
{
  const int g = (n + DOT_TH - 1) / DOT_TH;

  return g < DOT_CTAS ? g : DOT_CTAS;
}

/* the scalars sc of the start (mode 0: u = r, v = z, w = b, p = z), <p, q> (mode 1:
 * u = p, v = q), the next direction (mode 2: u = r, v = z, w = r_prev) or the
 * residual alone (mode 3: u = r) */
extern "C" cudaError_t
ncg_launch_pcg_dots (int mode, const double *u, const double *v, const double *w, const double *D, double *p, int n,
                     double *sc, cudaStream_t s)
{
  double *part   = sc + NCG_PCG_NSC;
  int32_t *count = (int32_t *) (part + 3 * DOT_CTAS);
  const int g    = _dots_grid (n);

  if (mode == 0)
    ncg_pdl_launch (_pcg_dots_kernel<0>, g, DOT_TH, 0, s, u, v, w, D, p, n, sc, part, count);
  else if (mode == 1)
    ncg_pdl_launch (_pcg_dots_kernel<1>, g, DOT_TH, 0, s, u, v, w, D, p, n, sc, part, count);
  else if (mode == 2)
    ncg_pdl_launch (_pcg_dots_kernel<2>, g, DOT_TH, 0, s, u, v, w, D, p, n, sc, part, count);
  else
    ncg_pdl_launch (_pcg_dots_kernel<3>, g, DOT_TH, 0, s, u, v, w, D, p, n, sc, part, count);

  return cudaGetLastError ();
}

extern "C" cudaError_t
ncg_launch_pcg_step (double *x, double *r, double *rprev, const double *p, const double *q, const double *D, int n,
                     double *sc, cudaStream_t s)
{
  double *part   = sc + NCG_PCG_NSC;
  int32_t *count = (int32_t *) (part + 3 * DOT_CTAS);

  ncg_pdl_launch (_pcg_step_kernel, _dots_grid (n), DOT_TH, 0, s, x, r, rprev, p, q, D, n, sc, part, count);

  return cudaGetLastError ();
}

extern "C" cudaError_t
ncg_launch_pcg_dir (double *p, const double *z, int n, double *sc, cudaStream_t s)
{
  ncg_pdl_launch (_pcg_dir_kernel, (n + 255) / 256, 256, 0, s, p, z, n, sc);

  return cudaGetLastError ();
}

/* ------------------------------------------------------------------------ */
/* The FP64 NNLS solve's fallbacks when the normal equations of a set are    */
/* not positive definite (ncm_nnls.c:573-638, dispatch :655-666): a general  */
/* symmetric solve (the dsysv step; here Gaussian elimination with partial  */
/* pivoting on the full symmetric matrix) and, when that meets an exactly    */
/* zero pivot, the least-squares solve of A_P x = f by Householder QR (the  */
/* dgels step).  Both follow the oracle's operation order with explicitly   */
/* rounded operations (no FMA contraction), so the same inputs give the same */
/* bits: pivots are chosen by exact comparisons (the lowest row among equal  */
/* magnitudes), each reduction is one thread's sequential sum.  One launch  */
/* per elimination or reflection step; these are rare paths, sized for      */
/* correctness, not speed.                                                   */
/* ------------------------------------------------------------------------ */

/* the lower triangle of an upper-stored symmetric n x n matrix, in place */
__global__ void
_sym_mirror_kernel (double *A, int n)
{
  const int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;

  if (e >= (int64_t) n * n)
    return;

  const int r = (int) (e / n), c = (int) (e % n);

  if (c < r)
    A[e] = A[(size_t) c * n + r];
}

#define GE_PIV_TH 256

/* step k: the pivot row (largest |A[r][k]|, r >= k, lowest r among equals),
 * then the swap of rows k and p and of b[k], b[p]; *info = k + 1 when the
 * column is exactly zero */
__global__ void __launch_bounds__ (GE_PIV_TH)
_ge_pivot_kernel (double *A, int n, int k, double *b, int32_t *info)
{
  __shared__ double sv[GE_PIV_TH];
  __shared__ int si[GE_PIV_TH];
  const int t = threadIdx.x;

  if (*info)
    return;

  double amax = -1.0;
  int p       = n;

  for (int r = k + t; r < n; r += GE_PIV_TH)
  {
    const double v = fabs (A[(size_t) r * n + k]);

    if (v > amax)
    {
      amax = v;
      p    = r;
    }
  }

  sv[t] = amax;
  si[t] = p;
  __syncthreads ();

  for (int o = GE_PIV_TH / 2; o > 0; o >>= 1)
  {
    if (t < o && (sv[t + o] > sv[t] || (sv[t + o] == sv[t] && si[t + o] < si[t])))
    {
      sv[t] = sv[t + o];
      si[t] = si[t + o];
    }

    __syncthreads ();
  }

  amax = sv[0];
  p    = si[0];

  if (amax == 0.0)
  {
    if (t == 0)
      *info = k + 1;

    return;
  }

  if (p != k)
  {
    for (int c = t; c < n; c += GE_PIV_TH)
    {
      const double x = A[(size_t) k * n + c];

      A[(size_t) k * n + c] = A[(size_t) p * n + c];
      A[(size_t) p * n + c] = x;
    }

    if (t == 0)
    {
      const double x = b[k];

      b[k] = b[p];
      b[p] = x;
    }
  }
}

#define GE_UP_RX 32
#define GE_UP_RY 8

/* step k: rows r > k minus f_r times row k over the columns c > k (column k
 * below the diagonal is never read again), b[r] minus f_r b[k];
 * f_r = A[r][k] / A[k][k], rows with f_r = 0 untouched */
__global__ void __launch_bounds__ (GE_UP_RX * GE_UP_RY)
_ge_update_kernel (double *A, int n, int k, double *b, const int32_t *info)
{
  __shared__ double f[GE_UP_RY];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int r  = k + 1 + blockIdx.y * GE_UP_RY + ty;

  if (*info)
    return;

  if (tx == 0)
    f[ty] = (r < n) ? __ddiv_rn (A[(size_t) r * n + k], A[(size_t) k * n + k]) : 0.0;

  __syncthreads ();

  if (r >= n || f[ty] == 0.0)
    return;

  const double fr = f[ty];

  for (int c = k + 1 + blockIdx.x * GE_UP_RX + tx; c < n; c += gridDim.x * GE_UP_RX)
    A[(size_t) r * n + c] = __dsub_rn (A[(size_t) r * n + c], __dmul_rn (fr, A[(size_t) k * n + c]));

  if (blockIdx.x == 0 && tx == 0)
    b[r] = __dsub_rn (b[r], __dmul_rn (fr, b[k]));
}

/* back substitution of the eliminated system, one thread, the oracle's order */
__global__ void
_ge_backsub_kernel (const double *A, int n, double *b, const int32_t *info)
{
  if (*info || threadIdx.x != 0 || blockIdx.x != 0)
    return;

  for (int r = n - 1; r >= 0; r--)
  {
    double s = b[r];

    for (int c = r + 1; c < n; c++)
      s = __dsub_rn (s, __dmul_rn (A[(size_t) r * n + c], b[c]));

    b[r] = __ddiv_rn (s, A[(size_t) r * n + r]);
  }
}

extern "C" cudaError_t
ncg_launch_sysv (double *A, int n, double *b, int32_t *info, cudaStream_t s)
{
  if (n <= 0)
    return cudaSuccess;

  cudaError_t e = cudaMemsetAsync (info, 0, sizeof (int32_t), s);

  if (e != cudaSuccess)
    return e;

  _sym_mirror_kernel<<<(unsigned) (((int64_t) n * n + 255) / 256), 256, 0, s>>> (A, n);

  for (int k = 0; k < n; k++)
  {
    _ge_pivot_kernel<<<1, GE_PIV_TH, 0, s>>> (A, n, k, b, info);

    const int rows = n - k - 1;

    if (rows > 0)
    {
      const int gx = ((rows + GE_UP_RX - 1) / GE_UP_RX < 8) ? (rows + GE_UP_RX - 1) / GE_UP_RX : 8;
      dim3 grid ((unsigned) gx, (unsigned) ((rows + GE_UP_RY - 1) / GE_UP_RY));

      _ge_update_kernel<<<grid, dim3 (GE_UP_RX, GE_UP_RY), 0, s>>> (A, n, k, b, info);
    }
  }

  _ge_backsub_kernel<<<1, 32, 0, s>>> (A, n, b, info);

  return cudaGetLastError ();
}

/* Q = A[:, P] (nrows x np, row-major), y = f */
__global__ void
_qr_gather_kernel (const double *__restrict__ A, int nrows, int ncols, const int32_t *__restrict__ P, int np,
                   const double *__restrict__ f, double *__restrict__ Q, double *__restrict__ y)
{
  const int64_t e = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;

  if (e < (int64_t) nrows * np)
  {
    const int r = (int) (e / np), c = (int) (e % np);

    Q[e] = A[(size_t) r * ncols + P[c]];
  }

  if (e < nrows)
    y[e] = f[e];
}

/* reflection k, part 1 (one thread): restore the diagonal of step k - 1,
 * then nrm = |Q[k:, k]|, alpha = -sign(Q[k][k]) nrm, Q[k][k] -= alpha and
 * vtv = |Q[k:, k]|^2; sc = {alpha, vtv, skip} (skip when the column is zero) */
__global__ void
_qr_house_kernel (double *Q, int nrows, int np, int k, double *sc)
{
  if (threadIdx.x != 0 || blockIdx.x != 0)
    return;

  if (k > 0 && sc[2] == 0.0)
    Q[(size_t) (k - 1) * np + (k - 1)] = sc[0];

  double nrm = 0.0;

  for (int r = k; r < nrows; r++)
    nrm = __dadd_rn (nrm, __dmul_rn (Q[(size_t) r * np + k], Q[(size_t) r * np + k]));

  nrm = __dsqrt_rn (nrm);

  const double alpha = (Q[(size_t) k * np + k] > 0.0) ? -nrm : nrm;

  if (nrm == 0.0)
  {
    sc[2] = 1.0;

    return;
  }

  Q[(size_t) k * np + k] = __dsub_rn (Q[(size_t) k * np + k], alpha);

  double vtv = 0.0;

  for (int r = k; r < nrows; r++)
    vtv = __dadd_rn (vtv, __dmul_rn (Q[(size_t) r * np + k], Q[(size_t) r * np + k]));

  sc[0] = alpha;
  sc[1] = vtv;
  sc[2] = 0.0;
}

/* reflection k, part 2: one thread per column c > k (c = np: the right-hand
 * side y), s = 2 (v . q_c) / vtv with the sum in row order, q_c -= s v */
__global__ void
_qr_apply_kernel (double *Q, int nrows, int np, int k, double *y, const double *sc)
{
  const int c = k + 1 + blockIdx.x * blockDim.x + threadIdx.x;

  if (sc[2] != 0.0 || c > np)
    return;

  const double vtv = sc[1];
  double s         = 0.0;

  if (c < np)
  {
    for (int r = k; r < nrows; r++)
      s = __dadd_rn (s, __dmul_rn (Q[(size_t) r * np + k], Q[(size_t) r * np + c]));

    s = __ddiv_rn (__dmul_rn (2.0, s), vtv);

    for (int r = k; r < nrows; r++)
      Q[(size_t) r * np + c] = __dsub_rn (Q[(size_t) r * np + c], __dmul_rn (s, Q[(size_t) r * np + k]));
  }
  else
  {
    for (int r = k; r < nrows; r++)
      s = __dadd_rn (s, __dmul_rn (Q[(size_t) r * np + k], y[r]));

    s = __ddiv_rn (__dmul_rn (2.0, s), vtv);

    for (int r = k; r < nrows; r++)
      y[r] = __dsub_rn (y[r], __dmul_rn (s, Q[(size_t) r * np + k]));
  }
}

/* the last diagonal, then R x = y by back substitution (one thread); a zero
 * diagonal gives x = 0 for that variable */
__global__ void
_qr_backsub_kernel (double *Q, int np, int kmax, const double *y, const double *sc, double *x)
{
  if (threadIdx.x != 0 || blockIdx.x != 0)
    return;

  if (kmax > 0 && sc[2] == 0.0)
    Q[(size_t) (kmax - 1) * np + (kmax - 1)] = sc[0];

  for (int k = np - 1; k >= 0; k--)
  {
    double s = y[k];

    for (int c = k + 1; c < np; c++)
      s = __dsub_rn (s, __dmul_rn (Q[(size_t) k * np + c], x[c]));

    x[k] = (Q[(size_t) k * np + k] != 0.0) ? __ddiv_rn (s, Q[(size_t) k * np + k]) : 0.0;
  }
}

extern "C" cudaError_t
ncg_launch_gels (const double *A, int nrows, int ncols, const int32_t *P, int np, const double *f, double *Q,
                 double *y, double *sc, double *x, cudaStream_t s)
{
  if (np <= 0)
    return cudaSuccess;

  const int64_t tot = (int64_t) nrows * np > nrows ? (int64_t) nrows * np : nrows;
  const int kmax    = np < nrows ? np : nrows;
  cudaError_t e;

  _qr_gather_kernel<<<(unsigned) ((tot + 255) / 256), 256, 0, s>>> (A, nrows, ncols, P, np, f, Q, y);

  if ((e = cudaMemsetAsync (sc, 0, 3 * sizeof (double), s)) != cudaSuccess)
    return e;

  for (int k = 0; k < kmax; k++)
  {
    _qr_house_kernel<<<1, 32, 0, s>>> (Q, nrows, np, k, sc);
    _qr_apply_kernel<<<(unsigned) ((np - k + 127) / 128), 128, 0, s>>> (Q, nrows, np, k, y, sc);
  }

  _qr_backsub_kernel<<<1, 32, 0, s>>> (Q, np, kmax, y, sc, x);

  return cudaGetLastError ();
}

/* ---- row sums of a square interpolation matrix (the AMISE of the LOO fit,
 * ncm_stats_dist.c:581-598): rowx[i] = sum_{j != i} IM[i][j] in column order
 * per lane, diag[i] = IM[i][i]; one warp per row */
__global__ void
_im_rowsums_kernel (const double *__restrict__ IM, int n, double *__restrict__ rowx, double *__restrict__ diag)
{
  const int warp = (int) ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;

  if (warp >= n)
    return;

  const double *row = IM + (size_t) warp * n;
  double s = 0.0;

  for (int j = lane; j < n; j += 32)
    if (j != warp)
      s += row[j];

  for (int o = 16; o > 0; o >>= 1)
    s += __shfl_xor_sync (0xffffffffu, s, o);

  if (lane == 0)
  {
    rowx[warp] = s;
    diag[warp] = row[warp];
  }
}

extern "C" cudaError_t
ncg_launch_im_rowsums (const double *IM, int n, double *rowx, double *diag, cudaStream_t s)
{
  if (n <= 0)
    return cudaSuccess;

  _im_rowsums_kernel<<<(unsigned) ((n + 7) / 8), 256, 0, s>>> (IM, n, rowx, diag);

  return cudaGetLastError ();
}
