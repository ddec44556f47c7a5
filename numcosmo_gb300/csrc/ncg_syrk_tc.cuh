/*
 * ncg_syrk_tc.cuh -- the operand pack of the tensor-core symmetric rank-K
 * update (ncg_syrk_tc.cu): layout constants and the writers shared with the
 * FP32 Cholesky's panel solve (ncg_linalg.cu), which packs its panel as it
 * finishes it.
 *
 * For each 128-column tile t and 32-row K-chunk c the pack holds a 32 KB block
 * at ((t * nkc) + c) * 32 KB: the TF32 hi part of the 128 x 32 sub-matrix in
 * the K-major core-matrix layout of ncg_tc_ptx.cuh (LBO 2048), then the lo
 * part (value - hi, rounded to TF32).
 */
#ifndef NCG_SYRK_TC_CUH
#define NCG_SYRK_TC_CUH

#include "ncg_tc_ptx.cuh"

#define SK_T 128                     /* output tile edge (MMA M and N)       */
#define SK_KC 32                     /* K rows per chunk                     */
#define SK_LBO (SK_T / 8 * 128)      /* 2048: K-adjacent core matrices       */
#define SK_HALF (SK_KC / 4 * SK_LBO) /* 16 KB: hi (or lo) of a 128 x 32 block */
#define SK_BLOCK (2 * SK_HALF)       /* 32 KB per tile and chunk             */
#define SK_STAGE (2 * SK_BLOCK)      /* A block + B block                    */
/* one float4 of four consecutive k of column-row `row`, split hi / lo */
static __device__ __forceinline__ void
_put_split4 (float *blk, int row, int k4, double v0, double v1, double v2, double v3)
{
  const uint32_t off = _cm_off (row, k4, SK_LBO) >> 2;
  const float h0 = _tf32 ((float) v0), h1 = _tf32 ((float) v1), h2 = _tf32 ((float) v2), h3 = _tf32 ((float) v3);

  *(float4 *) (blk + off) = make_float4 (h0, h1, h2, h3);
  *(float4 *) (blk + SK_HALF / 4 + off) =
    make_float4 (_tf32 ((float) (v0 - (double) h0)), _tf32 ((float) (v1 - (double) h1)),
                 _tf32 ((float) (v2 - (double) h2)), _tf32 ((float) (v3 - (double) h3)));
}

/* the same from FP32 values, where v - hi is exact in FP32: no FP64 conversions,
 * which take 64 cycles of the sub-partition's FP64 pipe each here */
static __device__ __forceinline__ void
_put_split4f (float *blk, int row, int k4, float v0, float v1, float v2, float v3)
{
  const uint32_t off = _cm_off (row, k4, SK_LBO) >> 2;
  const float h0 = _tf32 (v0), h1 = _tf32 (v1), h2 = _tf32 (v2), h3 = _tf32 (v3);

  *(float4 *) (blk + off) = make_float4 (h0, h1, h2, h3);
  *(float4 *) (blk + SK_HALF / 4 + off) = make_float4 (_tf32 (v0 - h0), _tf32 (v1 - h1), _tf32 (v2 - h2), _tf32 (v3 - h3));
}

#endif /* NCG_SYRK_TC_CUH */
