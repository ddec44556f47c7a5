/*
 * ncg_pdl.cuh -- launches that overlap the end of the kernel before them in the
 * stream (programmatic dependent launch): in the chains of short kernels of the
 * mixed weight fit the start of a grid, 1 to 2 us, is hidden behind its predecessor
 * (fit d=12 N=4096 41.5 -> 38.4 ms, half-move d=8 N=512 3.8 -> 3.3 ms), and between
 * the FP64 eval and its merge (one point 27.0 -> 24.4 us, 1000 points 97.0 -> 92.7 us,
 * KDE d=4 n=1000).  Kernels that fill an SM let the next grid in only as they
 * leave: the FP64 fit's product and panel kernels, d=12 N=2048, took 38.4 instead
 * of 32.7 ms with the next grid's CTAs resident from their start, and 26.1 instead
 * of 29.6 ms like this; the rank-K updates of the FP32 factor gain 2 % of the mixed
 * fit over the early form, its panels 1 % of the half-move with the early form.
 *
 * A kernel launched by ncg_pdl_launch begins with ncg_pdl_enter or ncg_pdl_wait
 * (before any access to global memory): it returns once every kernel before it in
 * the stream has finished and its writes can be seen, since each of those waited in
 * the same way before it let the next one start.  Loads through a `__restrict__` pointer, const or not, may be
 * moved by the compiler as if nothing else wrote there, also ahead of that wait:
 * the zero that they return, added to every such parameter, ties its loads to
 * the wait and leaves the pointer what it is to the compiler (hidden pointers cost
 * the inverses' kernel twice its time, its loads no longer ran ahead of its stores).
 */
#ifndef NCG_PDL_CUH
#define NCG_PDL_CUH

#include <cuda_runtime.h>

static __device__ __forceinline__ size_t
ncg_pdl_enter (void)
{
  size_t zero;

  asm volatile ("griddepcontrol.wait;\n\t"
                "griddepcontrol.launch_dependents;\n\t"
                "mov.u64 %0, 0;"
                : "=l"(zero)::"memory");

  return zero;
}

/* the two halves, for kernels that fill an SM: the next grid is let in late, when
 * this one's CTAs leave (called by one thread of a CTA or by all), and waits here
 * before its first access to global memory */
static __device__ __forceinline__ size_t
ncg_pdl_wait (void)
{
  size_t zero;

  asm volatile ("griddepcontrol.wait;\n\t"
                "mov.u64 %0, 0;"
                : "=l"(zero)::"memory");

  return zero;
}

static __device__ __forceinline__ void
ncg_pdl_next (void)
{
  asm volatile ("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... K, typename... A>
static cudaError_t
ncg_pdl_launch (void (*kernel) (K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
  cudaLaunchAttribute at[1];
  cudaLaunchConfig_t cfg = {};

  at[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;

  cfg.gridDim          = grid;
  cfg.blockDim         = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream           = s;
  cfg.attrs            = at;
  cfg.numAttrs         = 1;

  return cudaLaunchKernelEx (&cfg, kernel, args...);
}

#endif /* NCG_PDL_CUH */
