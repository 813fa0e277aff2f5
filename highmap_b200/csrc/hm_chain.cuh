/*
 * hm_chain.cuh - launches of a solve chained by programmatic dependent
 * launch.
 *
 * A solve is a chain of launches, each reading what the one before wrote.
 * Ordinary launches leave the GPU idle from a kernel's last CTA to the next
 * one's first instruction and its descriptor fetches: 5 of the 8.5 us of a
 * virtual-pipes step at 256^2.  A chained launch may start its CTAs while
 * the last CTAs of the kernel before it still run; they do what does not
 * depend on it (barrier set-up, descriptor prefetch, loads of the call's
 * constant inputs) and then wait in chain_wait until that kernel has
 * completed and its writes are visible.  Submitting one costs the host 3.3
 * us instead of 4.1.  Measured, ordinary to chained: virtual pipes 256^2
 * 8.4 -> 6.4 us per step, 1024^2 22.9 -> 20.5; sediment deposition 1024^2
 * 328 -> 285 us a call; thermal 4096^2 x 500 29.7 -> 27.7 ms.
 *
 * Rules kept by every kernel of a chain:
 *   - chain_wait by every thread before it reads anything an earlier launch
 *     of the chain wrote and before any global write.  It ends with the
 *     trigger that lets the next launch start: triggered before the wait,
 *     several future launches start at once and fill the SMs with waiting
 *     CTAs (9.5 instead of 8.4 us per step at 256^2);
 *   - grids an earlier launch wrote are read through pointers that came out
 *     of produced(), by plain loads: the compiler may move non-coherent
 *     loads (const __restrict__, __ldg) across the wait;
 *   - the first launch of a call is an ordinary one, so what came before the
 *     call is complete when any launch of the chain starts.
 */
#ifndef HM_CHAIN_CUH
#define HM_CHAIN_CUH

#include <cuda_runtime.h>

#include <utility>

namespace hm
{

__device__ __forceinline__ void chain_wait()
{
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

/* p after chain_wait, opaque to the compiler */
template <class T>
__device__ __forceinline__ T *produced(T *p)
{
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

/* launch k on s, chained to the launch before it on s or not */
template <class... P, class... A>
inline void chain_launch(bool chained, void (*k)(P...), dim3 grid, dim3 block, cudaStream_t s, A &&...args)
{
  cudaLaunchConfig_t  cfg = {};
  cudaLaunchAttribute   attr[1];
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained ? 1 : 0;
  (void)cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...); /* reported by HM_LAUNCH_CHECK */
}

} // namespace hm

#endif
