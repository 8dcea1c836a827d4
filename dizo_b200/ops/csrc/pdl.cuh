// Programmatic dependent launch: a kernel launched with `pdl_launch(..., dependent = true)` may start while its
// predecessor in the stream still runs, once every CTA of the predecessor has executed pdl_trigger() (or exited).
// It must execute pdl_wait() before it touches anything the predecessor writes or reads; the wait returns when the
// predecessor has completed and its memory is visible, and because every kernel of such a chain waits before it
// finishes, so has everything launched before it.  Both instructions do nothing in a kernel launched the ordinary way.
//
// A whole chain of such kernels can be resident while its first one still writes (each triggers before it waits): the norm
// behind a staging sweep, the projection behind the norm and so on, with the weights of all of them in the sweep's output.
// Memory that is written during a kernel's lifetime may not be read with non-coherent loads, so a kernel that calls
// pdl_wait() has no ld.global.nc, no __ldg and no `const __restrict__` parameter (through which the compiler may issue
// either), for weights and biases no more than for activations.  The exception is ld_table(): constants that nothing rewrites.
//
// The GEMMs, the attention forward, the norms and the sweeps always launch this way (a kernel launched the ordinary way in
// between serialises as before): the launch latency and the set-up of barriers, TMEM and tables run beside the predecessor's
// tail.  OPT-125m training step 2.88 -> 2.55 ms, OPT-350m graph replay 3.97 -> 3.73, OPT-2.7b 44.5 -> 44.3, scoring with
// OPT-1.3b 10.5 -> 10.0.
//
// A kernel that allocates TMEM triggers after its allocation: its dependents are then only resident beside CTAs that
// already own their columns, so an allocation can never wait for a CTA that waits for it.
#pragma once
#include <cuda_runtime.h>

namespace dz {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A constant that no kernel of the process rewrites (quantiles, rotary angles).
template <class T>
__device__ __forceinline__ T ld_table(const T* p) { return __ldg(p); }

// Launch with an optional cluster of `cluster_x` CTAs along x, optionally as a programmatic dependent.
template <class... Params, class... Args>
inline cudaError_t pdl_launch(void (*kern)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                              int cluster_x, bool dependent, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster_x > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (dependent) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, Params(args)...);
}

}  // namespace dz
