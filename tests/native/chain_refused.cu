// The chain of selections (csrc/cuda/sparse_chain.cu) where its cooperative launch is
// refused, as when less of the GPU is free than the queries say.  The refusal is the
// host's: the launch is not made.
#include <cuda_runtime.h>

#include "sparse_core.cuh"
#include "sync.cuh"

template <typename K, typename A>
static cudaError_t launch_unless_cooperative(const cudaLaunchConfig_t* c, K kern, const A& a) {
  for (unsigned i = 0; i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributeCooperative) return cudaErrorCooperativeLaunchTooLarge;
  return cudaLaunchKernelEx(c, kern, a);
}
#define cudaLaunchKernelEx launch_unless_cooperative
#include "sparse_chain.cu"
