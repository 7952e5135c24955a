// The chain of selections (csrc/cuda/sparse_chain.cu) whose grid barriers expire: each waits
// for one CTA more than there are, for 20 us.
#include <cuda_runtime.h>

#include "sparse_core.cuh"
#include "sync.cuh"

#define grid_barrier(words, gen, ctas, ns, status, code, wait) \
  grid_barrier(words, gen, (ctas) + 1u, 20000ull, status, code, wait)
#include "sparse_chain.cu"
