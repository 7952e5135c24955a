// Runs the selection's emit stage on a list that every CTA believes to have a length of
// its own, which is what CTAs see behind a grid barrier that expired.
#include "sparse_core.cuh"

using namespace hipress;

__global__ void __launch_bounds__(kSpThreads) emit_views_kernel(SelUnit unit, const uint32_t* counts, uint8_t* out) {
  extern __shared__ __align__(16) unsigned char raw[];
  SelSmem& sm = *reinterpret_cast<SelSmem*>(raw);
  EmitDst d = {};
  d.n = 1;
  d.out[0] = out;
  const ListState ls = {counts[blockIdx.x], 0u, unit.low};
  const uint32_t nx = emit_slices(ls.count, gridDim.x);
  if (blockIdx.x < nx) emit_slice(kGradDrop, unit, ls, d, sm, blockIdx.x, nx);
}

extern "C" int emit_views(float* a, uint32_t n, uint32_t k, uint32_t* ws, float* list, uint32_t cap, uint32_t low,
                          const uint32_t* counts, int ctas, uint8_t* out, void* stream) {
  SelUnit u = {};
  u.a = a;
  u.n = n;
  u.k = u.kmax = k;
  u.ws = ws;
  u.cv = list;
  u.cap = cap;
  u.low = low;
  cudaError_t e = cudaFuncSetAttribute(emit_views_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(SelSmem));
  if (e != cudaSuccess) return (int)e;
  emit_views_kernel<<<ctas, kSpThreads, sizeof(SelSmem), (cudaStream_t)stream>>>(u, counts, out);
  return (int)cudaGetLastError();
}

extern "C" int emit_workspace_words() { return kWsWords; }
