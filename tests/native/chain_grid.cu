// The size of the emitting launch of a chain (csrc/cuda/sparse_chain.cu), without a GPU.
#include "sparse_chain.cu"

// units arrays of n elements of which kmax are sent; 0 when a chain does not take them
extern "C" uint32_t chain_ctas(int units, uint32_t n, uint32_t kmax, int per_sm, int sms, uint32_t* emitters) {
  static hipress::ChainArgs A;
  A.units = units;
  for (int i = 0; i < units; ++i) {
    A.unit[i].s.n = n;
    A.unit[i].s.kmax = kmax;
    A.unit[i].s.stride = 4;
  }
  if (!hipress::chain_place(A, per_sm, sms)) return 0;
  *emitters = A.units * A.emitters;
  return A.ctas;
}
