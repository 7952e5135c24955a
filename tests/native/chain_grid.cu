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
  *emitters = A.emitting;
  return A.ctas;
}

// arrays of which k[i] are sent: how many CTAs emit the list of each, counted from the
// groups they are in; 0 when a group's number is wrong
extern "C" int chain_shares(int units, const uint32_t* n, const uint32_t* k, int per_sm, int sms, uint32_t* ctas) {
  static hipress::ChainArgs A;
  A.units = units;
  for (int i = 0; i < units; ++i) {
    A.unit[i].s.n = n[i];
    A.unit[i].s.kmax = k[i];
    A.unit[i].s.stride = 4;
    ctas[i] = 0;
  }
  if (!hipress::chain_place(A, per_sm, sms)) return 0;
  for (uint32_t g = 0; g < A.emitting / hipress::kChainLists; ++g) {
    const hipress::ChainEmitters& e = A.emitters[g];
    if (e.unit >= units || e.group != ctas[e.unit] / hipress::kChainLists) return 0;
    ctas[e.unit] += hipress::kChainLists;
  }
  for (uint32_t g = 0; g < A.emitting / hipress::kChainLists; ++g)
    if (A.emitters[g].groups * hipress::kChainLists != ctas[A.emitters[g].unit]) return 0;
  return A.ctas;
}
