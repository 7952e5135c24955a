// The selection of sparse_core.cuh as a chain of launches, for callers that wait for nobody
// (the stand-alone encode, buckets of a job of one rank): sample, collect with a CTA per half tile, emit.  SMs do not run
// at one speed, and equal shares of a persistent grid leave the fast ones idle for a tenth
// of the pass; a new CTA goes to whichever SM is free.  The collect begins while the sample
// ends, and its CTAs that start ahead of the bound update their tile before they wait for
// it; the emit is cooperative, and begins when the collect has ended.
#pragma once
#include "sparse_core.cuh"
#include "sync.cuh"

namespace hipress {

// An array's list is in parts, because its counter takes 20 ns a reservation; a CTA emits
// each, and those of a bucket's forty arrays fit the GPU at once.
constexpr uint32_t kChainLists = 7;

struct ChainUnit {
  SelUnit s;
  uint32_t* counts;     // of the parts of its list, kChainLists lines of 32 words
  uint32_t tile0;       // tiles of the units before it, and sampled tiles
  uint32_t sample0;
  float* add;           // where its pairs go, besides a payload (EmitDst)
  float* set;
};
// A group of kChainLists CTAs that emit a list, one each of its parts: number `group` of
// `groups`.  In a table, and not in ChainUnit, whose 120 bytes are read by all threads at
// once: with 128 the emitting launch of 40 arrays took 1 us longer.
struct ChainEmitters {
  uint8_t unit, group, groups;
};
constexpr uint32_t kChainGroups = 64;   // two CTAs on each of 148 SMs are 42
constexpr int kChainUnits = HP_MAX_SEGS;   // at most kSpThreads: a thread looks at each
struct ChainArgs {
  ChainUnit unit[kChainUnits];
  int units, alg;
  float momentum, scale;
  uint8_t* payload;      // of the only unit, or null
  uint32_t* barrier;     // kBarrierWords of zeros
  uint32_t *status, code;   // what a barrier that expires records, and where
  uint32_t* gave_up;     // zero until a CTA's barrier expires, for the chains of one bucket; or null
  ChainEmitters emitters[kChainGroups];
  uint32_t emitting;     // CTAs of these groups
  uint32_t tiles;
  uint32_t stretch;      // half tiles that lie between those of two neighbouring CTAs, or 0: in order
  uint32_t ctas;         // of the emitting launch; those behind the emitters wait for a list that came out short
};

// CTAs of the emitting launch that an SM holds at once, 0 when the kernels cannot run
int chain_per_sm(int dev);
// Whether an array of n elements, of which k are sent, is better served by the persistent
// kernels.  Of at most one tile: a single CTA of theirs meets no barrier, and is one launch
// instead of three (encode, us, persistent / chain: 300 elements, 10 % 17.0 / 19.6, 4096
// elements, 1 % 18.1 / 20.0; 4097 elements 19.8 / 18.1).  Of more than 42 M, when few of a
// tile's elements are candidates: a CTA per half tile spends longer on the bound, its barriers
// and its reservation than on them, where theirs look after several tiles (DGC, 0.1 %,
// normal values: 33 M 147 / 147, 50 M 204 / 211, 67 M 261 / 274, 134 M 472 / 525; GradDrop
// 33 M 96 / 97, 67 M 163 / 174, 134 M 296 / 322).  With more candidates their list's one
// counter is the longer wait, the sooner the fewer bytes an element moves: 67 M, DGC, 0.3 %
// 279 / 288 with normal, 290 / 285 with heavy-tailed values, 0.5 % 300 / 299, 328 / 295;
// GradDrop, 0.15 % 168 / 174, 186 / 175, 0.2 % 180 / 176, 202 / 175; without an update 0.02 %
// 79 / 85, 0.1 % 98 / 84.  mode: of the update (see pass0_body).
inline bool chain_is_slower(int mode, uint64_t n, uint64_t k) {
  const uint64_t few = mode == 2 ? 400 : (mode == 1 ? 900 : 2000);
  return n <= (uint64_t)kSelTile || (n > 10240ull * kSelTile && k * few <= n);
}
// Places the units' tiles and samples behind one another; per_sm: what chain_per_sm says,
// sms: those of the stream.  False when the lists cannot be shared out.
bool chain_place(ChainArgs& A, int per_sm, int sms);
// The three launches (mode of the update: see pass0_body); counters, lists' counts and
// barrier words are zero before them.  Where the emitting launch is refused (less of the GPU
// is ours than the queries said) five plain ones make up for it.
cudaError_t chain_select(int mode, const ChainArgs& A, cudaStream_t st);

}  // namespace hipress
