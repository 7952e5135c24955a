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
// elements, 1 % 18.1 / 20.0; 4097 elements 19.8 / 18.1).  Without DGC's momentum, of more than
// 42 M, when few of a tile's elements are candidates: a CTA per half tile spends longer on the
// bound, its barriers and its reservation than on them, where theirs look after several tiles
// (GradDrop, 0.1 %, normal values: 33 M 96 / 97, 67 M 163 / 171, 134 M 297 / 319).  With more
// candidates their list's one counter is the longer wait (67 M, GradDrop, 0.2 % 181 / 174 with
// normal, 201 / 174 with heavy-tailed values; without an update 0.02 % 79 / 85, 0.1 % 98 / 84),
// and DGC, which moves more bytes, gains throughout (0.1 %: 20 M 103 / 84, 67 M 262 / 224,
// 134 M 474 / 426).  mode: of the update (see pass0_body).
inline bool chain_is_slower(int mode, uint64_t n, uint64_t k) {
  return n <= (uint64_t)kSelTile || (mode != 2 && n > 10240ull * kSelTile && k * (mode == 1 ? 900 : 2000) <= n);
}
// Places the units' tiles and samples behind one another; per_sm: what chain_per_sm says,
// sms: those of the stream.  False when the lists cannot be shared out.
bool chain_place(ChainArgs& A, int per_sm, int sms);
// The three launches (mode of the update: see pass0_body); counters, lists' counts and
// barrier words are zero before them.  Where the emitting launch is refused (less of the GPU
// is ours than the queries said) five plain ones make up for it.
cudaError_t chain_select(int mode, const ChainArgs& A, cudaStream_t st);

}  // namespace hipress
