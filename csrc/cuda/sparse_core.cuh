// Device code of the top-k (DGC / GradDrop) compressor, shared by the
// stand-alone kernels (sparse_ops.cu) and the fused parameter-server kernels
// (fused_sparse.cu): radix-histogram passes, threshold search, block-aggregated
// compaction and scatter.  `cta` / `nctas` say which share of the work the calling
// CTA takes, so one launch can serve many (tensor, chunk) units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "hipress/capi.h"
#include "hipress/common.h"

namespace hipress {

// Two CTAs of 512 threads per SM in the grid-wide kernels: every CTA arrives at the same
// barrier counter, adds to the same histograms and reserves room in the same lists, and
// such an access to one address takes 10 to 25 ns of its own, so 444 CTAs of 256 threads
// spent 4.5 us per barrier.  One CTA per SM leaves HBM idle while it waits at its tile's
// end: the kernel of ResNet-50's compressed tensors through DGC and PS takes 197 us
// instead of 180.
constexpr int kSpThreads = 512;
constexpr uint32_t kSpTile = 16 * kSpThreads;   // elements per tile of the whole-array passes
constexpr int kBins = 4096;
// workspace words: 3 histograms, then counters
constexpr int kWsOutCount = 3 * kBins + 0;
constexpr int kWsTieCount = 3 * kBins + 1;
constexpr int kWsDone = 3 * kBins + 2;
constexpr int kWsSampled = 3 * kBins + 3;     // sampled tiles that are done
constexpr int kWsCandCount = 3 * kBins + 4;   // candidates collected by the update pass
constexpr int kWsOverflow = 3 * kBins + 5;    // they did not fit: use the full passes
constexpr int kWsLow = 3 * kBins + 6;         // magnitude key from which an element is a candidate
constexpr int kWsCand2Count = 3 * kBins + 7;  // candidates in the bin of the k-th largest
constexpr int kWsTicket = 3 * kBins + 8;      // stand-alone kernel: tile ticket, status
constexpr int kWsStatus = 3 * kBins + 9;
constexpr int kWsWords = 3 * kBins + 16;
// a list selection uses the first histogram for its candidates' digits, the room of the
// other two for the sample's keys
constexpr int kWsKeys = kBins;
constexpr uint32_t kMaxKeys = 2 * kBins;

__device__ __forceinline__ uint32_t digit_of(uint32_t key, int pass) {
  return pass == 0 ? (key >> 19) : (pass == 1 ? ((key >> 8) & 0x7FFu) : (key & 0xFFu));
}

struct FindSmem {
  uint32_t sums[kSpThreads / 32];
  uint2 res;
};

// Largest bin of a histogram of kBins bins whose suffix count reaches k, and krem = how
// many of the k fall in that bin, i.e. k - count(bins > bin); (0, 0) when fewer than k are
// counted.  `hist` is in shared or in global memory, where other CTAs' atomics wrote it.
// A warp sums 512 consecutive bins, read without bank conflicts; the warp in whose bins
// the k-th lies narrows it down to a row of 128, a lane and a bin.  (With 16 bins in a row
// per thread, every read of a histogram in shared memory was a 16-way conflict and a
// call took 0.9 us.)
static __device__ __noinline__ void find_bin(const uint32_t* hist, uint32_t k, FindSmem& fs, uint32_t& bin,
                                             uint32_t& krem) {
  constexpr int kRows = kBins / (kSpThreads * 4);  // rows of 128 bins per warp
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4 c[kRows];
  uint32_t rows[kRows], all = 0;
  const uint32_t* from = hist + warp * (kRows * 128) + lane * 4;
  if ((reinterpret_cast<uintptr_t>(hist) & 15) == 0) {
#pragma unroll
    for (int j = 0; j < kRows; ++j)
      asm volatile("ld.volatile.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(c[j].x), "=r"(c[j].y), "=r"(c[j].z), "=r"(c[j].w)
                   : "l"(from + j * 128)
                   : "memory");
  } else {   // a caller's workspace may lie on any word
#pragma unroll 1
    for (int j = 0; j < kRows; ++j) {
      const volatile uint32_t* w = from + j * 128;
      const uint4 v = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
      for (int q = 0; q < kRows; ++q)
        if (q == j) c[q] = v;
    }
  }
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    rows[j] = __reduce_add_sync(0xffffffffu, c[j].x + c[j].y + c[j].z + c[j].w);
    all += rows[j];
  }
  if (lane == 0) fs.sums[warp] = all;
  if (threadIdx.x == 0) fs.res = make_uint2(0u, 0u);
  __syncthreads();
  // elements in the bins of higher warps
  uint32_t above =
      __reduce_add_sync(0xffffffffu, lane > warp && lane < kSpThreads / 32 ? fs.sums[lane & (kSpThreads / 32 - 1)] : 0u);
  if (above < k && k <= above + all) {
    int row = kRows - 1;
    uint4 v = c[kRows - 1];
#pragma unroll
    for (int j = kRows - 1; j > 0; --j)
      if (row == j && above + rows[j] < k) {
        above += rows[j];
        row = j - 1;
        v = c[j - 1];
      }
    const uint32_t mine = v.x + v.y + v.z + v.w;
    uint32_t suffix = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_down_sync(0xffffffffu, suffix, o);
      if (lane + o < 32) suffix += y;
    }
    above += suffix - mine;   // in the bins of higher lanes too
    if (above < k && k <= above + mine) {
      uint32_t b = 3;
      if (above + v.w < k) { above += v.w; b = 2;
        if (above + v.z < k) { above += v.z; b = 1;
          if (above + v.y < k) { above += v.y; b = 0; } } }
      fs.res = make_uint2(warp * (kRows * 128) + row * 128 + lane * 4 + b, k - above);
    }
  }
  __syncthreads();
  const uint2 r = fs.res;
  bin = r.x;
  krem = r.y;
  __syncthreads();
}

__device__ __forceinline__ void flush_hist(const uint32_t* sh, uint32_t* __restrict__ gh) {
#pragma unroll
  for (int i = 0; i < kBins / 4; i += kSpThreads) {
    const uint4 c = reinterpret_cast<const uint4*>(sh)[i + threadIdx.x];
    uint32_t* to = gh + 4 * (i + threadIdx.x);
    if (c.x) atomicAdd(to, c.x);
    if (c.y) atomicAdd(to + 1, c.y);
    if (c.z) atomicAdd(to + 2, c.z);
    if (c.w) atomicAdd(to + 3, c.w);
  }
}

__device__ __forceinline__ float4 ld4(const float* p, uint64_t i, uint64_t n, bool vec) {
  if (vec && i + 3 < n) return *reinterpret_cast<const float4*>(p + i);
  float4 v;
  v.x = i < n ? p[i] : 0.0f;
  v.y = i + 1 < n ? p[i + 1] : 0.0f;
  v.z = i + 2 < n ? p[i + 2] : 0.0f;
  v.w = i + 3 < n ? p[i + 3] : 0.0f;
  return v;
}
__device__ __forceinline__ void st4(float* p, uint64_t i, uint64_t n, bool vec, float4 v) {
  if (vec && i + 3 < n) {
    *reinterpret_cast<float4*>(p + i) = v;
    return;
  }
  if (i < n) p[i] = v.x;
  if (i + 1 < n) p[i + 1] = v.y;
  if (i + 2 < n) p[i + 2] = v.z;
  if (i + 3 < n) p[i + 3] = v.w;
}

// MODE 0: select only (a already holds the accumulator)
// MODE 1: GradDrop  a += g
// MODE 2: DGC       u = m*u + g ; a += u
template <int MODE>
static __device__ __noinline__ void pass0_body(const float* __restrict__ g, float* __restrict__ a,
                                           float* __restrict__ u, uint64_t n, float momentum,
                                           uint32_t* __restrict__ ws, uint32_t* sh, uint32_t cta,
                                           uint32_t nctas) {
  for (int i = threadIdx.x; i < kBins; i += kSpThreads) sh[i] = 0;
  __syncthreads();
  const bool vec = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(g) |
                     reinterpret_cast<uintptr_t>(u)) & 15) == 0;
  const uint64_t stride = (uint64_t)nctas * kSpThreads * 4;
  for (uint64_t i = ((uint64_t)cta * kSpThreads + threadIdx.x) * 4; i < n; i += stride) {
    float4 av = ld4(a, i, n, vec);
    if (MODE == 1) {
      const float4 gv = ld4(g, i, n, vec);
      av.x = av.x + gv.x; av.y = av.y + gv.y; av.z = av.z + gv.z; av.w = av.w + gv.w;
      st4(a, i, n, vec, av);
    } else if (MODE == 2) {
      const float4 gv = ld4(g, i, n, vec);
      float4 uv = ld4(u, i, n, vec);
      uv.x = __fmaf_rn(momentum, uv.x, gv.x);
      uv.y = __fmaf_rn(momentum, uv.y, gv.y);
      uv.z = __fmaf_rn(momentum, uv.z, gv.z);
      uv.w = __fmaf_rn(momentum, uv.w, gv.w);
      av.x = av.x + uv.x; av.y = av.y + uv.y; av.z = av.z + uv.z; av.w = av.w + uv.w;
      st4(u, i, n, vec, uv);
      st4(a, i, n, vec, av);
    }
    const float e[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q < n) atomicAdd(&sh[abs_key(e[q]) >> 19], 1u);
  }
  __syncthreads();
  flush_hist(sh, ws);
}

// One copy of the code for both digit passes (PASS is a run-time value) and one per
// body below: the persistent kernels call every body from several phases, and inlined
// copies made them so large that cold instruction fetches showed in the phase times.
static __device__ __noinline__ void pass_body(int PASS, const float* __restrict__ a, uint64_t n,
                                          uint32_t k, uint32_t* __restrict__ ws, uint32_t* sh,
                                          FindSmem& fs, uint32_t cta, uint32_t nctas) {
  for (int i = threadIdx.x; i < kBins; i += kSpThreads) sh[i] = 0;
  uint32_t bin0, k1, bin1 = 0, k2;
  find_bin(ws, k, fs, bin0, k1);
  if (PASS == 2) find_bin(ws + kBins, k1, fs, bin1, k2);
  const uint32_t prefix = PASS == 1 ? bin0 : ((bin0 << 11) | bin1);
  const int shift = PASS == 1 ? 19 : 8;
  const bool vec = (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  // four independent 16-byte loads per thread in flight
  const uint64_t tiles = (n + kSpTile - 1) / kSpTile;
  for (uint64_t t = cta; t < tiles; t += nctas) {
    float4 av[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      av[j] = ld4(a, t * kSpTile + (uint64_t)(j * kSpThreads + threadIdx.x) * 4, n, vec);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t i = t * kSpTile + (uint64_t)(j * kSpThreads + threadIdx.x) * 4;
      const float e[4] = {av[j].x, av[j].y, av[j].z, av[j].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t key = abs_key(e[q]);
        if (i + q < n && (key >> shift) == prefix) atomicAdd(&sh[digit_of(key, PASS)], 1u);
      }
    }
  }
  __syncthreads();
  flush_hist(sh, ws + PASS * kBins);
}
struct EmitSmem {
  uint32_t warp_tot[kSpThreads / 32];
  uint32_t base_gt;
  uint32_t base_eq;
  uint32_t tot;
};

// Where the pairs go: one payload per destination (several for a broadcast), which may be
// peer GPUs' memory, and on this GPU straight into an accumulator (`add`) or into the
// cleared result (`set`, scaled), with no payload in between.
struct EmitDst {
  uint8_t* out[HP_MAX_RANKS];
  int n;
  float* add;
  float* set;
  float scale;
};
// store one pair at place `pos` of every destination
__device__ __forceinline__ void put_pair(const EmitDst& dst, size_t val_off, uint32_t kmax, uint32_t pos,
                                         uint32_t idx, float val) {
  if (pos >= kmax) return;
#pragma unroll 1
  for (int d = 0; d < dst.n; ++d) {
    reinterpret_cast<uint32_t*>(dst.out[d] + 16)[pos] = idx;
    reinterpret_cast<float*>(dst.out[d] + val_off)[pos] = val;
  }
  if (dst.add) atomicAdd(dst.add + idx, val);
  if (dst.set) dst.set[idx] = val * dst.scale;
}

// Compaction of the whole array, a tile per CTA iteration, 16 elements per thread.
// Returns true in thread 0 of the CTA that finished last, after it wrote the headers.
static __device__ __noinline__ bool emit_body(int alg, float* __restrict__ a, float* __restrict__ u,
                                          uint64_t n, uint32_t k, uint32_t kmax, const EmitDst& dst,
                                          uint32_t* __restrict__ ws, FindSmem& fs, EmitSmem& es,
                                          uint32_t cta, uint32_t nctas) {
  uint32_t bin0, k1, bin1, k2, bin2, need_eq;
  find_bin(ws, k, fs, bin0, k1);
  find_bin(ws + kBins, k1, fs, bin1, k2);
  find_bin(ws + 2 * kBins, k2, fs, bin2, need_eq);
  const uint32_t thr = (bin0 << 19) | (bin1 << 8) | bin2;
  if (thr == 0) need_eq = 0;  // zeros are never sent
  const size_t val_off = 16 + align_up(4ull * kmax, 16);
  const bool vec = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(u)) & 15) == 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  const uint64_t tiles = (n + kSpTile - 1) / kSpTile;
  for (uint64_t t = cta; t < tiles; t += nctas) {
    // The loops over a thread's 16 elements stay rolled (and the second one loads the
    // values again, from cache) on purpose: this body runs once or a few times per
    // launch, so its time is instruction fetch, not arithmetic -- fully unrolled it
    // took 13 us per tile, most of it waiting for code.
    uint32_t flag = 0;  // 2 bits per element: bit0 greater, bit1 equal
    uint32_t cnt = 0;   // low 16: greater, high 16: equal
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const uint64_t i = t * kSpTile + (uint64_t)(j * kSpThreads + threadIdx.x) * 4;
      const float4 av = ld4(a, i, n, vec);
      const float e4[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t key = abs_key(e4[q]);
        if (i + q < n) {
          if (key > thr) { flag |= 1u << (2 * (4 * j + q)); cnt += 1u; }
          else if (key == thr && need_eq) { flag |= 2u << (2 * (4 * j + q)); cnt += 1u << 16; }
        }
      }
    }
    // block exclusive scan of the packed counts
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) es.warp_tot[warp] = inc;
    __syncthreads();
    uint32_t wbase = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < kSpThreads / 32; ++w) {
      const uint32_t wt = es.warp_tot[w];
      if (w < warp) wbase += wt;
      tot += wt;
    }
    const uint32_t excl = wbase + inc - cnt;
    if (tot == 0) {       // uniform across the CTA
      __syncthreads();
      continue;
    }
    const uint32_t tot_gt = tot & 0xFFFFu, tot_eq = tot >> 16;
    if (threadIdx.x == 0) {
      uint32_t acc_eq = 0, beq = 0;
      if (tot_eq) {
        beq = atomicAdd(ws + kWsTieCount, tot_eq);
        acc_eq = beq >= need_eq ? 0u : min(tot_eq, need_eq - beq);
      }
      es.base_eq = acc_eq;  // number of ties this tile may send
      es.base_gt = (tot_gt + acc_eq) ? atomicAdd(ws + kWsOutCount, tot_gt + acc_eq) : 0u;
    }
    __syncthreads();
    const uint32_t base = es.base_gt, acc_eq = es.base_eq;
    uint32_t pg = base + (excl & 0xFFFFu);             // next slot for a "greater" element
    uint32_t rank_eq = excl >> 16;                     // tie rank inside this tile
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const uint32_t fj = (flag >> (8 * j)) & 255u;
      if (fj == 0) continue;
      const uint64_t i = t * kSpTile + (uint64_t)(j * kSpThreads + threadIdx.x) * 4;
      const float4 av = ld4(a, i, n, vec);
      const float e4[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t f = (fj >> (2 * q)) & 3u;
        uint32_t pos = 0xFFFFFFFFu;
        if (f & 1u) pos = pg++;
        else if (f & 2u) {
          if (rank_eq < acc_eq) pos = base + tot_gt + rank_eq;
          ++rank_eq;
        }
        if (pos < kmax) {
          put_pair(dst, val_off, kmax, pos, (uint32_t)(i + q), e4[q]);
          a[i + q] = 0.0f;
          if (u) u[i + q] = 0.0f;
        }
      }
    }
    __syncthreads();
  }
  // last CTA writes the header
  __syncthreads();
  if (threadIdx.x == 0) {
    // device scope is enough here: the one thread that finds itself last publishes
    // the unit (header, then a system-scope release of the flag by the caller), and
    // release is cumulative over what it has observed through this counter
    __threadfence();
    const uint32_t ticket = atomicAdd(ws + kWsDone, 1u);
    if (ticket == nctas - 1) {
      __threadfence();
      const uint32_t sent = atomicAdd(ws + kWsOutCount, 0u);
      WireHeader h;
      h.n = (uint32_t)n;
      h.alg = (uint8_t)alg;
      h.bitwidth = 0;
      h.flags = 0;
      h.a = __uint_as_float(thr);
      h.b = sent < kmax ? sent : kmax;
      for (int d = 0; d < dst.n; ++d)
        *reinterpret_cast<uint4*>(dst.out[d]) = *reinterpret_cast<const uint4*>(&h);
      return true;
    }
  }
  return false;
}

// ---------------------------------------------------------------------------
// Exact top-k with ONE pass over the arrays.  A selection used to read the accumulator
// again after the update to split it at a threshold bin, and every element went through
// a shared-memory histogram; both are gone:
//
//   sample   every stride-th tile of the array is updated first; each contributes its
//            largest keys to a short list, and the element of the rank that k scales to
//            (with a margin) is `low`, below which an element is almost surely not among
//            the k largest and above which about 1.1 to 1.5 k are.  Exact keys, not a
//            histogram: an accumulator in steady state is dense just below the last
//            threshold, and a bin there can hold many times k elements.
//   collect  the other tiles are updated; elements of at least `low` are appended to a
//            candidate list with a histogram of their distance from `low` (the sampled
//            tiles' from shared memory).  The list holds the k largest exactly when it
//            has k elements.
//   emit     every CTA takes a slice of the list, sends what lies above the histogram bin
//            of the k-th largest and moves what lies in that bin to a second list, a few
//            dozen elements; the CTA that comes last selects exactly among those and
//            writes the header.
//
// State is read and written once: HBM bound at 20 bytes per element for DGC, 12 for
// GradDrop (encodes at 0.1 %: DGC 5.2 TB/s of those bytes at 67 M elements, GradDrop 3.6
// and 4.8 at 25 M and 67 M; the kernel of a PS bucket with ResNet-50's 25.5 M elements takes
// 182 us, 98 of them this pass over its arrays).  A list that came out shorter than k or
// longer than its room (a sample that misled, or massive ties) makes the launch fall back
// to histogram passes over the whole array.
//
// Up to a few million elements the time is a chain of latencies instead: two grid
// barriers, and steps of a few dependent L2 accesses each (about 0.7 us an atomic).  So
// bins are fine where the k-th largest is to be expected, which leaves one digit to
// resolve; counters that are read together lie together; and slices send without a
// barrier behind the histogram.
constexpr uint32_t kMinSampled = 4;     // tiles of an array that are sampled at least
constexpr uint32_t kMaxSampled = 128;   // and at most: 0.5 M elements
constexpr uint32_t kSelTile = 8 * kSpThreads;  // elements per tile: two float4 of each array per thread

// One array to select from.
struct SelUnit {
  const float* g;
  float* a;
  float* u;
  float* clear;    // result that the update clears behind its reads (it may be g), or null
  uint32_t* ws;
  float* cv;       // candidate list: `cap` values, then `cap` indices; a second list of the
                   // same size behind it
  uint32_t n, k, kmax, cap;
  uint32_t stride, sampled;  // every stride-th tile is sampled: how many that is
  uint32_t top;              // keys a sampled tile contributes at least
  uint32_t run;              // tiles between two looks at the candidates' buffer
  uint32_t low;              // the candidates' lower bound, once the sample is complete
};
__device__ __forceinline__ uint32_t* list_indices(const SelUnit& s) { return reinterpret_cast<uint32_t*>(s.cv + s.cap); }
__device__ __forceinline__ float* list2_values(const SelUnit& s) { return s.cv + 2 * (size_t)s.cap; }
__device__ __forceinline__ uint32_t* list2_indices(const SelUnit& s) {
  return reinterpret_cast<uint32_t*>(s.cv + 3 * (size_t)s.cap);
}
// room of each of the two lists in `pairs` pairs
HP_HD uint32_t list_cap(uint64_t pairs) { return (uint32_t)(pairs / 2 < 0x7FFFFFFFull ? pairs / 2 : 0x7FFFFFFFull); }
// How an array is sampled when ctas CTAs share `total` tiles: about one tile for every
// CTA, and no more than leaves every tile room for several times the keys it will hold of
// the k largest (`top`), and half as many again.
// `run`: tiles after which a CTA looks whether its candidates have to leave its buffer,
// such that they seldom find it full (then each takes an atomic on the list's counter).
constexpr int kCollectBuf = 1024;  // candidates a CTA gathers before it reserves room in the lists
struct Sampling {
  uint32_t stride, top, run;
};
HP_HD Sampling sampling(uint32_t tiles, uint64_t total, uint32_t ctas, uint64_t n, uint64_t k) {
  const uint64_t hits = n && k ? (kSelTile * k + n - 1) / n : 1;   // of one tile among the k largest
  Sampling p;
  p.top = (uint32_t)(24 + 4 * hits < kSelTile / 2 ? 24 + 4 * hits : kSelTile / 2);
  p.run = (uint32_t)(kCollectBuf / 4 / hits < 2 ? 2 : kCollectBuf / 4 / hits) & ~1u;
  uint64_t share = ((uint64_t)tiles * ctas) / (total ? total : 1);
  if (share > kMaxKeys * 2 / 3 / p.top) share = kMaxKeys * 2 / 3 / p.top;   // `top` rounded up to whole bins
  if (share < kMinSampled) share = kMinSampled;
  if (share > kMaxSampled) share = kMaxSampled;
  p.stride = share >= tiles ? 1u : (uint32_t)((tiles + share - 1) / share);
  return p;
}

// First digit of a candidate.  Its distance from `low` in steps of 2^10 keys (1/8192 of
// the magnitude), the last bin for everything more than half an octave above, where the
// k-th largest is not to be expected.  Finer than needed to find the k-th: the counts of
// most candidates fall within a few percent above `low`, and the atomics on neighbouring
// words follow one another (steps of 2^12 took 320 us instead of 187 for 1 % of 67 M).
// When all non-zero elements are candidates (low == 1) they may span any range: the
// leading 12 bits then.
__device__ __forceinline__ uint32_t cand_digit(uint32_t key, uint32_t low) {
  return low <= 1u ? key >> 19 : min((key - low) >> 10, (uint32_t)kBins - 1u);
}

// counters that are read together behind the update pass
struct ListState {
  uint32_t count, overflow, low;
};
__device__ __forceinline__ ListState list_state(const SelUnit& s) {
  const uint4 v = __ldcg(reinterpret_cast<const uint4*>(s.ws + kWsCandCount));
  return {v.x, v.y, v.z};
}
// the list lacks some of the k largest
__device__ __forceinline__ bool selection_failed(const SelUnit& s, const ListState& l) {
  return l.overflow != 0u || (l.count < s.k && l.low > 1u);
}

struct SelSmem {
  union {
    uint32_t hist[kBins];            // sample; emit: the last digits
    struct {
      float val[kCollectBuf];
      uint32_t idx[kCollectBuf];
      uint16_t unit[kCollectBuf];
    } buf;                           // collect
  };
  float stash[2][kSelTile];          // sample to collect
  FindSmem fs;
  uint32_t count, base, base2, ticket, flag;
  uint32_t sent, ties;
};

__device__ __forceinline__ void clear_hist(uint32_t* sh) {
#pragma unroll
  for (int b = 0; b < kBins / 4; b += kSpThreads)
    reinterpret_cast<uint4*>(sh)[b + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
}

// Loads T consecutive tiles from t and applies the update (MODE as in pass0_body), all
// loads before the first store.  Tiles not in `mask` are left out; what lies past the end
// reads as zero, and a zero is never sent.
template <int MODE, int T, bool FULL>
__device__ __forceinline__ void update_tiles_impl(const SelUnit& s, float momentum, uint64_t i0, bool vec,
                                                  uint32_t mask, float4 (&av)[2 * T]) {
  auto on = [&](int j) { return FULL || (mask >> (j / 2) & 1u); };
  auto ld4 = [&](const float* p, uint64_t i, uint32_t n, bool v) {
    return FULL ? *reinterpret_cast<const float4*>(p + i) : hipress::ld4(p, i, n, v);
  };
  auto st4 = [&](float* p, uint64_t i, uint32_t n, bool v, const float4& x) {
    if (FULL) *reinterpret_cast<float4*>(p + i) = x;
    else hipress::st4(p, i, n, v, x);
  };
  float4 gv[2 * T], uv[2 * T];
#pragma unroll
  for (int j = 0; j < 2 * T; ++j) {
    const uint64_t i = i0 + j * kSpThreads * 4;
    av[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!on(j)) continue;
    av[j] = ld4(s.a, i, s.n, vec);
    if (MODE >= 1) gv[j] = ld4(s.g, i, s.n, vec);
    if (MODE == 2) uv[j] = ld4(s.u, i, s.n, vec);
  }
#pragma unroll
  for (int j = 0; j < 2 * T; ++j) {
    const uint64_t i = i0 + j * kSpThreads * 4;
    float4& v = av[j];
    if (!on(j)) continue;
    if (MODE == 1) {
      v.x = v.x + gv[j].x; v.y = v.y + gv[j].y; v.z = v.z + gv[j].z; v.w = v.w + gv[j].w;
      st4(s.a, i, s.n, vec, v);
    } else if (MODE == 2) {
      float4 w;
      w.x = __fmaf_rn(momentum, uv[j].x, gv[j].x);
      w.y = __fmaf_rn(momentum, uv[j].y, gv[j].y);
      w.z = __fmaf_rn(momentum, uv[j].z, gv[j].z);
      w.w = __fmaf_rn(momentum, uv[j].w, gv[j].w);
      v.x = v.x + w.x; v.y = v.y + w.y; v.z = v.z + w.z; v.w = v.w + w.w;
      st4(s.u, i, s.n, vec, w);
      st4(s.a, i, s.n, vec, v);
    }
  }
  if (MODE >= 1 && s.clear) {
#pragma unroll
    for (int j = 0; j < 2 * T; ++j)
      if (on(j)) st4(s.clear, i0 + j * kSpThreads * 4, s.n, vec, make_float4(0.f, 0.f, 0.f, 0.f));
  }
}
template <int MODE, int T>
__device__ __forceinline__ void update_tiles(const SelUnit& s, float momentum, uint32_t t, uint32_t mask,
                                             float4 (&av)[2 * T]) {
  const bool vec = ((reinterpret_cast<uintptr_t>(s.a) | (MODE >= 1 ? reinterpret_cast<uintptr_t>(s.g) : 0) |
                     (MODE >= 1 ? reinterpret_cast<uintptr_t>(s.clear) : 0) |
                     (MODE == 2 ? reinterpret_cast<uintptr_t>(s.u) : 0)) & 15) == 0;
  const uint64_t i0 = (uint64_t)t * kSelTile + threadIdx.x * 4;
  // one test for the tiles: with one per load the loads did not overlap as they should
  if (vec && mask == (1u << T) - 1u && (uint64_t)(t + T) * kSelTile <= s.n)
    update_tiles_impl<MODE, T, true>(s, momentum, i0, vec, mask, av);
  else
    update_tiles_impl<MODE, T, false>(s, momentum, i0, vec, mask, av);
}

// Sampled tile number i of an array: update, values into `stash`, the largest keys into
// the array's list.  The CTA that completes the sample picks the candidates' lower bound.
template <int MODE>
static __device__ __noinline__ void sample_body(const SelUnit& s, float momentum, SelSmem& sm, uint32_t i,
                                                float* stash) {
  clear_hist(sm.hist);
  float4 av[2];
  update_tiles<MODE, 1>(s, momentum, i * s.stride, 1u, av);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    reinterpret_cast<float4*>(stash)[j * kSpThreads + threadIdx.x] = av[j];
    const float e[4] = {av[j].x, av[j].y, av[j].z, av[j].w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t key = abs_key(e[q]);
      if (key) atomicAdd(&sm.hist[key >> 19], 1u);
    }
  }
  if (threadIdx.x == 0) sm.count = 0;
  __syncthreads();
  uint32_t bin, rem;
  find_bin(sm.hist, s.top, sm.fs, bin, rem);   // bin 0 when the tile has fewer
  const uint32_t edge = bin ? bin << 19 : 1u;
  uint32_t at[8];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float e[4] = {av[j].x, av[j].y, av[j].z, av[j].w};
#pragma unroll
    for (int q = 0; q < 4; ++q) at[4 * j + q] = abs_key(e[q]) >= edge ? atomicAdd(&sm.count, 1u) : kMaxKeys;
  }
  // places of its own: a reservation behind 100 others took 2 us.  Keys that find no room
  // are left out, which lowers the bound: safe.
  const uint32_t room = kMaxKeys / s.sampled;
  uint32_t* keys = s.ws + kWsKeys;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float e[4] = {av[j].x, av[j].y, av[j].z, av[j].w};
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (at[4 * j + q] < room) keys[i * room + at[4 * j + q]] = abs_key(e[q]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t done;   // release the CTA's keys, acquire those of the CTAs before
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(done) : "l"(s.ws + kWsSampled) : "memory");
    sm.flag = done == s.sampled - 1;
  }
  __syncthreads();
  if (!sm.flag) return;
  // the CTA that completes the sample: the first 24 bits of the rank-th largest key
  uint32_t rank = s.k;
  if (s.stride > 1) {
    // k scaled to the sample, plus five standard deviations, plus a tenth because
    // neighbouring elements are not independent
    const float hits = __fdividef((float)s.k * (float)(s.sampled * kSelTile), (float)s.n);
    float dev;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(dev) : "f"(hits));
    rank = (uint32_t)(1.1f * hits + 5.0f * dev + 4.0f);
  }
  uint32_t prefix = 0, mine[kMaxKeys / kSpThreads];
#pragma unroll
  for (uint32_t q = 0; q < kMaxKeys / kSpThreads; ++q) mine[q] = __ldcg(keys + q * kSpThreads + threadIdx.x);
#pragma unroll 1
  for (int shift = 19; shift > 0; shift -= 12) {
    clear_hist(sm.hist);
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < kMaxKeys / kSpThreads; ++q)   // a place not taken holds zero
      if (mine[q] && (mine[q] >> shift >> 12) == prefix) atomicAdd(&sm.hist[(mine[q] >> shift) & (kBins - 1)], 1u);
    __syncthreads();
    find_bin(sm.hist, rank, sm.fs, bin, rem);
    if (rem == 0) break;   // fewer keys than that: all that is not zero is a candidate
    rank = rem;
    prefix = (prefix << 12) | bin;
  }
  const uint32_t low = rem ? max(prefix << 7, 1u) : 1u;
  if (threadIdx.x == 0) s.ws[kWsLow] = low;
}

// Items [0, total).  Below kShareAll per CTA in equal shares: the tickets of all CTAs
// follow one another, 25 ns each, and took longer than the SMs' unequal speed costs.
// Above, seven eighths in equal shares, the rest in short stretches taken from
// *word by whichever of the ctas CTAs is free -- SMs do not run at one speed, and equal
// shares alone leave the fast ones waiting, while handing out everything made the ticket
// word the bottleneck.  One array, 296 CTAs, us per launch with equal shares / handed out:
//   tiles per CTA          5.4        20.8       32.4       54         108         216
//   GradDrop encode      48.1/49.2  85.0/87.0  110/113    167/171    292/288     538/536
//   GradDrop, PS bucket  94.2/99.3  171/179    221/229    342/347    605/597    1142/1121
//   DGC, ring bucket     70.7/75.7  144/146    198/202    319/321    601/587    1160/1144
// At 81 tiles the two are within 2 % of one another, either way.  The next stretch is asked for before the current one is worked
// on, by predicated instructions (an `if` around them split thread 0 from its warp, and
// the two halves then counted twice at the barriers that follow).  f(lo, hi) runs with
// the whole CTA; `slot` is shared memory.
constexpr uint32_t kShareAll = 96;
template <typename F>
__device__ __forceinline__ void hand_out(uint32_t* word, uint32_t total, uint32_t cta, uint32_t ctas, uint32_t& slot,
                                         F f) {
  if (total < kShareAll * ctas) {
    const uint32_t lo = (uint32_t)((uint64_t)total * cta / ctas), hi = (uint32_t)((uint64_t)total * (cta + 1) / ctas);
    if (lo < hi) f(lo, hi);
    return;
  }
  const uint32_t share = total / ctas * 7u / 8u, dealt = share * ctas;
  uint32_t stretch = (total - dealt) / (2u * ctas) + 1u;
  if (stretch > 2u) stretch = (stretch + 2u) & ~3u;   // whole groups of tiles
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(&slot);
  uint32_t next = 0;
  auto take = [&] {
    asm volatile("{\n.reg .pred p;\nsetp.eq.u32 p, %1, 0;\n@p atom.add.relaxed.gpu.global.u32 %0, [%2], %3;\n}"
                 : "+r"(next) : "r"(threadIdx.x), "l"(word), "r"(stretch) : "memory");
  };
  take();
  uint32_t lo = cta * share, hi = lo + share;
#pragma unroll 1
  for (;;) {
    if (lo < hi) f(lo, hi);
    asm volatile("{\n.reg .pred p;\nsetp.eq.u32 p, %1, 0;\n@p st.shared.u32 [%2], %0;\n}" ::"r"(next),
                 "r"(threadIdx.x), "r"(at) : "memory");
    __syncthreads();
    lo = dealt + *(volatile uint32_t*)&slot;
    __syncthreads();
    if (lo >= total) break;
    hi = min(lo + stretch, total);
    take();
  }
}

// one candidate into the CTA's buffer, or, when that is full, straight into its list
__device__ __forceinline__ void collect_one(const SelUnit& s, uint32_t uid, SelSmem& sm, uint32_t low, float v,
                                            uint32_t i) {
  const uint32_t p = atomicAdd(&sm.count, 1u);
  if (p < (uint32_t)kCollectBuf) {
    sm.buf.val[p] = v;
    sm.buf.idx[p] = i;
    sm.buf.unit[p] = (uint16_t)uid;
    return;
  }
  const uint32_t pos = atomicAdd(s.ws + kWsCandCount, 1u);
  atomicAdd(s.ws + cand_digit(abs_key(v), low), 1u);
  if (pos < s.cap) {
    s.cv[pos] = v;
    list_indices(s)[pos] = i;
  } else {
    s.ws[kWsOverflow] = 1u;
  }
}
// the elements of T tiles that reach `low`
template <int T>
__device__ __forceinline__ void collect_tiles(const SelUnit& s, uint32_t uid, SelSmem& sm, uint32_t t,
                                              const float4 (&av)[2 * T]) {
  const uint32_t low = s.low;
#pragma unroll
  for (int j = 0; j < 2 * T; ++j) {
    const float e[4] = {av[j].x, av[j].y, av[j].z, av[j].w};
    const uint32_t most = max(max(abs_key(e[0]), abs_key(e[1])), max(abs_key(e[2]), abs_key(e[3])));
    if (most < low) continue;
    const uint32_t i = t * kSelTile + (j * kSpThreads + threadIdx.x) * 4;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (abs_key(e[q]) >= low) collect_one(s, uid, sm, low, e[q], i + q);
  }
}

// Tiles [t0, t1) of one array without the sampled ones, T at a time: 4 to 6 loads of
// 16 bytes per thread are what keeps HBM busy with 32 warps per SM.
template <int MODE>
static __device__ __noinline__ void collect_body(const SelUnit& s, uint32_t uid, float momentum, SelSmem& sm,
                                                 uint32_t t0, uint32_t t1) {
  constexpr uint32_t T = MODE == 0 ? 2 : 1;
  uint32_t phase = t0 % s.stride;   // 0: a sampled tile
#pragma unroll 1
  for (uint32_t t = t0; t < t1; t += T) {
    uint32_t mask = 0;
#pragma unroll
    for (uint32_t q = 0; q < T; ++q) {
      if (phase != 0 && t + q < t1) mask |= 1u << q;
      if (++phase == s.stride) phase = 0;
    }
    float4 av[2 * T];
    update_tiles<MODE, T>(s, momentum, t, mask, av);
    collect_tiles<T>(s, uid, sm, t, av);
  }
}

// Sampled tile number i again, updated before: from its stash, or (again) read once more.
static __device__ __noinline__ void collect_sampled(const SelUnit& s, uint32_t uid, SelSmem& sm, uint32_t i,
                                                    const float* stash, bool again) {
  const uint32_t t = i * s.stride;
  float4 av[2];
  if (again) {
    update_tiles<0, 1>(s, 0.0f, t, 1u, av);
  } else {
#pragma unroll
    for (int j = 0; j < 2; ++j) av[j] = reinterpret_cast<const float4*>(stash)[j * kSpThreads + threadIdx.x];
  }
  collect_tiles<1>(s, uid, sm, t, av);
}

// Append the CTA's gathered candidates to their lists, and their first digits to the
// lists' histograms.  A warp's entries mostly belong to one list: one reservation for each
// group of lanes with the same list.  unit(uid) gives the array.
template <typename F>
__device__ __forceinline__ void collect_flush(SelSmem& sm, F unit) {
  __syncthreads();
  const uint32_t n = min(sm.count, (uint32_t)kCollectBuf);
  bool same = true;
#pragma unroll
  for (uint32_t p = threadIdx.x; p < (uint32_t)kCollectBuf; p += kSpThreads) same &= p >= n || sm.buf.unit[p] == sm.buf.unit[0];
  if (__syncthreads_and(same)) {   // one reservation for the CTA
    if (threadIdx.x == 0 && n) sm.base = atomicAdd(unit(sm.buf.unit[0]).ws + kWsCandCount, n);
    const SelUnit& s = unit(n ? sm.buf.unit[0] : 0u);
    const uint32_t low = s.low;
    __syncthreads();
#pragma unroll 1
    for (uint32_t p = threadIdx.x; p < n; p += kSpThreads) {
      const float v = sm.buf.val[p];
      const uint32_t pos = sm.base + p;
      atomicAdd(s.ws + cand_digit(abs_key(v), low), 1u);
      if (pos < s.cap) {
        s.cv[pos] = v;
        list_indices(s)[pos] = sm.buf.idx[p];
      } else {
        s.ws[kWsOverflow] = 1u;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) sm.count = 0;
    __syncthreads();
    return;
  }
#pragma unroll 1
  for (uint32_t p0 = 0; p0 < n; p0 += kSpThreads) {
    const uint32_t p = p0 + threadIdx.x;
    const bool have = p < n;
    const uint32_t mask = __ballot_sync(0xffffffffu, have);
    if (have) {
      const uint32_t uid = sm.buf.unit[p], lane = threadIdx.x & 31;
      const float v = sm.buf.val[p];
      const SelUnit& s = unit(uid);
      const uint32_t low = s.low;
      const uint32_t group = __match_any_sync(mask, uid);
      const int lead = __ffs(group) - 1;
      uint32_t pos = 0;
      if ((int)lane == lead) pos = atomicAdd(s.ws + kWsCandCount, (uint32_t)__popc(group));
      atomicAdd(s.ws + cand_digit(abs_key(v), low), 1u);
      pos = __shfl_sync(group, pos, lead) + __popc(group & ((1u << lane) - 1u));
      if (pos < s.cap) {
        s.cv[pos] = v;
        list_indices(s)[pos] = sm.buf.idx[p];
      } else {
        s.ws[kWsOverflow] = 1u;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) sm.count = 0;
  __syncthreads();
}

// CTAs that share a list of L elements
__device__ __forceinline__ uint32_t emit_slices(uint32_t L, uint32_t most) {
  const uint32_t n = L / kSpThreads + 1u;
  return n < most ? n : most;
}

// Places [lo, hi) of one array's candidate list, one of nx spans.  True in thread 0 of the CTA that finished
// last, behind the headers.
// A CTA whose barrier expired goes on, and may have read another count than the others:
// their slices then overlap, and together hold more than the lists have room for.  So a
// list is read up to its room and no further, and so is the second one written.
static __device__ __noinline__ bool emit_span(int alg, const SelUnit& s, const ListState& ls, const EmitDst& dst,
                                              SelSmem& sm, uint32_t lo, uint32_t hi, uint32_t nx) {
  const uint32_t L = min(ls.count, s.cap), low = ls.low;   // no overflow: the list holds all of them
  const size_t val_off = 16 + align_up(4ull * s.kmax, 16);
  const bool every = L <= s.k;                 // all candidates are sent
  uint32_t bin0 = 0, rem = 0, least = 0xFFFFFFFFu;
  if (!every) find_bin(s.ws, s.k, sm.fs, bin0, rem);
  // four candidates per thread: the reservations of all CTAs on the two counters follow
  // one another, 25 ns each
  constexpr int kPer = 4;
#pragma unroll 1
  for (uint32_t p0 = lo; p0 < hi; p0 += kPer * kSpThreads) {
    if (threadIdx.x == 0) sm.sent = sm.ties = 0;
    __syncthreads();
    float v[kPer];
    uint32_t idx[kPer], at[kPer];   // place of those sent, behind kKeep of those kept
    constexpr uint32_t kKeep = 0x80000000u, kNone = 0xFFFFFFFFu;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const uint32_t p = p0 + q * kSpThreads + threadIdx.x;
      v[q] = p < hi ? __ldcg(s.cv + p) : 0.0f;
      idx[q] = p < hi ? __ldcg(list_indices(s) + p) : 0u;
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      at[q] = kNone;
      if (p0 + q * kSpThreads + threadIdx.x < hi) {
        const uint32_t key = abs_key(v[q]), d = cand_digit(key, low);
        least = min(least, key);
        if (every || d > bin0) at[q] = atomicAdd(&sm.sent, 1u);
        else if (d == bin0) at[q] = kKeep | atomicAdd(&sm.ties, 1u);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0 && sm.sent) sm.base = atomicAdd(s.ws + kWsOutCount, sm.sent);
    if (threadIdx.x == 32 && sm.ties) sm.base2 = atomicAdd(s.ws + kWsCand2Count, sm.ties);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      if (at[q] == kNone) continue;
      if (at[q] & kKeep) {
        const uint32_t pos = sm.base2 + (at[q] & ~kKeep);
        if (pos < s.cap) {
          list2_values(s)[pos] = v[q];
          list2_indices(s)[pos] = idx[q];
        }
      } else if (idx[q] < s.n) {
        put_pair(dst, val_off, s.kmax, sm.base + at[q], idx[q], v[q]);
        s.a[idx[q]] = 0.0f;
        if (s.u) s.u[idx[q]] = 0.0f;
      }
    }
  }
  if (every) {   // the least key sent is the threshold: kept as the largest complement
    least = __reduce_min_sync(0xffffffffu, least);
    if ((threadIdx.x & 31) == 0) atomicMax(s.ws + kWsTieCount, ~least);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t done;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(done) : "l"(s.ws + kWsDone) : "memory");
    sm.flag = done == nx - 1;
  }
  __syncthreads();
  if (!sm.flag) return false;
  // The last CTA: among the elements of the k-th's bin, `rem` are sent.  What is left of
  // their keys is 10 bits in a fine bin, 19 in a bin of the leading bits, and up to 31 in
  // the last fine bin.
  const uint32_t L2 = every ? 0u : min(__ldcg(s.ws + kWsCand2Count), s.cap);
  if (threadIdx.x == 0) sm.sent = __ldcg(s.ws + kWsOutCount), sm.ties = 0;
  const uint32_t start = low <= 1u ? bin0 << 19 : low + (bin0 << 10);
  int shift = low <= 1u ? 7 : (bin0 == (uint32_t)kBins - 1u ? 19 : 0), bits = 12;
  uint32_t prefix = 0;
  const bool pick = L2 != 0u;
  if (pick) {
#pragma unroll 1
    for (;;) {
      clear_hist(sm.hist);
      __syncthreads();
#pragma unroll 1
      for (uint32_t p = threadIdx.x; p < L2; p += kSpThreads) {
        const uint32_t rest = abs_key(__ldcg(list2_values(s) + p)) - start;
        if ((rest >> shift >> bits) == prefix) atomicAdd(&sm.hist[(rest >> shift) & ((1u << bits) - 1u)], 1u);
      }
      __syncthreads();
      uint32_t b;
      find_bin(sm.hist, rem, sm.fs, b, rem);
      prefix = (prefix << bits) | b;
      if (shift == 0) break;
      bits = shift == 19 ? 12 : 7;
      shift = shift == 19 ? 7 : 0;
    }
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t p = threadIdx.x; p < L2; p += kSpThreads) {
    const float v = __ldcg(list2_values(s) + p);
    const uint32_t idx = __ldcg(list2_indices(s) + p), rest = abs_key(v) - start;
    bool send = rest > prefix;
    if (rest == prefix) send = atomicAdd(&sm.ties, 1u) < rem;
    if (send && idx < s.n) {
      put_pair(dst, val_off, s.kmax, atomicAdd(&sm.sent, 1u), idx, v);
      s.a[idx] = 0.0f;
      if (s.u) s.u[idx] = 0.0f;
    }
  }
  __syncthreads();
  if (threadIdx.x != 0) return false;
  WireHeader h;
  h.n = s.n;
  h.alg = (uint8_t)alg;
  h.bitwidth = 0;
  h.flags = 0;
  // zero when fewer than k are not zero
  h.a = __uint_as_float(!every ? start + prefix : (L < s.k ? 0u : ~__ldcg(s.ws + kWsTieCount)));
  h.b = sm.sent < s.kmax ? sm.sent : s.kmax;
#pragma unroll 1
  for (int d = 0; d < dst.n; ++d) *reinterpret_cast<uint4*>(dst.out[d]) = *reinterpret_cast<const uint4*>(&h);
  return true;
}

// slice x of nx of a list without gaps
__device__ __forceinline__ bool emit_slice(int alg, const SelUnit& s, const ListState& ls, const EmitDst& dst, SelSmem& sm,
                                           uint32_t x, uint32_t nx) {
  const uint32_t L = min(ls.count, s.cap), per = (L + nx - 1) / nx, lo = min(x * per, L), hi = min(lo + per, L);
  return emit_span(alg, s, ls, dst, sm, lo, hi, nx);
}

// out[idx] (+)= val * scale ; indices come from another rank: bounds-checked
static __device__ __noinline__ void scatter_body(const uint8_t* __restrict__ payload,
                                             float* __restrict__ out, uint64_t n, uint32_t kmax,
                                             float scale, int accumulate, uint32_t cta,
                                             uint32_t nctas) {
  const WireHeader* h = reinterpret_cast<const WireHeader*>(payload);
  uint32_t k = __ldcg(&h->b);
  if (k > kmax) k = kmax;
  const uint32_t* idx = reinterpret_cast<const uint32_t*>(payload + 16);
  const float* val = reinterpret_cast<const float*>(payload + 16 + align_up(4ull * kmax, 16));
  for (uint32_t j = cta * kSpThreads + threadIdx.x; j < k; j += nctas * kSpThreads) {
    const uint32_t i = __ldcg(idx + j);
    const float d = __ldcg(val + j) * scale;
    if (i < n) {
      if (accumulate == 2) atomicAdd(out + i, d);  // several payloads may hit one index
      else out[i] = accumulate ? out[i] + d : d;
    }
  }
}

}  // namespace hipress
