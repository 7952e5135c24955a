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

constexpr int kSpThreads = 256;
constexpr int kBins = 4096;
// workspace words: 3 histograms, then counters
constexpr int kWsOutCount = 3 * kBins + 0;
constexpr int kWsTieCount = 3 * kBins + 1;
constexpr int kWsDone = 3 * kBins + 2;
constexpr int kWsCandCount = 3 * kBins + 3;   // candidates collected by the update pass
constexpr int kWsOverflow = 3 * kBins + 4;    // they did not fit: use the full passes
constexpr int kWsLow = 3 * kBins + 5;         // magnitude key from which an element is a candidate
constexpr int kWsSampled = 3 * kBins + 6;     // slices of the sample that are done
constexpr int kWsCand2Count = 3 * kBins + 7;  // candidates left after the first digit
constexpr int kWsTicket = 3 * kBins + 8;      // stand-alone kernel: tile ticket, status
constexpr int kWsStatus = 3 * kBins + 9;
constexpr int kWsWords = 3 * kBins + 16;

__device__ __forceinline__ uint32_t digit_of(uint32_t key, int pass) {
  return pass == 0 ? (key >> 19) : (pass == 1 ? ((key >> 8) & 0x7FFu) : (key & 0xFFu));
}

struct FindSmem {
  alignas(16) uint32_t counts[kBins / kSpThreads];
  uint32_t sums[kSpThreads / 32];
  uint32_t owner, above;
};

// Largest bin of a histogram of kBins bins whose suffix count reaches k, and krem = how
// many of the k fall in that bin, i.e. k - count(bins > bin); (0, 0) when fewer than k are
// counted.  `hist` is in shared or in global memory, where other CTAs' atomics wrote it.
// Thread t sums bins 16t .. 16t+15; the thread in whose bins the k-th lies hands its
// sixteen counts to everybody, and every warp finds the bin among them.
static __device__ __noinline__ void find_bin(const uint32_t* hist, uint32_t k, FindSmem& fs, uint32_t& bin,
                                             uint32_t& krem) {
  constexpr int per = kBins / kSpThreads;  // 16
  uint4 c[per / 4];
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < per / 4; ++i) {
    asm volatile("ld.volatile.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(c[i].x), "=r"(c[i].y), "=r"(c[i].z), "=r"(c[i].w)
                 : "l"(hist + threadIdx.x * per + 4 * i)
                 : "memory");
    sum += c[i].x + c[i].y + c[i].z + c[i].w;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t v = sum;   // suffix sum over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_down_sync(0xffffffffu, v, o);
    if (lane + o < 32) v += y;
  }
  if (lane == 0) fs.sums[warp] = v;
  if (threadIdx.x == 0) fs.owner = 0xFFFFFFFFu;
  __syncthreads();
  const uint32_t higher = lane > warp && lane < kSpThreads / 32 ? fs.sums[lane] : 0u;
  const uint32_t above = v - sum + __reduce_add_sync(0xffffffffu, higher);  // in the bins of higher threads
  if (above < k && k <= above + sum) {
    fs.owner = threadIdx.x;
    fs.above = above;
#pragma unroll
    for (int i = 0; i < per / 4; ++i) *reinterpret_cast<uint4*>(fs.counts + 4 * i) = c[i];
  }
  __syncthreads();
  const uint32_t owner = fs.owner;
  bin = krem = 0;
  if (owner != 0xFFFFFFFFu) {
    const uint32_t mine = lane < per ? fs.counts[lane & (per - 1)] : 0u;
    uint32_t w = mine;
#pragma unroll
    for (int o = 1; o < per; o <<= 1) {
      const uint32_t y = __shfl_down_sync(0xffffffffu, w, o);
      if (lane + o < per) w += y;
    }
    const uint32_t acc = fs.above + w - mine;
    const uint32_t hit = __ballot_sync(0xffffffffu, lane < per && acc < k && k <= acc + mine);
    const int at = __ffs(hit) - 1;
    bin = owner * per + at;
    krem = k - __shfl_sync(0xffffffffu, acc, at);
  }
  __syncthreads();
}

__device__ __forceinline__ void flush_hist(const uint32_t* sh, uint32_t* __restrict__ gh) {
#pragma unroll 1
  for (int i = threadIdx.x; i < kBins; i += kSpThreads) {
    const uint32_t c = sh[i];
    if (c) atomicAdd(gh + i, c);
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
static __device__ __noinline__ void pass_body_rt(int PASS, const float* __restrict__ a, uint64_t n,
                                          uint32_t k, uint32_t* __restrict__ ws, uint32_t* sh,
                                          FindSmem& fs, uint32_t cta, uint32_t nctas) {
  for (int i = threadIdx.x; i < kBins; i += kSpThreads) sh[i] = 0;
  uint32_t bin0, k1, bin1 = 0, k2;
  find_bin(ws, k, fs, bin0, k1);
  if (PASS == 2) find_bin(ws + kBins, k1, fs, bin1, k2);
  const uint32_t prefix = PASS == 1 ? bin0 : ((bin0 << 11) | bin1);
  const int shift = PASS == 1 ? 19 : 8;
  const bool vec = (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  // 4096-element tiles, four independent 16-byte loads per thread in flight
  const uint64_t tiles = (n + 4095) / 4096;
  for (uint64_t t = cta; t < tiles; t += nctas) {
    float4 av[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      av[j] = ld4(a, t * 4096 + (uint64_t)(j * kSpThreads + threadIdx.x) * 4, n, vec);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t i = t * 4096 + (uint64_t)(j * kSpThreads + threadIdx.x) * 4;
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
template <int PASS>
__device__ __forceinline__ void pass_body(const float* __restrict__ a, uint64_t n, uint32_t k,
                                          uint32_t* __restrict__ ws, uint32_t* sh, FindSmem& fs,
                                          uint32_t cta, uint32_t nctas) {
  pass_body_rt(PASS, a, n, k, ws, sh, fs, cta, nctas);
}

struct EmitSmem {
  uint32_t warp_tot[kSpThreads / 32];
  uint32_t base_gt;
  uint32_t base_eq;
  uint32_t tot;
};

// where the pairs go: one payload per destination (several for a broadcast);
// destinations may be peer GPUs' memory
struct EmitDst {
  uint8_t* out[HP_MAX_RANKS];
  int n;
};

// Compaction of the whole array.  Tile = 4096 elements per CTA iteration, 16 per thread.
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

  const uint64_t tiles = (n + 4095) / 4096;
  for (uint64_t t = cta; t < tiles; t += nctas) {
    // The loops over a thread's 16 elements stay rolled (and the second one loads the
    // values again, from cache) on purpose: this body runs once or a few times per
    // launch, so its time is instruction fetch, not arithmetic -- fully unrolled it
    // took 13 us per tile, most of it waiting for code.
    uint32_t flag = 0;  // 2 bits per element: bit0 greater, bit1 equal
    uint32_t cnt = 0;   // low 16: greater, high 16: equal
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const uint64_t i = t * 4096 + (uint64_t)(j * kSpThreads + threadIdx.x) * 4;
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
      const uint64_t i = t * 4096 + (uint64_t)(j * kSpThreads + threadIdx.x) * 4;
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
          for (int d = 0; d < dst.n; ++d) {
            reinterpret_cast<uint32_t*>(dst.out[d] + 16)[pos] = (uint32_t)(i + q);
            reinterpret_cast<float*>(dst.out[d] + val_off)[pos] = e4[q];
          }
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
//   sample   every stride-th tile of the array is updated first; the histogram of its
//            magnitudes gives a `low` below which an element is almost surely not among
//            the k largest, and above which about 1.1 to 1.7 k are
//   collect  the other tiles are updated; elements of at least `low` are appended to a
//            candidate list with the histogram of their first digit (the sampled tiles'
//            from shared memory).  The list holds the k largest exactly when it has k
//            elements.
//   finish   digit by digit on the list: the exact threshold, the pairs, the header.  A
//            long list first goes through one distributed step (refine) that sends what
//            lies above the first digit's bin and keeps what lies in it.
//
// State is read and written once: HBM bound at 20 bytes per element for DGC, 12 for
// GradDrop.  A list that came out shorter than k or longer than its room (a sample that
// misled, or massive ties) makes the launch fall back to histogram passes over the
// whole array.
//
// Up to a few million elements the time is not memory but instruction fetch: most of
// this code runs once or twice per launch, and code that is not in the instruction cache
// comes in at a few instructions per 0.1 us (one CTA on 4000 elements: 1900 instructions
// per warp took 25 us, half of all warp-cycles waiting for one).  Hence one out-of-line
// copy of every step, rolled loops where a step runs once, 32-bit arithmetic, and sizes
// worked out on the host.
constexpr uint32_t kFinishKeys = 8192;  // list length up to which a CTA keeps the keys in shared memory
constexpr uint32_t kFinishList = 12288; // longest list that is finished without a refine step
constexpr uint32_t kMinSampled = 4;     // tiles of an array that are sampled at least
constexpr uint32_t kSelTile = 4096;     // elements per tile: 16 per thread

// One array to select from.
struct SelUnit {
  const float* g;
  float* a;
  float* u;
  uint32_t* ws;
  float* cv;       // candidate list: `cap` values, then `cap` indices; a second list of the
                   // same size behind it
  uint32_t n, k, kmax, cap;
  uint32_t stride, sampled;  // every stride-th tile is sampled: how many that is
};
__device__ __forceinline__ uint32_t* list_indices(const SelUnit& s) { return reinterpret_cast<uint32_t*>(s.cv + s.cap); }
__device__ __forceinline__ float* list2_values(const SelUnit& s) { return s.cv + 2 * (size_t)s.cap; }
__device__ __forceinline__ uint32_t* list2_indices(const SelUnit& s) {
  return reinterpret_cast<uint32_t*>(s.cv + 3 * (size_t)s.cap);
}
// room of each of the two lists in `pairs` pairs; keeps every list on 16 bytes
HP_HD uint32_t list_cap(uint64_t pairs) {
  return (uint32_t)(pairs / 2 < 0x7FFFFFFCull ? pairs / 2 : 0x7FFFFFFCull) & ~3u;
}
// stride of the sampled tiles of an array when ctas CTAs share `total` tiles: about a
// sampled tile for every CTA
HP_HD uint32_t sample_stride(uint32_t tiles, uint64_t total, uint32_t ctas) {
  uint64_t share = ((uint64_t)tiles * ctas) / (total ? total : 1);
  if (share < kMinSampled) share = kMinSampled;
  return share >= tiles ? 1u : (uint32_t)((tiles + share - 1) / share);
}

constexpr int kCollectBuf = 1024;  // candidates a CTA gathers before it reserves room in the lists

struct SelSmem {
  union {
    uint32_t hist[kBins];            // sample; finish: digit histograms
    struct {
      float val[kCollectBuf];
      uint32_t idx[kCollectBuf];
      uint16_t unit[kCollectBuf];
    } buf;                           // collect
  };
  union {
    uint32_t keys[kFinishKeys];      // finish
    float stash[2][kSelTile];        // sample to collect
  };
  FindSmem fs;
  uint32_t count, base, ticket, flag;
  uint32_t sent, ties;
};

__device__ __forceinline__ void clear_hist(uint32_t* sh) {
#pragma unroll 1
  for (int b = threadIdx.x; b < kBins / 4; b += kSpThreads)
    reinterpret_cast<uint4*>(sh)[b] = make_uint4(0u, 0u, 0u, 0u);
}

// The update of one element.  MODE as in pass0_body.
template <int MODE>
__device__ __forceinline__ float update_value(float v, float g, float& u, float momentum) {
  if (MODE == 1) v = v + g;
  if (MODE == 2) {
    u = __fmaf_rn(momentum, u, g);
    v = v + u;
  }
  return v;
}

// Loads tile t and applies the update, all loads before the first store; put(j, v) gets
// float4 number j * 256 + thread.  A tile that is not full or not on 16 bytes goes
// element by element; what lies past the end reads as zero, and a zero is never sent.
template <int MODE, typename F>
__device__ __forceinline__ void update_tile(const SelUnit& s, float momentum, uint32_t t, F put) {
  const size_t base = (size_t)t * kSelTile;
  const bool vec = ((reinterpret_cast<uintptr_t>(s.a) | (MODE >= 1 ? reinterpret_cast<uintptr_t>(s.g) : 0) |
                     (MODE == 2 ? reinterpret_cast<uintptr_t>(s.u) : 0)) & 15) == 0;
  if (vec && base + kSelTile <= s.n) {
    float4 av[4], gv[4], uv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t i = base + (j * kSpThreads + threadIdx.x) * 4;
      av[j] = *reinterpret_cast<const float4*>(s.a + i);
      if (MODE >= 1) gv[j] = *reinterpret_cast<const float4*>(s.g + i);
      if (MODE == 2) uv[j] = *reinterpret_cast<const float4*>(s.u + i);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t i = base + (j * kSpThreads + threadIdx.x) * 4;
      float4& v = av[j];
      v.x = update_value<MODE>(v.x, gv[j].x, uv[j].x, momentum);
      v.y = update_value<MODE>(v.y, gv[j].y, uv[j].y, momentum);
      v.z = update_value<MODE>(v.z, gv[j].z, uv[j].z, momentum);
      v.w = update_value<MODE>(v.w, gv[j].w, uv[j].w, momentum);
      if (MODE == 2) *reinterpret_cast<float4*>(s.u + i) = uv[j];
      if (MODE >= 1) *reinterpret_cast<float4*>(s.a + i) = v;
      put(j, v);
    }
  } else {
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      float e[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const size_t i = base + (j * kSpThreads + threadIdx.x) * 4 + q;
        e[q] = 0.0f;
        if (i < s.n) {
          float w = MODE == 2 ? s.u[i] : 0.0f;
          e[q] = update_value<MODE>(s.a[i], MODE >= 1 ? s.g[i] : 0.0f, w, momentum);
          if (MODE == 2) s.u[i] = w;
          if (MODE >= 1) s.a[i] = e[q];
        }
      }
      put(j, make_float4(e[0], e[1], e[2], e[3]));
    }
  }
}

template <int MODE>
static __device__ __noinline__ void update_to_stash(const SelUnit& s, float momentum, uint32_t t, float* stash) {
  update_tile<MODE>(s, momentum, t, [&](int j, const float4& v) {
    reinterpret_cast<float4*>(stash)[j * kSpThreads + threadIdx.x] = v;
  });
}

// Sampled tile number i of an array: update, values into `stash`, magnitudes into the
// array's sample histogram.  The CTA that completes the sample turns it into the
// candidates' lower bound.
static __device__ __noinline__ void sample_body(int mode, const SelUnit& s, float momentum, SelSmem& sm, uint32_t i,
                                                float* stash) {
  const uint32_t t = i * s.stride;
  if (mode == 0) update_to_stash<0>(s, momentum, t, stash);
  else if (mode == 1) update_to_stash<1>(s, momentum, t, stash);
  else update_to_stash<2>(s, momentum, t, stash);
  clear_hist(sm.hist);
  __syncthreads();
#pragma unroll 1
  for (uint32_t p = threadIdx.x; p < kSelTile; p += kSpThreads) {
    const uint32_t key = abs_key(stash[p]);
    if (key) atomicAdd(&sm.hist[key >> 19], 1u);
  }
  __syncthreads();
  flush_hist(sm.hist, s.ws);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t done;   // release the CTA's counts, acquire those of the CTAs before
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(done) : "l"(s.ws + kWsSampled) : "memory");
    sm.flag = done == s.sampled - 1;
  }
  __syncthreads();
  if (!sm.flag) return;
  uint32_t rank = s.k;
  if (s.stride > 1) {
    // k scaled to the sample, plus five standard deviations, plus a tenth because
    // neighbouring elements are not independent
    const float hits = __fdividef((float)s.k * (float)(s.sampled * kSelTile), (float)s.n);
    float dev;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(dev) : "f"(hits));
    rank = (uint32_t)(1.1f * hits + 5.0f * dev + 4.0f);
  }
  uint32_t bin, rem;
  find_bin(s.ws, rank, sm.fs, bin, rem);   // bin 0 when fewer than rank are counted
  if (threadIdx.x == 0) s.ws[kWsLow] = bin ? bin << 19 : 1u;   // zeros are never sent
  __syncthreads();
}

// Items [0, total) in stretches, taken from *word by whichever of the ctas CTAs is free:
// SMs do not run at one speed, and equal shares leave the fast ones waiting.  f(lo, hi)
// runs with the whole CTA; `slot` is shared memory.  (Asking for the next stretch before
// working on the current one split thread 0 from its warp, and the two halves then
// counted twice at the barriers that follow.)
template <typename F>
__device__ __forceinline__ void hand_out(uint32_t* word, uint32_t total, uint32_t ctas, uint32_t& slot, F f) {
  const uint32_t stretch = total / (4u * ctas) + 1u;
#pragma unroll 1
  for (;;) {
    if (threadIdx.x == 0) slot = atomicAdd(word, stretch);
    __syncthreads();
    const uint32_t lo = slot;
    __syncthreads();
    if (lo >= total) break;
    f(lo, min(lo + stretch, total));
  }
}

// one candidate into the CTA's buffer, or, when that is full, straight into its list
static __device__ __noinline__ void collect_one(const SelUnit& s, uint32_t uid, SelSmem& sm, float v, uint32_t i) {
  const uint32_t p = atomicAdd(&sm.count, 1u);
  if (p < (uint32_t)kCollectBuf) {
    sm.buf.val[p] = v;
    sm.buf.idx[p] = i;
    sm.buf.unit[p] = (uint16_t)uid;
    return;
  }
  const uint32_t pos = atomicAdd(s.ws + kWsCandCount, 1u);
  atomicAdd(s.ws + kBins + (abs_key(v) >> 19), 1u);
  if (pos < s.cap) {
    s.cv[pos] = v;
    list_indices(s)[pos] = i;
  } else {
    s.ws[kWsOverflow] = 1u;
  }
}

// Tiles [t0, t1) of one array without the sampled ones.
template <int MODE>
static __device__ __noinline__ void collect_body(const SelUnit& s, uint32_t uid, float momentum, SelSmem& sm,
                                                 uint32_t t0, uint32_t t1) {
  const uint32_t low = __ldcg(s.ws + kWsLow);
  uint32_t phase = t0 % s.stride;   // 0: a sampled tile
#pragma unroll 1
  for (uint32_t t = t0; t < t1; ++t) {
    const bool skip = phase == 0;
    if (++phase == s.stride) phase = 0;
    if (skip) continue;
    update_tile<MODE>(s, momentum, t, [&](int j, const float4& v) {
      const uint32_t most = max(max(abs_key(v.x), abs_key(v.y)), max(abs_key(v.z), abs_key(v.w)));
      if (most < low) return;
      const uint32_t i = t * kSelTile + (j * kSpThreads + threadIdx.x) * 4;
      if (abs_key(v.x) >= low) collect_one(s, uid, sm, v.x, i);
      if (abs_key(v.y) >= low) collect_one(s, uid, sm, v.y, i + 1);
      if (abs_key(v.z) >= low) collect_one(s, uid, sm, v.z, i + 2);
      if (abs_key(v.w) >= low) collect_one(s, uid, sm, v.w, i + 3);
    });
  }
}

// Sampled tile number i again, updated before: from its stash, or (again) read once more.
static __device__ __noinline__ void collect_sampled(const SelUnit& s, uint32_t uid, SelSmem& sm, uint32_t i,
                                                    float* stash, bool again) {
  const uint32_t t = i * s.stride, low = __ldcg(s.ws + kWsLow);
  if (again) update_to_stash<0>(s, 0.0f, t, stash);
  __syncthreads();
#pragma unroll 1
  for (uint32_t p = threadIdx.x; p < kSelTile; p += kSpThreads) {
    const float v = stash[p];
    if (abs_key(v) >= low) collect_one(s, uid, sm, v, t * kSelTile + p);
  }
  __syncthreads();
}

// Append the CTA's gathered candidates to their lists, and their first digits to the
// lists' histograms.  A warp's entries mostly belong to one list: one reservation for each
// group of lanes with the same list.  unit(uid) gives the array.
template <typename F>
__device__ __forceinline__ void collect_flush(SelSmem& sm, F unit) {
  __syncthreads();
  const uint32_t n = min(sm.count, (uint32_t)kCollectBuf);
#pragma unroll 1
  for (uint32_t p0 = 0; p0 < n; p0 += kSpThreads) {
    const uint32_t p = p0 + threadIdx.x;
    const bool have = p < n;
    const uint32_t mask = __ballot_sync(0xffffffffu, have);
    if (have) {
      const uint32_t uid = sm.buf.unit[p], lane = threadIdx.x & 31;
      const float v = sm.buf.val[p];
      const SelUnit s = unit(uid);
      const uint32_t group = __match_any_sync(mask, uid);
      const int lead = __ffs(group) - 1;
      uint32_t pos = 0;
      if ((int)lane == lead) pos = atomicAdd(s.ws + kWsCandCount, (uint32_t)__popc(group));
      atomicAdd(s.ws + kBins + (abs_key(v) >> 19), 1u);
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

// store one pair at place `pos` of every destination's payload
__device__ __forceinline__ void put_pair(const EmitDst& dst, size_t val_off, uint32_t kmax, uint32_t pos,
                                         uint32_t idx, float val) {
  if (pos >= kmax) return;
#pragma unroll 1
  for (int d = 0; d < dst.n; ++d) {
    reinterpret_cast<uint32_t*>(dst.out[d] + 16)[pos] = idx;
    reinterpret_cast<float*>(dst.out[d] + val_off)[pos] = val;
  }
}

// Slice x of nx of a list too long for one CTA: pairs above the first digit's bin are
// sent (and their state cleared), pairs in it move to the second list.  The finds of a
// stretch are counted in shared memory so that the global counters are touched twice
// per CTA and stretch.
static __device__ __noinline__ void refine_body(const SelUnit& s, const EmitDst& dst, SelSmem& sm, uint32_t x,
                                                uint32_t nx) {
  const uint32_t L = min(__ldcg(s.ws + kWsCandCount), s.cap);
  uint32_t bin0, rem;
  find_bin(s.ws + kBins, min(s.k, L), sm.fs, bin0, rem);
  const size_t val_off = 16 + align_up(4ull * s.kmax, 16);
  const uint32_t per = (L + nx - 1) / nx, lo = min(x * per, L), hi = min(lo + per, L);
#pragma unroll 1
  for (uint32_t p0 = lo; p0 < hi; p0 += 4 * kSpThreads) {
    if (threadIdx.x == 0) sm.sent = sm.ties = 0;
    __syncthreads();
    float v[4];
    uint32_t at[4], idx[4];
    int what[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t p = p0 + j * kSpThreads + threadIdx.x;
      v[j] = p < hi ? __ldcg(s.cv + p) : 0.0f;
      idx[j] = p < hi ? __ldcg(list_indices(s) + p) : 0u;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t bin = abs_key(v[j]) >> 19;
      const bool have = p0 + j * kSpThreads + threadIdx.x < hi;
      what[j] = !have || bin < bin0 ? 0 : (bin > bin0 ? 1 : 2);
      at[j] = what[j] == 1 ? atomicAdd(&sm.sent, 1u) : (what[j] == 2 ? atomicAdd(&sm.ties, 1u) : 0u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      sm.base = sm.sent ? atomicAdd(s.ws + kWsOutCount, sm.sent) : 0u;
      sm.ticket = sm.ties ? atomicAdd(s.ws + kWsCand2Count, sm.ties) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (what[j] == 1 && idx[j] < s.n) {
        put_pair(dst, val_off, s.kmax, sm.base + at[j], idx[j], v[j]);
        s.a[idx[j]] = 0.0f;
        if (s.u) s.u[idx[j]] = 0.0f;
      } else if (what[j] == 2) {
        const uint32_t pos = sm.ticket + at[j];   // never more than the first list holds
        if (pos < s.cap) {
          list2_values(s)[pos] = v[j];
          list2_indices(s)[pos] = idx[j];
        }
      }
    }
    __syncthreads();
  }
}

// Slice x of nx of the finish of one array.  The nx CTAs all work out the exact threshold
// of the list (the second one after a refine step) -- its keys are a few kilobytes in L2,
// and repeating the three digits costs less than a barrier after them -- and each sends
// its share of the pairs.  True in thread 0 of the CTA that finished last, behind the
// headers.  Every step runs once per launch, so its time is latency and instruction
// fetch: one copy of the digit search, rolled loops.
static __device__ __noinline__ bool finish_body(int alg, const SelUnit& s, const EmitDst& dst, SelSmem& sm,
                                                bool refined, uint32_t x, uint32_t nx) {
  const uint32_t all = min(__ldcg(s.ws + kWsCandCount), s.cap);
  const uint32_t k = min(s.k, all);          // fewer than k non-zero elements: all of them
  const uint32_t L = refined ? min(__ldcg(s.ws + kWsCand2Count), s.cap) : all;
  const float* cv = refined ? list2_values(s) : s.cv;
  const uint32_t* ci = refined ? list2_indices(s) : list_indices(s);
  const size_t val_off = 16 + align_up(4ull * s.kmax, 16);
  // keys into shared memory, eight a thread in flight; past L whatever the list's room holds
#pragma unroll 1
  for (uint32_t p = threadIdx.x * 4; p < L && p < kFinishKeys; p += 8 * kSpThreads) {
    const uint32_t q = p + 4 * kSpThreads;
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(cv + p));
    uint4 w = v;
    if (q < L) w = __ldcg(reinterpret_cast<const uint4*>(cv + q));
    *reinterpret_cast<uint4*>(sm.keys + p) =
        make_uint4(v.x & 0x7FFFFFFFu, v.y & 0x7FFFFFFFu, v.z & 0x7FFFFFFFu, v.w & 0x7FFFFFFFu);
    *reinterpret_cast<uint4*>(sm.keys + q) =
        make_uint4(w.x & 0x7FFFFFFFu, w.y & 0x7FFFFFFFu, w.z & 0x7FFFFFFFu, w.w & 0x7FFFFFFFu);
  }
  auto key_at = [&](uint32_t p) { return p < kFinishKeys ? sm.keys[p] : abs_key(__ldcg(cv + p)); };
  uint32_t prefix, rem;
  find_bin(s.ws + kBins, k, sm.fs, prefix, rem);
  // the remaining digits: 11 bits, then 8
#pragma unroll 1
  for (int d = 0; d < 2; ++d) {
    const int low = d == 0 ? 8 : 0, bits = d == 0 ? 11 : 8;
    clear_hist(sm.hist);
    __syncthreads();
#pragma unroll 1
    for (uint32_t p = threadIdx.x; p < L; p += kSpThreads) {
      const uint32_t key = key_at(p);
      if ((key >> (low + bits)) == prefix) atomicAdd(&sm.hist[(key >> low) & ((1u << bits) - 1u)], 1u);
    }
    __syncthreads();
    uint32_t bin, r;
    find_bin(sm.hist, rem, sm.fs, bin, r);
    prefix = (prefix << bits) | bin;
    rem = r;
  }
  const uint32_t thr = prefix, need = rem;   // `need` of the elements equal to thr are sent
  const uint32_t per = (L + nx - 1) / nx, lo = min(x * per, L), hi = min(lo + per, L);
#pragma unroll 1
  for (uint32_t p0 = lo; p0 < hi; p0 += kSpThreads) {
    if (threadIdx.x == 0) sm.sent = sm.ties = 0;
    __syncthreads();
    const uint32_t p = p0 + threadIdx.x;
    const uint32_t key = p < hi ? key_at(p) : 0u;
    const bool more = p < hi && key > thr, tie = p < hi && key == thr;
    uint32_t idx = 0, at = 0;
    float val = 0.0f;
    if (more || tie) {
      idx = __ldcg(ci + p);
      val = __ldcg(cv + p);
      at = more ? atomicAdd(&sm.sent, 1u) : atomicAdd(&sm.ties, 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      // of this stretch's ties those that come early enough in the launch are sent
      uint32_t ok = 0;
      if (sm.ties && need) {
        const uint32_t before = atomicAdd(s.ws + kWsTieCount, sm.ties);
        ok = before < need ? min(sm.ties, need - before) : 0u;
      }
      sm.ties = ok;
      sm.base = sm.sent + ok ? atomicAdd(s.ws + kWsOutCount, sm.sent + ok) : 0u;
    }
    __syncthreads();
    const bool send = more || (tie && at < sm.ties);
    if (send && idx < s.n) {
      put_pair(dst, val_off, s.kmax, sm.base + (more ? at : sm.sent + at), idx, val);
      s.a[idx] = 0.0f;
      if (s.u) s.u[idx] = 0.0f;
    }
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x != 0) return false;
  __threadfence();
  if (atomicAdd(s.ws + kWsDone, 1u) != nx - 1) return false;
  __threadfence();
  const uint32_t sent = atomicAdd(s.ws + kWsOutCount, 0u);
  WireHeader h;
  h.n = s.n;
  h.alg = (uint8_t)alg;
  h.bitwidth = 0;
  h.flags = 0;
  h.a = all < s.k ? 0.0f : __uint_as_float(thr);
  h.b = sent < s.kmax ? sent : s.kmax;
#pragma unroll 1
  for (int d = 0; d < dst.n; ++d) *reinterpret_cast<uint4*>(dst.out[d]) = *reinterpret_cast<const uint4*>(&h);
  return true;
}
// CTAs that share the finish of a list of L elements
__device__ __forceinline__ uint32_t finish_slices(uint32_t L, uint32_t most) {
  const uint32_t n = L / 256u + 1u;
  return n < most ? n : most;
}

// The sample misled: the list lacks some of the k largest.
__device__ __forceinline__ bool selection_failed(const SelUnit& s) {
  const uint32_t c = __ldcg(s.ws + kWsCandCount);
  return __ldcg(s.ws + kWsOverflow) != 0u || (c < s.k && __ldcg(s.ws + kWsLow) > 1u);
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
