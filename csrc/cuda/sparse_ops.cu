// Sparse (top-k) compression for DGC and GradDrop on sm_100a.
//
// With room for a candidate list (the usual call) an encode is three launches: sample, update
// + collect with a CTA per half tile, which begins while the sample ends, and emit
// (sparse_chain.cuh).  One persistent kernel with grid barriers does the same for calls that
// limit the CTAs (max_ctas), and for those that it is better at (chain_is_slower); in the
// others equal shares leave the faster SMs idle, and the arrays stand still while the sample
// is worked out.  DGC encode and decode at 0.1 %, us, persistent / chain (B200): 64 K elements
// 26.7 / 24.8, 1 M 36.8 / 30.3, 3 M 51.4 / 42.1, 10 M at 1 % 98.4 / 75.9, 20 M 122.7 / 104.7.
// The emitting launch is cooperative, because where a list came out short its CTAs count
// the digits together, and sized for the SMs that the stream may use.  Barriers are
// bounded (kGridBarrierNs); if a kernel that holds SMs for longer than that comes between
// the CTAs, the payload may lack elements, and the workspace's status word (kWsStatus) is set.
//
// Without it (the allocation-free entry point) four launches read the array once each:
//   pass 0   state update fused with the first radix histogram
//              DGC      : u = m*u + g ; v += u        (momentum correction)
//              GradDrop : r += g
//   pass 1,2 histograms of bits 18..8 and 7..0 among elements matching the prefix so far
//   emit     compaction of (index,value) pairs, sent entries of v (and u) zeroed
//
// The selection is exact: every |v_i| above the k-th largest magnitude is sent,
// plus entries equal to it until k are sent (which of several equal entries is
// unspecified on the GPU; the CPU oracle takes the lowest indices).  Zeros are
// never sent.  Pair order inside the payload is unspecified.
//
// Reference parity: DGC and GradDrop are two of the five built-in algorithms of
// mark14wu/hipress (README.md:9; --comp_alg dgc README.md:180); CompLL planned
// sort/copy_if for them (src/CompLL/GCGen/unit.py:24-29) but has no translation
// rule, so there is no reference kernel to compare with.
#include "partition.cuh"
#include "sparse_chain.cuh"
#include "sparse_core.cuh"
#include "sync.cuh"
#include "hipress/noalloc.h"

namespace hipress {

template <int MODE>
__global__ void __launch_bounds__(kSpThreads)
sparse_pass0_kernel(const float* __restrict__ g, float* __restrict__ a, float* __restrict__ u,
                    uint64_t n, float momentum, uint32_t* __restrict__ ws) {
  __shared__ __align__(16) uint32_t sh[kBins];
  pass0_body<MODE>(g, a, u, n, momentum, ws, sh, blockIdx.x, gridDim.x);
}

template <int PASS>
__global__ void __launch_bounds__(kSpThreads)
sparse_pass_kernel(const float* __restrict__ a, uint64_t n, uint32_t k,
                   uint32_t* __restrict__ ws) {
  __shared__ __align__(16) uint32_t sh[kBins];
  __shared__ FindSmem fs;
  pass_body(PASS, a, n, k, ws, sh, fs, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(kSpThreads)
sparse_emit_kernel(int alg, float* __restrict__ a, float* __restrict__ u, uint64_t n, uint32_t k,
                   uint32_t kmax, uint8_t* __restrict__ out, uint32_t* __restrict__ ws) {
  __shared__ FindSmem fs;
  __shared__ EmitSmem es;
  EmitDst d = {};
  d.n = 1;
  d.out[0] = out;
  emit_body(alg, a, u, n, k, kmax, d, ws, fs, es, blockIdx.x, gridDim.x);
}

// ---- the whole encode in one cooperative launch, as wide as the caller allows
struct SelArgs {
  SelUnit unit;
  int alg, mode;
  float momentum;
  uint8_t* out;
};

union SelOrPassSmem {
  SelSmem sel;
  uint32_t hist[kBins];   // whole-array passes
  EmitSmem emit;
};

__global__ void __launch_bounds__(kSpThreads, 2) sparse_encode_kernel(const __grid_constant__ SelArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SelOrPassSmem& sm = *reinterpret_cast<SelOrPassSmem*>(smem_raw);
  __shared__ WaitState wst;
  __shared__ FindSmem fs;
  __shared__ SelUnit s;
  if (threadIdx.x == 0) s = A.unit;
  const uint32_t G = gridDim.x, c = blockIdx.x;
  uint32_t gen = 0;
  wait_init(wst);
  auto barrier = [&]() {
    grid_barrier(s.ws + kWsWords, gen, G, kGridBarrierNs, s.ws + kWsStatus, 1u, wst);
  };
  const uint32_t tiles = (s.n - 1) / kSelTile + 1;
  uint32_t mine = 0;   // sampled tiles of this CTA: the first two stay in shared memory
#pragma unroll 1
  for (uint32_t i = c; i < s.sampled; i += G, ++mine) {
    float* stash = sm.sel.stash[mine < 1 ? 0 : 1];
    if (A.mode == 0) sample_body<0>(s, A.momentum, sm.sel, i, stash);
    else if (A.mode == 1) sample_body<1>(s, A.momentum, sm.sel, i, stash);
    else sample_body<2>(s, A.momentum, sm.sel, i, stash);
    __syncthreads();
  }
  barrier();
  if (threadIdx.x == 0) {
    sm.sel.count = 0;
    s.low = __ldcg(s.ws + kWsLow);
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t i = c, r = 0; r < mine; i += G, ++r)
    collect_sampled(s, 0, sm.sel, i, sm.sel.stash[r < 1 ? 0 : 1], r >= 1 && mine > 2);
  auto self = [&](uint32_t) -> const SelUnit& { return s; };
  if (s.stride > 1)
    hand_out(s.ws + kWsTicket, tiles, c, G, sm.sel.ticket, [&](uint32_t t0, uint32_t t1) {
#pragma unroll 1
      for (uint32_t t = t0; t < t1; t += s.run) {
        const uint32_t end = min(t + s.run, t1);
        if (A.mode == 0) collect_body<0>(s, 0, A.momentum, sm.sel, t, end);
        else if (A.mode == 1) collect_body<1>(s, 0, A.momentum, sm.sel, t, end);
        else collect_body<2>(s, 0, A.momentum, sm.sel, t, end);
        if (__syncthreads_or(sm.sel.count > (uint32_t)kCollectBuf / 2)) collect_flush(sm.sel, self);
      }
    });
  collect_flush(sm.sel, self);
  barrier();
  EmitDst d = {};
  d.n = 1;
  d.out[0] = A.out;
  const ListState ls = list_state(s);   // the same in every CTA: its writers are behind the barrier
  if (!selection_failed(s, ls)) {
    const uint32_t nx = emit_slices(ls.count, G);
    if (c < nx) emit_slice(A.alg, s, ls, d, sm.sel, c, nx);
    return;
  }
  // whole-array passes
  for (uint32_t i = c * kSpThreads + threadIdx.x; i < 3u * kBins; i += G * kSpThreads) s.ws[i] = 0;
  barrier();
  pass0_body<0>(nullptr, s.a, nullptr, s.n, 0.0f, s.ws, sm.hist, c, G);
  barrier();
  pass_body(1, s.a, s.n, s.k, s.ws, sm.hist, fs, c, G);
  barrier();
  pass_body(2, s.a, s.n, s.k, s.ws, sm.hist, fs, c, G);
  barrier();
  emit_body(A.alg, s.a, s.u, s.n, s.k, s.kmax, d, s.ws, fs, sm.emit, c, G);
}

__global__ void __launch_bounds__(kSpThreads)
sparse_scatter_kernel(const uint8_t* __restrict__ payload, float* __restrict__ out, uint64_t n,
                      uint32_t kmax, float scale, int accumulate) {
  scatter_body(payload, out, n, kmax, scale, accumulate, blockIdx.x, gridDim.x);
}

// Decode of a short payload in one launch: every CTA clears its share of the result and
// then looks through all pairs for those that fall into it (at most kScanPairs, read from
// L2), instead of a memset, a wait and a scatter.
constexpr uint32_t kScanPairs = 4096;
__global__ void __launch_bounds__(kSpThreads)
sparse_decode_kernel(const uint8_t* __restrict__ payload, float* __restrict__ out, uint64_t n, uint32_t kmax,
                     float scale) {
  const uint64_t per = ((n + gridDim.x - 1) / gridDim.x + 3) & ~3ull;
  const uint64_t lo = min((uint64_t)blockIdx.x * per, n), hi = min(lo + per, n);
  const bool vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  for (uint64_t i = lo + threadIdx.x * 4; i < hi; i += kSpThreads * 4)
    st4(out, i, hi, vec, make_float4(0.f, 0.f, 0.f, 0.f));
  __syncthreads();
  const WireHeader* h = reinterpret_cast<const WireHeader*>(payload);
  const uint32_t k = min(__ldcg(&h->b), kmax);
  const uint32_t* idx = reinterpret_cast<const uint32_t*>(payload + 16);
  const float* val = reinterpret_cast<const float*>(payload + 16 + align_up(4ull * kmax, 16));
  for (uint32_t p0 = 0; p0 < k; p0 += 4 * kSpThreads) {
    uint32_t i[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t p = p0 + j * kSpThreads + threadIdx.x;
      i[j] = p < k ? __ldcg(idx + p) : 0xFFFFFFFFu;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i[j] >= lo && i[j] < hi) out[i[j]] = __ldcg(val + p0 + j * kSpThreads + threadIdx.x) * scale;
  }
}

}  // namespace hipress

using namespace hipress;

extern "C" {

// minimum scratch (histograms + counters); with room for two candidate lists of
// 4 * kmax pairs each on top, the encoder reads the state once, in the update
uint64_t hp_sparse_workspace_bytes() { return (uint64_t)kWsWords * 4; }
uint64_t hp_sparse_workspace_bytes_for(uint64_t kmax) {
  return (uint64_t)(kWsWords + kBarrierWords + 32 * kChainLists) * 4 + (8 * kmax + 4096) * 8;
}

// ws_bytes beyond the histogram block is used for the candidate lists; when there
// is none (the allocation-free entry point) the three full-array passes run.
static int sparse_encode_impl(int alg, const float* g, float* a, float* u, uint64_t n, uint64_t k,
                              uint64_t kmax, float momentum, int update, uint8_t* out,
                              uint32_t* ws, uint64_t ws_bytes, int max_ctas, cudaStream_t st) {
  if (n == 0 || n > 0xFFFFF000ull || k < 1 || k > n || k > kmax || kmax > 0xFFFFFFFFull)
    return HP_ERR_BAD_ARG;
  if (alg != kDgc && alg != kGradDrop) return HP_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(out) & 15) return HP_ERR_BAD_ARG;
  if (update && !g) return HP_ERR_BAD_ARG;
  if (update && alg == kDgc && !u) return HP_ERR_BAD_ARG;
  const uint64_t tiles = (n + kSelTile - 1) / kSelTile;
  float* uu = alg == kDgc ? u : nullptr;
  const int mode = !update ? 0 : (alg == kGradDrop ? 1 : 2);
  // histograms and counters, then the barrier words and the candidate lists
  constexpr uint32_t kParts = 32 * kChainLists;   // counts of a list's parts
  const uint64_t head = (uint64_t)(kWsWords + kBarrierWords + kParts) * 4;
  const uint64_t pairs = ws_bytes > head ? (ws_bytes - head) / 8 : 0;
  const bool listed = pairs >= 1024 && (reinterpret_cast<uintptr_t>(ws) & 15) == 0;   // counters are read as uint4
  cudaError_t e = cudaMemsetAsync(ws, 0, listed ? head : (size_t)kWsWords * 4, st);
  if (e != cudaSuccess) return (int)e;
  if (listed) {
    const size_t smem = sizeof(SelOrPassSmem);
    static int per_sm[64] = {}, all_sms[64] = {};   // CTAs an SM holds at once and SMs, per device
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    int per = dev >= 0 && dev < 64 ? per_sm[dev] : 0, sms = per ? all_sms[dev] : 0;
    if (per == 0) {
      e = cudaFuncSetAttribute((const void*)sparse_encode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return (int)e;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sparse_encode_kernel, kSpThreads, smem);
      if (e != cudaSuccess) return (int)e;
      if (per < 1 || sms < 1) return HP_ERR_RESIDENCY;
      if (dev >= 0 && dev < 64) {
        all_sms[dev] = sms;
        per_sm[dev] = per;
      }
    }
    int cap = per * stream_sms(st, sms);   // the stream may own only some of the SMs
    if (max_ctas <= 0 && !chain_is_slower(mode, n, k) && chain_per_sm(dev) > 0) {
      ChainArgs C = {};
      SelUnit& V = C.unit[0].s;
      V.g = g;
      V.a = a;
      V.u = uu;
      V.ws = ws;
      V.cv = reinterpret_cast<float*>(ws + kWsWords + kBarrierWords + kParts);
      V.n = (uint32_t)n;
      V.k = (uint32_t)k;
      V.kmax = (uint32_t)kmax;
      V.cap = list_cap(pairs);
      const Sampling cs = sampling((uint32_t)tiles, tiles, (uint32_t)cap, n, k);
      V.stride = cs.stride;
      V.top = cs.top;
      C.unit[0].counts = ws + kWsWords + kBarrierWords;
      C.units = 1;
      C.alg = alg;
      C.momentum = momentum;
      C.payload = out;
      C.barrier = ws + kWsWords;
      C.status = ws + kWsStatus;
      C.code = 1u;
      if (chain_place(C, chain_per_sm(dev), stream_sms(st, sms)))
        return (int)chain_select(mode, C, st);
    }
    if (max_ctas > 0 && max_ctas < cap) cap = max_ctas;
    const int grid = (int)(tiles < (uint64_t)cap ? tiles : (uint64_t)cap);
    SelArgs A = {};
    SelUnit& U = A.unit;
    U.g = g;
    U.a = a;
    U.u = uu;
    U.clear = nullptr;
    U.ws = ws;
    U.cv = reinterpret_cast<float*>(ws + kWsWords + kBarrierWords + kParts);
    U.n = (uint32_t)n;
    U.k = (uint32_t)k;
    U.kmax = (uint32_t)kmax;
    U.cap = list_cap(pairs);
    const Sampling sp = sampling((uint32_t)tiles, tiles, (uint32_t)grid, n, k);
    U.stride = sp.stride;
    U.top = sp.top;
    U.run = sp.run;
    U.sampled = ((uint32_t)tiles + U.stride - 1) / U.stride;
    A.alg = alg;
    A.mode = mode;
    A.momentum = momentum;
    A.out = out;
    void* args[] = {(void*)&A};
    e = cudaLaunchCooperativeKernel((const void*)sparse_encode_kernel, dim3(grid), dim3(kSpThreads), args, smem, st);
    if (e != cudaErrorCooperativeLaunchTooLarge) return (int)e;
    // less of the GPU is ours than the queries said: the launches that need no co-residency
    cudaGetLastError();
  }
  if (max_ctas <= 0) max_ctas = 148 * 4;
  const int grid = (int)(tiles < (uint64_t)max_ctas ? tiles : (uint64_t)max_ctas);
  if (mode == 0) sparse_pass0_kernel<0><<<grid, kSpThreads, 0, st>>>(g, a, u, n, momentum, ws);
  else if (mode == 1) sparse_pass0_kernel<1><<<grid, kSpThreads, 0, st>>>(g, a, u, n, momentum, ws);
  else sparse_pass0_kernel<2><<<grid, kSpThreads, 0, st>>>(g, a, u, n, momentum, ws);
  sparse_pass_kernel<1><<<grid, kSpThreads, 0, st>>>(a, n, (uint32_t)k, ws);
  sparse_pass_kernel<2><<<grid, kSpThreads, 0, st>>>(a, n, (uint32_t)k, ws);
  sparse_emit_kernel<<<grid, kSpThreads, 0, st>>>(alg, a, uu, n, (uint32_t)k, (uint32_t)kmax, out, ws);
  return (int)cudaGetLastError();
}

// a: accumulator (DGC v / GradDrop residual).  update=1 applies the state update
// with g first; update=0 selects from a as it is (server / ring re-selection).
int hp_cuda_sparse_encode(int alg, const float* g, float* a, float* u, uint64_t n, uint64_t k,
                          uint64_t kmax, float momentum, int update, uint8_t* out, void* workspace,
                          uint64_t workspace_bytes, int max_ctas, void* stream) {
  if (workspace_bytes < (uint64_t)kWsWords * 4) return HP_ERR_BAD_ARG;
  return sparse_encode_impl(alg, g, a, u, n, k, kmax, momentum, update, out,
                            static_cast<uint32_t*>(workspace), workspace_bytes, max_ctas,
                            (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Allocation-free variant (see hipress/noalloc.h): the scratch lives in this
// file-scope device array.  In host code the name below is only a handle for
// the runtime, never a device address; the address each GPU gave the array is
// fetched once per device with cudaGetSymbolAddress and passed to the kernels.
static __device__ __align__(256) uint32_t g_noalloc_scratch[kWsWords];

static uint32_t* g_noalloc_ptr[64];  // per device, filled on the first call there

uint64_t hp_cuda_noalloc_scratch_bytes(void) { return (uint64_t)kWsWords * 4; }

int hp_cuda_sparse_encode_noalloc(int alg, const float* g, float* a, float* u, uint64_t n,
                                  uint64_t k, uint64_t kmax, float momentum, int update,
                                  uint8_t* out, int max_ctas, void* stream) {
  if (n > HP_NOALLOC_MAX_ELEMS) return HP_ERR_TOO_LARGE;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64) return HP_ERR_BAD_ARG;
  if (!g_noalloc_ptr[dev]) {  // set-up: once per device, with that device current
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return (int)e;
    if (!p) return HP_ERR_BAD_ARG;
    g_noalloc_ptr[dev] = static_cast<uint32_t*>(p);
  }
  return sparse_encode_impl(alg, g, a, u, n, k, kmax, momentum, update, out, g_noalloc_ptr[dev],
                            (uint64_t)kWsWords * 4, max_ctas, (cudaStream_t)stream);
}

// accumulate=0: out is zero-filled first.  accumulate=1: out[idx] += val*scale.
int hp_cuda_sparse_decode(const uint8_t* payload, float* out, uint64_t n, uint64_t kmax,
                          float scale, int accumulate, void* stream) {
  if (n == 0) return 0;
  if (reinterpret_cast<uintptr_t>(payload) & 15) return HP_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (!accumulate && kmax && kmax <= kScanPairs) {
    const uint64_t tiles = (n + 4095) / 4096;
    sparse_decode_kernel<<<(int)(tiles < 148 * 8 ? tiles : 148 * 8), kSpThreads, 0, st>>>(payload, out, n, (uint32_t)kmax, scale);
    return (int)cudaGetLastError();
  }
  if (!accumulate) {
    cudaError_t e = cudaMemsetAsync(out, 0, n * sizeof(float), st);
    if (e != cudaSuccess) return (int)e;
  }
  if (kmax == 0) return 0;
  int grid = (int)((kmax + kSpThreads - 1) / kSpThreads);
  if (grid > 148 * 8) grid = 148 * 8;
  sparse_scatter_kernel<<<grid, kSpThreads, 0, st>>>(payload, out, n, (uint32_t)kmax, scale,
                                                      accumulate);
  return (int)cudaGetLastError();
}

}  // extern "C"
