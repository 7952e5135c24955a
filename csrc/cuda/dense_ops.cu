// Stand-alone dense (quantising) compression ops for onebit, TBQ and TernGrad:
// one encode kernel (optionally merging an incoming payload, the ring "recv ->
// decode -> merge -> encode" chain of CaSync) and one decode / decode-accumulate
// kernel.  They are the building blocks of the unfused baseline and the public
// per-tensor API; the fused ring / PS kernels reuse the same tile code.
//
// Reference parity: op pair Encode(gradient, compressed, params) /
// Decode(compressed, gradient), in place, caller-allocated buffers
// (src/CompLL/GCGen/output/TernGradEncode/TernGradEncode.cc:10-24).
#include "dense_tile.cuh"
#include "hipress/capi.h"

namespace hipress {

// Where the parts of a payload lie, worked out on the host.
struct PayloadPtrs {
  float* meta;
  uint8_t* codes;
};

// These kernels may be resident before the launch in front of them in the stream has ended
// (programmatic launch): what a small tensor's call waits for is mostly the launch itself,
// and calls follow one another (decode, decode, ..., encode: 20.4 -> 17.8 us for four and
// one of 1 M elements; a hop of 16.8 M, whose first tiles wait in place, 34.9 -> 33.0).
// The result is zero, and the
// tile index needs it, so that no load of what an earlier launch wrote can be moved up.
__device__ __forceinline__ uint32_t after_earlier_launches() {
  uint32_t zero;
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(zero)::"memory");
  return zero;
}

// One tile per CTA unless the caller limits the grid: SMs do not run at one speed, and
// with a block per tile the hardware gives the next tile to whichever is free (TBQ
// encode with an incoming payload, 16.8 M elements: 38.8 us with 1184 CTAs striding over
// the tiles, 31.0 us = 6.75 TB/s with a CTA per tile).
// TernGrad without state needs few registers and has a long chain between a tile's loads
// and its stores: six CTAs per SM hide it better than four (67.1 M elements 66 -> 61 us);
// the others are at HBM speed with four and slightly slower with more.
template <int ALG, int B, bool IN, bool RES>
__global__ void __launch_bounds__(kThreads, ALG == kTernGrad && !RES ? 6 : 4)
dense_encode_kernel(const float* __restrict__ g, float* __restrict__ r, const PayloadPtrs in,
                    const PayloadPtrs out, const WireHeader hdr, uint32_t n, uint32_t tiles, DenseParams P,
                    uint32_t tensor_id, uint64_t elem_offset) {
  __shared__ TileSmem s;
  const uint32_t first = blockIdx.x + after_earlier_launches();
  if (first == 0) {
    uint4* head = reinterpret_cast<uint4*>(out.meta) - 1;   // the header ends where the metadata starts
    if (threadIdx.x == 0) *head = *reinterpret_cast<const uint4*>(&hdr);
    // zero the padding behind the tile metadata so payload bytes are deterministic
    const uint32_t used = tiles * dense_meta_floats(ALG), padded = (used + 3) & ~3u;
    if (used + threadIdx.x < padded) out.meta[used + threadIdx.x] = 0.0f;
  }
  for (uint32_t t = first; t < tiles; t += gridDim.x) {
    const uint32_t start = t * kTile;
    const int m = (int)min((uint32_t)kTile, n - start);
    const bool full =
        m == kTile && ((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(RES ? r : nullptr)) & 15) == 0;
    // every load of the tile goes out before the first one is used
    float x[kIter][4], rr[kIter][4], im[2];
    uint32_t inf[kIter];
    if (full) load_tile_full(g + start, x);
    else load_tile(g + start, m, x);
    if (IN) {
      load_meta<ALG>(in.meta, t, im);
#pragma unroll
      for (int j = 0; j < kIter; ++j) inf[j] = load_frag<B>(in.codes + (size_t)t * (kTile * B / 8), j, m);
    }
    if (RES) {
      if (full) load_tile_full(r + start, rr);
      else load_tile(r + start, m, rr);
    }
    if (IN) {
#pragma unroll
      for (int j = 0; j < kIter; ++j) {
        float d[4];
        decode_frag<ALG, B>(inf[j], im, P.tau, d);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[j][e] = x[j][e] + d[e];
      }
    }
    if (RES) {
#pragma unroll
      for (int j = 0; j < kIter; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) x[j][e] = rr[j][e] + x[j][e];
    }
    float meta[2];
    uint32_t frag[kIter];
    encode_tile<ALG, B>(x, m, P, tensor_id, elem_offset + start, P.salt, s, 0, meta, frag, RES);
    if (RES) {
      if (full) store_tile_full(r + start, x);
      else store_tile(r + start, m, x);
    }
    store_codes<B>(out.codes + (size_t)t * (kTile * B / 8), m, frag);
    if (threadIdx.x == 0) {
      if (ALG == kOnebit) out.meta[t] = meta[0];
      if (ALG == kTernGrad) *reinterpret_cast<float2*>(out.meta + 2 * t) = make_float2(meta[0], meta[1]);
    }
    if (t + gridDim.x < tiles) __syncthreads();   // the reduction's shared memory is used again
  }
}

// Decode is write bound (4 B/element out, bits in), and a tile's payload load is exposed
// once per CTA: with a CTA per tile eight of them share an SM and hide it (16.8 M
// elements, TBQ: 14.5 us with four tiles per CTA, 12.4 us with one; 1 M elements
// decode-accumulate 6.2 -> 4.1 us, where four tiles per CTA left most SMs without work).
template <int ALG, int B, bool ACC>
__global__ void __launch_bounds__(kThreads)
dense_decode_kernel(const PayloadPtrs in, float* __restrict__ out, uint32_t n, uint32_t tiles, float tau,
                    float scale) {
  for (uint32_t t = blockIdx.x + after_earlier_launches(); t < tiles; t += gridDim.x) {
    const uint32_t start = t * kTile;
    const int m = (int)min((uint32_t)kTile, n - start);
    const bool full = tile_is_full_aligned(out, m);
    float meta[2], x[kIter][4];
    uint32_t fr[kIter];
    load_meta<ALG>(in.meta, t, meta);
#pragma unroll
    for (int j = 0; j < kIter; ++j) fr[j] = load_frag<B>(in.codes + (size_t)t * (kTile * B / 8), j, m);
    if (ACC) {
      if (full) load_tile_full(out + start, x);
      else load_tile(out + start, m, x);
    }
#pragma unroll
    for (int j = 0; j < kIter; ++j) {
      float d[4];
      decode_frag<ALG, B>(fr[j], meta, tau, d);
#pragma unroll
      for (int e = 0; e < 4; ++e) x[j][e] = ACC ? x[j][e] + d[e] * scale : d[e] * scale;
    }
    if (full) store_tile_full(out + start, x);
    else store_tile(out + start, m, x);
  }
}

static PayloadPtrs payload_ptrs(const uint8_t* base, int alg, uint64_t n) {
  uint8_t* p = const_cast<uint8_t*>(base);
  return {reinterpret_cast<float*>(p + 16), p + 16 + dense_meta_bytes(alg, n)};
}

static int grid_of(uint64_t tiles, int max_ctas) {
  return (int)(max_ctas > 0 && tiles > (uint64_t)max_ctas ? (uint64_t)max_ctas : tiles);
}

// A launch that may begin while the one before it in the stream ends.
template <typename... P, typename... A>
static int launch_early(void (*kern)(P...), int grid, cudaStream_t st, A... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3(kThreads);
  c.stream = st;
  c.attrs = at;
  c.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&c, kern, args...);
}

template <int ALG, int B>
static int launch_encode(const float* g, float* r, const uint8_t* in, uint8_t* out, uint64_t n,
                         const DenseParams& P, uint32_t tensor_id, uint64_t elem_offset,
                         int max_ctas, cudaStream_t st) {
  const uint32_t tiles = (uint32_t)num_tiles(n);
  WireHeader h;
  h.n = (uint32_t)n;
  h.alg = (uint8_t)ALG;
  h.bitwidth = (uint8_t)B;
  h.flags = dense_meta_floats(ALG) ? 1 : 0;
  h.a = ALG == kTbq ? P.tau : 0.0f;
  h.b = kTile;
  auto kern = in ? (r ? dense_encode_kernel<ALG, B, true, true> : dense_encode_kernel<ALG, B, true, false>)
                 : (r ? dense_encode_kernel<ALG, B, false, true> : dense_encode_kernel<ALG, B, false, false>);
  return launch_early(kern, grid_of(tiles, max_ctas), st, g, r, payload_ptrs(in, ALG, n), payload_ptrs(out, ALG, n),
                      h, (uint32_t)n, tiles, P, tensor_id, elem_offset);
}

template <int ALG, int B>
static int launch_decode(const uint8_t* p, float* out, uint64_t n, float tau, float scale,
                         int acc, int max_ctas, cudaStream_t st) {
  const uint32_t tiles = (uint32_t)num_tiles(n);
  auto kern = acc ? dense_decode_kernel<ALG, B, true> : dense_decode_kernel<ALG, B, false>;
  return launch_early(kern, grid_of(tiles, max_ctas), st, payload_ptrs(p, ALG, n), out, (uint32_t)n, tiles, tau, scale);
}

}  // namespace hipress

using namespace hipress;

#define HP_DISPATCH_DENSE(alg, bits, CALL)                         \
  do {                                                             \
    if (alg == kOnebit && bits == 1) { CALL(kOnebit, 1); }         \
    else if (alg == kTbq && bits == 2) { CALL(kTbq, 2); }          \
    else if (alg == kTernGrad && bits == 1) { CALL(kTernGrad, 1); }\
    else if (alg == kTernGrad && bits == 2) { CALL(kTernGrad, 2); }\
    else if (alg == kTernGrad && bits == 4) { CALL(kTernGrad, 4); }\
    else if (alg == kTernGrad && bits == 8) { CALL(kTernGrad, 8); }\
    else return HP_ERR_BAD_ARG;                                    \
  } while (0)

extern "C" {

int hp_cuda_dense_encode(int alg, int bits, const float* g, float* r, const uint8_t* in_payload,
                         uint8_t* out, uint64_t n, float tau, uint64_t seed, uint32_t step,
                         uint32_t salt, uint32_t tensor_id, uint64_t elem_offset, int max_ctas,
                         void* stream) {
  if (n == 0) return 0;
  if (n > 0xFFFFF000ull || (elem_offset & 3)) return HP_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(in_payload) & 15))
    return HP_ERR_BAD_ARG;
  DenseParams P{tau, step, salt, (uint32_t)seed, (uint32_t)(seed >> 32)};
  cudaStream_t st = (cudaStream_t)stream;
#define CALL(A, B) return launch_encode<A, B>(g, r, in_payload, out, n, P, tensor_id, elem_offset, max_ctas, st)
  HP_DISPATCH_DENSE(alg, bits, CALL);
#undef CALL
  return 0;
}

int hp_cuda_dense_decode(int alg, int bits, const uint8_t* payload, float* out, uint64_t n,
                         float tau, float scale, int accumulate, int max_ctas, void* stream) {
  if (n == 0) return 0;
  if (n > 0xFFFFF000ull || (reinterpret_cast<uintptr_t>(payload) & 15)) return HP_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
#define CALL(A, B) return launch_decode<A, B>(payload, out, n, tau, scale, accumulate, max_ctas, st)
  HP_DISPATCH_DENSE(alg, bits, CALL);
#undef CALL
  return 0;
}

}  // extern "C"
