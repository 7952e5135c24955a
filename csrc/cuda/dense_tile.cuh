// Tile-level device code shared by the stand-alone encode/decode kernels and by
// the fused ring / parameter-server kernels.
//
// A tile is kTile (4096) consecutive fp32 elements handled by one 256-thread
// CTA: every thread keeps 16 elements in registers (four float4 at float4-index
// j*256+tid), so the residual add, the per-tile scale or min/max reduction, the
// quantisation and the residual write-back all happen on one pass over HBM
// (12 B/element with error feedback, 4 B/element without).  The reference does
// this with two synchronising thrust::reduce calls, a thrust::transform with
// one thread per output byte and four host memcpys per tensor
// (src/CompLL/GCGen/output/TernGradEncode/TernGradEncode_body.h:115-123).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "hipress/common.h"

namespace hipress {

constexpr int kThreads = 256;
constexpr int kIter = kTile / (kThreads * 4);  // float4 per thread per tile
static_assert(kIter * kThreads * 4 == kTile, "tile must split evenly");

struct TileSmem {
  double red_d[2][kThreads / 32];
  float2 red_f[2][kThreads / 32];
};

// ------------------------------------------------------------------ memory ops
__device__ __forceinline__ void load_tile(const float* __restrict__ p, int m,
                                          float (&x)[kIter][4]) {
  const bool vec = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
#pragma unroll
  for (int j = 0; j < kIter; ++j) {
    const int i0 = 4 * (j * kThreads + (int)threadIdx.x);
    if (vec && i0 + 3 < m) {
      const float4 v = *reinterpret_cast<const float4*>(p + i0);
      x[j][0] = v.x; x[j][1] = v.y; x[j][2] = v.z; x[j][3] = v.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[j][e] = (i0 + e < m) ? p[i0 + e] : 0.0f;
    }
  }
}

__device__ __forceinline__ void store_tile(float* __restrict__ p, int m,
                                           const float (&x)[kIter][4]) {
  const bool vec = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
#pragma unroll
  for (int j = 0; j < kIter; ++j) {
    const int i0 = 4 * (j * kThreads + (int)threadIdx.x);
    if (vec && i0 + 3 < m) {
      *reinterpret_cast<float4*>(p + i0) = make_float4(x[j][0], x[j][1], x[j][2], x[j][3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (i0 + e < m) p[i0 + e] = x[j][e];
    }
  }
}

// a full tile at a 16-byte aligned address: no per-element checks
__device__ __forceinline__ void load_tile_full(const float* __restrict__ p, float (&x)[kIter][4]) {
#pragma unroll
  for (int j = 0; j < kIter; ++j) {
    const float4 v = reinterpret_cast<const float4*>(p)[j * kThreads + (int)threadIdx.x];
    x[j][0] = v.x; x[j][1] = v.y; x[j][2] = v.z; x[j][3] = v.w;
  }
}
__device__ __forceinline__ void store_tile_full(float* __restrict__ p, const float (&x)[kIter][4]) {
#pragma unroll
  for (int j = 0; j < kIter; ++j)
    reinterpret_cast<float4*>(p)[j * kThreads + (int)threadIdx.x] =
        make_float4(x[j][0], x[j][1], x[j][2], x[j][3]);
}
__device__ __forceinline__ bool tile_is_full_aligned(const float* p, int m) {
  return m == kTile && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// Code fragment = the 4*B bits of the four elements of one float4.
// Payload bytes that another GPU wrote are read with ld.global.cg (L2 only).
template <int B>
__device__ __forceinline__ uint32_t load_frag(const uint8_t* __restrict__ codes, int j, int m) {
  const int f = j * kThreads + (int)threadIdx.x;
  if (4 * f >= m) return 0u;
  if (B == 1) {
    const uint32_t b = __ldcg(codes + (f >> 1));
    return (f & 1) ? (b >> 4) : (b & 15u);
  } else if (B == 2) {
    return __ldcg(codes + f);
  } else if (B == 4) {
    return __ldcg(reinterpret_cast<const unsigned short*>(codes) + f);
  } else {
    return __ldcg(reinterpret_cast<const unsigned int*>(codes) + f);
  }
}

__device__ __forceinline__ int tile_code_bytes(int m, int bits) {
  return (int)align_up(((uint32_t)m * bits + 7) / 8, 16);
}

// The code bytes of one tile, straight from the registers: a warp's row is 16 to 128
// consecutive bytes, so the stores are as wide as the codes allow and need no shared
// memory and no barrier.  Bytes behind the last code of a partial tile are zero up to
// the next multiple of 16.
template <int B>
__device__ __forceinline__ void store_codes(uint8_t* __restrict__ dst, int m, const uint32_t (&frag)[kIter]) {
  const int nbytes = tile_code_bytes(m, B);
#pragma unroll
  for (int j = 0; j < kIter; ++j) {
    const int f = j * kThreads + (int)threadIdx.x;
    if (B == 1) {
      const uint32_t hi = __shfl_down_sync(0xffffffffu, frag[j], 1);
      if (!(threadIdx.x & 1) && (f >> 1) < nbytes) dst[f >> 1] = (uint8_t)(frag[j] | (hi << 4));
    } else if (f * B / 2 < nbytes) {
      if (B == 2) dst[f] = (uint8_t)frag[j];
      else if (B == 4) reinterpret_cast<uint16_t*>(dst)[f] = (uint16_t)frag[j];
      else reinterpret_cast<uint32_t*>(dst)[f] = frag[j];
    }
  }
}

// ------------------------------------------------------------- block reductions
// All 256 threads must call; every thread returns the same value.  One barrier each:
// `buf` (0 or 1) picks the shared array, and two calls with no other barrier in between
// take different ones.
__device__ __forceinline__ double block_sum(double v, TileSmem& s, int buf) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s.red_d[buf][threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) t += s.red_d[buf][w];
  return t;
}

// Warp level: one redux.sync.{min,max}.f32 each (the fp32 forms of the warp
// reduction are sm_100a instructions) instead of five shuffle + compare rounds; every
// warp reduces the eight partial results the same way.
__device__ __forceinline__ void block_minmax(float& mn, float& mx, TileSmem& s, int buf) {
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(mn) : "f"(mn));
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(mx) : "f"(mx));
  if ((threadIdx.x & 31) == 0) s.red_f[buf][threadIdx.x >> 5] = make_float2(mn, mx);
  __syncthreads();
  const float2 v = s.red_f[buf][threadIdx.x & (kThreads / 32 - 1)];
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(mn) : "f"(v.x));
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(mx) : "f"(v.y));
}

// ------------------------------------------------------------------ algorithms
// decode the four elements of fragment j into d[0..3]
template <int ALG, int B>
__device__ __forceinline__ void decode_frag(uint32_t frag, const float (&meta)[2], float tau,
                                            float (&d)[4]) {
  constexpr uint32_t mask = (1u << B) - 1u;
  float gap = 0.0f;
  if (ALG == kTernGrad) gap = tern_gap(meta[0], meta[1], B);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (ALG == kTernGrad) {
      // the code as a float without a shift or a conversion (which run at an eighth of
      // the rate of a multiply-add): its bits are or-ed in place into the mantissa of
      // 2^23, and one exact multiply-add takes the place value and the 2^23 off again
      const int sh = B == 8 ? 0 : e * B;
      const uint32_t bits = B == 8 ? __byte_perm(frag, 0x4B000000u, 0x7650u | e)
                                   : ((frag & (mask << sh)) | 0x4B000000u);
      const float place = 1.0f / (float)(1u << sh);
      const float q = fmaf(__uint_as_float(bits), place, -8388608.0f * place);
      d[e] = fmaf(q, gap, meta[0]);   // tern_value
    } else if (ALG == kTbq) {
      // tbq_value of the 2-bit code at bits 2e, 2e+1 by testing the bits in place
      // (bit 1: non-zero level, bit 0: positive)
      const bool nz = (frag & (2u << (e * B))) != 0u, pos = (frag & (1u << (e * B))) != 0u;
      d[e] = nz ? (pos ? tau : -tau) : 0.0f;
    } else {
      d[e] = onebit_value((frag >> (e * B)) & mask, meta[0]);
    }
  }
}

// three-input minimum / maximum (sm_100a); like fminf / fmaxf they skip NaNs
__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Four TernGrad codes (tern_code of x[0..3] with the draws rnd16(v[e], half)) as the
// fragment of one float4.  Bound by the integer pipe, which runs at half the rate of the
// multiply-adds, and by the conversion unit at an eighth, so the work is moved off both:
//   * up to 4 bits the position t = (x - min) * scale16 stays below 2^20, and its floor
//     comes from adding 2^23 rounding down.  The product is taken 2^(16+B) smaller
//     (exact), so that the saturating multiply maps NaN to 0 and infinity to a clamped
//     code for free, and the multiply-add that adds 2^23 scales it back.  `scale` is
//     scale16 / 2^(16+B) then.  8-bit positions need 24 bits: they are converted.
//   * the draw is added and the sum clamped in one instruction; the code is byte 2
//   * bytes are gathered with permutes, and for 1 and 2 bits packed with one dot product
template <int B>
__device__ __forceinline__ uint32_t tern_frag(const float (&x)[4], float mn, float scale, const Philox4& rnd,
                                              uint32_t half) {
  constexpr uint32_t qmax = (1u << B) - 1u;
  uint32_t w[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t u16 = rnd16(rnd.v[e], half);
    if (B == 8) {
      w[e] = __viaddmin_u32((uint32_t)f2i_floor_sat((x[e] - mn) * scale), u16, (qmax << 16) | 0xFFFFu);
    } else {
      const float y = __fmaf_rd(__saturatef((x[e] - mn) * scale), (float)(1u << (16 + B)), 8388608.0f);
      w[e] = __viaddmin_u32(__float_as_uint(y), u16, 0x4B00FFFFu | (qmax << 16));
    }
  }
  const uint32_t c = __byte_perm(__byte_perm(w[0], w[1], 0x0062), __byte_perm(w[2], w[3], 0x0062), 0x5410);
  if (B == 8) return c;
  if (B == 4) return __byte_perm(c | (c >> 4), 0u, 0x4420);
  return __dp4a(c, B == 2 ? 0x40100401u : 0x08040201u, 0u);
}

// Quantise the register tile x (m valid elements).  On return frag[] holds the
// code fragments (zero for elements past m), meta[] the tile metadata, and x the
// quantisation error x - decode(code) of every valid element (left untouched by
// TernGrad when the caller keeps no residual: want_err = false).
template <int ALG, int B, bool FULL, bool ERR>
__device__ __forceinline__ void encode_tile_impl(float (&x)[kIter][4], int m, const DenseParams& P,
                                                 uint32_t tensor_id, uint64_t elem0, uint32_t salt,
                                                 TileSmem& s, int buf, float (&meta)[2],
                                                 uint32_t (&frag)[kIter]) {
  meta[0] = 0.0f;
  meta[1] = 0.0f;
  if (ALG == kOnebit) {
    double part = 0.0;
#pragma unroll
    for (int j = 0; j < kIter; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (FULL || 4 * (j * kThreads + (int)threadIdx.x) + e < m) part += (double)fabsf(x[j][e]);
    const double tot = block_sum(part, s, buf);
    meta[0] = (float)(tot / (double)m);
  } else if (ALG == kTernGrad) {
    float mn = INFINITY, mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < kIter; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (FULL || 4 * (j * kThreads + (int)threadIdx.x) + e < m) {
          mn = fminf(mn, x[j][e]);
          mx = fmaxf(mx, x[j][e]);
        }
    block_minmax(mn, mx, s, buf);
    meta[0] = mn;
    meta[1] = mx;
  }
  float gap = 0.0f, scale16 = 0.0f;
  if (ALG == kTernGrad) {
    gap = tern_gap(meta[0], meta[1], B);
    scale16 = tern_scale16(gap);
  }
  // TernGrad: one Philox call per pair of rows (see rnd16_counter); a tile that does
  // not start on a 2048-element boundary of its tensor cannot share calls
  const bool paired = ALG != kTernGrad || (elem0 & 2047u) == 0;
  Philox4 rnd;
#pragma unroll
  for (int j = 0; j < kIter; ++j) {
    const int i0 = 4 * (j * kThreads + (int)threadIdx.x);
    uint32_t half = 0u;
    if (ALG == kTernGrad) {
      const uint64_t ge = elem0 + (uint64_t)i0;
      half = paired ? (uint32_t)(j & 1) : rnd16_half(ge);
      if (!paired || !(j & 1))
        rnd = philox4x32(rnd16_counter(ge), tensor_id, P.step, salt, P.seed_lo, P.seed_hi);
    }
    uint32_t f = 0u;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (FULL || i0 + e < m) {
        uint32_t c;
        float d;
        if (ALG == kOnebit) {
          c = onebit_code(x[j][e]);
          d = onebit_value(c, meta[0]);
        } else if (ALG == kTbq) {
          // tbq_code and tbq_value of it from one pair of compares
          const bool pos = x[j][e] >= P.tau, neg = x[j][e] <= -P.tau;
          c = pos ? 3u : (neg ? 2u : 0u);
          d = pos ? P.tau : (neg ? -P.tau : 0.0f);
        } else {
          c = tern_code(x[j][e], meta[0], scale16, rnd16(rnd.v[e], half), B);
          d = ERR ? tern_value(c, meta[0], gap) : 0.0f;
        }
        f |= c << (e * B);
        if (ERR) x[j][e] = x[j][e] - d;
      }
    }
    frag[j] = f;
  }
}

// The usual TernGrad tile: full, no residual, on a 2048-element boundary of its tensor.
// The draws do not depend on the data, so they are made while its loads are in flight.
template <int B>
__device__ __forceinline__ void tern_encode_full(float (&x)[kIter][4], const DenseParams& P, uint32_t tensor_id,
                                                 uint64_t elem0, uint32_t salt, TileSmem& s, int buf,
                                                 float (&meta)[2], uint32_t (&frag)[kIter]) {
  static_assert(kIter == 4, "one draw serves two rows");
  Philox4 rnd[2];
#pragma unroll
  for (int p = 0; p < 2; ++p)
    rnd[p] = philox4x32(rnd16_counter(elem0 + 4u * (2 * p * kThreads + threadIdx.x)), tensor_id, P.step, salt,
                        P.seed_lo, P.seed_hi);
  float mn = fmin3(x[0][0], x[0][1], x[0][2]), mx = fmax3(x[0][0], x[0][1], x[0][2]);
  mn = fminf(mn, x[0][3]);
  mx = fmaxf(mx, x[0][3]);
#pragma unroll
  for (int j = 1; j < kIter; ++j)
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      mn = fmin3(mn, x[j][e], x[j][e + 1]);
      mx = fmax3(mx, x[j][e], x[j][e + 1]);
    }
  if (mn != mn) { mn = INFINITY; mx = -INFINITY; }   // sixteen NaNs
  block_minmax(mn, mx, s, buf);
  meta[0] = mn;
  meta[1] = mx;
  const float scale16 = tern_scale16(tern_gap(mn, mx, B));
  const float scale = B == 8 ? scale16 : scale16 * (1.0f / (float)(1u << (16 + B)));
  if (scale16 == 0.0f || scale >= 1.17549435e-38f) {
#pragma unroll
    for (int j = 0; j < kIter; ++j) frag[j] = tern_frag<B>(x[j], mn, scale, rnd[j >> 1], j & 1);
  } else {
    // a scale that is no longer a normal number (the tile spans more than about 2^120)
    // would lose bits: element by element
#pragma unroll
    for (int j = 0; j < kIter; ++j) {
      uint32_t f = 0u;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        f |= tern_code(x[j][e], mn, scale16, rnd16(rnd[j >> 1].v[e], j & 1), B) << (e * B);
      frag[j] = f;
    }
  }
}

// Quantises what the codes of a full tile decode to once more (the server's pass over one
// rank's push), from the codes alone.  Level L decodes to mn + L*gap, so the new extremes
// are the values of levels 0 and qmax, and the position of level L is 65536*L plus a
// rounding error `off` that is the same for the whole tile: the new code is L unless the
// draw u16 is within `off` of its end of the range.  A thread whose sixteen draws stay clear
// of both ends keeps its codes; the others (1 in 4096 when off is -1) take the element-wise
// way.  Instead of a decode, a minimum and maximum and sixteen roundings that is a pair of
// packed minima per draw, and no draw at all where every level is exact.  One rank, PS,
// 60 M elements, us per bucket: 1 bit 100.5 -> 74.8, 2 bits 103.6 -> 77.9, 8 bits 98.5 -> 90.9
// (8 bytes an element at the copy rate: 73).
// A tile without a gap (all zero, as the rows of an embedding that a batch did not touch, or
// of another constant) has codes of zero only, which decode to its minimum: both extremes of
// the new codes, zero again.  60 M elements, all constant, us, with every tile quantised
// twice / without this shortcut / with it: 1 bit 112 / 125 / 76, 2 bits 131 / 156 / 84, 8
// bits 125 / 154 / 82.
// False (for the whole CTA, nothing changed) when the tile is not finite, spans less than its
// values resolve, or lost its largest level to a draw.
template <int B>
__device__ __forceinline__ bool tern_requantise(uint32_t (&frag)[kIter], float (&meta)[2], const DenseParams& P,
                                                uint32_t tensor_id, uint64_t elem0, uint32_t salt, TileSmem& s) {
  constexpr uint32_t qmax = (1u << B) - 1u;
  static_assert(qmax < (uint32_t)kThreads, "a thread per level");
  const float mn = meta[0], gap = tern_gap(meta[0], meta[1], B);
  if (gap == 0.0f) {
    meta[0] = meta[1] = tern_value(0u, mn, gap);
    return true;
  }
  uint32_t top = 0u;   // a code of all ones; level 0 is there, it is the minimum's
#pragma unroll
  for (int j = 0; j < kIter; ++j) {
    uint32_t f = frag[j];
    if (B >= 2) f &= f >> 1;
    if (B >= 4) f &= f >> 2;
    if (B == 8) f &= f >> 4;
    top |= f & (B == 1 ? 0xFu : (B == 2 ? 0x55u : (B == 4 ? 0x1111u : 0x01010101u)));
  }
  const float mn2 = tern_value(0u, mn, gap), mx2 = tern_value(qmax, mn, gap);
  const float scale2 = tern_scale16(tern_gap(mn2, mx2, B));
  // every warp looks at all levels, or, when they are 256, at its 32 of them
  const uint32_t L = B == 8 ? threadIdx.x : threadIdx.x & 31;
  int lo = 0, hi = 0;
  if (L <= qmax) {
    lo = f2i_floor_sat((tern_value(L, mn, gap) - mn2) * scale2) - (int)(L << 16);
    hi = max(lo, 0);
    lo = min(lo, 0);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  int2* offs = reinterpret_cast<int2*>(s.red_d[0]);   // unused by TernGrad
  if (B == 8 && (threadIdx.x & 31) == 0) offs[threadIdx.x >> 5] = make_int2(lo, hi);
  const bool reached = __syncthreads_or(top != 0u);
  if (B == 8) {
    const int2 o = offs[threadIdx.x & (kThreads / 32 - 1)];
    lo = __reduce_min_sync(0xffffffffu, o.x);
    hi = __reduce_max_sync(0xffffffffu, o.y);
  }
  if (!(reached && gap > 0.0f && gap < INFINITY && lo >= -64 && hi <= 64)) return false;
  meta[0] = mn2;
  meta[1] = mx2;
  if (lo == 0 && hi == 0) return true;
  Philox4 rnd[2];
#pragma unroll
  for (int p = 0; p < 2; ++p)
    rnd[p] = philox4x32(rnd16_counter(elem0 + 4u * (2 * p * kThreads + threadIdx.x)), tensor_id, P.step, salt,
                        P.seed_lo, P.seed_hi);
  uint32_t least = rnd[0].v[0], most = rnd[0].v[0];
#pragma unroll
  for (int q = 1; q < 8; ++q) {
    least = __vminu2(least, rnd[q >> 2].v[q & 3]);
    most = __vmaxu2(most, rnd[q >> 2].v[q & 3]);
  }
  if ((int)min(least & 0xFFFFu, least >> 16) + lo < 0 || (int)max(most & 0xFFFFu, most >> 16) + hi > 0xFFFF) {
#pragma unroll
    for (int j = 0; j < kIter; ++j) {
      uint32_t f = 0u;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        f |= tern_code(tern_value((frag[j] >> (e * B)) & qmax, mn, gap), mn2, scale2, rnd16(rnd[j >> 1].v[e], j & 1), B)
             << (e * B);
      frag[j] = f;
    }
  }
  return true;
}

template <int ALG, int B>
__device__ __forceinline__ void encode_tile(float (&x)[kIter][4], int m, const DenseParams& P,
                                            uint32_t tensor_id, uint64_t elem0, uint32_t salt,
                                            TileSmem& s, int buf, float (&meta)[2],
                                            uint32_t (&frag)[kIter], bool want_err = true) {
  if (ALG == kTernGrad) {
    if (!want_err && m == kTile && (elem0 & 2047u) == 0)
      tern_encode_full<B>(x, P, tensor_id, elem0, salt, s, buf, meta, frag);
    else if (!want_err)
      encode_tile_impl<ALG, B, false, false>(x, m, P, tensor_id, elem0, salt, s, buf, meta, frag);
    else
      encode_tile_impl<ALG, B, false, true>(x, m, P, tensor_id, elem0, salt, s, buf, meta, frag);
  } else {
    if (m == kTile) encode_tile_impl<ALG, B, true, true>(x, m, P, tensor_id, elem0, salt, s, buf, meta, frag);
    else encode_tile_impl<ALG, B, false, true>(x, m, P, tensor_id, elem0, salt, s, buf, meta, frag);
  }
}

// read tile metadata that may have been written by a peer
template <int ALG>
__device__ __forceinline__ void load_meta(const float* meta, uint32_t t, float (&m)[2]) {
  m[0] = 0.0f;
  m[1] = 0.0f;
  if (ALG == kOnebit) m[0] = __ldcg(meta + t);
  if (ALG == kTernGrad) {
    m[0] = __ldcg(meta + 2 * t);
    m[1] = __ldcg(meta + 2 * t + 1);
  }
}

}  // namespace hipress
