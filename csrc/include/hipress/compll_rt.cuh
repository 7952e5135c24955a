// Run-time support for code generated by hipress_b200.compll: unaligned header
// access, sub-byte vector reads and the per-element random source.  Compiles as
// device code under nvcc and as plain C++ for the generator's CPU target, so both
// targets of one DSL function draw the same random numbers and pack the same bits.
#pragma once
#include <stdint.h>
#include <string.h>

#include "hipress/common.h"

#if defined(__CUDACC__)
#define COMPLL_FN __device__ __forceinline__
#else
#define COMPLL_FN static inline
#endif

// header fields sit at arbitrary byte offsets (the DSL's concat packs them
// back to back), so they are moved bytewise
template <typename T>
COMPLL_FN T compll_load(const uint8_t* p) {
  T v;
  uint8_t* d = reinterpret_cast<uint8_t*>(&v);
#pragma unroll
  for (int i = 0; i < (int)sizeof(T); ++i) d[i] = p[i];
  return v;
}

template <typename T>
COMPLL_FN void compll_store(uint8_t* p, T v) {
  const uint8_t* s = reinterpret_cast<const uint8_t*>(&v);
#pragma unroll
  for (int i = 0; i < (int)sizeof(T); ++i) p[i] = s[i];
}

// element i of a vector of `bits`-wide unsigned values packed LSB-first
COMPLL_FN uint32_t compll_get_bits(const uint8_t* v, uint64_t i, uint32_t bits) {
  const uint64_t bit = i * bits;
  return (v[bit >> 3] >> (bit & 7)) & ((1u << bits) - 1u);
}

// uniform in [0,1): Philox4x32-7 keyed by the seed, counter = (element / 4, call
// site); element i takes word i % 4 of the call, so code that handles four
// consecutive elements per thread pays one call for the four.
COMPLL_FN hipress::Philox4 compll_rand4(uint64_t seed, uint64_t group, uint32_t site) {
  return hipress::philox4x32((uint32_t)group, (uint32_t)(group >> 32), site, 0u, (uint32_t)seed,
                             (uint32_t)(seed >> 32));
}
COMPLL_FN float compll_rand01(uint64_t seed, uint64_t elem, uint32_t site) {
  return hipress::u01(compll_rand4(seed, elem >> 2, site).v[elem & 3]);
}

// Quotients with one divisor, rounded as `/` rounds them, from a product and three fused
// multiply-adds.  hi + lo is 1/b to about 47 bits (hi rounded to nearest), so q is within
// one unit of a/b, the remainder a - b*q is exact, and q + remainder * hi rounds to the
// nearest float (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990; the two-part reciprocal is from N. Brisebarre, J.-M. Muller
// and S. K. Raina, "Accelerating correctly rounded floating-point division when the divisor
// is known in advance", 2004).  Holds while nothing overflows or gets subnormal: for b in
// [2^-60, 2^61) (`ok`) and |a| in [2^-63, 2^65) -- of anything else, zero included,
// compll_div sets the top bit of `bad`, and the caller divides instead.
struct CompllDivisor {
  float b, hi, lo;
  bool ok;
};
COMPLL_FN CompllDivisor compll_divisor(float b) {
  CompllDivisor d;
  d.b = b;
  d.hi = 1.0f / b;
  d.lo = fmaf(-b, d.hi, 1.0f) * d.hi;
  d.ok = b >= 0x1p-60f && b < 0x1p61f;
  return d;
}
COMPLL_FN float compll_div(float a, const CompllDivisor& d, uint32_t& bad) {
  uint32_t bits;
  memcpy(&bits, &a, 4);
  bad |= (bits << 1) - (64u << 24);   // its exponent, from 0 where the quotient is exact
  const float q = fmaf(a, d.hi, a * d.lo);
  return fmaf(fmaf(-d.b, q, a), d.hi, q);
}

#if defined(__CUDACC__)
// ---- support of the fused (one launch per function) target --------------------
// a bit width known when the code is compiled
template <uint32_t W>
struct CompllWidth {
  __device__ constexpr operator uint32_t() const { return W; }
};
template <bool V>
struct CompllFlag {
  __device__ constexpr operator bool() const { return V; }
};
// Philox4x32-7 of one seed: the keys of the rounds are made once, not for every call (two
// additions a round, a tenth of TernGradEncode's instructions)
struct CompllRand {
  uint32_t k0[hipress::kPhiloxRounds], k1[hipress::kPhiloxRounds];
  __device__ __forceinline__ explicit CompllRand(uint64_t seed) {
#pragma unroll
    for (int r = 0; r < hipress::kPhiloxRounds; ++r) {
      k0[r] = (uint32_t)seed + r * 0x9E3779B9u;
      k1[r] = (uint32_t)(seed >> 32) + r * 0xBB67AE85u;
    }
  }
  // compll_rand4 of a group below 2^32
  __device__ __forceinline__ hipress::Philox4 operator()(uint32_t group, uint32_t site) const {
    uint32_t c0 = group, c1 = 0u, c2 = site, c3 = 0u;
#pragma unroll
    for (int r = 0; r < hipress::kPhiloxRounds; ++r) {
      uint32_t hi0, lo0, hi1, lo1;
      hipress::philox_mulhilo(0xD2511F53u, c0, hi0, lo0);
      hipress::philox_mulhilo(0xCD9E8D57u, c2, hi1, lo1);
      c0 = hi1 ^ c1 ^ k0[r];
      c1 = lo1;
      c2 = hi0 ^ c3 ^ k1[r];
      c3 = lo0;
    }
    return hipress::Philox4{{c0, c1, c2, c3}};
  }
};
// Groups of four elements that lie in whole blocks of 256 groups, where every vector can
// be read and written 16 bytes at a time; none when a vector is off alignment or a group's
// number does not fit 31 bits.
__device__ __forceinline__ uint32_t compll_whole(uint64_t count, uint64_t addresses) {
  return (addresses & 15) == 0 && count < (1ull << 33) ? (uint32_t)(count / 1024) * 256u : 0u;
}
// four consecutive floats starting at element i0 (a multiple of 4) of a vector of n
__device__ __forceinline__ void compll_load4(const float* p, uint64_t i0, uint64_t n, float (&v)[4]) {
  if (i0 + 3 < n && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const float4 t = *reinterpret_cast<const float4*>(p + i0);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = i0 + e < n ? p[i0 + e] : 0.0f;
  }
}
__device__ __forceinline__ void compll_store4(float* p, uint64_t i0, uint64_t n, const float (&v)[4]) {
  if (i0 + 3 < n && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    *reinterpret_cast<float4*>(p + i0) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (i0 + e < n) p[i0 + e] = v[e];
  }
}
template <typename T>
__device__ __forceinline__ void compll_load4(const T* p, uint64_t i0, uint64_t n, T (&v)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] = i0 + e < n ? p[i0 + e] : T(0);
}
template <typename T>
__device__ __forceinline__ void compll_store4(T* p, uint64_t i0, uint64_t n, const T (&v)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (i0 + e < n) p[i0 + e] = v[e];
}

// The 4*bits-bit fragment of group q (elements 4q .. 4q+3) of a sub-byte vector: one
// aligned 32-bit load when the address allows, byte loads otherwise; bytes at or past
// `nbytes` read as zero.  Element e of the group is (frag >> (e * bits)) & mask.
__device__ __forceinline__ uint32_t compll_load_frag(const uint8_t* v, uint64_t nbytes, uint64_t q,
                                                     uint32_t bits) {
  const uint64_t bit = q * 4u * bits;
  const uint64_t off = bit >> 3;
  if (off >= nbytes) return 0u;
  const uint32_t width = 4u * bits;             // 4, 8, 16 or 32 bits
  uint32_t w;
  if (width == 32 && off + 4 <= nbytes && (reinterpret_cast<uintptr_t>(v + off) & 3) == 0) {
    w = *reinterpret_cast<const uint32_t*>(v + off);
  } else if (width >= 16 && off + width / 8 <= nbytes && (reinterpret_cast<uintptr_t>(v + off) & 1) == 0) {
    w = *reinterpret_cast<const uint16_t*>(v + off);
    if (width == 32) w |= (uint32_t)*reinterpret_cast<const uint16_t*>(v + off + 2) << 16;
  } else {
    const uint32_t nb = width <= 8 ? 1u : width / 8u;
    w = 0u;
    for (uint32_t b = 0; b < nb && off + b < nbytes; ++b) w |= (uint32_t)v[off + b] << (8 * b);
  }
  w >>= (uint32_t)(bit & 7);
  return width >= 32 ? w : (w & ((1u << width) - 1u));
}

// Warp-level packing of a sub-byte vector.  Every lane of the warp calls with the
// 4*bits-bit fragment `frag` of its group q of four elements (0 beyond the end);
// lanes cooperate through shuffles so that whole 32-bit words leave the warp.
// `dst` is the vector's first byte, `nbytes` its length: nothing past it is written.
__device__ __forceinline__ void compll_pack_store(uint8_t* dst, uint64_t nbytes, uint64_t q,
                                                  uint32_t frag, uint32_t bits) {
  if ((reinterpret_cast<uintptr_t>(dst) & 3) != 0) {
    // behind a header of an odd length: every lane stores its own one, two or four bytes,
    // or with one bit every second lane a byte
    if (bits == 1) {
      const uint32_t hi = __shfl_down_sync(0xffffffffu, frag, 1);
      if (!(q & 1) && q / 2 < nbytes) dst[q / 2] = (uint8_t)(frag | (hi << 4));
      return;
    }
    const uint64_t off = q * bits / 2;
    const uint32_t nb = bits / 2;
    uint8_t* p = dst + off;
    if (nb >= 2 && (reinterpret_cast<uintptr_t>(p) & 1) == 0 && off + nb <= nbytes) {
      *reinterpret_cast<uint16_t*>(p) = (uint16_t)frag;
      if (nb == 4) *reinterpret_cast<uint16_t*>(p + 2) = (uint16_t)(frag >> 16);
    } else {
      for (uint32_t b = 0; b < nb && off + b < nbytes; ++b) p[b] = (uint8_t)(frag >> (8 * b));
    }
    return;
  }
  const uint32_t lanes = 8u / bits;            // lanes per 32-bit word: 8, 4, 2, 1
  uint32_t w = frag;
  for (uint32_t s = 1, sh = 4u * bits; s < lanes; s <<= 1, sh <<= 1) {
    const uint32_t o = __shfl_down_sync(0xffffffffu, w, s);
    w |= o << sh;
  }
  if ((q & (lanes - 1)) != 0) return;           // only the first lane of a word stores
  const uint64_t off = q * bits / 2;            // byte offset of group q: 4 * bits / 8 per group
  if (off >= nbytes) return;
  uint8_t* p = dst + off;
  if (off + 4 <= nbytes && (reinterpret_cast<uintptr_t>(p) & 3) == 0) {
    *reinterpret_cast<uint32_t*>(p) = w;
  } else {
    for (uint32_t b = 0; b < 4 && off + b < nbytes; ++b) p[b] = (uint8_t)(w >> (8 * b));
  }
}

// The same for a warp whose groups are all complete: no bounds.
__device__ __forceinline__ void compll_pack_full(uint8_t* dst, uint32_t q, uint32_t frag, uint32_t bits) {
  const uint32_t low = (uint32_t)reinterpret_cast<uintptr_t>(dst) & 3u;
  if (bits == 8 && low == 0) {
    reinterpret_cast<uint32_t*>(dst)[q] = frag;
  } else if (bits >= 4 && (low & 1u) == 0) {
    uint16_t* p = reinterpret_cast<uint16_t*>(dst + (uint64_t)q * (bits / 2));
    p[0] = (uint16_t)frag;
    if (bits == 8) p[1] = (uint16_t)(frag >> 16);
  } else if (bits == 1 || low == 0) {
    const uint32_t lanes = low == 0 ? 8u / bits : 2u;   // whose bits go out together
    for (uint32_t s = 1, sh = 4u * bits; s < lanes; s <<= 1, sh <<= 1) frag |= __shfl_down_sync(0xffffffffu, frag, s) << sh;
    if ((q & (lanes - 1)) != 0) return;
    if (low == 0) reinterpret_cast<uint32_t*>(dst)[q / lanes] = frag;
    else dst[q / 2] = (uint8_t)frag;
  } else {
    for (uint32_t b = 0; b < bits / 2; ++b) dst[(uint64_t)q * (bits / 2) + b] = (uint8_t)(frag >> (8 * b));
  }
}

// Barrier over the blocks of a cooperative launch.  `word` counts arrivals, word[32] is
// the number of the last complete barrier (both zero when the kernel starts), `gen` is
// the caller's running barrier number.  Bounded: after
// about a second of polling a block gives up, raises `*err` and goes on.
__device__ __forceinline__ void compll_grid_sync(unsigned int* word, unsigned int& gen,
                                                 unsigned int* err) {
  __syncthreads();
  ++gen;
  if (threadIdx.x == 0) {
    unsigned int before, v;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(word) : "memory");
    unsigned int* flag = word + 32;   // polled apart from the word everybody adds to
    if (before == gen * gridDim.x - 1) {
      __threadfence();
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(gen) : "memory");
    } else {
      unsigned long long spins = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v >= gen) break;
        if (++spins > (1ull << 23)) {
          *err = 1u;
          break;
        }
      }
    }
  }
  __syncthreads();
}
#endif
