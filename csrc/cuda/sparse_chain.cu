// Kernels and launches of the chain of selections (sparse_chain.cuh).
#include "sparse_chain.cuh"

namespace hipress {

constexpr int kChainThreads = 256;
constexpr uint32_t kChainTile = kSelTile / 2;   // two float4 of each array per thread
constexpr uint32_t kStretches = 16;
constexpr uint32_t kNoBase = 0xFFFFFFFFu;       // no places of a list

__device__ __forceinline__ void after_launches_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_launch_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Half tile h of an array: update, and what reaches the bound into its list, from part
// `part` on.
// HBM bound on large arrays; 256 threads and two vectors of each array per thread leave room
// for five CTAs on an SM, whose starts and ends overlap (six: no change), and for 48
// registers a thread, with which DGC's six loads are in flight together (20 M elements, DGC,
// ring: 97 us, 4.9 TB/s with the sample and the emit; 113 when compiled to 40).
template <int MODE>
__device__ __forceinline__ void chain_collect(const SelUnit& s, uint32_t* counts, float momentum, uint32_t h, uint32_t part) {
  __shared__ float val[kChainTile];
  __shared__ uint32_t idx[kChainTile];
  __shared__ uint32_t count, base;
  const bool vec = ((reinterpret_cast<uintptr_t>(s.a) | (MODE >= 1 ? reinterpret_cast<uintptr_t>(s.g) : 0) |
                     (MODE >= 1 ? reinterpret_cast<uintptr_t>(s.clear) : 0) |
                     (MODE == 2 ? reinterpret_cast<uintptr_t>(s.u) : 0)) & 15) == 0;
  const uint64_t i0 = (uint64_t)h * kChainTile + threadIdx.x * 4;
  const bool full = vec && (uint64_t)(h + 1) * kChainTile <= s.n;
  constexpr int kStep = kChainThreads * 4;
  float4 av[2], gv[2], uv[2];
  if (threadIdx.x == 0) count = 0;
  if (full) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      av[j] = *reinterpret_cast<const float4*>(s.a + i0 + j * kStep);
      if (MODE >= 1) gv[j] = *reinterpret_cast<const float4*>(s.g + i0 + j * kStep);
      if (MODE == 2) uv[j] = *reinterpret_cast<const float4*>(s.u + i0 + j * kStep);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      av[j] = ld4(s.a, i0 + j * kStep, s.n, vec);
      if (MODE >= 1) gv[j] = ld4(s.g, i0 + j * kStep, s.n, vec);
      if (MODE == 2) uv[j] = ld4(s.u, i0 + j * kStep, s.n, vec);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint64_t i = i0 + j * kStep;
    float4& v = av[j];
    if (MODE == 1) {
      v.x = v.x + gv[j].x; v.y = v.y + gv[j].y; v.z = v.z + gv[j].z; v.w = v.w + gv[j].w;
    } else if (MODE == 2) {
      float4& w = uv[j];
      w.x = __fmaf_rn(momentum, w.x, gv[j].x);
      w.y = __fmaf_rn(momentum, w.y, gv[j].y);
      w.z = __fmaf_rn(momentum, w.z, gv[j].z);
      w.w = __fmaf_rn(momentum, w.w, gv[j].w);
      v.x = v.x + w.x; v.y = v.y + w.y; v.z = v.z + w.z; v.w = v.w + w.w;
      if (full) *reinterpret_cast<float4*>(s.u + i) = w;
      else st4(s.u, i, s.n, vec, w);
    }
    if (MODE >= 1) {
      if (full) *reinterpret_cast<float4*>(s.a + i) = v;
      else st4(s.a, i, s.n, vec, v);
      if (s.clear) {
        if (full) *reinterpret_cast<float4*>(s.clear + i) = make_float4(0.f, 0.f, 0.f, 0.f);
        else st4(s.clear, i, s.n, vec, make_float4(0.f, 0.f, 0.f, 0.f));
      }
    }
  }
  after_launches_before();   // the bound
  const uint32_t low = __ldcg(s.ws + kWsLow), room = s.cap / kChainLists;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float e[4] = {av[j].x, av[j].y, av[j].z, av[j].w};
    if (max(max(abs_key(e[0]), abs_key(e[1])), max(abs_key(e[2]), abs_key(e[3]))) < low) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (abs_key(e[q]) < low) continue;
      const uint32_t p = atomicAdd(&count, 1u);
      val[p] = e[q];
      idx[p] = (uint32_t)i0 + j * kStep + q;
    }
  }
  __syncthreads();
  const uint32_t n = count;
  if (n == 0) return;
  // What finds no room in its part goes to the next one, so that an array whose large values
  // lie together (the rows of an embedding that a batch touched, a block of a matrix's
  // columns) fills all of the list: it overflowed at a seventh.  That it did is written by the
  // CTAs that find out, not by those that read it: thousands of stores to one word follow one
  // another (65 K large values of 6.6 M, GradDrop at 0.1 %, us: 194 with them, 104 without).
  uint32_t done = 0, of = part;
#pragma unroll 1
  for (uint32_t t = 0; done < n; ++t) {
    if (threadIdx.x == 0) {
      const bool known = t > 0 && __ldcg(s.ws + kWsOverflow) != 0u;
      if (t == kChainLists && !known) s.ws[kWsOverflow] = 1u;
      base = known || t == kChainLists ? kNoBase : atomicAdd(counts + 32 * of, n - done);
    }
    __syncthreads();
    const uint32_t at = base;
    if (at == kNoBase) return;
    const uint32_t end = at < room ? min(n, done + room - at) : done;
#pragma unroll 1
    for (uint32_t p = done + threadIdx.x; p < end; p += kChainThreads) {
      const float v = val[p];
      const uint32_t to = of * room + at + p - done;
      atomicAdd(s.ws + cand_digit(abs_key(v), low), 1u);
      s.cv[to] = v;
      list_indices(s)[to] = idx[p];
    }
    done = end;
    of = of + 1 == kChainLists ? 0 : of + 1;
    __syncthreads();
  }
}

__device__ __forceinline__ uint32_t chain_unit(const ChainArgs& A, uint32_t ChainUnit::* first, uint32_t i) {
  uint32_t lo = 0, hi = (uint32_t)A.units;
#pragma unroll 1
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (A.unit[mid].*first <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <int MODE>
__global__ void __launch_bounds__(kSpThreads, 2) chain_sample_kernel(const __grid_constant__ ChainArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SelSmem& sm = *reinterpret_cast<SelSmem*>(smem_raw);
  __shared__ SelUnit s;
  const uint32_t y = chain_unit(A, &ChainUnit::sample0, blockIdx.x);
  if (threadIdx.x == 0) s = A.unit[y].s;
  __syncthreads();
  after_launches_before();
  let_next_launch_begin();   // what lies before this launch is complete: the next one may read it too
  sample_body<MODE>(s, A.momentum, sm, blockIdx.x - A.unit[y].sample0, sm.stash[0]);
}

template <int MODE>
__global__ void __launch_bounds__(kChainThreads, 5) chain_collect_kernel(const __grid_constant__ ChainArgs A) {
  uint32_t b = blockIdx.x;
  if (A.stretch != 0u) {
    b = b % kStretches * A.stretch + b / kStretches;
    if (b >= 2 * A.tiles) return;
  }
  const uint32_t t = b / 2, y = chain_unit(A, &ChainUnit::tile0, t);
  const ChainUnit& u = A.unit[y];
  const uint32_t h = b - 2 * u.tile0, part = b % kChainLists;
  if (MODE != 0 && (t - u.tile0) % u.s.stride == 0) {
    after_launches_before();   // the sample's update
    chain_collect<0>(u.s, u.counts, 0.0f, h, part);
  } else {
    chain_collect<MODE>(u.s, u.counts, A.momentum, h, part);
  }
}

__device__ __forceinline__ ListState chain_state(const ChainUnit& u) {
  ListState l = {0u, __ldcg(u.s.ws + kWsOverflow), __ldcg(u.s.ws + kWsLow)};
#pragma unroll
  for (uint32_t p = 0; p < kChainLists; ++p) l.count += min(__ldcg(u.counts + 32 * p), u.s.cap / kChainLists);
  return l;
}

union ChainSmem {
  SelSmem sel;
  uint32_t hist[kBins];
  EmitSmem emit;
};

// Where the pairs of an array go; thread 0 fills `s` and `dst` in.  A CTA that has given up
// on a barrier may pick other elements than the largest, and leaves the result alone.
__device__ __forceinline__ void chain_aim(const ChainArgs& A, const ChainUnit& to, bool gave_up, SelUnit& s, EmitDst& dst) {
  if (threadIdx.x == 0) {
    s = to.s;
    dst.n = A.payload ? 1 : 0;
    dst.out[0] = A.payload;
    dst.add = to.add;
    dst.set = gave_up ? nullptr : to.set;
    dst.scale = A.scale;
  }
  __syncthreads();
}

// One of the passes over whole arrays, of the n arrays listed in `which` (or the first n):
// -1 clears the histograms, 0 to 2 count a digit each, 3 sends.  Between two of them all CTAs
// are done with the one before.  The arrays share the CTAs: each has histograms of its own,
// and its passes are short.
__device__ __forceinline__ void chain_pass(const ChainArgs& A, int pass, const uint8_t* which, uint32_t n, bool gave_up,
                                           SelUnit& s, EmitDst& dst, ChainSmem& sm, FindSmem& fs) {
  const uint32_t G = max(gridDim.x / n, 1u);
#pragma unroll 1
  for (uint32_t v = blockIdx.x; v < n * G; v += gridDim.x) {
    const uint32_t c = v % G;
    chain_aim(A, A.unit[which ? which[v / G] : v / G], gave_up, s, dst);
    if (pass < 0) {
      for (uint32_t i = c * kSpThreads + threadIdx.x; i < 3u * kBins; i += G * kSpThreads) s.ws[i] = 0;
    } else if (pass == 0) {
      pass0_body<0>(nullptr, s.a, nullptr, s.n, 0.0f, s.ws, sm.hist, c, G);
    } else if (pass < 3) {
      pass_body(pass, s.a, s.n, s.k, s.ws, sm.hist, fs, c, G);
    } else {
      emit_body(A.alg, s.a, s.u, s.n, s.k, s.kmax, dst, s.ws, fs, sm.emit, c, G);
    }
    __syncthreads();   // s and dst
  }
}

__global__ void __launch_bounds__(kSpThreads, 2) chain_emit_kernel(const __grid_constant__ ChainArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ChainSmem& sm = *reinterpret_cast<ChainSmem*>(smem_raw);
  __shared__ SelUnit s;
  __shared__ EmitDst dst;
  __shared__ WaitState wst;
  __shared__ FindSmem fs;
  __shared__ uint8_t failed[kChainUnits];
  __shared__ uint32_t nfailed;
  const uint32_t before = A.gave_up ? __ldcg(A.gave_up) : 0u;   // the chain before this one
  if (blockIdx.x < A.emitting) {
    const ChainEmitters em = A.emitters[blockIdx.x / kChainLists];
    const ChainUnit& u = A.unit[em.unit];
    const ListState ls = chain_state(u);
    chain_aim(A, u, before != 0, s, dst);
    if (!selection_failed(s, ls)) {
      // a part each; of several groups each takes a span of all parts
      const uint32_t part = blockIdx.x % kChainLists, sub = em.group, subs = em.groups;
      const uint32_t room = s.cap / kChainLists, n = min(__ldcg(u.counts + 32 * part), room);
      const uint32_t per = (n + subs - 1) / subs, lo = min(sub * per, n), hi = min(lo + per, n);
      emit_span(A.alg, s, ls, dst, sm.sel, part * room + lo, part * room + hi, kChainLists * subs);
    }
  }
  // whole-array passes for the units whose list is not complete; every CTA decides the same
  const bool bad = threadIdx.x < (uint32_t)A.units &&
                   selection_failed(A.unit[threadIdx.x].s, chain_state(A.unit[threadIdx.x]));
  if (!__syncthreads_or(bad)) return;
  if (threadIdx.x < (uint32_t)A.units) failed[threadIdx.x] = bad;
  wait_init(wst);
  if (threadIdx.x == 0) {
    wst.poisoned = before != 0;
    nfailed = 0;
    for (int q = 0; q < A.units; ++q)
      if (failed[q]) failed[nfailed++] = (uint8_t)q;
  }
  __syncthreads();
  uint32_t gen = 0;
#pragma unroll 1
  for (int pass = -1; pass <= 3; ++pass) {
    chain_pass(A, pass, failed, nfailed, wst.poisoned, s, dst, sm, fs);
    if (pass < 3) grid_barrier(A.barrier, gen, gridDim.x, kGridBarrierNs, A.status, A.code, wst);
  }
  if (A.gave_up && threadIdx.x == 0 && wst.poisoned) *A.gave_up = 1u;
}

// One of those passes for all arrays, as a launch of its own.
__global__ void __launch_bounds__(kSpThreads, 2) chain_pass_kernel(const __grid_constant__ ChainArgs A, int pass) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ChainSmem& sm = *reinterpret_cast<ChainSmem*>(smem_raw);
  __shared__ SelUnit s;
  __shared__ EmitDst dst;
  __shared__ FindSmem fs;
  chain_pass(A, pass, nullptr, (uint32_t)A.units, A.gave_up && __ldcg(A.gave_up), s, dst, sm, fs);
}

// ------------------------------------------------------------------ host side
int chain_per_sm(int dev) {
  static int known[64] = {};
  if (dev < 0 || dev >= 64) return 0;
  if (known[dev]) return known[dev] - 1;
  int per = 0;
  const void* big[] = {(const void*)chain_sample_kernel<0>, (const void*)chain_sample_kernel<1>,
                       (const void*)chain_sample_kernel<2>, (const void*)chain_emit_kernel,
                       (const void*)chain_pass_kernel};
  bool ok = true;
  for (const void* k : big)
    ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChainSmem)) == cudaSuccess;
  ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, chain_emit_kernel, kSpThreads, sizeof(ChainSmem)) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    per = 0;
  }
  known[dev] = per + 1;
  return per;
}

// groups of kChainLists CTAs that emit a list in one round, four candidates a thread
static uint64_t groups_for(uint64_t kmax) { return (kmax + kmax / 2) / (4 * kSpThreads * kChainLists) + 1; }

bool chain_place(ChainArgs& A, int per_sm, int sms) {
  uint64_t tiles = 0, samples = 0, wanted = 0, n = 0, k = 0;
  for (int i = 0; i < A.units; ++i) {
    SelUnit& s = A.unit[i].s;
    if (s.n == 0) return false;
    const uint32_t t = (s.n - 1) / kSelTile + 1;
    s.sampled = (t + s.stride - 1) / s.stride;
    A.unit[i].tile0 = (uint32_t)tiles;
    A.unit[i].sample0 = (uint32_t)samples;
    tiles += t;
    samples += s.sampled;
    wanted += groups_for(s.kmax) - 1;
    n += s.n;
    k += s.kmax;
  }
  const uint32_t fit = (uint32_t)(per_sm * sms) / kChainLists, most = fit < kChainGroups ? fit : kChainGroups;
  if (most < (uint32_t)A.units || tiles > 0x3FFFFFFFull) return false;
  // A group for each list, and of those that are left as many more as its length asks for,
  // or where they are too few its share of them.  In equal shares the longest list kept few
  // CTAs busy: 20 M elements and 30 arrays of 500, DGC, ring, us, equal / by length
  // (persistent kernels): 0.1 % 129 / 120 (138), 1 % 230 / 137 (256), 10 % 1218 / 288 (1033).
  const uint64_t spare = most - (uint32_t)A.units;
  uint32_t group = 0;
  for (int i = 0; i < A.units; ++i) {
    const uint64_t more = groups_for(A.unit[i].s.kmax) - 1;
    const uint32_t own = 1 + (uint32_t)(wanted <= spare ? more : more * spare / wanted);
    for (uint32_t q = 0; q < own; ++q) A.emitters[group++] = {(uint8_t)i, (uint8_t)q, (uint8_t)own};
  }
  A.emitting = kChainLists * group;
  // An array's CTAs wait for one another where they count its candidates' first digits: at a
  // few words in an owner's sum, which holds little but what was pushed, and else where many
  // are sent.  Several arrays are taken at a time then, by the bucket's half tiles in sixteen
  // stretches side by side.  Two arrays of 10 M elements, us, one stretch / sixteen
  // (persistent kernels): PS, the sums alone, DGC, 1 % 222 / 197 (240), 3 % 355 / 290 (334);
  // ring, GradDrop, 0.1 % 81.2 / 82.0 (96), 1 % 93.9 / 93.2 (115), 3 % 170 / 129 (159), 10 %
  // 412 / 267 (303).  Half tiles of an update are fastest in order: one of 16 M elements, one
  // of 8 M and so on, DGC, ring, 0.1 % 150 / 152 (188), 1 % 185 / 186 (237), 3 % 241 / 232
  // (309).
  const bool sums = A.unit[0].s.g == nullptr;
  A.tiles = (uint32_t)tiles;
  A.stretch = A.units > 1 && (sums || k * 50 >= n) ? (uint32_t)((2 * tiles + kStretches - 1) / kStretches) : 0u;
  // One CTA per SM for the passes over whole arrays, up to a tile each.  Of 6.6 M elements,
  // 40 rows of 1024 not zero, GradDrop at 0.1 % (encode, us): the emitters alone 658, one per
  // SM 88, two 78; but where no list comes out short two cost the 25 MB bucket 1.9 us, one
  // nothing.
  const uint64_t busy = A.emitting, wide = tiles < (uint64_t)sms ? tiles : (uint64_t)sms;
  A.ctas = (uint32_t)(busy > wide ? busy : wide);
  return true;
}

template <typename K>
static cudaError_t chain_launch(K kern, uint32_t grid, int threads, size_t smem, bool early, cudaStream_t st, const ChainArgs& A) {
  cudaLaunchAttribute at;
  at.id = early ? cudaLaunchAttributeProgrammaticStreamSerialization : cudaLaunchAttributeCooperative;
  if (early) at.val.programmaticStreamSerializationAllowed = 1;
  else at.val.cooperative = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, A);
}

template <int MODE>
static cudaError_t chain_select_mode(const ChainArgs& A, cudaStream_t st) {
  const ChainUnit& last = A.unit[A.units - 1];
  const uint32_t tiles = last.tile0 + (last.s.n - 1) / kSelTile + 1, samples = last.sample0 + last.s.sampled;
  cudaError_t e = chain_launch(chain_sample_kernel<MODE>, samples, kSpThreads, sizeof(SelSmem), true, st, A);
  const uint32_t halves = A.stretch ? kStretches * A.stretch : 2 * tiles;
  if (e == cudaSuccess) e = chain_launch(chain_collect_kernel<MODE>, halves, kChainThreads, 0, true, st, A);
  if (e == cudaSuccess)
    e = chain_launch(chain_emit_kernel, A.ctas, kSpThreads, sizeof(ChainSmem), false, st, A);
  if (e != cudaErrorCooperativeLaunchTooLarge) return e;
  // Less of the GPU is ours than the queries said, and the arrays are updated by now: what
  // the emitting CTAs do together, in launches that need no co-residency.
  cudaGetLastError();
  const uint32_t grid = tiles < 148u * 2u ? tiles : 148u * 2u;
  for (int pass = -1; pass <= 3; ++pass) chain_pass_kernel<<<grid, kSpThreads, sizeof(ChainSmem), st>>>(A, pass);
  return cudaGetLastError();
}

cudaError_t chain_select(int mode, const ChainArgs& A, cudaStream_t st) {
  return mode == 0 ? chain_select_mode<0>(A, st) : (mode == 1 ? chain_select_mode<1>(A, st) : chain_select_mode<2>(A, st));
}

}  // namespace hipress
