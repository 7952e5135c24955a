// Fused CaSync-PS and CaSync-Ring for the top-k algorithms (DGC, GradDrop): ONE
// persistent cooperative launch per bucket, no NCCL call, no host round trip.  The
// stages below run as grid-synchronised phases of that launch (a bounded barrier
// over the launch's own CTAs between phases that depend on one another); waiting
// across GPUs happens on release / acquire flags, as in the dense kernels.
//
//   push   : per (tensor, owner) unit: state update and exact top-k selection in one
//            pass over the arrays (sparse_core.cuh), the (index, value) pairs stored
//            straight into the owner GPU's inbox; the CTA that finishes a unit
//            releases the owner's flag.
//   server : the owner waits (bounded) for the N flags of a tensor, adds the N
//            sparse payloads into its accumulator (= server-side residual),
//            re-selects the top-k of the sum and stores the result into every
//            rank's inbox, releasing their flags.
//   pull   : every rank waits for each owner's flag and scatters value / N into the
//            result, which the update pass cleared.
//
// A job of one rank takes neither: its bucket is a chain of launches (launch_chain).
//
// All units of a bucket are batched in every phase, which is the "bulk
// synchronisation" of many small tensors: the update pass splits the bucket's tiles, not
// its tensors, over the CTAs (equal shares of the CTAs per tensor left ResNet-50's largest
// tensors on 15 CTAs each; see hand_out for how the tiles are split).  An earlier
// version ran every stage as a launch of its own: 19 launches per bucket for PS and
// 9 per ring hop, with a floor of about 0.2 ms per bucket from launch latency alone.
//
// Reference parity: DGC through the PS topology is the reference's ResNet-50
// style configuration (--comp_alg dgc, README.md:180; CaSync-PS cost shape
// src/SeCoPa/SeCoPa.py:75-89 of mark14wu/hipress).
#include <cuda_runtime.h>

#include "hipress/capi.h"
#include "partition.cuh"
#include "sparse_chain.cuh"
#include "sparse_core.cuh"
#include "sync.cuh"

namespace hipress {

struct SpSeg {
  const float* g;
  float* a;    // accumulator: DGC v / GradDrop residual
  float* u;    // DGC momentum or null
  float* out;  // averaged gradient (may alias g)
  float* sr;   // server accumulator for the owned chunk [chunk]
  uint32_t n, chunk, kmax, pay_off;
  uint32_t tiles;       // tiles of one chunk
  uint32_t k_last;      // pairs of the last chunk, which may be shorter
  Sampling sample;      // set at launch: depends on the grid
  uint32_t cap;         // candidate pairs per (tensor, chunk) unit, for both lists
  uint64_t cand_push;   // first push unit's candidate list, in pairs from the region start
  uint64_t cand_srv;    // the server unit's candidate list
};

struct SpBucket {
  SpSeg seg[HP_MAX_SEGS];
  int nseg;
  int alg;
  float ratio, momentum, inv_n;
  uint64_t slot_bytes;
  uint64_t cand_pairs;  // candidate pairs of all units of one rank
  uint32_t tiles_total; // tiles of one chunk summed over the tensors
};

__device__ __forceinline__ uint32_t sp_chunk_valid(uint32_t n, uint32_t chunk, int c) {
  const uint64_t start = (uint64_t)c * chunk;
  if (start >= n) return 0;
  const uint64_t rest = n - start;
  return (uint32_t)(rest < chunk ? rest : chunk);
}

__device__ __forceinline__ void write_empty_header(uint8_t* out, int alg) {
  WireHeader h;
  h.n = 0; h.alg = (uint8_t)alg; h.bitwidth = 0; h.flags = 0; h.a = 0.0f; h.b = 0;
  *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(&h);
}

// ------------------------------------------------------ persistent-kernel plumbing
struct UnitDst {
  EmitDst out;
  uint32_t* flag[HP_MAX_RANKS];
};
constexpr int kMaxUnits = HP_MAX_SEGS * HP_MAX_RANKS;

struct SpSmem {
  union {
    SelSmem sel;
    uint32_t sh[kBins];   // whole-array passes
    EmitSmem es;
  };
  FindSmem fs;
  WaitState wst;
  uint32_t ticket;
  UnitDst dst;
  SelUnit unit[kMaxUnits];
  uint32_t tile_at[kMaxUnits + 1], sample_at[kMaxUnits + 1];
};

// control words of one rank played by a launch, behind its histogram blocks; zero
// when the kernel starts (cleared with the histograms)
constexpr int kCtlStamps = 8;    // low 32 bits of %globaltimer: kernel start, then after every barrier
constexpr int kCtlTickets = 96;  // one per selection, cleared with the rest
constexpr int kCtlBarrier = 128;
constexpr int kCtlWords = kCtlBarrier + kBarrierWords;

struct SpCtx {
  int N, R, E;
  uint32_t G;            // CTAs that play this rank
  uint32_t* ws;          // histogram / counter blocks of this rank, kWsWords per unit
  uint8_t* cand;         // candidate lists of this rank
  uint32_t* ctl;         // control words of this rank
  uint32_t* status;
  uint32_t gen;          // barriers passed so far
};

// the flag value a CTA releases: its epoch, marked when it had given up on a wait
__device__ __forceinline__ uint32_t flag_value(const HpComm& cm, const SpSmem& sm) {
  return cm.epoch | (*(volatile const int*)&sm.wst.poisoned ? kGaveUp : 0u);
}

__device__ __forceinline__ void sp_barrier(const HpComm& cm, SpCtx& cx, SpSmem& sm) {
  // a peer may be late by up to one wait bound before a CTA reaches the barrier
  grid_barrier(cx.ctl + kCtlBarrier, cx.gen, cx.G, 2 * cm.timeout_ns + 1000000000ull, cx.status,
               HP_STATUS_TIMEOUT | (8u << 16) | (cx.gen & 255u), sm.wst);
  if (blockIdx.x == 0 && threadIdx.x == 0 && kCtlStamps + cx.gen < 64u)
    cx.ctl[kCtlStamps + cx.gen] = (uint32_t)global_timer_ns();
}

// extra stamps of CTA 0 inside a phase (profile words 64..)
__device__ __forceinline__ void sp_mark(const SpCtx& cx, int id) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && 64 + id < kCtlTickets)
    cx.ctl[64 + id] = (uint32_t)global_timer_ns();
}

// Phase driver: `units` work units, each cut into `per` slices; slice v of the phase
// goes to CTA v % G.  f(unit, slice, per) is what one CTA of the old one-launch-per-
// stage grid did.
template <typename F>
__device__ __forceinline__ void run_units(const SpCtx& cx, uint32_t units, uint32_t per, F f) {
  const uint32_t total = units * per;
  for (uint32_t v = blockIdx.x; v < total; v += cx.G) {
    f((int)(v / per), v % per, per);
    __syncthreads();  // shared memory is reused by the next slice
  }
}

__device__ __forceinline__ uint32_t slices_heavy(const SpCtx& cx, uint32_t units) {
  const uint32_t p = cx.G / (units ? units : 1);
  return p < 1 ? 1 : (p > 592 ? 592 : p);
}
__device__ __forceinline__ uint32_t slices_cap(const SpCtx& cx, uint32_t units, uint32_t cap) {
  const uint32_t p = slices_heavy(cx, units);
  return p > cap ? cap : p;
}

// ------------------------------------------------------------ units of a selection
// push : every (tensor, owner) pair, unit y = tensor * N + owner
// serve: the owned chunk of every tensor, y = tensor
// hop  : the chunk of every tensor that hop `hop` of the ring works on, y = tensor
// Every element of the gradient is read by exactly one push or hop, and the update clears
// the result behind that read (it may be the same buffer).
// The kind is a run-time value: the two selections of a PS launch and the hops of a ring
// run the same instructions, so all but the first find them in the instruction cache.
enum SelKind { kSelPush, kSelServe, kSelHop };

struct SelPhase {
  int kind, hop;
  uint32_t units;
  int mode;   // of the update: see pass0_body
};

__device__ __forceinline__ void unit_ref(const SpCtx& cx, const SelPhase& ph, uint32_t y, int& si, int& c) {
  si = (int)y;
  c = cx.R;
  if (ph.kind == kSelPush) {
    si = (int)(y / (uint32_t)cx.N);
    c = (int)(y % (uint32_t)cx.N);
  } else if (ph.kind == kSelHop) {
    c = cx.R - ph.hop;
    if (c < 0) c += cx.N;
  }
}

// Every unit's array, and prefix sums of the units' tiles and sampled tiles, in shared
// memory: worked out once per phase by all threads, looked up at every stretch of tiles.
static __device__ __noinline__ void set_units(const SpBucket& bk, const HpComm& cm, const SpCtx& cx,
                                              const SelPhase& ph, SpSmem& sm) {
  __syncthreads();
#pragma unroll 1
  for (uint32_t y = threadIdx.x; y < ph.units; y += kSpThreads) {
    int si, c;
    unit_ref(cx, ph, y, si, c);
    const SpSeg& sg = bk.seg[si];
    SelUnit& s = sm.unit[y];
    const size_t E = (size_t)cx.E, off = (size_t)c * sg.chunk;
    const uint32_t n = sp_chunk_valid(sg.n, sg.chunk, c), tiles = (n + kSelTile - 1) / kSelTile;
    s.n = n;
    s.k = n == sg.chunk ? sg.kmax : sg.k_last;   // only the last chunk is shorter
    s.kmax = sg.kmax;
    s.cap = list_cap(sg.cap);
    s.stride = sg.sample.stride;
    s.top = sg.sample.top;
    s.run = sg.sample.run;
    s.sampled = (tiles + s.stride - 1) / s.stride;
    uint64_t list = sg.cand_srv;
    uint32_t block = (uint32_t)(bk.nseg * cx.N) + y;
    s.g = nullptr;
    s.u = nullptr;
    s.clear = nullptr;
    if (ph.kind == kSelServe) {
      s.a = sg.sr + E * cm.emu_stride_sr;
    } else {
      s.g = sg.g + E * cm.emu_stride_g + off;
      s.a = sg.a + E * cm.emu_stride_r + off;
      if (sg.u) s.u = sg.u + E * cm.emu_stride_r + off;
      s.clear = sg.out + E * cm.emu_stride_out + off;
      list = sg.cand_push + (uint64_t)c * sg.cap;
      block = ph.kind == kSelPush ? y : (uint32_t)(ph.hop * bk.nseg + si);
    }
    s.ws = cx.ws + (size_t)block * kWsWords;
    s.cv = reinterpret_cast<float*>(cx.cand + list * 8);
    sm.tile_at[y + 1] = tiles;
    sm.sample_at[y + 1] = s.sampled;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t t0 = 0, s0 = 0;
#pragma unroll 1
    for (uint32_t b = 0; b < ph.units; b += 32) {
      const uint32_t y = b + threadIdx.x;
      uint32_t t = y < ph.units ? sm.tile_at[y + 1] : 0u, q = y < ph.units ? sm.sample_at[y + 1] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, t, o), c = __shfl_up_sync(0xffffffffu, q, o);
        if ((int)threadIdx.x >= o) {
          t += a;
          q += c;
        }
      }
      if (y < ph.units) {
        sm.tile_at[y + 1] = t0 + t;
        sm.sample_at[y + 1] = s0 + q;
      }
      t0 += __shfl_sync(0xffffffffu, t, 31);
      s0 += __shfl_sync(0xffffffffu, q, 31);
    }
    if (threadIdx.x == 0) sm.tile_at[0] = sm.sample_at[0] = 0;
  }
  __syncthreads();
}
// the unit in whose stretch of the prefix sums item t lies
__device__ __forceinline__ uint32_t unit_at(const uint32_t* at, uint32_t units, uint32_t t) {
  uint32_t lo = 0, hi = units;
#pragma unroll 1
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (at[mid] <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Where a unit's pairs go, and the flags that announce them: into sm.dst (whole CTA).
// What stays on this rank does not pass through its inbox: the push of the own chunk is
// added to the owner's accumulator, and a final chunk goes into the result.
__device__ __forceinline__ void unit_dst(const SpBucket& bk, const HpComm& cm, const SpCtx& cx, const SelPhase& ph,
                                         uint32_t y, SpSmem& sm) {
  const int N = cx.N, R = cx.R, q = (int)threadIdx.x;
  int si, c;
  unit_ref(cx, ph, y, si, c);
  const SpSeg& sg = bk.seg[si];
  const bool final_chunk = ph.kind == kSelServe || (ph.kind == kSelHop && ph.hop == N - 1);
  const bool own_push = ph.kind == kSelPush && c == R;
  const int slot = ph.kind == kSelPush ? R : (ph.kind == kSelServe ? N + R : (final_chunk ? N - 1 + R : ph.hop));
  const int n = final_chunk ? N - 1 : (own_push ? 0 : 1);
  __syncthreads();
  if (q == 0) {
    sm.dst.out.n = n;
    sm.dst.out.add = own_push ? sg.sr + cx.E * cm.emu_stride_sr : nullptr;
    // a CTA that has given up leaves the result alone
    sm.dst.out.set = final_chunk && !*(volatile int*)&sm.wst.poisoned ? sg.out + cx.E * cm.emu_stride_out + (size_t)c * sg.chunk : nullptr;
    sm.dst.out.scale = bk.inv_n;
  }
  if (q < n) {
    int to = (ph.kind == kSelPush ? c : R + 1) + q;
    if (to >= N) to -= N;
    sm.dst.out.out[q] = reinterpret_cast<uint8_t*>(cm.inbox[to]) + (size_t)slot * bk.slot_bytes + sg.pay_off;
    sm.dst.flag[q] = reinterpret_cast<uint32_t*>(cm.flags[to]) + (size_t)slot * bk.nseg + si;
  }
  __syncthreads();
}
// thread 0 of the CTA that completed the unit
__device__ __forceinline__ void unit_release(const HpComm& cm, const SpSmem& sm) {
  if (sm.dst.out.n == 0) return;
  __threadfence_system();
  const uint32_t v = flag_value(cm, sm);
#pragma unroll 1
  for (int q = 0; q < sm.dst.out.n; ++q) st_release_sys(sm.dst.flag[q], v);
}

// The selection of all units of one kind, the ticket-th of the launch: two barriers (more
// only when a sample misled).
static __device__ __noinline__ void select_units(const SpBucket& bk, const HpComm& cm, SpCtx& cx, SpSmem& sm, int kind,
                                                 int hop, int ticket) {
  SelPhase ph;
  ph.kind = kind;
  ph.hop = hop;
  ph.units = (uint32_t)bk.nseg * (kind == kSelPush ? (uint32_t)cx.N : 1u);
  ph.mode = kind == kSelServe ? 0 : (bk.alg == kDgc ? 2 : 1);
  const uint32_t units = ph.units;
  set_units(bk, cm, cx, ph, sm);
  const uint32_t samples = sm.sample_at[units];
  // sampled tiles of this CTA; the first two stay in shared memory until they are collected
  uint32_t mine = 0;
#pragma unroll 1
  for (uint32_t i = blockIdx.x; i < samples; i += cx.G, ++mine) {
    const uint32_t y = unit_at(sm.sample_at, units, i), j = i - sm.sample_at[y];
    float* stash = sm.sel.stash[mine < 1 ? 0 : 1];
    if (ph.mode == 0) sample_body<0>(sm.unit[y], bk.momentum, sm.sel, j, stash);
    else if (ph.mode == 1) sample_body<1>(sm.unit[y], bk.momentum, sm.sel, j, stash);
    else sample_body<2>(sm.unit[y], bk.momentum, sm.sel, j, stash);
    __syncthreads();
  }
  sp_barrier(cm, cx, sm);
  if (threadIdx.x == 0) sm.sel.count = 0;
  for (uint32_t y = threadIdx.x; y < units; y += kSpThreads) sm.unit[y].low = __ldcg(sm.unit[y].ws + kWsLow);
  __syncthreads();
#pragma unroll 1
  for (uint32_t i = blockIdx.x, r = 0; r < mine; i += cx.G, ++r) {
    const uint32_t y = unit_at(sm.sample_at, units, i);
    collect_sampled(sm.unit[y], y, sm.sel, i - sm.sample_at[y], sm.sel.stash[r < 1 ? 0 : 1], r >= 1 && mine > 2);
  }
  auto unit = [&](uint32_t y) -> const SelUnit& { return sm.unit[y]; };
  hand_out(cx.ctl + kCtlTickets + ticket, sm.tile_at[units], blockIdx.x, cx.G, sm.ticket, [&](uint32_t t, uint32_t end) {
    uint32_t y = unit_at(sm.tile_at, units, t);
#pragma unroll 1
    while (t < end) {
      while (sm.tile_at[y + 1] <= t) ++y;   // empty units
      const uint32_t base = sm.tile_at[y], t1 = min(min(sm.tile_at[y + 1], end), t + sm.unit[y].run);
      const SelUnit& s = sm.unit[y];
      if (s.stride > 1) {
        if (ph.mode == 0) collect_body<0>(s, y, bk.momentum, sm.sel, t - base, t1 - base);
        else if (ph.mode == 1) collect_body<1>(s, y, bk.momentum, sm.sel, t - base, t1 - base);
        else collect_body<2>(s, y, bk.momentum, sm.sel, t - base, t1 - base);
      }
      t = t1;
      if (__syncthreads_or(sm.sel.count > (uint32_t)kCollectBuf / 2)) collect_flush(sm.sel, unit);
    }
  });
  collect_flush(sm.sel, unit);
  sp_barrier(cm, cx, sm);
  // behind the barrier every CTA reads the same counters and decides the same
  int bad = 0;
#pragma unroll 1
  for (uint32_t y = threadIdx.x; y < units; y += kSpThreads)
    bad |= sm.unit[y].n && selection_failed(sm.unit[y], list_state(sm.unit[y]));
  const bool failed = __syncthreads_or(bad);
  const uint32_t share = slices_cap(cx, units, 64);
  run_units(cx, units, share, [&](int y, uint32_t x, uint32_t) {
    const SelUnit& s = sm.unit[y];
    const ListState ls = list_state(s);
    if (s.n && selection_failed(s, ls)) return;
    const uint32_t nx = s.n ? emit_slices(ls.count, share) : 1u;
    if (x >= nx) return;
    unit_dst(bk, cm, cx, ph, (uint32_t)y, sm);
    bool done = false;
    if (s.n == 0) {
      done = threadIdx.x == 0;
      if (done)
        for (int q = 0; q < sm.dst.out.n; ++q) write_empty_header(sm.dst.out.out[q], bk.alg);
    } else {
      done = emit_slice(bk.alg, s, ls, sm.dst.out, sm.sel, x, nx);
    }
    if (done) unit_release(cm, sm);
  });
  sp_mark(cx, ticket);
  if (!failed) return;
  // whole-array passes for the units whose sample misled: clear the histograms, count the
  // three digits, send
  const uint32_t heavy = slices_heavy(cx, units);
#pragma unroll 1
  for (int pass = -1; pass <= 3; ++pass) {
    run_units(cx, units, heavy, [&](int y, uint32_t x, uint32_t nx) {
      const SelUnit& s = sm.unit[y];
      if (s.n == 0 || !selection_failed(s, list_state(s))) return;
      if (pass < 0) {
        for (uint32_t i = x * kSpThreads + threadIdx.x; i < 3u * kBins; i += nx * kSpThreads) s.ws[i] = 0;
      } else if (pass == 0) {
        pass0_body<0>(nullptr, s.a, nullptr, s.n, 0.0f, s.ws, sm.sh, x, nx);
      } else if (pass < 3) {
        pass_body(pass, s.a, s.n, s.k, s.ws, sm.sh, sm.fs, x, nx);
      } else {
        unit_dst(bk, cm, cx, ph, (uint32_t)y, sm);
        if (emit_body(bk.alg, s.a, s.u, s.n, s.k, s.kmax, sm.dst.out, s.ws, sm.fs, sm.es, x, nx)) unit_release(cm, sm);
      }
    });
    if (pass < 3) sp_barrier(cm, cx, sm);
  }
}

// ---------------------------------------------------------------- incoming payloads
// PS owner: wait for the other ranks' pushes of tensor si and add them into the accumulator
__device__ __forceinline__ void serve_in(const SpBucket& bk, const HpComm& cm, const SpCtx& cx, SpSmem& sm, int si,
                                         uint32_t x, uint32_t nx) {
  const int N = cx.N, R = cx.R;
  const SpSeg& sg = bk.seg[si];
  const uint32_t len = sp_chunk_valid(sg.n, sg.chunk, R);
  const uint32_t* my_flags = reinterpret_cast<const uint32_t*>(cm.flags[R]);
  for (int q = 0; q < N; ++q)
    if (q != R)
      wait_flag(my_flags + (size_t)q * bk.nseg + si, cm.epoch, cm.timeout_ns, cx.status,
                HP_STATUS_TIMEOUT | (4u << 16) | ((uint32_t)q << 8) | (si & 255), sm.wst);
  if (len == 0) return;
  const uint8_t* inbox = reinterpret_cast<const uint8_t*>(cm.inbox[R]);
  for (int q = 0; q < N; ++q)
    if (q != R)
      scatter_body(inbox + (size_t)q * bk.slot_bytes + sg.pay_off, sg.sr + cx.E * cm.emu_stride_sr, len, sg.kmax,
                   1.0f, 2, x, nx);
}

// ring: wait for the predecessor's pairs of tensor si and add them into the accumulator
__device__ __forceinline__ void hop_in(const SpBucket& bk, const HpComm& cm, const SpCtx& cx, SpSmem& sm, int hop,
                                       int si, uint32_t x, uint32_t nx) {
  const SpSeg& sg = bk.seg[si];
  const int c = (cx.R - hop + cx.N) % cx.N;
  const uint32_t len = sp_chunk_valid(sg.n, sg.chunk, c);
  wait_flag(reinterpret_cast<const uint32_t*>(cm.flags[cx.R]) + (size_t)(hop - 1) * bk.nseg + si, cm.epoch,
            cm.timeout_ns, cx.status, HP_STATUS_TIMEOUT | (6u << 16) | ((uint32_t)(hop - 1) << 8) | (si & 255),
            sm.wst);
  if (len == 0) return;
  scatter_body(reinterpret_cast<const uint8_t*>(cm.inbox[cx.R]) + (size_t)(hop - 1) * bk.slot_bytes + sg.pay_off,
               sg.a + cx.E * cm.emu_stride_r + (size_t)c * sg.chunk, len, sg.kmax, 1.0f, 1, x, nx);
}

// ---------------------------------------------------------------- pull
// wait for the reduced chunk c that arrives in inbox slot `slot` and scatter value / N
// into the (zero-filled) result; unit y = seg * N + j.  A CTA that has given up leaves
// the result alone.
__device__ __forceinline__ void gather_stage(const SpBucket& bk, const HpComm& cm, const SpCtx& cx,
                                             SpSmem& sm, int si, int slot, int c, uint32_t phase,
                                             uint32_t x, uint32_t nx) {
  const SpSeg& sg = bk.seg[si];
  const uint32_t len = sp_chunk_valid(sg.n, sg.chunk, c);
  wait_flag(reinterpret_cast<const uint32_t*>(cm.flags[cx.R]) + (size_t)slot * bk.nseg + si, cm.epoch,
            cm.timeout_ns, cx.status,
            HP_STATUS_TIMEOUT | (phase << 16) | ((uint32_t)(slot & 255) << 8) | (si & 255), sm.wst);
  if (len == 0 || *(volatile int*)&sm.wst.poisoned) return;
  const uint8_t* p = reinterpret_cast<const uint8_t*>(cm.inbox[cx.R]) + (size_t)slot * bk.slot_bytes +
                     sg.pay_off;
  scatter_body(p, sg.out + cx.E * cm.emu_stride_out + (size_t)c * sg.chunk, len, sg.kmax, bk.inv_n, 0,
               x, nx);
}

// ------------------------------------------------------------- the two kernels
struct SpLaunch {
  uint8_t* ws;            // scratch of all ranks played by the launch
  uint64_t ws_rank_bytes; // per rank: histogram blocks, control words, candidate lists
  uint64_t hist_words;    // histogram words per rank (the control words follow)
  uint64_t hist_bytes;    // offset of the candidate lists inside a rank's scratch
};

__device__ __forceinline__ void sp_prologue(const HpComm& cm, const SpLaunch& L, SpCtx& cx,
                                            SpSmem& sm) {
  cx.N = cm.nranks;
  cx.R = cm.emulate ? (int)blockIdx.y : cm.rank;
  cx.E = cm.emulate ? (int)blockIdx.y : 0;
  cx.G = gridDim.x;
  uint8_t* base = L.ws + (size_t)cx.E * L.ws_rank_bytes;
  cx.ws = reinterpret_cast<uint32_t*>(base);
  cx.ctl = cx.ws + L.hist_words;
  cx.cand = base + L.hist_bytes;
  cx.status = reinterpret_cast<uint32_t*>(cm.status) + 4 * cx.E;
  cx.gen = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) cx.ctl[kCtlStamps] = (uint32_t)global_timer_ns();
  wait_init(sm.wst);
}

// CTA 0's last stamp and the number of barriers it passed (the other CTAs may still
// be scattering: the stamps are a profile of the phases, not a completion signal)
__device__ __forceinline__ void sp_epilogue(const SpCtx& cx) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (kCtlStamps + cx.gen + 1 < 64u)
      cx.ctl[kCtlStamps + cx.gen + 1] = (uint32_t)global_timer_ns();
    cx.ctl[1] = cx.gen;
  }
}

// PS: push (every rank selects per owner and stores the pairs into the owner's inbox),
// serve (the owner adds the payloads, re-selects, stores the result into every inbox),
// pull (every rank scatters value / N).  Five barriers.
__global__ void __launch_bounds__(kSpThreads, 2)
sp_ps_kernel(const __grid_constant__ SpBucket bk, const __grid_constant__ HpComm cm, const __grid_constant__ SpLaunch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SpSmem& sm = *reinterpret_cast<SpSmem*>(smem_raw);
  SpCtx cx;
  sp_prologue(cm, L, cx, sm);
  const int N = cx.N;
  const uint32_t nseg = (uint32_t)bk.nseg, units = nseg * (uint32_t)(N - 1);
  select_units(bk, cm, cx, sm, kSelPush, 0, 0);
  if (N > 1)
    run_units(cx, nseg, slices_cap(cx, nseg, 32),
              [&](int y, uint32_t x, uint32_t nx) { serve_in(bk, cm, cx, sm, y, x, nx); });
  sp_barrier(cm, cx, sm);
  select_units(bk, cm, cx, sm, kSelServe, 0, 1);
  if (N > 1)
    run_units(cx, units, slices_cap(cx, units, 16), [&](int y, uint32_t x, uint32_t nx) {
      const int j = (cx.R + 1 + y % (N - 1)) % N;
      gather_stage(bk, cm, cx, sm, y / (N - 1), N + j, j, 5u, x, nx);
    });
  sp_epilogue(cx);
}

// Ring: N hops of (add the predecessor's pairs, update and select, store into the
// successor's inbox), the last hop storing into every inbox; then every rank scatters
// the reduced chunks of the others.  Three barriers per hop.
__global__ void __launch_bounds__(kSpThreads, 2)
sp_ring_kernel(const __grid_constant__ SpBucket bk, const __grid_constant__ HpComm cm, const __grid_constant__ SpLaunch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SpSmem& sm = *reinterpret_cast<SpSmem*>(smem_raw);
  SpCtx cx;
  sp_prologue(cm, L, cx, sm);
  const int N = cx.N;
  const uint32_t nseg = (uint32_t)bk.nseg;
#pragma unroll 1
  for (int hop = 0; hop < N; ++hop) {
    if (hop > 0) {
      run_units(cx, nseg, slices_cap(cx, nseg, 32),
                [&](int y, uint32_t x, uint32_t nx) { hop_in(bk, cm, cx, sm, hop, y, x, nx); });
      sp_barrier(cm, cx, sm);
    }
    select_units(bk, cm, cx, sm, kSelHop, hop, hop);
  }
  // gather: rank src finalised chunk src + 1
  const uint32_t units = nseg * (uint32_t)(N - 1);
  if (N > 1)
    run_units(cx, units, slices_cap(cx, units, 16), [&](int y, uint32_t x, uint32_t nx) {
      const int src = (cx.R + 1 + y % (N - 1)) % N;
      gather_stage(bk, cm, cx, sm, y / (N - 1), N - 1 + src, (src + 1) % N, 7u, x, nx);
    });
  sp_epilogue(cx);
}

static int build_sp_bucket(int alg, float ratio, float momentum, const HpSeg* segs,
                           void* const* accs, void* const* us, int nseg, int nranks, SpBucket& bk) {
  if (nseg < 1 || nseg > HP_MAX_SEGS || nranks < 1 || nranks > HP_MAX_RANKS) return HP_ERR_BAD_ARG;
  if (alg != kDgc && alg != kGradDrop) return HP_ERR_BAD_ARG;
  uint64_t pay = 0, cand = 0, tiles = 0;
  for (int i = 0; i < nseg; ++i) {
    const uint64_t n = segs[i].n;
    if (n == 0 || n > 0xFFFFF000ull) return HP_ERR_BAD_ARG;
    const uint64_t chunk = align_up((n + nranks - 1) / nranks, kTile);
    SpSeg& d = bk.seg[i];
    d.g = static_cast<const float*>(segs[i].g);
    d.a = accs ? static_cast<float*>(accs[i]) : static_cast<float*>(segs[i].r);
    d.u = us ? static_cast<float*>(us[i]) : nullptr;
    d.out = static_cast<float*>(segs[i].out);
    d.sr = static_cast<float*>(segs[i].sr);
    d.n = (uint32_t)n;
    d.chunk = (uint32_t)chunk;
    d.kmax = (uint32_t)sparse_k(chunk, ratio);
    d.k_last = (uint32_t)sparse_k(n % chunk, ratio);
    d.pay_off = (uint32_t)pay;
    d.tiles = (uint32_t)((chunk + kSelTile - 1) / kSelTile);
    tiles += d.tiles;
    d.cap = (uint32_t)align_up(8ull * d.kmax + 4096, 32);
    d.cand_push = cand;
    cand += (uint64_t)d.cap * nranks;
    d.cand_srv = cand;
    cand += d.cap;
    pay += align_up(sparse_payload_bytes(d.kmax), 128);
    if (pay > 0xFFFFFFFFull) return HP_ERR_TOO_LARGE;
  }
  bk.nseg = nseg;
  bk.alg = alg;
  bk.ratio = ratio;
  bk.momentum = momentum;
  bk.inv_n = 1.0f / (float)nranks;
  bk.slot_bytes = pay;
  bk.cand_pairs = cand;
  if (tiles * (uint64_t)nranks > 0x7FFFFFFFull) return HP_ERR_TOO_LARGE;
  bk.tiles_total = (uint32_t)tiles;
  return 0;
}

// ------------------------------------------------------------------ host side
static uint64_t sp_hist_words(int nseg, int nranks) {
  return (uint64_t)(nseg * nranks + nseg) * kWsWords;   // the ring uses nseg * nranks of them
}

// words behind the control words that a job of one rank uses: the counts of its lists'
// parts, push and server, the server selection's barrier, and whether one expired
static uint64_t sp_chain_words(int nseg, int nranks) {
  return nranks == 1 ? 2ull * nseg * 32 * kChainLists + kBarrierWords + 1 : 0;
}
static uint64_t sp_cleared_words(int nseg, int nranks) {
  return sp_hist_words(nseg, nranks) + kCtlWords + sp_chain_words(nseg, nranks);
}

// A job of one rank waits for nobody: its selections run as chains of launches, in a PS the
// owner's sum behind the push.  The persistent kernels that follow do the same with grid
// barriers; us per step or bucket, persistent / chain (B200): ResNet-50, DGC, PS 203 / 171;
// GradDrop ring 6.6 M elements 56.0 / 39.8, 20 M at 1 % 128 / 95; DGC ring 3 M 49.0 / 34.4; DGC
// PS 64 K 52.1 / 37.7, 20 M 176 / 132; 24 arrays of 1 M in all, PS 61.7 / 47.6.
// False when the arrays do not fit a chain (and always with a limit on the CTAs).
static bool launch_chain(int topo, const SpBucket& bk, const HpComm& cm, uint8_t* ws, cudaStream_t st, int& rc) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || chain_per_sm(dev) == 0) return false;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  sms = stream_sms(st, sms);
  const int resident = chain_per_sm(dev) * sms;
  uint32_t* words = reinterpret_cast<uint32_t*>(ws);
  uint32_t* ctl = words + sp_hist_words(bk.nseg, 1);
  uint8_t* lists = ws + align_up(sp_cleared_words(bk.nseg, 1) * 4, 256);
  auto arrays = [&](ChainArgs& A, bool serve) {
    A.units = bk.nseg;
    A.alg = bk.alg;
    A.momentum = bk.momentum;
    A.scale = bk.inv_n;
    uint32_t* behind = ctl + kCtlWords + 2 * bk.nseg * 32 * kChainLists;
    A.barrier = serve ? behind : ctl + kCtlBarrier;
    A.gave_up = behind + kBarrierWords;
    A.status = reinterpret_cast<uint32_t*>(cm.status);
    A.code = HP_STATUS_TIMEOUT | (8u << 16);
    for (int i = 0; i < bk.nseg; ++i) {
      const SpSeg& sg = bk.seg[i];
      const int y = serve ? bk.nseg + i : i;
      ChainUnit& u = A.unit[i];
      u.s.g = serve ? nullptr : sg.g;
      u.s.a = serve ? sg.sr : sg.a;
      u.s.u = serve ? nullptr : sg.u;
      u.s.clear = serve ? nullptr : sg.out;
      u.s.ws = words + (size_t)y * kWsWords;
      u.s.cv = reinterpret_cast<float*>(lists + (serve ? sg.cand_srv : sg.cand_push) * 8);
      u.s.n = sg.n;
      u.s.k = sg.n == sg.chunk ? sg.kmax : sg.k_last;
      u.s.kmax = sg.kmax;
      u.s.cap = list_cap(sg.cap);
      const Sampling p = sampling(sg.tiles, bk.tiles_total, (uint32_t)resident, sg.chunk, sg.kmax);
      u.s.stride = p.stride;
      u.s.top = p.top;
      u.counts = ctl + kCtlWords + (size_t)y * 32 * kChainLists;
      u.add = topo == HP_TOPO_PS && !serve ? sg.sr : nullptr;
      u.set = topo == HP_TOPO_PS && !serve ? nullptr : sg.out;
    }
    return chain_place(A, chain_per_sm(dev), sms);
  };
  ChainArgs push = {}, sum = {};
  if (!arrays(push, false) || (topo == HP_TOPO_PS && !arrays(sum, true))) return false;
  cudaError_t e = cudaMemsetAsync(ws, 0, sp_cleared_words(bk.nseg, 1) * 4, st);
  if (e == cudaSuccess) e = chain_select(bk.alg == kDgc ? 2 : 1, push, st);
  if (e == cudaSuccess && topo == HP_TOPO_PS) e = chain_select(0, sum, st);
  rc = (int)e;
  return true;
}

static int launch_sparse(int topo, SpBucket& bk, const HpComm& cm, void* ws, int ctas,
                         cudaStream_t st) {
  int chained = 0;
  if (cm.nranks == 1 && ctas <= 0 && launch_chain(topo, bk, cm, static_cast<uint8_t*>(ws), st, chained)) return chained;
  const void* kern = topo == HP_TOPO_RING ? (const void*)sp_ring_kernel : (const void*)sp_ps_kernel;
  const int N = cm.nranks, nseg = bk.nseg;
  static int resident[2][64] = {};   // CTAs the GPU holds at once, per (topology, device)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  int cap = (dev >= 0 && dev < 64) ? resident[topo][dev] : 0;
  const size_t smem = sizeof(SpSmem);
  if (cap == 0) {
    int sms = 0, per_sm = 0;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSpThreads, smem);
    if (e != cudaSuccess) return (int)e;
    cap = per_sm * sms;
    if (cap < 1) return HP_ERR_RESIDENCY;
    if (dev >= 0 && dev < 64) resident[topo][dev] = cap;
  }
  const int ranks_here = cm.emulate ? N : 1;
  int G = ctas;
  if (G <= 0) {   // a CTA per tile of the bucket
    const uint64_t tiles = (uint64_t)bk.tiles_total * N;
    G = (int)(tiles < (uint64_t)cap ? tiles : (uint64_t)cap);
  }
  if (G > cap / ranks_here) G = cap / ranks_here;   // what the GPU holds at once
  if (G < 1) return HP_ERR_RESIDENCY;
  for (int i = 0; i < nseg; ++i)  // a sampled tile for every CTA, over the units of a push or of a hop
    bk.seg[i].sample = sampling(bk.seg[i].tiles, (uint64_t)bk.tiles_total * (topo == HP_TOPO_PS ? N : 1), (uint32_t)G,
                                bk.seg[i].chunk, bk.seg[i].kmax);
  SpLaunch L;
  L.ws = static_cast<uint8_t*>(ws);
  L.hist_words = sp_hist_words(nseg, N);
  L.hist_bytes = align_up(sp_cleared_words(nseg, N) * 4, 256);
  L.ws_rank_bytes = L.hist_bytes + bk.cand_pairs * 8;
  for (int r = 0; r < ranks_here; ++r) {  // histograms, counters and control words start at zero
    e = cudaMemsetAsync(L.ws + (size_t)r * L.ws_rank_bytes, 0, (L.hist_words + kCtlWords) * 4, st);
    if (e != cudaSuccess) return (int)e;
  }
  void* args[] = {(void*)&bk, (void*)&cm, (void*)&L};
  // cooperative: the CTAs of a launch wait for one another at the phase barriers
  e = cudaLaunchCooperativeKernel(kern, dim3(G, ranks_here), dim3(kSpThreads), args, smem, st);
  return (int)e;
}

}  // namespace hipress

using namespace hipress;

extern "C" {

// sizes a caller needs to reserve for a bucket of tensors with the given sizes
int hp_fused_sparse_layout(float ratio, const uint64_t* ns, int nseg, int nranks,
                           uint64_t* inbox_bytes, uint64_t* flag_words, uint64_t* ws_bytes) {
  if (nseg < 1 || nseg > HP_MAX_SEGS) return HP_ERR_BAD_ARG;
  HpSeg segs[HP_MAX_SEGS] = {};
  for (int i = 0; i < nseg; ++i) segs[i].n = ns[i];
  SpBucket bk;
  int rc = build_sp_bucket(kDgc, ratio, 0.f, segs, nullptr, nullptr, nseg, nranks, bk);
  if (rc) return rc;
  if (inbox_bytes) *inbox_bytes = bk.slot_bytes * 2ull * nranks;
  if (flag_words) *flag_words = 2ull * nranks * nseg;
  // per rank played by a launch: histogram blocks of the push (nseg * nranks) and
  // server (nseg) units, control words, candidate lists
  if (ws_bytes)
    *ws_bytes = align_up(sp_cleared_words(nseg, nranks) * 4, 256) + bk.cand_pairs * 8;
  return 0;
}

// One synchronisation of a bucket through the PS topology: one cooperative launch, or with
// one rank and ctas <= 0 two chains of three launches (launch_chain).
// segs[i].r is the accumulator (DGC v / GradDrop residual), us[i] the DGC momentum
// (or NULL), segs[i].sr the server accumulator of the owned chunk.  ws: scratch of
// hp_fused_sparse_layout().ws_bytes per rank played by this call.  ctas <= 0: the
// grid is sized from the bucket.
int hp_cuda_fused_sparse_ps(int alg, float ratio, float momentum, const HpSeg* segs,
                            void* const* us, int nseg, const HpComm* comm, void* ws, int ctas,
                            void* stream) {
  if (!comm || ctas > 1024) return HP_ERR_BAD_ARG;
  SpBucket bk;
  int rc = build_sp_bucket(alg, ratio, momentum, segs, nullptr, us, nseg, comm->nranks, bk);
  if (rc) return rc;
  return launch_sparse(HP_TOPO_PS, bk, *comm, ws, ctas, (cudaStream_t)stream);
}

// One synchronisation of a bucket through the ring topology: one cooperative launch, or with
// one rank and ctas <= 0 a chain of three (launch_chain).
// Same arguments as hp_cuda_fused_sparse_ps (segs[i].sr is not used).
int hp_cuda_fused_sparse_ring(int alg, float ratio, float momentum, const HpSeg* segs,
                              void* const* us, int nseg, const HpComm* comm, void* ws, int ctas,
                              void* stream) {
  if (!comm || ctas > 1024) return HP_ERR_BAD_ARG;
  SpBucket bk;
  int rc = build_sp_bucket(alg, ratio, momentum, segs, nullptr, us, nseg, comm->nranks, bk);
  if (rc) return rc;
  return launch_sparse(HP_TOPO_RING, bk, *comm, ws, ctas, (cudaStream_t)stream);
}

}  // extern "C"
