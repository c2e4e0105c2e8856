// ggks_pipeline.cuh -- host driver of the selection pipeline (templated on the
// input element type and the output value type).  Included by the
// per-type instantiation units.
#pragma once

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "ggks_front.cuh"
#include "ggks_internal.h"
#include "ggks_small.cuh"
#include "ggks_tiny.cuh"
#include "ggks_topk.cuh"
#include "ggks_window.cuh"

namespace ggks {

// keys of needed bins that one finishing CTA holds in shared memory (plus an
// equal scratch area for sorting a large bin)
template <class T>
static inline uint32_t cap_keys_for() {
  return sizeof(typename Traits<T>::K) == 4 ? 4096u : 2048u;
}
// bins (5 arrays), the gather buffer, a scratch half its size for sorting one
// large bin, per-bin key ranges: about 52 KB (f32) / 60 KB (f64), so that
// several finishing CTAs share an SM
template <class T>
static inline int finish_smem_bytes() {
  using K = typename Traits<T>::K;
  return (int)finish_smem_for<K>(cap_keys_for<T>());
}

// Shared memory asked for when there are no more slots than SMs: a CTA per SM.  The CTAs
// start as the ones of k_compact end, and with their own need four of them shared
// the first SM to be free (7.5 M few-valued floats, 11 slots of 28000 keys: 245 us a
// call, now 151; 3 to 150 small slots: the same).
constexpr int kFinAlone = 120 << 10;

static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// k_plan's shared memory: the table, the bucket prefix and flags for the
// largest bucket count, and room for 6144 per-slot request counters (both
// launchers raise the kernel's limit to this one value)
constexpr size_t kPlanSlotBytes = 6144 * 8;
constexpr int kPlanSmemMax = (int)(kLutPadded * sizeof(uint32_t) + (size_t)kMaxNb * 5 + 16 +
                                   kPlanSlotBytes);

// The words after the fine counts, cleared by k_sample with them where a path
// uses them: the window path's bins, cursors, large bins' first keys (64-bit) and
// flags, and counters, then the sample keys around thresholds (SliceOut, whose first
// words are cleared too).
constexpr uint32_t kWinBinsAt = kLutIdx, kWinCurAt = kWinBinsAt + kWinBins,
                   kWinFirstAt = kWinCurAt + kWinBins, kWinMixedAt = kWinFirstAt + 2 * kWinBins,
                   kWinCtlAt = kWinMixedAt + kWinBins, kFineWords = kWinCtlAt + 16;
static_assert(sizeof(WinCtl<uint64_t>) <= 64 && kWinFirstAt % 2 == 0 && kFineWords % 4 == 0,
              "the counters' place and alignment");

struct Plan {
  uint64_t n = 0;
  uint32_t num_req = 0;
  uint32_t S = 0;
  uint32_t nb_max = 0;   // buckets that the rows and arrays hold
  uint32_t nb_want = 0;  // buckets of a table that tracks no keys
  uint32_t G = 0;           // hist / compact grid
  bool unroll8 = true;      // tiles of 8 (else 4) vectors per thread in hist / compact
  uint32_t scan_tiles = 0;
  uint32_t cap_keys = 0;
  uint32_t fin_grid = 0;
  uint64_t surv_cap = 0;
  // arena offsets
  size_t out = 0, ctrl = 0, reqs = 0, hdr = 0, lut = 0, samples = 0, spans = 0, fine = 0, wpre = 0, partials = 0, sorted = 0,
         bpre = 0, bco = 0, ttot = 0, seg_bucket = 0, seg_off = 0, seg_size = 0, kstart = 0, kcnt = 0, fill = 0,
         kcur = 0, seg_lo = 0, seg_hi = 0, deferred = 0, req_bucket = 0, req_local = 0, klist = 0,
         pm_bits = 0, pm_bcount = 0, pm_bslot = 0, cand_cnt = 0, cand_tab = 0, reps = 0,
         bsingle = 0, bkey = 0, total = 0;
  // speculative compaction: the candidate pool is the survivor buffer from
  // surv_half on, cand_chunks chunks of kCandChunk keys
  uint64_t surv_half = 0;
  uint32_t cand_chunks = 0;
};
static_assert(sizeof(Ctrl) <= 256 && sizeof(Ctrl) % 4 == 0, "the control block's 256-byte slot");
// Host k lists are read from pinned host memory (k_sample, the small-vector
// kernels), and at most kPinOut results are written there by the finishing
// kernels; the control block goes up in the first kernel's parameters and comes
// back by k_finish's last CTA.  Such a call puts no copy on the stream.  More
// results come back in one copy (their scattered 4- and 8-byte stores would
// cross the link one by one).
// (2^20 floats, 101 k's: 72 -> 65 us a call; 5003 floats, 11 k's: 47 -> 43 us;
// 10 M floats, 257 k's: 96 -> 91 us.)
constexpr uint32_t kPinOut = 4096;

// The streaming passes' grid and buckets, and the arena's layout (rows: with the
// histogram's rows, up to 60 MB, which only the pipeline reads).  A CTA per 16384 elements up to one per
// SM: below 10 M elements a pass is its CTAs' fixed work and one or two tiles
// each, so more of them end sooner (65536 elements a CTA: 2^21 floats, 101 k's 63 us
// a call, now 52; 2^21 doubles 75 -> 60; 2^22 floats 63 -> 57).  A top-k that takes
// the pipeline keeps 65536 (cta_keys): its speculating passes keep a list per warp.
// n / 512 buckets, 8192 to kMaxNb, in the table: a CTA writes as many counts
// (n / 32: 55 us for 52 at 2^21 floats, 60 for 57 at 2^22, 70 for 68 at 10 M); the
// rows have room for n / 32, as tables that track single keys and dense ones need.
// Half as many, down to 8192, where there are more requests than buckets (above 2^25
// elements: n / 2^25 times as many, as survivors then cost more than slots): nearly
// every bucket holds one, whatever their number, and the plan and the finisher work
// by the slot (65536 k's of 2^24 floats / doubles 827 / 1041 us a call with 32768
// buckets, 479 / 721 with 8192; 20000 k's of 2^23 doubles 408 and 344 with 16384 and
// 8192; but 33000 k's of 2^27 doubles 3546 with 32768, 4292 with 8192).
template <class InT, class OutT>
static Plan make_plan(const Context &ctx, uint64_t n, uint32_t num_req, uint32_t cta_keys = 16384,
                      bool rows = true) {
  using K = typename Traits<InT>::K;
  Plan p;
  p.n = n;
  p.num_req = num_req;
  p.S = n <= kFrontSamples ? (uint32_t)n : kFrontSamples;
  auto buckets = [&](uint64_t want) {
    uint32_t nb = 8192;
    while (nb < kMaxNb && (uint64_t)nb * 2 <= want) nb *= 2;
    return nb;
  };
  p.nb_max = buckets(n / 32);
  p.nb_want = buckets(n / 512);
  const uint64_t many = std::max<uint64_t>(1, n >> 25);
  while (p.nb_want > 8192 && num_req >= p.nb_want * many) p.nb_want /= 2;
  const uint64_t g = (n + cta_keys - 1) / cta_keys;
  p.G = (uint32_t)(g < 1 ? 1 : (g > (uint64_t)ctx.sm_count ? ctx.sm_count : g));
  p.scan_tiles = (p.nb_max + kScanTile - 1) / kScanTile;
  // Tiles of 8 vectors per thread stream a little faster than tiles of 4, but
  // the grid's last round of tiles is then coarser: keep 8 unless 4 spreads
  // the tiles over the CTAs better by more than 1 % (the busiest CTA's tiles
  // against the average).
  {
    const double nv = (double)(n * sizeof(InT) / 16);
    auto spread = [&](double tile_v) {
      const double t = std::floor(nv / tile_v);
      return t < 1 ? 1e9 : std::ceil(t / p.G) * p.G / t;
    };
    p.unroll8 = spread(8.0 * 1024) <= spread(4.0 * 1024) * 1.01;
  }
  p.cap_keys = cap_keys_for<InT>();
  uint32_t slots_bound = num_req < p.nb_max ? num_req : p.nb_max;
  uint32_t fg = 5u * (uint32_t)ctx.sm_count;
  p.fin_grid = slots_bound < fg ? (slots_bound ? slots_bound : 1) : fg;
  uint64_t cap = n / 8;
  cap = cap < (1u << 20) ? (1u << 20) : cap;
  if (cap > n) cap = n;
  // survivors below surv_half; from there the candidate pool, which also
  // holds one partly filled chunk per histogram warp
  p.surv_half = (cap / 2) & ~(uint64_t)3;  // 16-byte aligned pool
  p.surv_cap = cap + (uint64_t)p.G * kCandWarps * kCandChunk;
  const uint64_t chunks = (p.surv_cap - p.surv_half) / kCandChunk;
  p.cand_chunks = (uint32_t)(chunks < 0xFFFFFFFFull ? chunks : 0xFFFFFFFFull);

  const size_t A = 256;
  size_t o = 0;
  p.out = o;
  o = align_up(o + (size_t)num_req * sizeof(OutT), A);
  p.ctrl = o;
  o += A;  // ctrl is followed directly by the requests (one upload)
  p.reqs = o;
  o = align_up(o + (size_t)num_req * sizeof(Req), A);
  p.hdr = o;
  o = align_up(o + sizeof(LutHeader<K>), A);
  p.lut = o;
  o = align_up(o + kLutPadded * sizeof(uint32_t), A);
  p.samples = o;
  o = align_up(o + (size_t)p.S * sizeof(K), A);
  p.spans = o;
  o = align_up(o + 2 * (size_t)front_ctas(p.S) * sizeof(K), A);
  p.fine = o;
  o = align_up(o + kFineWords * sizeof(uint32_t) + sizeof(SliceOut<K>), A);
  p.wpre = o;
  o = align_up(o + kWinBins * sizeof(uint32_t), A);
  p.partials = o;
  o = align_up(o + (rows ? (size_t)p.G * p.nb_max * sizeof(uint32_t) : 0), A);
  auto arr = [&](size_t &off, size_t elems, size_t esz) {
    off = o;
    o = align_up(o + elems * esz, A);
  };
  arr(p.sorted, kPlanFew, sizeof(Req));
  // (sized for a dense table's buckets)
  arr(p.bpre, kDenseKeys, 4);
  arr(p.bco, kDenseKeys / 8, 4);
  arr(p.ttot, kDenseKeys / kScanTile, 4);
  arr(p.seg_bucket, p.nb_max, 4);
  arr(p.seg_off, p.nb_max, 8);
  arr(p.seg_size, p.nb_max, 4);
  arr(p.kstart, p.nb_max, 4);
  arr(p.kcnt, p.nb_max, 4);
  arr(p.kcur, p.nb_max, 4);
  arr(p.fill, p.nb_max, 4);
  arr(p.seg_lo, p.nb_max, sizeof(K));
  arr(p.seg_hi, p.nb_max, sizeof(K));
  arr(p.deferred, p.nb_max, 4);
  arr(p.req_bucket, num_req, 4);
  arr(p.req_local, num_req, 4);
  arr(p.klist, num_req, sizeof(Req));
  // premapped plan (many requests): bucket bitmap and request counts, zeroed
  // together before each use, and the bucket -> slot map
  p.pm_bits = o;
  p.pm_bcount = o + (size_t)p.nb_max / 8;
  o = align_up(o + (size_t)p.nb_max / 8 + (size_t)p.nb_max * 4, A);
  arr(p.pm_bslot, p.nb_max, 4);
  arr(p.cand_cnt, (size_t)p.G * kCandWarps, 4);
  arr(p.cand_tab, (size_t)p.G * kCandWarps * kCandChunksPerWarp, 4);
  // single-key tracking of tables whose keys repeat often: each CTA's key per
  // bucket, and per bucket whether the vector holds one key there and which
  arr(p.reps, rows ? (size_t)p.G * p.nb_max : 0, sizeof(K));
  arr(p.bsingle, p.nb_max, 4);
  arr(p.bkey, p.nb_max, sizeof(K));
  p.total = o;
  return p;
}

// Raise a kernel's dynamic shared-memory limit on the current device.  The
// attribute belongs to the kernel as loaded on one device, so it is set once
// per device (the largest value asked for so far is remembered per device);
// the result of the setting is returned for the caller to check.
template <auto F>
static cudaError_t set_smem_max(int bytes) {
  static std::atomic<int> set_to[kMaxDevices];  // static storage: starts at zero
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool tracked = dev >= 0 && dev < kMaxDevices;
  if (tracked && set_to[dev].load(std::memory_order_acquire) >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute((const void *)F, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && tracked) {
    int cur = set_to[dev].load(std::memory_order_acquire);
    while (cur < bytes && !set_to[dev].compare_exchange_weak(cur, bytes)) {
    }
  }
  return e;
}

// Launches a pipeline kernel with programmatic stream serialization: it may be
// scheduled while the previous kernel in the stream still runs, and waits for
// that kernel in its own first instructions (pdl_start).  The arguments are
// converted to the kernel's parameter types.
template <class... P, class... A>
static cudaError_t launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                          A &&...args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Launches k_small as one cluster of kSmCtas CTAs, plainly (no programmatic
// serialization: it is the call's first kernel).
template <class... P, class... A>
static cudaError_t launch_small(void (*kern)(P...), cudaStream_t s, A &&...args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kSmCtas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kSmCtas);
  cfg.blockDim = dim3(kSmThreads);
  cfg.dynamicSmemBytes = kSmBytes;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Whether the current device can run k_small<InT, OutT> (once per device):
// its shared memory and the cluster size (16 CTAs, a non-portable size that
// must be allowed first) are set, and the occupancy calculator must find room
// for one such cluster.  false: the small-vector path is not used there.
template <class InT, class OutT>
static std::atomic<int> *small_state() {
  static std::atomic<int> state[kMaxDevices];  // 0 unknown, 1 ready, 2 unavailable
  return state;
}
template <class InT, class OutT>
static bool small_ready() {
  std::atomic<int> *state = small_state<InT, OutT>();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
  const int st = state[dev].load(std::memory_order_acquire);
  if (st) return st == 1;
  auto kern = k_small<InT, OutT>;
  bool ok = cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSmBytes) == cudaSuccess &&
            cudaFuncSetAttribute((const void *)kern,
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (ok) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kSmCtas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSmCtas);
    cfg.blockDim = dim3(kSmThreads);
    cfg.dynamicSmemBytes = kSmBytes;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    ok = cudaOccupancyMaxActiveClusters(&clusters, (const void *)kern, &cfg) == cudaSuccess &&
         clusters >= 1;
  }
  cudaGetLastError();  // a refused attribute or query leaves no error behind
  state[dev].store(ok ? 1 : 2, std::memory_order_release);
  return ok;
}

struct PassTimer {
  Context &ctx;
  cudaStream_t s;
  int pass;
  PassTimer(Context &c, cudaStream_t st, int p) : ctx(c), s(st), pass(p) {
    if (ctx.profiling & (1u << pass)) cudaEventRecord(ctx.ev0[pass], s);
  }
  ~PassTimer() {
    if (ctx.profiling & (1u << pass)) cudaEventRecord(ctx.ev1[pass], s);
    ctx.stats.launches++;
    ctx.stats.pass_launches[pass]++;
  }
};

static void collect_pass_times(Context &ctx, const bool *ran) {
  if (!ctx.profiling) return;
  for (int i = 0; i < GGKS_NUM_PASSES; ++i) {
    if (!ran[i] || !(ctx.profiling & (1u << i))) continue;
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, ctx.ev0[i], ctx.ev1[i]) == cudaSuccess) ctx.stats.pass_ms[i] += ms;
  }
}

// Rank windows for speculative compaction: one window over all requested
// ranks, or, for up to 64 requests, two windows split at the widest gap
// between neighbouring ranks.  The table builder widens them by the sample's
// error and turns speculation off when they would keep too many elements;
// windows spanning more than n / 16 ranks are not sent at all.
static inline void set_windows_any(Ctrl *ci, const Req *hr, uint32_t num_req) {
  if (num_req == 0) return;
  if (num_req > 64) {
    uint32_t lo = hr[0].rank, hi = hr[0].rank;
    for (uint32_t i = 1; i < num_req; ++i) {
      lo = hr[i].rank < lo ? hr[i].rank : lo;
      hi = hr[i].rank > hi ? hr[i].rank : hi;
    }
    ci->spec_nwin = 1;
    ci->spec_lo[0] = lo;
    ci->spec_hi[0] = hi;
    return;
  }
  uint32_t r[64];
  for (uint32_t i = 0; i < num_req; ++i) r[i] = hr[i].rank;
  std::sort(r, r + num_req);
  uint32_t cut = 0, gap = 0;  // the second window starts at r[cut] (0: one window)
  for (uint32_t i = 1; i < num_req; ++i)
    if (r[i] - r[i - 1] > gap) {
      gap = r[i] - r[i - 1];
      cut = i;
    }
  if (gap <= 1) cut = 0;
  ci->spec_nwin = cut ? 2 : 1;
  ci->spec_lo[0] = r[0];
  ci->spec_hi[0] = cut ? r[cut - 1] : r[num_req - 1];
  if (cut) {
    ci->spec_lo[1] = r[cut];
    ci->spec_hi[1] = r[num_req - 1];
  }
}
static inline void set_windows(Ctrl *ci, const Req *hr, uint32_t num_req, uint64_t n) {
  set_windows_any(ci, hr, num_req);
  uint64_t span = 0;
  for (uint32_t w = 0; w < ci->spec_nwin; ++w) span += ci->spec_hi[w] - ci->spec_lo[w] + 1;
  if (span > n / 16) ci->spec_nwin = 0;
}

// Top-k by a sampled threshold (ggks_topk.cuh): k_sample, k_bin, k_slice,
// k_filter, k_pick.  *missed: the candidates fell short (or did not fit), nothing is
// answered, and the caller runs the pipeline; d_in then holds the device copy
// of an ingested host vector.
template <class InT>
static int topk_threshold(Context &ctx, const InT *d_in, uint64_t n, uint32_t K, InT *d_out_user,
                          const InT **host_results, cudaStream_t s, const InT *ingest,
                          bool *missed) {
  using Kt = typename Traits<InT>::K;
  *missed = false;
  const Plan p = make_plan<InT, InT>(ctx, n, K, 16384u, false);
  cudaError_t e = ensure_arena(ctx, p.total);
  if (e != cudaSuccess) return from_cuda(e);
  e = ensure_surv(ctx, (size_t)p.surv_cap * sizeof(Kt));
  if (e != cudaSuccess) return from_cuda(e);
  char *A = ctx.arena;
  Ctrl *ctrl = reinterpret_cast<Ctrl *>(A + p.ctrl);
  Kt *tau = reinterpret_cast<Kt *>(A + p.hdr);
  Kt *samples = reinterpret_cast<Kt *>(A + p.samples);
  Kt *spans = reinterpret_cast<Kt *>(A + p.spans);
  uint32_t *fine = reinterpret_cast<uint32_t *>(A + p.fine);
  SliceOut<Kt> *slice = reinterpret_cast<SliceOut<Kt> *>(fine + kFineWords);
  Kt *arr = reinterpret_cast<Kt *>(ctx.surv);  // the candidate array
  const uint64_t arr_cap = p.surv_cap;
  InT *d_out = d_out_user;
  // pinned: [out | status]
  const size_t out_span = p.ctrl - p.out;
  e = ensure_pin(ctx, out_span + 256);
  if (e != cudaSuccess) return from_cuda(e);
  const bool want_host = host_results != nullptr;
  static_assert(kPickMax <= kPinOut, "k_pick writes its results in place");
  if (!d_out_user) d_out = reinterpret_cast<InT *>(ctx.pin_dev);
  const volatile uint32_t *h_status = reinterpret_cast<const uint32_t *>(ctx.pin + out_span);
  cudaError_t le = cudaSuccess;
  auto L = [&le](cudaError_t r) {
    if (le == cudaSuccess) le = r;
  };
  const int pick_smem = (int)pick_smem_bytes<Kt>();
  const int filt_smem = (int)(kCandWarps * kFiltBuf * sizeof(Kt));
  L(set_smem_max<k_pick<Kt, InT>>(pick_smem));
  L(set_smem_max<k_filter<InT, 8>>(filt_smem));
  L(set_smem_max<k_filter<InT, 4>>(filt_smem));
  bool ran[GGKS_NUM_PASSES] = {false, false, false, false, false, false};
  bool open = false;  // no threshold: every key is a candidate
  {
    PassTimer t(ctx, s, GGKS_PASS_SAMPLE);
    const uint32_t g = front_ctas(p.S);
    L(launch(k_sample<InT>, g, 1024, 0, s, ingest ? ingest : d_in, n, p.S, 0x5EEDu, samples, spans,
             fine, kFineWords + kSliceZeroWords, ctrl, Ctrl{}, ReqCopy{}));
    L(launch(k_bin<Kt>, g, 1024, 0, s, samples, p.S, spans, fine, ctrl));
    // the sample rank below the K-th largest's, with six standard deviations
    // and four ranks to spare
    const double pl = (double)(n - K) / (double)n, S = p.S;
    const double a = pl * S - (6.0 * std::sqrt(S * pl * (1.0 - pl)) + 4.0);
    open = !(a > 0.0);  // the window reaches the smallest sample
    SliceWant want{};
    want.rank[0] = open ? 0u : (a >= S - 1.0 ? p.S - 1u : (uint32_t)a);
    L(launch(k_slice<Kt, 1>, g, 1024, 0, s, samples, p.S, spans, fine, want, slice));
    ctx.stats.launches += 2;
    ran[GGKS_PASS_SAMPLE] = true;
  }
  {
    PassTimer t(ctx, s, GGKS_PASS_HIST);
    L(launch(p.unroll8 ? k_filter<InT, 8> : k_filter<InT, 4>, p.G, 1024, filt_smem, s,
             ingest ? ingest : d_in, n, slice, samples, p.S, open, tau, arr, arr_cap, &ctrl->cand_next,
             ingest ? const_cast<InT *>(d_in) : nullptr, ctrl));
    ran[GGKS_PASS_HIST] = true;
  }
  {
    PassTimer t(ctx, s, GGKS_PASS_FINISH);
    L(launch(k_pick<Kt, InT>, 1, 1024, pick_smem, s, arr, arr_cap, &ctrl->cand_next, tau, K,
             d_out, ctrl, reinterpret_cast<uint32_t *>(ctx.pin_dev + out_span)));
    ran[GGKS_PASS_FINISH] = true;
  }
  e = le != cudaSuccess ? le : cudaGetLastError();
  if (e != cudaSuccess) return from_cuda(e);
  if (want_host && d_out_user)
    e = cudaMemcpyAsync(ctx.pin, d_out, (size_t)K * sizeof(InT), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return from_cuda(e);
  collect_pass_times(ctx, ran);
  const uint32_t status = *h_status;
  if (status & ST_FATAL) return (status & ST_TIMEOUT) ? GGKS_TIMEOUT : GGKS_INTERNAL;
  if (status & ST_TOPK_MISS) {
    *missed = true;
    ctx.stats.topk_misses++;
    return GGKS_OK;
  }
  ctx.stats.topk_threshold_calls++;
  if (want_host) *host_results = reinterpret_cast<const InT *>(ctx.pin);
  return GGKS_OK;
}

// A top-k's large bins of distinct keys: up to kWinMaxDefer that a CTA can sort are
// (k_wbig); else one bin is selected from again for at most kWinMaxAgain values, or the
// pipeline answers.  (786000 values, most of them 0 to 2, some up to 150000, top-20000:
// 151 us a call by the pipeline after the window, now 75; 110 by the pipeline alone.  2^24
// floats, 0.1 % of them one value far out, top-20000: 222, by a recursive level 134, now
// 105; 3 M such floats, 17000 values of one bin: 163, by a recursive level 203, now 98.)
constexpr uint32_t kWinMaxDefer = 64;
constexpr uint32_t kWinMaxAgain = 4096;
// smallest vector whose clustered k's go to the window path before the one-launch one
constexpr uint64_t kWinFirstN = 1ull << 19;

// The window path's choice (ggks_window.cuh): the sample ranks around the
// requested ascending ranks [rlo, rhi] -- six standard deviations and four ranks
// outside them, or an open end -- and the candidates to expect.
struct WindowPlan {
  bool ok = false, lo_open = false, hi_open = false;
  SliceWant want{};
  double expect = 0.0;
};
// Taken for ranks that span at most n / 32 of a vector of more than 2^18
// elements (the pipeline's speculating pass and its further kernels cost more:
// 2^26 uint32, top-65536: 167 us a call, here 94; the median of 50 M floats 132,
// here 77; of a smaller vector the sample is a good part, and most calls on one
// take the one-launch path), when the window is closed on one side at least and the
// candidates, with half again to spare, fit the survivor buffer's lower half.
// A top-k also needs bins that a warp can sort: at most 32 keys on average.
static inline WindowPlan plan_window(const Plan &p, uint64_t rlo, uint64_t rhi, bool topk) {
  WindowPlan w;
  const double n = (double)p.n, S = p.S;
  if (p.n <= (1u << 18) || (rhi - rlo + 1) * 32 > p.n) return w;
  const double pl = rlo / n, ph = (rhi + 1) / n;
  const double a = pl * S - (6.0 * std::sqrt(S * pl * (1.0 - pl)) + 4.0);
  const double b = ph * S + (6.0 * std::sqrt(S * ph * (1.0 - ph)) + 4.0);
  w.lo_open = a <= 0.0;
  w.hi_open = b >= S - 1.0;
  if (w.lo_open && w.hi_open) return w;
  w.want.rank[0] = w.lo_open ? 0u : (uint32_t)a;
  w.want.rank[1] = w.hi_open ? p.S - 1u : (uint32_t)b;
  w.expect = ((w.hi_open ? S : b) - (w.lo_open ? 0.0 : a)) / S * n;
  w.ok = w.expect * 1.5 <= (double)p.surv_half && (!topk || w.expect <= 32.0 * kWinBins);
  return w;
}

// *missed: as in topk_threshold.
template <class InT>
static int select_window(Context &ctx, const InT *d_in, uint64_t n, const ReqSource &src,
                         uint32_t num_req, uint64_t rlo, uint64_t rhi, InT *d_out_user,
                         const InT **host_results, cudaStream_t s, const InT *ingest,
                         bool *missed) {
  using K = typename Traits<InT>::K;
  *missed = true;
  const Plan p = make_plan<InT, InT>(ctx, n, num_req, 16384u, false);
  const WindowPlan w = plan_window(p, rlo, rhi, src.topk);
  if (!w.ok) return GGKS_OK;
  cudaError_t e = ensure_arena(ctx, p.total);
  if (e != cudaSuccess) return from_cuda(e);
  e = ensure_surv(ctx, (size_t)p.surv_cap * sizeof(K));
  if (e != cudaSuccess) return from_cuda(e);
  char *A = ctx.arena;
  Ctrl *ctrl = reinterpret_cast<Ctrl *>(A + p.ctrl);
  Req *reqs = reinterpret_cast<Req *>(A + p.reqs);
  K *samples = reinterpret_cast<K *>(A + p.samples);
  K *spans = reinterpret_cast<K *>(A + p.spans);
  uint32_t *fine = reinterpret_cast<uint32_t *>(A + p.fine);
  uint32_t *bins = fine + kWinBinsAt, *cur = fine + kWinCurAt;
  const BigBins big{reinterpret_cast<unsigned long long *>(fine + kWinFirstAt), fine + kWinMixedAt};
  WinCtl<K> *wc = reinterpret_cast<WinCtl<K> *>(fine + kWinCtlAt);
  SliceOut<K> *slice = reinterpret_cast<SliceOut<K> *>(fine + kFineWords);
  uint32_t *wpre = reinterpret_cast<uint32_t *>(A + p.wpre);
  K *arr = reinterpret_cast<K *>(ctx.surv), *placed = arr + p.surv_half;
  // pinned: [out | control block | requests | large bins]
  const bool want_host = host_results != nullptr;
  const size_t out_span = p.ctrl - p.out;
  const uint32_t room = src.h_k ? num_req : kWinMaxDefer;
  const size_t big_at = align_up(out_span + 256 + (src.h_k ? (size_t)num_req * sizeof(Req) : 0), 16);
  e = ensure_pin(ctx, big_at + room * sizeof(WinDefer));
  if (e != cudaSuccess) return from_cuda(e);
  Ctrl *h_ctrl = reinterpret_cast<Ctrl *>(ctx.pin + out_span);
  WinDefer *h_big = reinterpret_cast<WinDefer *>(ctx.pin + big_at);
  // results in place: at most kPlanFew of a k list, and a top-k's warps write
  // neighbouring ones (65536 uint32: 4 us a call less than by a copy)
  static_assert(kPlanFew <= kPinOut, "results of a k list");
  InT *d_out = d_out_user ? d_out_user : reinterpret_cast<InT *>(ctx.pin_dev);
  if (src.h_k) {
    Req *hr = reinterpret_cast<Req *>(ctx.pin + out_span + 256);
    for (uint32_t i = 0; i < num_req; ++i) {
      hr[i].rank = (uint32_t)(n - src.h_k[i]);
      hr[i].out = i;
    }
  }
  cudaError_t le = cudaSuccess;
  auto L = [&le](cudaError_t r) {
    if (le == cudaSuccess) le = r;
  };
  bool ran[GGKS_NUM_PASSES] = {false, false, false, false, false, false};
  const uint32_t g = front_ctas(p.S);
  {
    PassTimer t(ctx, s, GGKS_PASS_SAMPLE);
    const ReqCopy bring{src.h_k ? reinterpret_cast<const Req *>(ctx.pin_dev + out_span + 256) : nullptr,
                        reqs, src.h_k ? num_req : 0u};
    L(launch(k_sample<InT>, g + (bring.num + 1023) / 1024, 1024, 0, s, ingest ? ingest : d_in, n,
             p.S, 0x5EEDu, samples, spans, fine, kFineWords + kSliceZeroWords, ctrl, Ctrl{}, bring));
    L(launch(k_bin<K>, g, 1024, 0, s, samples, p.S, spans, fine, ctrl));
    L(launch(k_slice<K, 2>, g, 1024, 0, s, samples, p.S, spans, fine, w.want, slice));
    ctx.stats.launches += 2;
    ran[GGKS_PASS_SAMPLE] = true;
  }
  {
    const int smem = (int)wfilter_smem_bytes<K>();
    L(set_smem_max<k_wfilter<InT>>(smem));
    PassTimer t(ctx, s, GGKS_PASS_HIST);
    L(launch(k_wfilter<InT>, p.G, 1024, smem, s, ingest ? ingest : d_in, n, slice, samples, p.S, spans, g,
             w.lo_open, w.hi_open, wc, arr, p.surv_half, bins,
             ingest ? const_cast<InT *>(d_in) : nullptr));
    ran[GGKS_PASS_HIST] = true;
  }
  WinSlots<K> sl;
  sl.seg_off = reinterpret_cast<uint64_t *>(A + p.seg_off);
  sl.seg_size = reinterpret_cast<uint32_t *>(A + p.seg_size);
  sl.bin = reinterpret_cast<uint32_t *>(A + p.kstart);
  sl.seg_lo = reinterpret_cast<K *>(A + p.seg_lo);
  sl.seg_hi = reinterpret_cast<K *>(A + p.seg_hi);
  sl.klist = reinterpret_cast<Req *>(A + p.klist);
  {
    PassTimer t(ctx, s, GGKS_PASS_COMPACT);
    const uint32_t grid = (uint32_t)std::min<double>(ctx.sm_count, 1.0 + w.expect / 4096.0);
    L(set_smem_max<k_wplace<K>>((int)(kWinBins * 4)));
    L(launch(k_wplace<K>, grid, 1024, kWinBins * 4, s, arr, p.surv_half, n, src.topk ? num_req : 0u, w.lo_open,
             w.hi_open, reqs, num_req, wc, bins, cur, wpre, placed, p.surv_cap - p.surv_half, big, sl,
             ctrl));
    ran[GGKS_PASS_COMPACT] = true;
  }
  Ctrl *h_ctrl_dev = reinterpret_cast<Ctrl *>(ctx.pin_dev + out_span);
  WinDefer *deferred = reinterpret_cast<WinDefer *>(ctx.pin_dev + big_at);
  {
    PassTimer t(ctx, s, GGKS_PASS_FINISH);
    if (src.topk) {
      L(launch(k_wsort<K, InT>, 2u * (uint32_t)ctx.sm_count, kWinSortThreads, 0, s, placed, wc, bins,
               wpre, big, num_req, deferred, room, d_out, ctrl, h_ctrl_dev));
    } else {
      const int smem = finish_smem_bytes<InT>();
      L(set_smem_max<k_wfinish<K, InT>>(smem));
      L(launch(k_wfinish<K, InT>, num_req, kFinThreads, smem, s, placed, sl, big, deferred,
               p.cap_keys, d_out, ctrl, h_ctrl_dev));
    }
    ran[GGKS_PASS_FINISH] = true;
  }
  e = le != cudaSuccess ? le : cudaGetLastError();
  if (e != cudaSuccess) return from_cuda(e);
  auto pull = [&]() -> cudaError_t {  // results to host memory, and the synchronisation
    cudaError_t r = cudaSuccess;
    if (want_host && d_out_user)
      r = cudaMemcpyAsync(ctx.pin, d_out, (size_t)num_req * sizeof(InT), cudaMemcpyDeviceToHost, s);
    return r == cudaSuccess ? cudaStreamSynchronize(s) : r;
  };
  e = pull();
  if (e != cudaSuccess) return from_cuda(e);
  collect_pass_times(ctx, ran);
  const uint32_t status = *reinterpret_cast<const volatile uint32_t *>(&h_ctrl->status);
  if (status & ST_FATAL) return (status & ST_TIMEOUT) ? GGKS_TIMEOUT : GGKS_INTERNAL;
  // a miss: the pipeline answers (the streaming pass has written the device copy of an
  // ingested vector)
  const uint32_t D = (status & ST_DEFERRED) ? h_ctrl->deferred_count : 0u;
  bool sort = src.topk && D && D <= kWinMaxDefer;  // large bins that k_wbig can sort
  for (uint32_t i = 0; sort && i < D; ++i) sort = h_big[i].size <= win_big_max<K>();
  *missed = (status & ST_TOPK_MISS) != 0 ||
            (src.topk && !sort &&
             (D > 1 || (D && std::min(h_big[0].size, num_req - h_big[0].above) > kWinMaxAgain)));
  if (*missed) return GGKS_OK;
  if (sort) {
    const int smem = (int)wbig_smem_bytes<K>();
    e = set_smem_max<k_wbig<K, InT>>(smem);
    if (e != cudaSuccess) return from_cuda(e);
    k_wbig<K, InT><<<D, 1024, smem, s>>>(placed, deferred, num_req, d_out);
    ctx.stats.launches++;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = pull();
    if (e != cudaSuccess) return from_cuda(e);
  } else if (D) {
    // large bins of distinct keys: select from each again, on its keys
    int st = GGKS_OK;
    Context *ch = child_of(ctx, &st);
    if (!ch) return st;
    if (src.topk) {
      // a bin's largest keys are the outputs from the number of keys above it on (many
      // results: through the arena, see kPinOut)
      for (uint32_t i = 0; i < D; ++i) {
        const WinDefer &d = h_big[i];
        const uint32_t m = std::min(d.size, num_req - d.above);
        InT *o = (d_out_user ? d_out : reinterpret_cast<InT *>(A + p.out)) + d.above;
        ReqSource cs;
        cs.topk = true;
        ctx.stats.recursions++;
        st = select<K, InT>(*ch, placed + d.off, d.size, cs, m, o, nullptr, s, nullptr);
        if (st != GGKS_OK) return st;
        if (!d_out_user)
          e = cudaMemcpyAsync(ctx.pin + (size_t)d.above * sizeof(InT), o, (size_t)m * sizeof(InT),
                              cudaMemcpyDeviceToHost, s);
        if (e != cudaSuccess) return from_cuda(e);
      }
    } else {
      // the requests of one bin together, in the call's pinned requests (all read by now)
      std::sort(h_big, h_big + D, [](const WinDefer &a, const WinDefer &b) { return a.off < b.off; });
      Req *hr = reinterpret_cast<Req *>(ctx.pin + out_span + 256);
      const Req *dr = reinterpret_cast<const Req *>(ctx.pin_dev + out_span + 256);
      for (uint32_t i = 0; i < D; ++i) hr[i] = {h_big[i].rank, h_big[i].slot};
      for (uint32_t i = 0, j; i < D; i = j) {
        for (j = i + 1; j < D && h_big[j].off == h_big[i].off; ++j) {
        }
        ReqSource cs;
        cs.d_reqs = dr + i;
        ctx.stats.recursions++;
        st = select<K, InT>(*ch, placed + h_big[i].off, h_big[i].size, cs, j - i, d_out, nullptr, s,
                            nullptr);
        if (st != GGKS_OK) return st;
      }
    }
    e = pull();
    if (e != cudaSuccess) return from_cuda(e);
  }
  ctx.stats.spec_calls++;
  ctx.stats.spec_ctas += p.G;
  if (want_host) *host_results = reinterpret_cast<const InT *>(ctx.pin);
  return GGKS_OK;
}

// A small vector in one launch (ggks_tiny.cuh: one CTA, where the vector fits
// its registers; else ggks_small.cuh: one cluster): host k lists or a top-k of
// at most kSmMaxReq requests on a device vector of at most kSmMaxN
// (kSmMaxTopkN for a top-k) elements.
// *missed: the kernel met a case it leaves to the pipeline (nothing is
// answered; the caller runs the pipeline, which writes every output again).
// Arena: [phase stamps | cursors' starts]; pinned host memory,
// which the kernel reads and writes in place: [out | status | requests].
template <class InT, class OutT>
static int select_small(Context &ctx, const InT *d_in, uint64_t n, const ReqSource &src,
                        uint32_t num_req, OutT *d_out_user, const OutT **host_results,
                        cudaStream_t s, bool *missed) {
  using K = typename Traits<InT>::K;
  *missed = false;
  const size_t out_span = align_up((size_t)num_req * sizeof(OutT), 256);
  const size_t o_ctrl = 0, o_chk = o_ctrl + 256;
  cudaError_t e = ensure_pin(ctx, out_span + 256 + (size_t)num_req * sizeof(Req));
  if (e != cudaSuccess) return from_cuda(e);
  static_assert(kSmMaxReq <= kPinOut && kSmCtas * 4 <= 256,
                "requests, results and status in place");
  OutT *d_out = d_out_user ? d_out_user : reinterpret_cast<OutT *>(ctx.pin_dev);
  const volatile uint32_t *h_status = reinterpret_cast<const uint32_t *>(ctx.pin + out_span);
  // every call ends with a stream synchronisation: no earlier kernel still
  // reads or writes the pinned buffer
  Req *hr = reinterpret_cast<Req *>(ctx.pin + out_span + 256);
  for (uint32_t i = 0; i < num_req; ++i) {
    hr[i].rank = src.topk ? (uint32_t)(n - 1 - i) : (uint32_t)(n - src.h_k[i]);
    hr[i].out = i;
  }
  const Req *d_reqs = reinterpret_cast<const Req *>(ctx.pin_dev + out_span + 256);
  uint32_t *d_status = reinterpret_cast<uint32_t *>(ctx.pin_dev + out_span);
  const bool want_host = host_results != nullptr;
  // waits for the launch; statuses: words the kernel leaves in h_status
  auto finish = [&](uint32_t statuses, bool *miss) -> int {
    cudaError_t r = cudaGetLastError();
    if (r == cudaSuccess && want_host && d_out_user)
      r = cudaMemcpyAsync(ctx.pin, d_out, (size_t)num_req * sizeof(OutT), cudaMemcpyDeviceToHost,
                          s);
    if (r == cudaSuccess) r = cudaStreamSynchronize(s);
    if (r != cudaSuccess) return from_cuda(r);
    const bool ran[GGKS_NUM_PASSES] = {true, false, false, false, false, false};
    collect_pass_times(ctx, ran);
    uint32_t status = 0;
    for (uint32_t c = 0; c < statuses; ++c) status |= h_status[c];
    *miss = (status & ST_SMALL_MISS) != 0;
    if (!*miss) {
      ctx.stats.small_calls++;
      if (want_host) *host_results = reinterpret_cast<const OutT *>(ctx.pin);
    }
    return GGKS_OK;
  };
  // A vector that fits the registers of one CTA: one CTA.
  if (n <= tiny_max<K>()) {
    const int smem = (int)tiny_smem_bytes<K>(n);
    e = set_smem_max<k_tiny<InT, OutT>>((int)tiny_smem_bytes<K>(tiny_max<K>()));
    if (e != cudaSuccess) return from_cuda(e);
    {
      PassTimer t(ctx, s, GGKS_PASS_SAMPLE);
      k_tiny<InT, OutT><<<1, kTinyThreads, smem, s>>>(d_in, (uint32_t)n, d_reqs, num_req, d_out);
    }
    return finish(0, missed);
  }
  if (!small_ready<InT, OutT>()) {
    *missed = true;
    return GGKS_OK;
  }
  e = ensure_arena(ctx, o_chk + (size_t)kSmNb * kSmCtas * sizeof(uint32_t));
  if (e == cudaSuccess) e = ensure_surv(ctx, (size_t)n * sizeof(K));
  if (e != cudaSuccess) return from_cuda(e);
  char *A = ctx.arena;
  Ctrl *ctrl = reinterpret_cast<Ctrl *>(A + o_ctrl);
#ifdef GGKS_SMALL_TIMING
  cudaMemsetAsync(ctrl, 0, sizeof(Ctrl), s);
#endif
  {
    PassTimer t(ctx, s, GGKS_PASS_SAMPLE);
    e = launch_small(k_small<InT, OutT>, s, d_in, n, d_reqs, num_req, d_out,
                     reinterpret_cast<K *>(ctx.surv), ctx.surv_bytes / sizeof(K),
                     reinterpret_cast<uint32_t *>(A + o_chk), d_status, ctrl);
  }
  if (e != cudaSuccess) {
    // a cluster launch the device refuses (its SMs held by other work in a
    // way the occupancy query did not foresee): the pipeline runs instead,
    // and this device no longer tries the small path
    cudaGetLastError();
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices)
      small_state<InT, OutT>()[dev].store(2, std::memory_order_release);
    *missed = true;
    return GGKS_OK;
  }
  const int st = finish(kSmCtas, missed);
  if (st != GGKS_OK) return st;
#ifdef GGKS_SMALL_TIMING
  Ctrl tc;
  const Ctrl *h_ctrl = &tc;
  cudaMemcpy(&tc, ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost);
  fprintf(stderr, "ggks small timing n=%llu req=%u:", (unsigned long long)n, num_req);
  // stamp order: 0 start, 1 sampled, 2 table, 3 histograms, 8 totals, 9 scan,
  // 10 barrier, 11 prefix, 12 requests, 13 cursors, 4 barrier, 5 compacted,
  // 6 checked, 7 finished
  static const int order[14] = {0, 1, 2, 3, 8, 9, 10, 11, 12, 13, 4, 5, 6, 7};
  for (int i = 1; i < 14; ++i)
    fprintf(stderr, " %.2f",
            (double)(h_ctrl->t_ns[order[i]] - h_ctrl->t_ns[order[i - 1]]) * 1e-3);
  fprintf(stderr, " us; first CTA start %.2f us before CTA 0, last CTA end %.2f us after\n",
          (double)(h_ctrl->t_ns[0] - ~h_ctrl->t_ns[14]) * 1e-3,
          (double)(h_ctrl->t_ns[15] - h_ctrl->t_ns[7]) * 1e-3);
#endif
  if (*missed) ctx.stats.small_misses++;
  return GGKS_OK;
}

template <class InT, class OutT>
int select(Context &ctx, const InT *d_in, uint64_t n, const ReqSource &src, uint32_t num_req,
           OutT *d_out_user, const OutT **host_results, cudaStream_t s, const InT *ingest) {
  using K = typename Traits<InT>::K;
  if (ctx.depth > 12) return GGKS_INTERNAL;
  // the requests' ranks, where the window path may take them
  const bool window = ctx.depth == 0 && num_req >= 1 && !src.no_window &&
                      (src.topk ? !src.topk_pipeline : src.h_k && num_req <= kPlanFew);
  uint64_t rlo = n - num_req, rhi = n - 1;
  if (window && src.h_k) {
    const auto mm = std::minmax_element(src.h_k, src.h_k + num_req);
    rlo = n - *mm.second;
    rhi = n - *mm.first;
  }
  // clustered k's of a vector above 2^19: the window path is the faster one (one k,
  // 2^19 floats 44 us a call in one launch, 41 by a window; 2^20 53 and 42; 2^20
  // doubles 65 and 55; 400 K doubles 52 and 54)
  const bool window_first = window && src.h_k && n > kWinFirstN && rhi - rlo < n / 32;
  if constexpr (std::is_same<InT, OutT>::value) {
    bool missed = false;
    auto try_small = [&]() -> int {
      return select_small<InT, OutT>(ctx, d_in, n, src, num_req, d_out_user, host_results, s, &missed);
    };
    // a small device vector with host k's or a top-k: one launch, unless that
    // kernel leaves the case to the pipeline
    const bool small = ctx.depth == 0 && !ingest && !src.no_small && (src.h_k || src.topk) &&
                       num_req >= 1 && num_req <= kSmMaxReq &&
                       n <= (src.topk ? kSmMaxTopkN : kSmMaxN);
    if (small && !window_first) {
      const int st = try_small();
      if (st != GGKS_OK || !missed) return st;
    }
    if (src.topk && ctx.depth == 0 && num_req <= kPickMax && n > 65536 &&
        (uint64_t)num_req * 64 <= n && !src.topk_pipeline) {
      // a top-k of at most kPickMax values from a vector larger than the sample:
      // the threshold path, unless its candidates fall short
      const int st = topk_threshold<InT>(ctx, d_in, n, num_req, d_out_user, host_results, s,
                                         ingest, &missed);
      if (st != GGKS_OK || !missed) return st;
      ingest = nullptr;  // the filter pass wrote the device copy
    } else if (window) {
      // clustered ranks: the window path, unless its candidates fall short
      const uint64_t done = ctx.stats.launches;
      const int st = select_window<InT>(ctx, d_in, n, src, num_req, rlo, rhi, d_out_user,
                                        host_results, s, ingest, &missed);
      if (st != GGKS_OK || !missed) return st;
      if (ctx.stats.launches != done) {
        ctx.stats.topk_misses++;
        ingest = nullptr;  // the pass wrote the device copy
      }
      if (small && window_first) {
        const int st2 = try_small();
        if (st2 != GGKS_OK || !missed) return st2;
      }
    }
  }
  const Plan p = make_plan<InT, OutT>(ctx, n, num_req, src.topk ? 65536u : 16384u);
  cudaError_t e = ensure_arena(ctx, p.total);
  if (e != cudaSuccess) return from_cuda(e);
  e = ensure_surv(ctx, (size_t)p.surv_cap * sizeof(K));
  if (e != cudaSuccess) return from_cuda(e);
  char *A = ctx.arena;
  Ctrl *ctrl = reinterpret_cast<Ctrl *>(A + p.ctrl);
  Req *reqs = reinterpret_cast<Req *>(A + p.reqs);
  Req *sorted = reinterpret_cast<Req *>(A + p.sorted);
  LutHeader<K> *hdr = reinterpret_cast<LutHeader<K> *>(A + p.hdr);
  uint32_t *lut = reinterpret_cast<uint32_t *>(A + p.lut);
  K *samples = reinterpret_cast<K *>(A + p.samples);
  K *spans = reinterpret_cast<K *>(A + p.spans);
  uint32_t *fine = reinterpret_cast<uint32_t *>(A + p.fine);
  uint32_t *partials = reinterpret_cast<uint32_t *>(A + p.partials);
  uint32_t *bpre = reinterpret_cast<uint32_t *>(A + p.bpre);  // prefix inside 64-bucket tiles
  uint32_t *bco = reinterpret_cast<uint32_t *>(A + p.bco);    // every eighth of them
  uint32_t *ttot = reinterpret_cast<uint32_t *>(A + p.ttot);  // the tiles' totals
  uint32_t *seg_bucket = reinterpret_cast<uint32_t *>(A + p.seg_bucket);
  uint64_t *seg_off = reinterpret_cast<uint64_t *>(A + p.seg_off);
  uint32_t *seg_size = reinterpret_cast<uint32_t *>(A + p.seg_size);
  uint32_t *kstart = reinterpret_cast<uint32_t *>(A + p.kstart);
  uint32_t *kcnt = reinterpret_cast<uint32_t *>(A + p.kcnt);
  uint32_t *kcur = reinterpret_cast<uint32_t *>(A + p.kcur);
  uint32_t *fill = reinterpret_cast<uint32_t *>(A + p.fill);
  K *seg_lo = reinterpret_cast<K *>(A + p.seg_lo);
  K *seg_hi = reinterpret_cast<K *>(A + p.seg_hi);
  uint32_t *deferred = reinterpret_cast<uint32_t *>(A + p.deferred);
  uint32_t *req_bucket = reinterpret_cast<uint32_t *>(A + p.req_bucket);
  uint32_t *req_local = reinterpret_cast<uint32_t *>(A + p.req_local);
  Req *klist = reinterpret_cast<Req *>(A + p.klist);
  K *surv = reinterpret_cast<K *>(ctx.surv);
  K *cand = surv + p.surv_half;
  uint32_t *cand_cnt = reinterpret_cast<uint32_t *>(A + p.cand_cnt);
  uint32_t *cand_tab = reinterpret_cast<uint32_t *>(A + p.cand_tab);
  K *reps = reinterpret_cast<K *>(A + p.reps);
  uint32_t *bsingle = reinterpret_cast<uint32_t *>(A + p.bsingle);
  K *bkey = reinterpret_cast<K *>(A + p.bkey);
  // pinned host memory: [out | control block | requests]
  const bool want_host = host_results != nullptr;
  const size_t out_span = p.ctrl - p.out;  // == align_up(num_req * sizeof(OutT), 256)
  e = ensure_pin(ctx, out_span + 256 + (src.h_k ? (size_t)num_req * sizeof(Req) : 0));
  if (e != cudaSuccess) return from_cuda(e);
  Ctrl *h_ctrl = reinterpret_cast<Ctrl *>(ctx.pin + out_span);
  Ctrl *h_ctrl_dev = reinterpret_cast<Ctrl *>(ctx.pin_dev + out_span);
  const bool out_in_pin = !d_out_user && want_host && num_req <= kPinOut;
  const bool out_in_arena = !d_out_user && !out_in_pin;
  OutT *d_out = d_out_user    ? d_out_user
                : out_in_pin ? reinterpret_cast<OutT *>(ctx.pin_dev)
                             : reinterpret_cast<OutT *>(A + p.out);
  Ctrl ci{};  // the control block's initial words
  const Req *rq = src.d_reqs;  // where k_sample finds the requests (null: a top-k)
  if (src.h_k) {
    // every call ends with a stream synchronisation, so nothing of an earlier
    // one still reads the pinned buffer here
    Req *hr = reinterpret_cast<Req *>(ctx.pin + out_span + 256);
    for (uint32_t i = 0; i < num_req; ++i) {
      hr[i].rank = (uint32_t)(n - src.h_k[i]);
      hr[i].out = i;
    }
    set_windows(&ci, hr, num_req, n);
    rq = reinterpret_cast<const Req *>(ctx.pin_dev + out_span + 256);
  }
  if (src.topk && num_req && (uint64_t)num_req <= n / 16) {
    ci.spec_nwin = 1;
    ci.spec_lo[0] = n - num_req;
    ci.spec_hi[0] = n - 1;
  }
  bool ran[GGKS_NUM_PASSES] = {false, false, false, false, false, false};
  cudaError_t le = cudaSuccess;  // the first failed launch
  auto L = [&le](cudaError_t r) {
    if (le == cudaSuccess) le = r;
  };
  // ---- (b) sample + splitter table; the requests
  const bool few = num_req <= kPlanFew;
  const bool dense_ok = std::is_same<InT, uint32_t>::value && src.h_k && few && !ingest &&
                        !src.no_dense && ctx.depth == 0 && p.nb_max == kMaxNb;
  {
    PassTimer t(ctx, s, GGKS_PASS_SAMPLE);
    const uint32_t g = front_ctas(p.S);
    // device requests of a recursive level are read in place
    const ReqCopy bring{rq, reqs, src.d_reqs ? 0u : num_req};
    const Req *raw = src.d_reqs ? src.d_reqs : reqs;
    L(launch(k_sample<InT>, g + (bring.num + 1023) / 1024, 1024, 0, s, ingest ? ingest : d_in, n,
             p.S, 0x5EEDu, samples, spans, fine, kLutIdx, ctrl, ci, bring));
    L(launch(k_bin<K>, g, 1024, 0, s, samples, p.S, spans, fine, ctrl));
    const RankWindows win{ci.spec_nwin, {ci.spec_lo[0], ci.spec_lo[1]}, {ci.spec_hi[0], ci.spec_hi[1]}};
    const ReqCopy sort{raw, sorted, few ? num_req : 0u};
    L(launch(k_table<K>, 1 + sort_ctas(sort.num), kTableThreads, 0, s, samples, p.S, spans, fine, n,
             win, hdr, lut, p.nb_max, p.nb_want, p.cand_chunks, p.G, dense_ok, ctrl, sort));
    rq = few ? sorted : raw;
    ctx.stats.launches += 2;
    ran[GGKS_PASS_SAMPLE] = true;
  }
  // ---- (c) histogram
  {
    const int smem = (int)(kRepWords * sizeof(uint32_t) + (size_t)p.nb_max * 4);
    L(set_smem_max<k_hist<InT, 8>>((int)(kRepWords * sizeof(uint32_t) + (size_t)kMaxNb * 4)));
    L(set_smem_max<k_hist<InT, 4>>((int)(kRepWords * sizeof(uint32_t) + (size_t)kMaxNb * 4)));
    PassTimer t(ctx, s, GGKS_PASS_HIST);
    // with a mapped host vector, this pass also writes the device copy d_in
    L(launch(p.unroll8 ? k_hist<InT, 8> : k_hist<InT, 4>, p.G, 1024, smem, s, ingest ? ingest : d_in, n, hdr, lut, partials,
             p.nb_max, ctrl, ingest ? const_cast<InT *>(d_in) : nullptr, cand, cand_cnt, cand_tab,
             &ctrl->cand_next, reps));
    ran[GGKS_PASS_HIST] = true;
  }
  // ---- (d) reduce + decoupled look-back scan
  {
    PassTimer t(ctx, s, GGKS_PASS_SCAN);
    L(launch(k_colsum<K>, p.scan_tiles, kScanThreads, 0, s, partials, p.G, p.nb_max, hdr, bpre,
             bco, ttot, ctrl, reps, bsingle, bkey));
    ran[GGKS_PASS_SCAN] = true;
  }
  // ---- (e) plan
  {
    // per-slot request counters in shared memory unless the requests are premapped
    const int smem = (int)(align_up(kLutPadded * sizeof(uint32_t) + (size_t)p.nb_max * 5, 16) +
                           (num_req < kPremapMin ? kPlanSlotBytes : 0));
    L(set_smem_max<k_plan<InT, OutT>>(kPlanSmemMax));
    PassTimer t(ctx, s, GGKS_PASS_PLAN);
    Premap pm;
    const bool premap = num_req >= kPremapMin;
    uint32_t *pm_bits = reinterpret_cast<uint32_t *>(A + p.pm_bits);
    uint32_t *pm_bcount = reinterpret_cast<uint32_t *>(A + p.pm_bcount);
    uint32_t *pm_bslot = reinterpret_cast<uint32_t *>(A + p.pm_bslot);
    if (premap) {
      // many requests: map them with many CTAs (k_reqmap), place them with
      // many CTAs (k_reqplace); the plan CTA only numbers the slots
      e = cudaMemsetAsync(pm_bits, 0, (size_t)p.nb_max / 8 + (size_t)p.nb_max * 4, s);
      if (e != cudaSuccess) return from_cuda(e);
      L(set_smem_max<k_reqmap>((int)(kMaxNb * 4)));
      L(launch(k_reqmap, (num_req + kReqmapPerCta - 1) / kReqmapPerCta, 1024, p.nb_max * 4, s,
               bpre, ttot, ctrl, rq, num_req, req_bucket, req_local, pm_bits, pm_bcount));
      pm.bits = pm_bits;
      pm.bcount = pm_bcount;
      pm.bslot = pm_bslot;
    }
    if (few)
      L(launch(k_plan_few<InT>, 1, 1024, 0, s, hdr, lut, bpre, bco, ttot, n, rq, num_req, p.nb_max, ctrl,
               seg_bucket, seg_off, seg_size, kstart, kcnt, fill, seg_lo, seg_hi, klist, p.surv_cap,
               bsingle, bkey, p.surv_half));
    else
      L(launch(k_plan<InT, OutT>, 1, 1024, smem, s, hdr, lut, bpre, ttot, n, rq, num_req, p.nb_max,
               ctrl, seg_bucket, seg_off, seg_size, kstart, kcnt, kcur, fill, seg_lo, seg_hi,
               req_bucket, req_local, klist, p.surv_cap, pm, bsingle, bkey));
    if (premap) {
      L(launch(k_reqplace, (num_req + 1023) / 1024, 1024, 0, s, ctrl, rq, num_req, req_bucket,
               req_local, pm_bslot, kstart, kcur, klist));
      ctx.stats.launches += 2;
    }
    ran[GGKS_PASS_PLAN] = true;
  }
  uint64_t surv_cap = p.surv_cap;
  const K *cand_live = cand;  // no candidates once the survivor buffer is replaced
  auto launch_tail = [&]() {
    {
      const int smem = (int)compact_smem_bytes(p.nb_max);
      L(set_smem_max<k_compact<InT, 8>>((int)compact_smem_bytes(kMaxNb)));
      L(set_smem_max<k_compact<InT, 4>>((int)compact_smem_bytes(kMaxNb)));
      PassTimer t(ctx, s, GGKS_PASS_COMPACT);
      L(launch(p.unroll8 ? k_compact<InT, 8> : k_compact<InT, 4>, p.G, 1024, smem, s, d_in, n, hdr, lut, seg_bucket, seg_off,
               seg_size, partials, fill, p.nb_max, surv, surv_cap, ctrl, cand_live, cand_cnt,
               cand_tab, p.surv_half));
      ran[GGKS_PASS_COMPACT] = true;
    }
    {
      const int smem = p.fin_grid <= (uint32_t)ctx.sm_count ? kFinAlone : finish_smem_bytes<InT>();
      L(set_smem_max<k_finish<K, OutT>>(kFinAlone));
      PassTimer t(ctx, s, GGKS_PASS_FINISH);
      L(launch(k_finish<K, OutT>, p.fin_grid, kFinThreads, smem, s, surv, ctrl, seg_off, seg_size,
               seg_lo, seg_hi, kstart, kcnt, klist, deferred, p.cap_keys, d_out, h_ctrl_dev));
      ran[GGKS_PASS_FINISH] = true;
    }
  };
  launch_tail();
  e = le != cudaSuccess ? le : cudaGetLastError();
  if (e != cudaSuccess) return from_cuda(e);

  // k_finish leaves the control block (and few results) in pinned memory
  auto pull = [&](bool with_out) -> cudaError_t {
    cudaError_t r = cudaSuccess;
    if (with_out && !out_in_pin)
      r = cudaMemcpyAsync(ctx.pin, out_in_arena ? reinterpret_cast<const OutT *>(A + p.out) : d_out,
                          (size_t)num_req * sizeof(OutT), cudaMemcpyDeviceToHost, s);
    return r != cudaSuccess ? r : cudaStreamSynchronize(s);
  };
  e = pull(want_host);
  if (e != cudaSuccess) return from_cuda(e);
  collect_pass_times(ctx, ran);

  for (int round = 0; round < 4; ++round) {
    const Ctrl c = *h_ctrl;
    if (c.status & ST_FATAL) {
      return (c.status & ST_TIMEOUT) ? GGKS_TIMEOUT : GGKS_INTERNAL;
    }
    if (dense_ok && (c.status & ST_TOPK_MISS)) {
      // a dense table that cannot answer: the pipeline again, with an ordinary one
      ctx.stats.retries++;
      ReqSource again = src;
      again.no_dense = again.no_window = again.no_small = true;
      return select<InT, OutT>(ctx, d_in, n, again, num_req, d_out_user, host_results, s, nullptr);
    }
    if (c.status & ST_OVERFLOW) {
      // survivors did not fit: grow the buffer, re-run compaction + finish
      const uint64_t need = c.cap_needed + (c.cap_needed >> 3);
      e = ensure_surv(ctx, (size_t)need * sizeof(K));
      if (e != cudaSuccess) return from_cuda(e);
      surv = reinterpret_cast<K *>(ctx.surv);
      surv_cap = need;
      cand_live = nullptr;
      ctx.stats.retries++;
      e = cudaMemsetAsync(&ctrl->status, 0, sizeof(uint32_t), s);
      if (e != cudaSuccess) return from_cuda(e);
      for (int i = 0; i < GGKS_NUM_PASSES; ++i) ran[i] = false;
      launch_tail();
      if (le != cudaSuccess) return from_cuda(le);
      e = pull(want_host);
      if (e != cudaSuccess) return from_cuda(e);
      collect_pass_times(ctx, ran);
      continue;
    }
    if (c.status & ST_DEFERRED) {
      // oversized segments: select each again, recursively, on its keys
      const uint32_t D = c.deferred_count, ns = c.num_slots;
      std::vector<uint32_t> dl(D), sz(ns), ks(ns), kc(ns);
      std::vector<uint64_t> so(ns);
      e = cudaMemcpyAsync(dl.data(), deferred, D * 4, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaMemcpyAsync(sz.data(), seg_size, ns * 4, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaMemcpyAsync(so.data(), seg_off, ns * 8, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaMemcpyAsync(ks.data(), kstart, ns * 4, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaMemcpyAsync(kc.data(), kcnt, ns * 4, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return from_cuda(e);
      int st = GGKS_OK;
      Context *ch = child_of(ctx, &st);
      if (!ch) return st;
      for (uint32_t d = 0; d < D; ++d) {
        const uint32_t slot = dl[d];
        ReqSource cs;
        cs.d_reqs = klist + ks[slot];
        ctx.stats.recursions++;
        st = select<K, OutT>(*ch, surv + so[slot], sz[slot], cs, kc[slot], d_out, nullptr, s,
                             nullptr);
        if (st != GGKS_OK) return st;
      }
      if (want_host) {
        e = pull(true);
        if (e != cudaSuccess) return from_cuda(e);
      }
    }
    break;
  }
  ctx.stats.survivors += h_ctrl->total_surv;
  ctx.stats.spec_calls += h_ctrl->spec_on;
  ctx.stats.spec_ctas += h_ctrl->spec_ctas;
  if (want_host) *host_results = reinterpret_cast<const OutT *>(ctx.pin);
  return GGKS_OK;
}

}  // namespace ggks
