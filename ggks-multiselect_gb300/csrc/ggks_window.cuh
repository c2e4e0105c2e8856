// ggks_window.cuh -- clustered ranks (one k, k's close together, a long top-k) by a
// sampled window: one streaming pass keeps the keys that can hold the requested
// ranks and counts the keys below them, and the requests are answered from those.
//
// The reference computes every selection over the whole vector twice
// (bucketMultiselect.cu:571-574, :780-797).  Here, when the requests' ranks lie
// within a small part of the order:
//   k_sample, k_bin, k_slice (ggks_front.cuh): the sample, and its keys around
//             the window's two ends;
//   k_wfilter takes as the window [tlo, thi] the sample keys six standard
//             deviations and four ranks outside the requests' extreme ranks (an
//             end past the sample is open) and streams the vector once: keys
//             inside go to one contiguous candidate array and are counted in
//             kWinBins equal-width bins, keys below are counted, and so are
//             the copies of end keys that much of the vector holds;
//   k_wplace  every CTA takes the bins' prefix, finds the bins that hold the
//             requested ranks, and the candidates of those bins go to the
//             places of their ranks (bin by bin, unordered inside a bin);
//   k_wsort   (top-k) a warp per bin sorts and writes its values, descending; or
//   k_wfinish (requests) a CTA per request selects inside its bin;
//   large bins hold copies of one key, or the host selects from their keys again.
// No second read of the vector, no splitter table, no bucket atomics per key:
// the pass does two or three compares per key and is bound by HBM, where the
// speculating histogram pass (ggks_device.cuh) did a table lookup, a shared
// atomic and a vote: 50 M floats, their median: 81 us, now 43; the call 132 ->
// 77 us.
// Correctness never rests on the prediction: k_wplace checks that the candidates
// were all kept, fill their bins exactly and hold every requested rank; else the
// call reports ST_TOPK_MISS and the caller runs the pipeline.
#pragma once

#include "ggks_front.cuh"
#include "ggks_tiny.cuh"

namespace ggks {

constexpr int kWinBinBits = 13;
constexpr uint32_t kWinBins = 1u << kWinBinBits;
constexpr uint32_t kWinCol = 16;    // keys of one lane's column (k_wfilter)
constexpr uint32_t kWinSort = 256;  // keys of a bin that a warp sorts (k_wsort)
// Large bins of requests: more keys than kWinFlat may be copies of one key (a value's,
// in few-valued vectors), which needs no selection: 256 values in 2^26 floats, their
// median 287 us a call by selecting from the copies, now 108.  More than win_slot_max
// distinct ones (a gap in the distribution puts all candidates on one side into one
// bin) take one CTA longer than a recursive level, about 50 us: 2^26 floats in
// +-[1, 2), median: 505 us a call by one CTA and then the pipeline, now 155; 169 in
// the pipeline.
constexpr uint32_t kWinFlat = 2048;
template <class K>
__host__ __device__ constexpr uint32_t win_slot_max() {
  return (256u << 10) / (uint32_t)sizeof(K);
}
static_assert(1024 * kWinCol >= 2 * kSliceBuf, "the samples around the ends fit the columns");

// The window's bins: [copies of key_lo] [inner equal-width bins] [copies of key_hi].
// The two one-key bins exist where the window's closed ends are counted rather than
// kept (popular()): their copies are no candidates, and what lies between is never
// more than the window's ranks.
template <class K>
struct WinMap {
  K lo;                   // bin(k) = has_lo + (k - lo) >> shift, clamped to the inner bins
  K key_lo, key_hi;
  uint32_t shift, inner;  // inner may be 0 (counted ends with no key between them)
  bool has_lo, has_hi, lo_open, hi_open;
  __device__ __forceinline__ uint32_t nbins() const { return inner + has_lo + has_hi; }
  // bin of a candidate; keys outside [lo, ...] (beyond the sampled extremes, at an open
  // end) go to the end bins
  __device__ __forceinline__ uint32_t bin(K k) const {
    const K j = (k - lo) >> shift;
    return has_lo + (k < lo ? 0u : j < (K)inner ? (uint32_t)j : inner - 1u);
  }
  // bins one key wide; an end bin at an open end also holds the keys beyond the
  // sampled extremes
  __device__ __forceinline__ bool one_key(uint32_t b) const {
    return (has_lo && b == 0) || (has_hi && b + 1 == nbins()) ||
           (shift == 0 && !(lo_open && b == 0) && !(hi_open && b + 1 == nbins()));
  }
  // such a bin's key
  __device__ __forceinline__ K key(uint32_t b) const {
    return has_lo && b == 0 ? key_lo : has_hi && b + 1 == nbins() ? key_hi : lo + (K)(b - has_lo);
  }
};

// The map and what k_wfilter counted (device; len and below are zero on entry).
template <class K>
struct WinCtl {
  uint32_t len;    // candidates
  uint32_t below;  // keys below the window
  uint32_t total;  // keys in all bins: the candidates and the counted ends (k_wplace)
  uint32_t first;  // first bin that a top-k needs (k_wplace)
  uint32_t big;    // needed bins of more than kWinSort keys exist (k_wplace)
  uint32_t ends;   // 1: has_lo, 2: has_hi
  K lo, key_lo, key_hi;
  uint32_t shift, inner;
  __device__ __forceinline__ WinMap<K> map(bool lo_open, bool hi_open) const {
    return {lo, key_lo, key_hi, shift, inner, (ends & 1u) != 0, (ends & 2u) != 0, lo_open, hi_open};
  }
};

// One warp's candidates: each lane keeps its own in a column of shared memory --
// a predicated store and increment per key, no votes -- and when a column could
// fill up the warp moves all of them to the array with one atomic on its length,
// counting them in the CTA's bins on the way.  (With a vote and a position per
// kept key, as k_filter does, a window of 2.4 % of the keys took the pass from
// 36 to 52 us at 50 M floats: nearly every vector holds some.)
template <class K>
struct WinWarp {
  K *col;            // this lane's column: entry c at col[32 c]
  uint32_t cnt = 0;  // keys in it
  K *arr;
  uint64_t cap;
  uint32_t *len;
  uint32_t *bins;  // the CTA's
  WinMap<K> map;
  __device__ __forceinline__ void put(K k, bool keep) {
    if (keep) col[32 * cnt++] = k;
  }
  // every lane calls this after at most four puts
  __device__ __forceinline__ void check() {
    if (__any_sync(0xffffffffu, cnt > kWinCol - 4)) flush();
  }
  __device__ __forceinline__ void flush() {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t total = __reduce_add_sync(0xffffffffu, cnt);
    const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
    uint32_t base = 0;
    if (lane == 0 && total) base = atomicAdd(len, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (uint32_t c = 0; c < most; ++c) {
      const bool have = cnt > c;
      const uint32_t m = __ballot_sync(0xffffffffu, have);
      if (have) {
        const K k = col[32 * c];
        atomicAdd(&bins[map.bin(k)], 1u);
        const uint64_t at = (uint64_t)base + __popc(m & ((1u << lane) - 1u));
        if (at < cap) arr[at] = k;
      }
      base += __popc(m);
    }
    cnt = 0;
  }
};

template <class K>
__host__ __device__ constexpr size_t wfilter_smem_bytes() {
  return kWinBins * 4 + (size_t)1024 * kWinCol * sizeof(K);
}

// What a thread counted: keys below the window (COUNT: neither end open -- a window
// that is open below has none, one that is open above has all keys outside it),
// and copies of its end keys (ENDS).
struct WinCount {
  uint32_t below = 0, lo = 0, hi = 0;
};

// Grid and tiles as k_hist; 1024 threads.  Keeps the keys of [in, in + width] (ENDS:
// none at all where `none`).  copy_to: as in k_filter.
template <class T, bool COUNT, bool ENDS, bool INGEST>
__device__ __forceinline__ void wfilter_body(const T *__restrict__ x, uint64_t n,
                                             typename Traits<T>::K tlo, typename Traits<T>::K thi,
                                             typename Traits<T>::K in,
                                             typename Traits<T>::K width, bool none,
                                             T *__restrict__ copy_to,
                                             WinWarp<typename Traits<T>::K> &ww, WinCount &wcnt) {
  using K = typename Traits<T>::K;
  using V = typename Traits<T>::Vec;
  constexpr int PV = Traits<T>::kPerVec;
  constexpr int UNROLL = 4;
  const Span<T> sp = split_span(x, n);
  const V *xv = reinterpret_cast<const V *>(x + sp.head);
  V *cv = reinterpret_cast<V *>(copy_to + sp.head);
  const uint64_t tile_v = (uint64_t)blockDim.x * UNROLL;
  const uint64_t ntiles = sp.nvec / tile_v;
  uint32_t below = 0, at_lo = 0, at_hi = 0;
  auto one = [&](K k, bool valid) {
    if (COUNT || ENDS) below += valid && k < tlo ? 1u : 0u;
    if (ENDS) {
      at_lo += valid && k == tlo ? 1u : 0u;
      at_hi += valid && k == thi ? 1u : 0u;
    }
    ww.put(k, valid && !(ENDS && none) && (K)(k - in) <= width);
  };
  for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint64_t off = tile * tile_v + threadIdx.x;
    V v[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      v[u] = INGEST ? xv[off + (uint64_t)u * blockDim.x] : ldg_stream(xv + off + (uint64_t)u * blockDim.x);
    if (INGEST) {
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) cv[off + (uint64_t)u * blockDim.x] = v[u];
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      K k[PV];
      vec_keys<T>(v[u], k);
#pragma unroll
      for (int e = 0; e < PV; ++e) one(k[e], true);
      ww.check();
    }
  }
  // leftover vectors and the scalar head / tail: every lane runs every round
  if (blockIdx.x == (uint32_t)(ntiles % gridDim.x)) {
    for (uint64_t vb = ntiles * tile_v; vb < sp.nvec; vb += blockDim.x) {
      const uint64_t vi = vb + threadIdx.x;
      const bool valid = vi < sp.nvec;
      V vv{};
      if (valid) {
        vv = INGEST ? xv[vi] : ldg_stream(xv + vi);
        if (INGEST) cv[vi] = vv;
      }
      K k[PV];
      vec_keys<T>(vv, k);
#pragma unroll
      for (int e = 0; e < PV; ++e) one(k[e], valid);
      ww.check();
    }
    auto scalar = [&](uint64_t e0, uint64_t e1) {
      for (uint64_t eb = e0; eb < e1; eb += blockDim.x) {
        const uint64_t e = eb + threadIdx.x;
        const bool valid = e < e1;
        K k = 0;
        if (valid) {
          const T v = x[e];
          if (INGEST) copy_to[e] = v;
          k = Traits<T>::key(v);
        }
        one(k, valid);
        ww.check();
      }
    };
    scalar(0, sp.head);
    scalar(sp.tail0, n);
  }
  wcnt.below = below;
  wcnt.lo = at_lo;
  wcnt.hi = at_hi;
}

// bins: kWinBins words, zero on entry.
template <class T>
__global__ void __launch_bounds__(1024, 1)
    k_wfilter(const T *x, uint64_t n, const SliceOut<typename Traits<T>::K> *slice,
              const typename Traits<T>::K *samples, uint32_t S,
              const typename Traits<T>::K *spans, uint32_t parts, bool lo_open,
              bool hi_open, WinCtl<typename Traits<T>::K> *wc,
              typename Traits<T>::K *__restrict__ arr, uint64_t cap, uint32_t *__restrict__ bins_g,
              T *__restrict__ copy_to) {
  pdl_trigger();
  using K = typename Traits<T>::K;
  extern __shared__ uint4 smem_raw[];
  uint32_t *bins = reinterpret_cast<uint32_t *>(smem_raw);
  __shared__ RankShared<K> s_rank;
  __shared__ uint32_t s_below[32];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  fill_words(bins, kWinBins, 0u);
  pdl_wait();
  const SampleSpan<K> sp = sample_span<K>(spans, parts);
  // (the candidates' columns lend their space)
  K *cols = reinterpret_cast<K *>(bins + kWinBins), ends[2];
  const bool open[2] = {lo_open, hi_open};
  uint32_t same[2];
  rank_keys<2, K>(slice, samples, S, open, cols, s_rank, ends, same);
  const K tlo = lo_open ? K(0) : ends[0], thi = hi_open ? KeyMax<K>::v : ends[1];
  // counted ends: all closed ones, where one is popular or both are the same key
  const bool counted = (!lo_open && popular(same[0], S)) || (!hi_open && popular(same[1], S)) ||
                       tlo == thi;
  WinWarp<K> ww;
  WinMap<K> &map = ww.map;
  map.has_lo = counted && !lo_open;
  map.has_hi = counted && !hi_open && !(map.has_lo && thi == tlo);
  map.lo_open = lo_open;
  map.hi_open = hi_open;
  map.key_lo = tlo;
  map.key_hi = thi;
  // the kept keys [in, out], if any
  const K in = map.has_lo ? tlo + 1 : tlo, out = map.has_hi ? thi - 1 : thi;
  const bool none = in > out || (map.has_lo && in == 0) || (map.has_hi && thi == 0);
  // at an open end the bins reach the range and 64 keys past the sampled extreme, for
  // the keys the sample missed: of 65536 values, 1024 copies each, it misses the
  // largest in one vector of three; a tail's few hundred largest keys lie past it,
  // and in one end bin they need a recursive level (2^26 doubles, top-20000: N(100, 1)
  // 205 us a call with a quarter of the range, now 138; Cauchy 204, now 137)
  K lo = lo_open ? sp.kmin : in, hi = hi_open ? sp.kmax : out;
  const K span = hi > lo ? hi - lo : K(0), more = span < KeyMax<K>::v - 64 ? span + 64 : span;
  if (lo_open) lo = lo > more ? lo - more : K(0);
  if (hi_open) hi = hi < KeyMax<K>::v - more ? hi + more : KeyMax<K>::v;
  map.lo = lo;
  const K range = hi > lo ? hi - lo : K(0);
  const int bl = bitlen<K>(range);
  map.shift = bl > kWinBinBits ? (uint32_t)(bl - kWinBinBits) : 0u;
  if (counted && (range >> map.shift) + 1 > (K)(kWinBins - 2)) map.shift++;  // room for the ends
  map.inner = none ? 0u : (uint32_t)(range >> map.shift) + 1u;
  ww.col = cols + warp * (32 * kWinCol) + lane;
  ww.arr = arr;
  ww.cap = cap;
  ww.len = &wc->len;
  ww.bins = bins;
  if (blockIdx.x == 0 && tid == 0) {
    wc->lo = map.lo;
    wc->key_lo = map.key_lo;
    wc->key_hi = map.key_hi;
    wc->shift = map.shift;
    wc->inner = map.inner;
    wc->ends = (map.has_lo ? 1u : 0u) | (map.has_hi ? 2u : 0u);
  }
  const K width = out - in;
  WinCount wcnt;
  if (copy_to) {
    if (counted)
      wfilter_body<T, false, true, true>(x, n, tlo, thi, in, width, none, copy_to, ww, wcnt);
    else if (lo_open || hi_open)
      wfilter_body<T, false, false, true>(x, n, tlo, thi, in, width, none, copy_to, ww, wcnt);
    else
      wfilter_body<T, true, false, true>(x, n, tlo, thi, in, width, none, copy_to, ww, wcnt);
  } else if (counted) {
    wfilter_body<T, false, true, false>(x, n, tlo, thi, in, width, none, nullptr, ww, wcnt);
  } else if (lo_open || hi_open) {
    wfilter_body<T, false, false, false>(x, n, tlo, thi, in, width, none, nullptr, ww, wcnt);
  } else {
    wfilter_body<T, true, false, false>(x, n, tlo, thi, in, width, none, nullptr, ww, wcnt);
  }
  ww.flush();
  const uint32_t nbins = map.nbins();
  const uint32_t below = __reduce_add_sync(0xffffffffu, wcnt.below);
  const uint32_t at_lo = __reduce_add_sync(0xffffffffu, wcnt.lo);
  const uint32_t at_hi = __reduce_add_sync(0xffffffffu, wcnt.hi);
  if (lane == 0) {
    s_below[warp] = below;
    if (map.has_lo && at_lo) atomicAdd(&bins[0], at_lo);
    if (map.has_hi && at_hi) atomicAdd(&bins[nbins - 1], at_hi);
  }
  __syncthreads();
  for (uint32_t b = tid; b < nbins; b += blockDim.x)
    if (bins[b]) atomicAdd(&bins_g[b], bins[b]);
  if (warp == 0) {
    const uint32_t all = __reduce_add_sync(0xffffffffu, s_below[lane]);
    if (lane == 0 && all) atomicAdd(&wc->below, all);
  }
}

// Whether a large bin holds one key: first[b] is one of its keys (big_first), mixed[b]
// is set when another one is met (also by the largest 8-byte key, which first[]
// cannot tell from no key).  Zero on entry.
struct BigBins {
  unsigned long long *first;
  uint32_t *mixed;
};
__device__ __forceinline__ unsigned long long big_first(uint32_t k) { return (1ull << 32) | k; }
__device__ __forceinline__ unsigned long long big_first(uint64_t k) { return ~k; }
template <class K>
__device__ __forceinline__ K big_key(unsigned long long f) {
  return sizeof(K) == 4 ? (K)f : (K)~f;
}

// The slots that k_wfinish reads, one per request (k_wplace).
template <class K>
struct WinSlots {
  uint64_t *seg_off;
  uint32_t *seg_size, *bin;
  K *seg_lo, *seg_hi;
  Req *klist;
};

// Bins that hold requested ranks: their candidates go to placed[prefix of the bin
// ...), which holds the keys of local ranks (rank - below) prefix ... .  kk > 0:
// a top-k (every bin from the one of the kk-th largest up); else num_req requests,
// whose slots CTA 0 writes.  Large bins (of more than kWinSort or kWinFlat keys): also
// whether they hold one key, in big.  cur: kWinBins entries, zero on entry; pre_g: the
// bins' prefix, written by CTA 0 for a top-k.
template <class K>
__global__ void __launch_bounds__(1024, 1)
    k_wplace(const K *arr, uint64_t cap, uint64_t n, uint32_t kk, bool lo_open,
             bool hi_open, const Req *reqs, uint32_t num_req, WinCtl<K> *wc,
             const uint32_t *bins_g, uint32_t *cur, uint32_t *__restrict__ pre_g,
             K *__restrict__ placed, uint64_t placed_cap, BigBins big_bins, WinSlots<K> sl,
             Ctrl *ctrl) {
  pdl_start();
  extern __shared__ uint4 smem_raw[];
  uint32_t *cnt = reinterpret_cast<uint32_t *>(smem_raw);  // the CTA's keys per bin, then their place
  __shared__ __align__(16) uint32_t pre[kWinBins];
  __shared__ uint32_t need[kWinBins / 32], mix[kWinBins / 32];  // needed bins; bins of several keys
  __shared__ uint32_t s_scan[32];
  __shared__ bool s_miss, s_any;
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t C = wc->len;
  const WinMap<K> map = wc->map(lo_open, hi_open);
  const uint32_t nbins = map.nbins();
  constexpr uint32_t kPer = kWinBins / 1024;
  uint32_t c[kPer], sum = 0;
#pragma unroll
  for (uint32_t q = 0; q < kPer / 4; ++q) {
    const uint4 v = reinterpret_cast<const uint4 *>(bins_g)[tid * (kPer / 4) + q];
    c[4 * q] = v.x; c[4 * q + 1] = v.y; c[4 * q + 2] = v.z; c[4 * q + 3] = v.w;
    sum += v.x + v.y + v.z + v.w;
  }
  if (tid < kWinBins / 32) need[tid] = mix[tid] = 0;
  if (tid == 0) s_miss = s_any = false;
  fill_words(cnt, kWinBins, 0u);
  uint32_t total;
  uint32_t run = block_excl_scan(sum, s_scan, &total);
  bool big = false;
#pragma unroll
  for (uint32_t q = 0; q < kPer; ++q) {
    pre[tid * kPer + q] = run;
    run += c[q];
  }
  __syncthreads();
  auto count_of = [&](uint32_t b) -> uint32_t {
    return (b + 1 < kWinBins ? pre[b + 1] : total) - pre[b];
  };
  // the counted ends' copies take no places: a bin's begin at pre - off
  const uint32_t off = map.has_lo ? count_of(0) : 0u;
  const uint32_t copies = off + (map.has_hi ? count_of(nbins - 1) : 0u);
  // keys below the window: none below an open low end, all outside the window below an
  // open high end, else counted
  const uint64_t below = lo_open ? 0u : hi_open ? n - total : wc->below;
  const bool bad = (uint64_t)C > cap || (uint64_t)C > placed_cap || total - copies != C ||
                   (kk && (total < kk || !hi_open));
  // the last bin whose prefix is <= r, for r < total (never an empty one)
  auto bin_at = [&](uint32_t r) -> uint32_t {
    uint32_t b = 0;
#pragma unroll
    for (uint32_t step = kWinBins / 2; step; step >>= 1)
      if (pre[b + step] <= r && b + step < nbins) b += step;
    return b;
  };
  uint32_t first = 0;
  if (!bad && kk) {
    first = bin_at(total - kk);
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q) {
      const uint32_t b = tid * kPer + q;
      big |= b >= first && c[q] > kWinSort;
      if (b >= first && c[q] && !map.one_key(b)) s_any = true;
    }
  }
  big = __syncthreads_or(big);
  if (!bad && !kk && tid < num_req) {
    const Req q = reqs[tid];
    if (q.rank < below || q.rank - below >= total) {
      s_miss = true;
    } else {
      const uint32_t r = (uint32_t)(q.rank - below), b = bin_at(r);
      const bool one = map.one_key(b);
      if (!one) {
        atomicOr(&need[b >> 5], 1u << (b & 31));
        s_any = true;
      }
      if (blockIdx.x == 0) {
        const uint32_t j = b - map.has_lo;  // among the inner bins
        sl.seg_off[tid] = pre[b] - off;
        sl.seg_size[tid] = one ? 0u : count_of(b);  // 0: a flat slot, answered from seg_lo
        // an end bin also holds the keys beyond the sampled extremes
        sl.seg_lo[tid] = one ? map.key(b) : b == 0 && lo_open ? K(0) : map.lo + ((K)j << map.shift);
        sl.seg_hi[tid] = j + 1 >= map.inner ? KeyMax<K>::v : map.lo + (((K)j + 1) << map.shift) - K(1);
        sl.bin[tid] = b;
        Req e;
        e.rank = r - pre[b];
        e.out = q.out;
        sl.klist[tid] = e;
      }
    }
  }
  __syncthreads();
  const bool miss = bad || s_miss;
  if (blockIdx.x == 0) {
    if (tid == 0) {
      if (miss) atomicOr(&ctrl->status, ST_TOPK_MISS);
      ctrl->num_slots = num_req;
      ctrl->total_surv = C;
      wc->total = total;
      wc->first = first;
      wc->big = big ? 1u : 0u;
    }
    if (kk)
      for (uint32_t b = tid; b < kWinBins; b += blockDim.x) pre_g[b] = pre[b];
  }
  if (miss || !s_any) return;
  // The candidates of needed bins: a key's place among the CTA's in its bin by one
  // shared atomic, the CTA's places in the bin by one global atomic per bin and round.
  // (Few-valued vectors put hundreds of thousands of keys into a handful of bins;
  // warps that took their places with an atomic each queued on them: clustered k's
  // of 256 values in 2^26 floats 171 us a call, now 130.)  A bin that meets more keys
  // than it counted keeps its places and the call is a miss.
  bool over = false;
  constexpr uint32_t U = 8;
  for (uint32_t i0 = blockIdx.x * 1024 * U; i0 < C; i0 += gridDim.x * 1024 * U) {
    K k[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t i = i0 + 1024 * u + tid;
      k[u] = i < C ? __ldcg(arr + i) : K(0);
    }
    uint32_t at[U];  // place in the CTA's part of the bin; kNoSlot: not needed
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t b = map.bin(k[u]);
      const bool want = i0 + 1024 * u + tid < C &&
                        (kk ? b >= first && !map.one_key(b) : ((need[b >> 5] >> (b & 31)) & 1u) != 0u);
      at[u] = want ? atomicAdd(&cnt[b], 1u) : kNoSlot;
      // the first key of a large bin, taken by one lane for all of a bin's lanes
      const bool large = want && count_of(b) > (kk ? kWinSort : kWinFlat);
      if (!__any_sync(0xffffffffu, large)) continue;
      unsigned long long one = large ? __ldcg(big_bins.first + b) : 1ull;
      const unsigned long long mine = big_first(k[u]);
      for (uint32_t round = 0; round < 32; ++round) {  // (each settles a lane at least)
        const uint32_t none = __ballot_sync(0xffffffffu, one == 0);
        if (!none) break;
        const int leader = __ffs(none) - 1;
        unsigned long long got = 0;
        if ((int)lane == leader) {
          got = atomicCAS(big_bins.first + b, 0ull, mine);
          got = got ? got : mine ? mine : ~0ull;  // (the largest 8-byte key: no first key)
        }
        got = __shfl_sync(0xffffffffu, got, leader);
        const uint32_t bin = __shfl_sync(0xffffffffu, b, leader);
        if (one == 0 && b == bin) one = got;
      }
      const uint32_t bit = 1u << (b & 31);
      if (large && one != mine && !(mix[b >> 5] & bit)) atomicOr(&mix[b >> 5], bit);
    }
    __syncthreads();
    for (uint32_t b = tid; b < nbins; b += 1024) {
      if (cnt[b]) cnt[b] = atomicAdd(&cur[b], cnt[b]);
      if (mix[b >> 5] & (1u << (b & 31))) big_bins.mixed[b] = 1u;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      if (at[u] == kNoSlot) continue;
      const uint32_t b = map.bin(k[u]), p = cnt[b] + at[u];
      if (p < count_of(b))
        placed[pre[b] - off + p] = k[u];
      else
        over = true;
    }
    if (i0 + gridDim.x * 1024 * U < C) {  // another round
      __syncthreads();
      fill_words(cnt, kWinBins, 0u);
      __syncthreads();
    }
  }
  if (over) atomicOr(&ctrl->status, ST_TOPK_MISS);
}

// A large bin of distinct keys, left to a recursive level: its places, and for a
// request its slot and rank, for a top-k the number of keys above the bin.
struct WinDefer {
  uint64_t off;
  uint32_t size, slot, rank, above;
};
// (one thread calls this; list: host memory, the first `room` are kept)
__device__ __forceinline__ void win_defer(Ctrl *ctrl, WinDefer *list, uint32_t room,
                                          const WinDefer &d) {
  const uint32_t at = atomicAdd(&ctrl->deferred_count, 1u);
  if (at < room) list[at] = d;
  atomicOr(&ctrl->status, ST_DEFERRED);
}

// The last CTA leaves the call's status and its large bins' number in host memory.
// Every thread calls this last.
__device__ __forceinline__ void win_leave(Ctrl *ctrl, Ctrl *host_ctrl) {
  __syncthreads();
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(&ctrl->fin_done, 1u) != gridDim.x - 1) return;
  __threadfence();
  host_ctrl->deferred_count = __ldcg(&ctrl->deferred_count);
  host_ctrl->status = __ldcg(&ctrl->status);
}

// Requests' values from their bins, a CTA per request.  Large bins of one key need no
// selection, those of more than win_slot_max distinct ones go to a recursive level.
template <class K, class OutT>
__global__ void __launch_bounds__(kFinThreads)
    k_wfinish(const K *placed, WinSlots<K> sl, BigBins big_bins, WinDefer *__restrict__ deferred,
              uint32_t bcap, OutT *__restrict__ out, Ctrl *ctrl, Ctrl *__restrict__ host_ctrl) {
  pdl_start();
  extern __shared__ uint4 smem_raw[];
  const uint32_t i = blockIdx.x;
  // (only ST_DEFERRED is set meanwhile)
  if (!(ctrl->status & (ST_FATAL | ST_TOPK_MISS))) {
    const uint32_t size = sl.seg_size[i], b = sl.bin[i];
    const bool done =
        size > kWinFlat && !big_bins.mixed[b]
            ? finish_slot<K, OutT>(placed, 0u, big_key<K>(big_bins.first[b]), K(0), sl.klist + i, 1u,
                                   bcap, reinterpret_cast<uint32_t *>(smem_raw), out)
            : size <= win_slot_max<K>() &&
                  finish_slot<K, OutT>(placed + sl.seg_off[i], size, sl.seg_lo[i], sl.seg_hi[i],
                                       sl.klist + i, 1u, bcap,
                                       reinterpret_cast<uint32_t *>(smem_raw), out);
    if (!done && threadIdx.x == 0)
      win_defer(ctrl, deferred, gridDim.x, {sl.seg_off[i], size, i, sl.klist[i].rank, 0u});
  }
  win_leave(ctrl, host_ctrl);
}

// A top-k's large bins of distinct keys (win_big_max keys at most), a CTA of 1024
// threads each; launched only where k_wsort left some.  A bin's keys go to the places
// of 4096 parts of their range in shared memory, and one thread sorts each part; where
// a part holds more than kWinPart keys (another gap) the whole bin is sorted by the
// CTA's network (about 1 us a step: 22000 of 3 M floats, the call 226 us, by parts 98).
constexpr uint32_t kWinParts = 4096, kWinPart = 32;
template <class K>
__host__ __device__ constexpr uint32_t win_big_max() {
  return (128u << 10) / (uint32_t)sizeof(K);
}
template <class K>
__host__ __device__ constexpr size_t wbig_smem_bytes() {
  return 2 * kWinParts * 4 + (size_t)win_big_max<K>() * sizeof(K);
}
template <class K, class OutT>
__global__ void __launch_bounds__(1024, 1)
    k_wbig(const K *placed, const WinDefer *list, uint32_t kk, OutT *__restrict__ out) {
  extern __shared__ uint4 smem_raw[];
  uint32_t *cnt = reinterpret_cast<uint32_t *>(smem_raw), *start = cnt + kWinParts;
  K *a = reinterpret_cast<K *>(start + kWinParts);
  __shared__ K s_key[33];
  __shared__ uint32_t s_scan[32];
  const WinDefer d = list[blockIdx.x];
  const uint32_t tid = threadIdx.x, c = d.size;
  if (c > win_big_max<K>()) return;
  auto each = [&](auto &&fn) {
    constexpr uint32_t U = 8;
    for (uint32_t i0 = tid; i0 < c; i0 += U * 1024) {
      K k[U];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) k[u] = i0 + 1024 * u < c ? __ldcg(placed + d.off + i0 + 1024 * u) : K(0);
#pragma unroll
      for (uint32_t u = 0; u < U; ++u)
        if (i0 + 1024 * u < c) fn(i0 + 1024 * u, k[u]);
    }
  };
  fill_words(cnt, kWinParts, 0u);
  K lo = KeyMax<K>::v, hi = 0;
  each([&](uint32_t, K k) {
    lo = k < lo ? k : lo;
    hi = k > hi ? k : hi;
  });
  lo = block_reduce(lo, [](K u, K v) { return u < v ? u : v; }, s_key);
  hi = block_reduce(hi, [](K u, K v) { return u > v ? u : v; }, s_key);
  const int bl = bitlen<K>(hi - lo);
  const uint32_t sh = bl > 12 ? (uint32_t)(bl - 12) : 0u;
  each([&](uint32_t, K k) { atomicAdd(&cnt[(uint32_t)((k - lo) >> sh)], 1u); });
  __syncthreads();
  const uint4 c4 = reinterpret_cast<const uint4 *>(cnt)[tid];
  uint32_t all;
  const uint32_t pre = block_excl_scan(c4.x + c4.y + c4.z + c4.w, s_scan, &all);
  reinterpret_cast<uint4 *>(start)[tid] = make_uint4(pre, pre + c4.x, pre + c4.x + c4.y, pre + c4.x + c4.y + c4.z);
  // (parts one key wide need no sort)
  const bool crowded = __syncthreads_or(sh && max(max(c4.x, c4.y), max(c4.z, c4.w)) > kWinPart);
  if (crowded) {
    each([&](uint32_t i, K k) { a[i] = k; });
    __syncthreads();
    cta_sort_any<K>(a, c);
  } else {
    each([&](uint32_t, K k) {
      const uint32_t b = (uint32_t)((k - lo) >> sh);
      a[start[b] + atomicSub(&cnt[b], 1u) - 1u] = k;
    });
    __syncthreads();
    for (uint32_t b = tid; sh && b < kWinParts; b += 1024) {
      const uint32_t p0 = start[b], p1 = b + 1 < kWinParts ? start[b + 1] : c;
      for (uint32_t p = p0 + 1; p < p1; ++p) {
        const K v = a[p];
        uint32_t r = p;
        for (; r > p0 && a[r - 1] > v; --r) a[r] = a[r - 1];
        a[r] = v;
      }
    }
    __syncthreads();
  }
  for (uint32_t i = tid; i < c && d.above + i < kk; i += 1024)
    out[d.above + i] = Traits<OutT>::value(a[c - 1 - i]);
}

// A top-k's values from the placed bins: a warp per bin from wc->first up, the
// values in descending order to out[0 .. kk).  A large bin of distinct keys is left
// to k_wbig or a recursive level.
constexpr uint32_t kWinSortThreads = 256;
template <class K, class OutT>
__global__ void __launch_bounds__(kWinSortThreads)
    k_wsort(const K *placed, const WinCtl<K> *wc, const uint32_t *bins_g,
            const uint32_t *pre_g, BigBins big_bins, uint32_t kk, WinDefer *__restrict__ deferred,
            uint32_t room, OutT *__restrict__ out, Ctrl *ctrl, Ctrl *__restrict__ host_ctrl) {
  pdl_start();
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  // (one value for the whole warp, whose lanes meet in shuffles below, whatever other
  // CTAs set meanwhile)
  const uint32_t status = __shfl_sync(0xffffffffu, ctrl->status, 0);
  if (!(status & (ST_FATAL | ST_TOPK_MISS))) {
    const uint32_t C = wc->total, first = wc->first;
    const WinMap<K> map = wc->map(false, true);
    const uint32_t nbins = map.nbins(), off = map.has_lo ? bins_g[0] : 0u;
    const uint32_t warps = gridDim.x * (kWinSortThreads / 32);
    // position p of the window's order is the (C - p)-th largest
    auto put = [&](uint32_t p, K k) {
      const uint32_t i = C - 1 - p;
      if (i < kk) out[i] = Traits<OutT>::value(k);
    };
    auto sorted = [&](auto regs, uint32_t p0, uint32_t c) {
      constexpr int R = decltype(regs)::value;
      K v[R];
#pragma unroll
      for (int r = 0; r < R; ++r)
        v[r] = r * 32 + lane < c ? __ldcg(placed + p0 - off + r * 32 + lane) : KeyMax<K>::v;
      warp_bitonic_regs<K, R>(v);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r * 32 + lane < c) put(p0 + r * 32 + lane, v[r]);
    };
    for (uint32_t b = first + blockIdx.x * (kWinSortThreads / 32) + (tid >> 5); b < nbins; b += warps) {
      const uint32_t c = bins_g[b], p0 = pre_g[b];
      if (c == 0) continue;
      if (map.one_key(b)) {
        for (uint32_t j = lane; c <= kWinSort && j < c; j += 32) put(p0 + j, map.key(b));
      } else if (c <= 32)
        sorted(std::integral_constant<int, 1>{}, p0, c);
      else if (c <= 64)
        sorted(std::integral_constant<int, 2>{}, p0, c);
      else if (c <= kWinSort)
        sorted(std::integral_constant<int, (int)(kWinSort / 32)>{}, p0, c);
      else if (lane == 0 && big_bins.mixed[b])
        win_defer(ctrl, deferred, room, {p0 - off, c, b, 0u, C - p0 - c});
    }
    // copies of one key: every thread writes its share of the outputs in large bins
    if (wc->big) {
      for (uint32_t i = blockIdx.x * kWinSortThreads + tid; i < kk; i += gridDim.x * kWinSortThreads) {
        const uint32_t p = C - 1 - i;
        uint32_t b = 0;
        for (uint32_t step = kWinBins / 2; step; step >>= 1)
          if (b + step < nbins && pre_g[b + step] <= p) b += step;
        if (bins_g[b] > kWinSort && (map.one_key(b) || !big_bins.mixed[b]))
          out[i] = Traits<OutT>::value(map.one_key(b) ? map.key(b) : big_key<K>(big_bins.first[b]));
      }
    }
  }
  win_leave(ctrl, host_ctrl);
}

}  // namespace ggks
