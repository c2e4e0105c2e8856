// window_kernels.cpp -- the sampled-window kernels and the splitter table on the host
// CPU (see cuda_on_host.h), as plain C functions for tests/test_window_host.py and
// tests/test_table_host.py.
#include "cuda_on_host.h"

#include "ggks_window.cuh"

using namespace ggks;

namespace {

template <class T>
struct Front {
  using K = typename Traits<T>::K;
  std::vector<K> samples, spans;
  std::vector<uint32_t> fine;
  SliceOut<K> slice;
  Ctrl ctrl;
};

// k_sample, k_bin, k_slice, k_wfilter over x[0 .. n), n <= kFrontSamples: every
// element is a sample, so the window's ends are the keys of ranks r0 and r1.
template <class T>
int filter(const T *x, uint64_t n, uint32_t r0, uint32_t r1, bool lo_open, bool hi_open,
           uint32_t grid, typename Traits<T>::K *arr, uint64_t cap, uint32_t *bins, uint64_t *out) {
  using K = typename Traits<T>::K;
  static Front<T> f;
  const uint32_t S = (uint32_t)n, g = front_ctas(S);
  f.samples.assign(S, 0);
  f.spans.assign(2 * g, 0);
  f.fine.assign(kLutIdx, ~0u);
  std::memset(&f.slice, 0, sizeof(f.slice));
  WinCtl<K> wc;
  std::memset(&wc, 0, sizeof(wc));
  SliceWant want;
  want.rank[0] = r0;
  want.rank[1] = r1;
  const K *samples = f.samples.data(), *spans = f.spans.data();
  bool ok = emu::launch(g, 1024, 0, [&] {
    k_sample<T>(x, n, S, 1u, f.samples.data(), f.spans.data(), f.fine.data(), kLutIdx, &f.ctrl,
                Ctrl{}, ReqCopy{});
  });
  ok = ok && emu::launch(g, 1024, 0, [&] { k_bin<K>(samples, S, spans, f.fine.data(), &f.ctrl); });
  ok = ok && emu::launch(g, 1024, 0, [&] {
         k_slice<K, 2>(samples, S, spans, f.fine.data(), want, &f.slice);
       });
  ok = ok && emu::launch(grid, 1024, wfilter_smem_bytes<K>(), [&] {
         k_wfilter<T>(x, n, &f.slice, samples, S, spans, g, lo_open, hi_open, &wc, arr, cap, bins, nullptr);
       });
  out[0] = wc.len;
  out[1] = wc.below;
  out[2] = wc.lo;
  out[3] = wc.shift;
  out[4] = wc.inner;
  out[5] = wc.ends;
  out[6] = wc.key_lo;
  out[7] = wc.key_hi;
  return ok ? 0 : 1;
}

// The table of x[0 .. n), n <= kFrontSamples (every element is a sample), and where it
// puts each of keys[0 .. m): the bucket and that bucket's smallest key.
template <class T>
int table(const T *x, uint64_t n, uint32_t nb_max, const typename Traits<T>::K *keys, uint32_t m,
          uint32_t *bucket, typename Traits<T>::K *first, uint32_t *nb) {
  using K = typename Traits<T>::K;
  const uint32_t S = (uint32_t)n, g = front_ctas(S);
  std::vector<K> samples(S), spans(2 * g);
  std::vector<uint32_t> fine(kLutIdx, ~0u), lut(kLutPadded, 0);
  LutHeader<K> h;
  Ctrl ctrl{};
  bool ok = emu::launch(g, 1024, 0, [&] {
    k_sample<T>(x, n, S, 1u, samples.data(), spans.data(), fine.data(), kLutIdx, &ctrl, Ctrl{},
                ReqCopy{});
  });
  ok = ok && emu::launch(g, 1024, 0, [&] {
         k_bin<K>(samples.data(), S, spans.data(), fine.data(), &ctrl);
       });
  ok = ok && emu::launch(1, kTableThreads, 0, [&] {
         k_table<K>(samples.data(), S, spans.data(), fine.data(), n, RankWindows{}, &h, lut.data(),
                    nb_max, nb_max, 0u, 1u, false, &ctrl, ReqCopy{});
       });
  if (!ok) return 1;
  const KeyTable<K> kt(h);
  for (uint32_t i = 0; i < m; ++i) {
    bucket[i] = bucket_of<K>(keys[i], kt, lut.data());
    first[i] = bucket_lo<K>(bucket[i], h.base, h.shift, lut.data(), sv_slices<K>() + 1 + h.low);
  }
  *nb = h.nb;
  return 0;
}

// k_wplace over the candidates arr[0 .. len) and the given bin counts, and, with out
// given, k_wsort (a top-k, kk > 0) or k_wfinish.
template <class K>
int place(const K *arr, uint32_t len, uint64_t n, uint32_t below, K lo, uint32_t shift,
          uint32_t nbins, const uint32_t *bins, uint32_t kk, const uint32_t *ranks,
          uint32_t num_req, uint32_t grid, K *placed, uint64_t placed_cap, K *out,
          uint32_t *status) {
  WinCtl<K> wc;
  std::memset(&wc, 0, sizeof(wc));
  wc.len = len;
  wc.below = below;
  wc.lo = lo;
  wc.shift = shift;
  wc.inner = nbins;
  std::vector<uint32_t> cur(kWinBins, 0), pre(kWinBins, 0);
  std::vector<unsigned long long> first(kWinBins, 0);
  std::vector<uint32_t> mixed(kWinBins, 0);
  const BigBins big{first.data(), mixed.data()};
  const uint32_t slots = num_req ? num_req : 1;
  std::vector<uint64_t> seg_off(slots);
  std::vector<uint32_t> seg_size(slots), bin(slots);
  std::vector<WinDefer> deferred(kWinBins);
  std::vector<K> seg_lo(slots), seg_hi(slots);
  std::vector<Req> klist(slots), reqs(slots);
  for (uint32_t i = 0; i < num_req; ++i) {
    reqs[i].rank = ranks[i];
    reqs[i].out = i;
  }
  WinSlots<K> sl{seg_off.data(), seg_size.data(), bin.data(),
                 seg_lo.data(),  seg_hi.data(),   klist.data()};
  Ctrl ctrl{}, host_ctrl{};
  bool ok = emu::launch(grid, 1024, kWinBins * 4, [&] {
    k_wplace<K>(arr, len, n, kk, false, kk != 0, reqs.data(), num_req, &wc, bins, cur.data(),
                pre.data(), placed, placed_cap, big, sl, &ctrl);
  });
  if (out && kk)
    ok = ok && emu::launch(grid, kWinSortThreads, 0, [&] {
           k_wsort<K, K>(placed, &wc, bins, pre.data(), big, kk,
                         deferred.data(), 4u, out, &ctrl, &host_ctrl);
         });
  else if (out)
    ok = ok && emu::launch(num_req, kFinThreads, finish_smem_for<K>(4096), [&] {
           k_wfinish<K, K>(placed, sl, big, deferred.data(), 4096u, out,
                           &ctrl, &host_ctrl);
         });
  *status = out ? host_ctrl.status : ctrl.status;
  return ok ? 0 : 1;
}

}  // namespace

extern "C" {

int emu_table_u32(const uint32_t *x, uint64_t n, uint32_t nb_max, const uint32_t *keys, uint32_t m,
                  uint32_t *bucket, uint32_t *first, uint32_t *nb) {
  return table<uint32_t>(x, n, nb_max, keys, m, bucket, first, nb);
}
int emu_table_f64(const double *x, uint64_t n, uint32_t nb_max, const uint64_t *keys, uint32_t m,
                  uint32_t *bucket, uint64_t *first, uint32_t *nb) {
  return table<double>(x, n, nb_max, keys, m, bucket, first, nb);
}
int emu_big_u32(const uint32_t *placed, uint64_t off, uint32_t size, uint32_t above, uint32_t kk,
                uint32_t *out) {
  const WinDefer d{off, size, 0, 0, above};
  return emu::launch(1, 1024, wbig_smem_bytes<uint32_t>(),
                     [&] { k_wbig<uint32_t, uint32_t>(placed, &d, kk, out); })
             ? 0
             : 1;
}
int emu_sort_u64(uint64_t *a, uint32_t c, uint32_t threads) {
  return emu::launch(1, threads, 0, [&] { cta_sort_any<uint64_t>(a, c); }) ? 0 : 1;
}

int emu_filter_f32(const float *x, uint64_t n, uint32_t r0, uint32_t r1, int lo_open, int hi_open,
                   uint32_t grid, uint32_t *arr, uint64_t cap, uint32_t *bins, uint64_t *out) {
  return filter<float>(x, n, r0, r1, lo_open, hi_open, grid, arr, cap, bins, out);
}
int emu_filter_u32(const uint32_t *x, uint64_t n, uint32_t r0, uint32_t r1, int lo_open,
                   int hi_open, uint32_t grid, uint32_t *arr, uint64_t cap, uint32_t *bins,
                   uint64_t *out) {
  return filter<uint32_t>(x, n, r0, r1, lo_open, hi_open, grid, arr, cap, bins, out);
}
int emu_filter_f64(const double *x, uint64_t n, uint32_t r0, uint32_t r1, int lo_open,
                   int hi_open, uint32_t grid, uint64_t *arr, uint64_t cap, uint32_t *bins,
                   uint64_t *out) {
  return filter<double>(x, n, r0, r1, lo_open, hi_open, grid, arr, cap, bins, out);
}
int emu_place_u32(const uint32_t *arr, uint32_t len, uint64_t n, uint32_t below, uint32_t lo,
                  uint32_t shift, uint32_t nbins, const uint32_t *bins, uint32_t kk,
                  const uint32_t *ranks, uint32_t num_req, uint32_t grid, uint32_t *placed,
                  uint64_t placed_cap, uint32_t *out, uint32_t *status) {
  return place<uint32_t>(arr, len, n, below, lo, shift, nbins, bins, kk, ranks, num_req, grid,
                         placed, placed_cap, out, status);
}

}  // extern "C"
