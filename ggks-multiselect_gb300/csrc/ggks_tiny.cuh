// ggks_tiny.cuh -- the selection of a tiny vector by one CTA.
//
// A vector of at most tiny_max<K>() elements fits the registers of one CTA
// (32 keys of 4 bytes or 16 of 8 per thread), so nothing of the bucket
// algorithm needs a sample, a splitter table or an exchange between CTAs:
//
//   load    every key into registers; the smallest and largest key below and
//           above the middle of the key space (for floats: the negatives, the
//           two zeros apart, the positives);
//   count   one histogram of at most kTinyBins equal-width bins over the two
//           occupied ranges laid end to end, with the two middle keys between
//           them.  The gaps, for floats every exponent between the smallest
//           magnitudes and zero, take no bins: 2^15 normal floats leave 17
//           keys in the fullest binade's bins;
//   scan    the bins' exclusive prefix: the first rank of each;
//   place   each request finds its bin; the keys of requested bins go to the
//           positions of their bin's ranks in shared memory;
//   sort    a warp per requested bin, in registers (at most tiny_bin<K> keys) or,
//           when it holds few distinct keys, by counting their copies; the
//           CTA together for a larger one;
//   answer  each request reads its own rank.
//
// Bound: latency, about eight block barriers.  A call's device time at 5003
// floats, 11 k's: about 6 us, against 31 us for the cluster kernel
// (ggks_small.cuh), whose sampling, table build and cluster barriers cost the
// same at every size.
#pragma once

#include "ggks_device.cuh"

namespace ggks {

constexpr uint32_t kTinyThreads = 1024;
constexpr int kTinyBinBits = 13;
constexpr uint32_t kTinyBins = 1u << kTinyBinBits;
// keys of a bin sorted by a warp in registers.  Floats in [0, 1) with some far out spread
// over 150 binades' bins: 30000 of them put 400 to 560 into a bin (such a vector missed at 256:
// 101 k's 87 us a call, now 45; 57 in the cluster kernel alone)
template <class K>
__host__ __device__ constexpr uint32_t tiny_bin() {
  return sizeof(K) == 4 ? 1024u : 256u;
}
// larger bins are sorted by the CTA, one after the other (616 doubles, most of them within
// 1e-7 of one value: by the cluster kernel after this one 89 us a call, now 29; 53 by the
// cluster kernel alone): at most so many
template <class K>
__host__ __device__ constexpr uint32_t tiny_big() {
  return sizeof(K) == 4 ? 32u : 64u;
}
constexpr uint32_t kTinyMaxReq = kTinyThreads;

// keys per thread, and the longest vector
template <class K>
__host__ __device__ constexpr uint32_t tiny_per() {
  return sizeof(K) == 4 ? 32u : 16u;
}
template <class K>
__host__ __device__ constexpr uint32_t tiny_max() {
  return tiny_per<K>() * kTinyThreads;
}
// dynamic shared memory: the bins, then n keys
template <class K>
__host__ __device__ constexpr size_t tiny_smem_bytes(uint64_t n) {
  return kTinyBins * 4 + (((size_t)n * sizeof(K) + 15) & ~(size_t)15);
}

// Sorts the 32 R keys held by a warp, key r * 32 + lane in v[r], ascending.
template <class K, int R>
__device__ __forceinline__ void warp_bitonic_regs(K (&v)[R]) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (uint32_t k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (uint32_t r = 0; r < R; ++r) {
        const uint32_t i = r * 32 + lane;
        if (j >= 32) {
          const uint32_t o = r ^ (j >> 5);
          if (o > r) {
            const bool up = (i & k) == 0;
            const K a = v[r], b = v[o];
            v[r] = (a < b) == up ? a : b;
            v[o] = (a < b) == up ? b : a;
          }
        } else {
          const K o = __shfl_xor_sync(0xffffffffu, v[r], j);
          const bool up = (i & k) == 0, lower = (lane & j) == 0;
          const K mn = v[r] < o ? v[r] : o, mx = v[r] < o ? o : v[r];
          v[r] = lower == up ? mn : mx;
        }
      }
    }
  }
}

// Sorts a[0, c) (shared memory, c <= 32 R) in place by one warp.
template <class K, int R>
__device__ __forceinline__ void warp_sort_smem(K *a, uint32_t c) {
  const uint32_t lane = threadIdx.x & 31;
  K v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = r * 32 + lane < c ? a[r * 32 + lane] : KeyMax<K>::v;
  warp_bitonic_regs<K, R>(v);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r * 32 + lane < c) a[r * 32 + lane] = v[r];
}

// Sorts a[0, c) (shared memory) in place by one warp when it holds few distinct
// keys (integer-valued floats, counts: a bin then holds hundreds of copies of
// two or three): one pass over the keys finds the next larger one and counts
// its copies, lane i keeping the i-th; the runs are written at the end.
// Returns false, with the keys as they were, when there are more than 32
// distinct keys or the passes would visit more than kTinyVisits keys.
constexpr uint32_t kTinyVisits = 32768;
template <class K>
__device__ __forceinline__ bool warp_sort_runs(K *a, uint32_t c) {
  const uint32_t lane = threadIdx.x & 31;
  K run_key = 0, above = 0;  // lane i: the i-th distinct key, and how many keys it holds
  uint32_t run_cnt = 0, seen = 0, runs = 0;
  while (seen < c) {
    if (runs == 32 || (runs + 1) * c > kTinyVisits + c) return false;
    K mn = KeyMax<K>::v;
    uint32_t cnt = 0;
    for (uint32_t j = lane; j < c; j += 32) {
      const K v = a[j];
      if (runs == 0 || v > above) {
        cnt = v < mn ? 1u : cnt + (v == mn ? 1u : 0u);
        mn = v < mn ? v : mn;
      }
    }
    K g = mn;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const K t = __shfl_xor_sync(0xffffffffu, g, o);
      g = t < g ? t : g;
    }
    cnt = __reduce_add_sync(0xffffffffu, mn == g ? cnt : 0u);
    if (lane == runs) {
      run_key = g;
      run_cnt = cnt;
    }
    above = g;
    seen += cnt;
    ++runs;
    // more than 32 runs to come: two passes tell
    if (runs == 2 && seen * 16 < c) return false;
  }
  uint32_t at = 0;
  for (uint32_t i = 0; i < runs; ++i) {
    const K v = __shfl_sync(0xffffffffu, run_key, i);
    const uint32_t m = __shfl_sync(0xffffffffu, run_cnt, i);
    for (uint32_t j = lane; j < m; j += 32) a[at + j] = v;
    at += m;
  }
  return true;
}

// x: device vector of n elements, 1 <= n <= tiny_max<K>(); reqs: num_req
// requests (ascending 0-based rank below n, output index; num_req <=
// kTinyMaxReq); out: outputs.  reqs and out may lie in host memory.  One CTA of
// kTinyThreads threads, tiny_smem_bytes<K>(n) of shared memory.
template <class T, class OutT>
__global__ void __launch_bounds__(kTinyThreads, 1)
    k_tiny(const T *__restrict__ x, uint32_t n, const Req *__restrict__ reqs, uint32_t num_req,
           OutT *__restrict__ out) {
  using K = typename Traits<T>::K;
  constexpr uint32_t kPer = tiny_per<K>();
  // the keys of -0.0 and +0.0: kMid and kMid + 1
  constexpr K kMid = KeyMax<K>::v >> 1;
  extern __shared__ uint4 smem_raw[];
  uint32_t *bins = reinterpret_cast<uint32_t *>(smem_raw);  // counts, then prefix, then cursors
  K *buf = reinterpret_cast<K *>(bins + kTinyBins);         // requested bins' keys at their ranks
  __shared__ K s_span[4][32];
  __shared__ uint32_t s_w[33];
  __shared__ uint32_t s_need[kTinyBins / 32];  // requested bins
  __shared__ uint32_t s_off[kTinyMaxReq], s_cnt[kTinyMaxReq];  // their segments of buf
  static_assert(tiny_max<K>() / (tiny_bin<K>() + 1) < tiny_big<K>(), "every large bin");
  __shared__ uint32_t s_nbin, s_nbig, s_big[tiny_big<K>()];  // requested bins; the large ones
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  Req q;
  q.rank = 0;
  q.out = 0;
  if (tid < num_req) q = reqs[tid];
  K k[kPer];
#pragma unroll
  for (uint32_t u = 0; u < kPer; ++u) {
    const uint32_t i = u * kTinyThreads + tid;
    if (i < n) k[u] = Traits<T>::key(x[i]);
  }
  fill_words(bins, kTinyBins, 0u);
  if (tid < kTinyBins / 32) s_need[tid] = 0;
  if (tid == 0) {
    s_nbin = 0;
    s_nbig = 0;
  }
  // the occupied ranges [lo[h], hi[h]] below and above the two middle keys
  K lo[2] = {KeyMax<K>::v, KeyMax<K>::v}, hi[2] = {0, 0};
#pragma unroll
  for (uint32_t u = 0; u < kPer; ++u) {
    if (u * kTinyThreads >= n) break;
    if (u * kTinyThreads + tid < n) {
      const K v = k[u];
      const bool dn = v < kMid, up = v > kMid + 1;
      lo[0] = dn && v < lo[0] ? v : lo[0];
      hi[0] = dn && v > hi[0] ? v : hi[0];
      lo[1] = up && v < lo[1] ? v : lo[1];
      hi[1] = up && v > hi[1] ? v : hi[1];
    }
  }
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {  // lanes of a warp, then the warps
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const K a = __shfl_xor_sync(0xffffffffu, lo[h], o);
        const K z = __shfl_xor_sync(0xffffffffu, hi[h], o);
        lo[h] = a < lo[h] ? a : lo[h];
        hi[h] = z > hi[h] ? z : hi[h];
      }
    }
    if (pass == 0) {
      if (lane == 0) {
        s_span[0][warp] = lo[0];
        s_span[1][warp] = hi[0];
        s_span[2][warp] = lo[1];
        s_span[3][warp] = hi[1];
      }
      __syncthreads();
      lo[0] = s_span[0][lane];
      hi[0] = s_span[1][lane];
      lo[1] = s_span[2][lane];
      hi[1] = s_span[3][lane];
    }
  }
  // d(key) = the key's position with the ranges laid end to end, the two
  // middle keys between them (an empty range has no length); the largest
  // position fits K, the ranges being disjoint
  const K len0 = lo[0] <= hi[0] ? hi[0] - lo[0] + 1 : K(0);
  const K off1 = len0 + 2 - lo[1];  // modulo the key width
  const K dmax = lo[1] <= hi[1] ? hi[1] + off1 : len0 + 1;
  const int bl = bitlen<K>(dmax);
  const uint32_t sh = bl > kTinyBinBits ? (uint32_t)(bl - kTinyBinBits) : 0u;
  const uint32_t nb = (uint32_t)(dmax >> sh) + 1u;  // <= kTinyBins
  auto bin_of = [&](K v) -> uint32_t {
    const K d = v < kMid ? v - lo[0] : v > kMid + 1 ? v + off1 : v - kMid + len0;
    return (uint32_t)(d >> sh);
  };
#pragma unroll
  for (uint32_t u = 0; u < kPer; ++u) {
    if (u * kTinyThreads >= n) break;
    if (u * kTinyThreads + tid < n) atomicAdd(&bins[bin_of(k[u])], 1u);
  }
  __syncthreads();
  smem_excl_scan(bins, nb, s_w);  // ends with a barrier

  // requests: the last bin whose prefix is <= the rank (never an empty one)
  if (tid < num_req) {
    const uint32_t top = nb > 1 ? 1u << (31 - __clz(nb - 1)) : 0u;
    uint32_t b = 0;
    for (uint32_t step = top; step; step >>= 1) {
      const uint32_t m = b + step;
      if (m < nb && bins[m] <= q.rank) b = m;
    }
    const uint32_t bit = 1u << (b & 31);
    if (!(atomicOr(&s_need[b >> 5], bit) & bit)) {  // the bin's first request
      const uint32_t at = atomicAdd(&s_nbin, 1u);
      s_off[at] = bins[b];
      s_cnt[at] = (b + 1 < nb ? bins[b + 1] : n) - bins[b];
    }
  }
  __syncthreads();
#pragma unroll
  for (uint32_t u = 0; u < kPer; ++u) {
    if (u * kTinyThreads >= n) break;
    if (u * kTinyThreads + tid < n) {
      const uint32_t b = bin_of(k[u]);
      if (s_need[b >> 5] & (1u << (b & 31))) buf[atomicAdd(&bins[b], 1u)] = k[u];
    }
  }
  __syncthreads();
  const uint32_t nbin = sh ? s_nbin : 0u;  // bins one key wide need no sort
  for (uint32_t i = warp; i < nbin; i += kTinyThreads / 32) {
    K *a = buf + s_off[i];
    const uint32_t c = s_cnt[i];
    if (c <= 1) continue;
    if (c <= 32) {
      warp_sort_smem<K, 1>(a, c);
    } else if (c <= 64) {
      warp_sort_smem<K, 2>(a, c);
    } else if (!warp_sort_runs<K>(a, c)) {
      if (c <= 128)
        warp_sort_smem<K, 4>(a, c);
      else if (c <= 256)
        warp_sort_smem<K, 8>(a, c);
      else if (c <= 512 && tiny_bin<K>() >= 512)
        warp_sort_smem<K, 16>(a, c);
      else if (c <= tiny_bin<K>())
        warp_sort_smem<K, (int)(tiny_bin<K>() / 32)>(a, c);
      else if (lane == 0)
        s_big[atomicAdd(&s_nbig, 1u)] = i;
    }
  }
  __syncthreads();
  for (uint32_t i = 0; i < s_nbig; ++i) cta_sort_any<K>(buf + s_off[s_big[i]], s_cnt[s_big[i]]);
  if (tid < num_req) out[q.out] = Traits<OutT>::value(buf[q.rank]);
}

}  // namespace ggks
