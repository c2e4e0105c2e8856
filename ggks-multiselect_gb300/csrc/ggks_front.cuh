// ggks_front.cuh -- the first kernels of a single-vector call: sampling, and what
// is built from the sample.
//
//   k_sample  kFrontSamples keys at hashed positions, gathered by the whole GPU
//   k_bin     the sample counted in 4096 fine slices of its span
//   k_table   the splitter table (LUT) of the pipeline, by one CTA
//   k_slice   the samples of the fine slices that hold given sample ranks (a
//             top-k's threshold, a window's ends)
//
// Workspace: [fine counts kLutIdx words][window path's bins and counters][SliceOut].
//
// Bound: latency.  A kernel boundary under programmatic dependent launch costs
// about 0.9 us here, less than any other way for CTAs to wait for one another:
// one kernel that binned, then found its last CTA by a ticket and let it build
// took 10.4 us after k_sample's 2.8 (5.4 us of them to the last CTA's start);
// one cluster of 16 CTAs exchanging spans and counts through distributed shared
// memory took 11.5 us, and its gather, 65536 random sectors through one GPC's
// address translation, 2.3 us at 10 M elements but 9 us at 2^28.
// k_sample, k_bin and k_table take 2.3, 1.7 and 3.2 us, the last two 9.2 with the
// boundaries (10.4 + 0.9 before); top-1024 of 2^26: k_filter starts 8.1 us after
// k_sample (15.2 before).
#pragma once

#include <cstddef>

#include "ggks_device.cuh"

namespace ggks {

constexpr uint32_t kFrontSamples = 65536;
// far-apart sample pairs compared, and how many times 1 / buckets of them must
// hold one key before a table tracks single-key buckets (a rule of one hit in
// 4096 pairs for 32768 buckets also met one in 17 vectors of 65536 values, whose
// histogram pass then took 1.6 times as long for nothing)
constexpr uint32_t kFarPairs = 32768;
constexpr uint32_t kFarTimes = 4;

// the sample's launch shape: 1024 samples per CTA
__host__ __device__ constexpr uint32_t front_ctas(uint32_t S) { return (S + 1023) / 1024; }

// Requests to bring to dst: from src in host or device memory, or (null) those of
// a top-k of n elements (output i receives the (i + 1)-th largest, i.e.
// ascending rank n - 1 - i; multiselectTimingFunctions.cu:207-209 builds
// k = 1..K for this).  num 0: none.
struct ReqCopy {
  const Req *src;
  Req *dst;
  uint32_t num;
};

// Grid: front_ctas(S), and a CTA per 1024 requests to bring.
// Each thread gathers one sample (pairs of neighbouring elements at hashed
// positions, every element when S = n); each CTA leaves its samples' smallest
// and largest key in spans (two keys per CTA).  zero_words words (the fine
// counts, and what follows them) are cleared and the control block set to init, which travels in the launch's parameters: no
// copy or clearing precedes the call's first kernel.
template <class T>
__global__ void __launch_bounds__(1024)
    k_sample(const T *x, uint64_t n, uint32_t S, uint32_t seed,
             typename Traits<T>::K *__restrict__ samples, typename Traits<T>::K *__restrict__ spans,
             uint32_t *__restrict__ zero, uint32_t zero_words, Ctrl *ctrl,
             const __grid_constant__ Ctrl init, const __grid_constant__ ReqCopy req) {
  pdl_start();
  using K = typename Traits<T>::K;
  __shared__ K s_span[2][32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t ctas = front_ctas(S);
  if (blockIdx.x >= ctas) {
    const uint32_t q = (blockIdx.x - ctas) * 1024 + tid;
    Req r;
    r.rank = (uint32_t)(n - 1 - q);
    r.out = q;
    if (q < req.num) req.dst[q] = req.src ? req.src[q] : r;
    return;
  }
  const uint32_t i = blockIdx.x * 1024 + tid;
  K lo = KeyMax<K>::v, hi = 0;
  if (i < S) {
    // pairs of neighbouring elements: samples 2q and 2q + 1 are neighbours, so
    // the collision estimate sees runs of equal buckets (sorted input) as the
    // passes' warps do
    const uint64_t pos =
        (uint64_t)S >= n
            ? i
            : (((uint64_t)hash32((i >> 1) * 0x9E3779B9u + seed) * (n - 1)) >> 32) + (i & 1u);
    const K k = Traits<T>::key(x[pos]);
    samples[i] = k;
    lo = k;
    hi = k;
  }
  for (uint32_t j = i; j < zero_words; j += ctas * 1024) zero[j] = 0;
  if (blockIdx.x == 0 && tid < sizeof(Ctrl) / 4)
    reinterpret_cast<uint32_t *>(ctrl)[tid] = reinterpret_cast<const uint32_t *>(&init)[tid];
  auto warp_span = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const K a = __shfl_xor_sync(0xffffffffu, lo, o), z = __shfl_xor_sync(0xffffffffu, hi, o);
      lo = a < lo ? a : lo;
      hi = z > hi ? z : hi;
    }
  };
  warp_span();
  if (lane == 0) {
    s_span[0][warp] = lo;
    s_span[1][warp] = hi;
  }
  __syncthreads();
  if (warp == 0) {
    lo = s_span[0][lane];
    hi = s_span[1][lane];
    warp_span();
    if (lane == 0) {
      spans[2 * blockIdx.x] = lo;
      spans[2 * blockIdx.x + 1] = hi;
    }
  }
}

// The sample's smallest and largest key, and the width of its fine slices;
// every warp finds them for itself (loads through L1: thousands of warps asking
// L2 for the same sectors at once queue on them).
template <class K>
struct SampleSpan {
  K kmin, kmax;
  uint32_t shift;  // fine slice of a key: (key - kmin) >> shift
};
template <class K>
__device__ __forceinline__ SampleSpan<K> sample_span(const K *__restrict__ spans, uint32_t parts) {
  K lo = KeyMax<K>::v, hi = 0;
  for (uint32_t i = threadIdx.x & 31; i < parts; i += 32) {
    const K a = spans[2 * i], z = spans[2 * i + 1];
    lo = a < lo ? a : lo;
    hi = z > hi ? z : hi;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const K a = __shfl_xor_sync(0xffffffffu, lo, o), z = __shfl_xor_sync(0xffffffffu, hi, o);
    lo = a < lo ? a : lo;
    hi = z > hi ? z : hi;
  }
  const int bl = bitlen<K>(hi - lo);
  return {lo, hi, bl > kLutIdxBits ? (uint32_t)(bl - kLutIdxBits) : 0u};
}

// Grid of front_ctas(S): every CTA counts its 1024 samples and adds them to
// fine.  Also the far-apart pairs (q, q + S/2) holding one key: does the vector
// hold many copies of a key?
template <class K>
__global__ void __launch_bounds__(1024)
    k_bin(const K *samples, uint32_t S, const K *spans, uint32_t *fine,
          Ctrl *ctrl) {
  pdl_trigger();
  __shared__ uint32_t cnt[kLutIdx];
  const uint32_t tid = threadIdx.x, i = blockIdx.x * 1024 + tid;
  fill_words(cnt, kLutIdx, 0u);
  pdl_wait();
  const K k = i < S ? __ldcg(samples + i) : K(0);
  const uint32_t npairs = min(S / 2, kFarPairs);
  const K far = i < npairs ? __ldcg(samples + i + S / 2) : K(0);
  const SampleSpan<K> sp = sample_span<K>(spans, gridDim.x);
  __syncthreads();
  if (i < S) atomicAdd(&cnt[(uint32_t)((k - sp.kmin) >> sp.shift)], 1u);
  const uint32_t same = __popc(__ballot_sync(0xffffffffu, i < npairs && far == k));
  if ((tid & 31) == 0 && same) atomicAdd(&ctrl->same_key, same);
  __syncthreads();
#pragma unroll
  for (uint32_t q = 0; q < kLutIdx / 1024; ++q) {
    const uint32_t c = cnt[tid + 1024 * q];
    if (c) atomicAdd(&fine[tid + 1024 * q], c);
  }
}

// ---------------------------------------------------------------------------
// the splitter table
// ---------------------------------------------------------------------------
// One CTA builds the table of sv_slices<K>() slices (build_table).  A slice is a
// run of 2^fold fine slices and its density is its largest fine count times
// 2^fold, so that a slice whose keys crowd into part of its range (the slice
// holding the sampled maximum, whose keys stop there; a steep stretch of a
// distribution) gets buckets as narrow as its densest part needs.  Tables whose
// keys repeat often get at most dup_nb_cap buckets, which the histogram pass
// then tracks.  The call's rank windows (win) become the candidate buckets of
// speculative compaction (cand_cap: chunks in the candidate pool, 0 for none; G:
// histogram CTAs).
struct RankWindows {
  uint32_t num;
  uint64_t lo[2], hi[2];  // ascending 0-based ranks, inclusive
};
// The CTAs after the first (sort_ctas) sort the call's requests meanwhile.
constexpr uint32_t kTableThreads = 512;

// At most kPlanFew requests are sorted by rank meanwhile, kSortPer per CTA with
// 16 threads each: every CTA reads all ranks into shared memory (s, kPlanFew
// words), and the threads of a request count those before it (equal ranks by
// index), its position in the sorted list.  About 2.5 us for 1001 k's, less than
// the table (with four threads each 5.5, one CTA's bitonic network 4).
constexpr uint32_t kSortTeam = 16;
constexpr uint32_t kSortPer = kTableThreads / kSortTeam;
__host__ __device__ constexpr uint32_t sort_ctas(uint32_t num_req) {
  return (num_req + kSortPer - 1) / kSortPer;
}
static __device__ __forceinline__ void sort_requests(const ReqCopy &rc, uint32_t cta, uint32_t *s) {
  const uint32_t tid = threadIdx.x;
  const uint32_t me = cta * kSortPer + tid / kSortTeam;
  Req mine;
  mine.rank = mine.out = 0;
  if (me < rc.num) mine = rc.src[me];
  const uint32_t nvec = (rc.num + 3) / 4;
  for (uint32_t i = tid; i < 4 * nvec; i += kTableThreads)
    s[i] = i < rc.num ? rc.src[i].rank : 0xFFFFFFFFu;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t v = tid % kSortTeam; v < nvec; v += kSortTeam) {
    const uint4 o = reinterpret_cast<const uint4 *>(s)[v];
    if (4 * v <= me && me < 4 * v + 4) {  // the request's own vector
      before += (o.x < mine.rank || (o.x == mine.rank && 4 * v + 0 < me)) ? 1u : 0u;
      before += (o.y < mine.rank || (o.y == mine.rank && 4 * v + 1 < me)) ? 1u : 0u;
      before += (o.z < mine.rank || (o.z == mine.rank && 4 * v + 2 < me)) ? 1u : 0u;
      before += (o.w < mine.rank || (o.w == mine.rank && 4 * v + 3 < me)) ? 1u : 0u;
    } else {  // equal ranks count before the request's index, not after (no rank is ~0)
      const uint32_t lim = 4 * v < me ? mine.rank + 1 : mine.rank;
      before += (o.x < lim ? 1u : 0u) + (o.y < lim ? 1u : 0u) + (o.z < lim ? 1u : 0u) +
                (o.w < lim ? 1u : 0u);
    }
  }
#pragma unroll
  for (uint32_t o = 1; o < kSortTeam; o <<= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (me < rc.num && tid % kSortTeam == 0) rc.dst[before] = mine;
}

template <class K>
__global__ void __launch_bounds__(kTableThreads, 1)
    k_table(const K *samples, uint32_t S, const K *spans,
            const uint32_t *fine_g, uint64_t n, const __grid_constant__ RankWindows win,
            LutHeader<K> *hdr, uint32_t *__restrict__ lut, uint32_t nb_max, uint32_t nb_want,
            uint32_t cand_cap,
            uint32_t G, bool dense_ok, Ctrl *ctrl, const __grid_constant__ ReqCopy sort) {
  pdl_trigger();
  constexpr int kBits = sv_bits<K>();
  constexpr uint32_t nsl = sv_slices<K>();
  constexpr int SPT = (int)(nsl / kTableThreads);  // slices per thread
  static_assert(nsl % kTableThreads == 0 && kLutIdx == 8 * kTableThreads, "shares of the slices");
  __shared__ __align__(16) uint32_t fine[kLutIdx];
  __shared__ uint32_t tab[sv_entries<K>()];
  __shared__ TableShared ts;
  __shared__ uint32_t s_scan[32];
  __shared__ uint32_t s_same;
  __shared__ uint32_t s_sp[8];  // per window: first bucket, last bucket, first / end sample rank
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  if (blockIdx.x > 0) {
    static_assert(kLutIdx >= kPlanFew, "the ranks fit");
    pdl_wait();
    sort_requests(sort, blockIdx.x - 1, fine);
    return;
  }
  table_init(ts);
  if (tid == 0) s_same = 0;
  pdl_wait();
  // everything in one round of loads: the counts, the spans, pairs of
  // neighbouring elements (for the collision estimate)
  constexpr uint32_t kNear = 4;  // pairs per thread
  const uint32_t near_pairs = min(S / 2, kNear * kTableThreads);
  uint4 c4[2];
#pragma unroll
  for (int q = 0; q < 2; ++q)
    c4[q] = __ldcg(reinterpret_cast<const uint4 *>(fine_g) + tid + q * kTableThreads);
  K na[kNear], nb2[kNear];
#pragma unroll
  for (uint32_t q = 0; q < kNear; ++q) {
    const uint32_t i = tid + q * kTableThreads;
    na[q] = i < near_pairs ? __ldcg(samples + 2 * i) : K(0);
    nb2[q] = i < near_pairs ? __ldcg(samples + 2 * i + 1) : K(0);
  }
  const uint32_t far_same = __ldcg(&ctrl->same_key);
  const SampleSpan<K> sp = sample_span<K>(spans, front_ctas(S));
  const K kmin = sp.kmin, kmax = sp.kmax;
#pragma unroll
  for (int q = 0; q < 2; ++q) reinterpret_cast<uint4 *>(fine)[tid + q * kTableThreads] = c4[q];
  // a table that tracks single-key buckets needs at most dup_cap of them; with
  // nb_max >= the final bucket count, this test holds whenever the dup flag will
  const uint32_t dup_cap = dup_nb_cap<K>(nb_max), far_pairs = min(S / 2, kFarPairs);
  const bool far = S >= 256;
  if (dup_cap && far && (uint64_t)far_same * nb_max >= kFarTimes * far_pairs && nb_max > dup_cap)
    nb_max = dup_cap;
  else
    nb_max = min(nb_max, nb_want);
  const int bl = bitlen<K>(kmax - kmin);
  const uint32_t shift = bl > kBits ? (uint32_t)(bl - kBits) : 0u;
  const uint32_t fold = shift - sp.shift;  // a slice is 2^fold fine slices
  int bcap = (int)(shift < (uint32_t)kMaxSubBits ? shift : (uint32_t)kMaxSubBits);
  if (bcap > 24 - kBits) bcap = 24 - kBits;
  __syncthreads();
  auto density = [&](uint32_t j) -> uint32_t {
    if (fold == 3) {  // every 4-byte key span of 2^12 or more
      const uint4 a = reinterpret_cast<const uint4 *>(fine)[2 * j];
      const uint4 b = reinterpret_cast<const uint4 *>(fine)[2 * j + 1];
      return max(max(max(a.x, a.y), max(a.z, a.w)), max(max(b.x, b.y), max(b.z, b.w))) << 3;
    }
    uint32_t m = 0;
    for (uint32_t i = j << fold; i < (j + 1) << fold; ++i) m = max(m, fine[i]);
    return m << fold;
  };
  LutHeader<K> h;
  if constexpr (sizeof(K) == 4) {
    // a dense table: two keys or more to a bucket otherwise, and no slice of keys
    // (with six standard deviations and ten samples to spare) that could fill a
    // CTA's 16-bit count
    if (dense_ok && bl == 16) {
      const float c = (float)density(tid);
      const bool full = (c + 6.0f * sqrtf(c) + 10.0f) * ((float)n / ((float)S * (float)G)) > kDenseFill;
      if (!__syncthreads_or(full)) {
        if (tid == 0) {
          // the range's spare keys, half on each side, within the keys there are
          const K spare = (kDenseKeys - 1u) - (kmax - kmin), left = min(kmin, spare / 2);
          const K right = min(KeyMax<K>::v - kmax, spare - left);
          h.base = kmin - min(kmin, spare - right);
          h.lo = h.base;
          h.hi = h.base + (K)(kDenseKeys - 1u);
          h.shift = 0;
          h.low = 0;
          h.nb = kDenseKeys;
          h.heavy = h.dup = h.spec = h.cand_cap = 0;
          h.spec_lo[0] = h.spec_lo[1] = 0;
          h.spec_len[0] = h.spec_len[1] = 0;
          h.dense = 1;
          *hdr = h;
          ctrl->nb = h.nb;
        }
        return;
      }
    }
  }
  table_place<K>(h, kmin, kmax, shift, nsl);
  const uint32_t nb = build_table<K, SPT>(density, nsl, h.low, shift, bcap, nb_max, lut, tab, ts);

  // Candidate windows.  The number of samples below the element of rank r is
  // about Binomial(S, r / n); each window [lo, hi] of ranks is widened to the
  // sample ranks E - 6 sd - 4 .. E + 6 sd + 4 of its ends, and the fine slices
  // holding those two samples bound its buckets.  A window reaching past the
  // sample's first or last key takes bucket 0 or the top bucket as well.  The
  // prediction only decides what the histogram pass keeps: compaction checks
  // that every segment's bucket was kept before it reads the candidates.
  const uint32_t nwin = cand_cap ? min(win.num, 2u) : 0u;
  uint32_t wa[2] = {0, 0}, wb[2] = {0, 0};
  bool wlo_open[2] = {false, false}, whi_open[2] = {false, false};
  if (nwin) {
    // single precision (float64 is slow on this part; sample ranks need about
    // one unit of 2^16)
    const float dn = (float)n, dS = (float)S;
#pragma unroll
    for (uint32_t w = 0; w < 2; ++w) {
      if (w >= nwin) break;
      const float pl = (float)win.lo[w] / dn;
      const float ph = fminf((float)(win.hi[w] + 1) / dn, 1.0f);
      const float a = pl * dS - (6.0f * sqrtf(dS * pl * (1.0f - pl)) + 4.0f);
      const float b = ph * dS + (6.0f * sqrtf(dS * ph * (1.0f - ph)) + 4.0f);
      wlo_open[w] = a <= 0.0f;
      whi_open[w] = b >= dS - 1.0f;
      wa[w] = wlo_open[w] ? 0u : (a >= dS - 1.0f ? S - 1u : (uint32_t)a);
      wb[w] = whi_open[w] ? S - 1u : (uint32_t)b;
    }
    // defaults (replaced below; no fine slice left unmatched): every bucket, every sample
    if (tid < 8) s_sp[tid] = (tid & 3) == 1 ? 0xFFFFFFFEu : ((tid & 3) == 3 ? S : 0u);
  }
  __syncthreads();  // the table
  const KeyTable<K> kt(h);
  auto bucket = [&](K k) { return bucket_of<K>(k, kt, tab); };
  if (nwin) {
    // the fine slices split the sample ranks [0, S) in order: eight per thread
    uint32_t fc[8], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      fc[q] = fine[8 * tid + q];
      sum += fc[q];
    }
    uint32_t all;
    uint32_t fpre = block_excl_scan(sum, s_scan, &all);
    const K span = kmax - kmin;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      if (fc[q] == 0) continue;
      const uint32_t jf = 8 * tid + q;
#pragma unroll
      for (uint32_t w = 0; w < 2; ++w) {
        if (w >= nwin) break;
        if (fpre <= wa[w] && wa[w] < fpre + fc[q]) {
          s_sp[4 * w + 0] = bucket(kmin + ((K)jf << sp.shift));
          s_sp[4 * w + 2] = fpre;
        }
        if (fpre <= wb[w] && wb[w] < fpre + fc[q]) {
          K dend = ((K)(jf + 1u) << sp.shift) - K(1);
          dend = dend < span ? dend : span;
          s_sp[4 * w + 1] = bucket(kmin + dend);
          s_sp[4 * w + 3] = fpre + fc[q];
        }
      }
      fpre += fc[q];
    }
  }
  // Warp-aggregated cursor updates in compaction pay off when lanes of a warp
  // often hit the same bucket (its atomics return positions, which lanes of
  // one address receive one at a time): the chance that two elements share a
  // bucket is estimated from pairs of neighbouring elements, which the passes'
  // warps see together.
  uint32_t near_same = 0;
#pragma unroll
  for (uint32_t q = 0; q < kNear; ++q)
    if (tid + q * kTableThreads < near_pairs && bucket(na[q]) == bucket(nb2[q])) ++near_same;
  near_same = __reduce_add_sync(0xffffffffu, near_same);
  if (lane == 0 && near_same) atomicAdd(&s_same, near_same);
  __syncthreads();
  if (tid == 0) {
    h.nb = nb;
    // collision chance >= 1/32: with 32 lanes, about 15 same-bucket pairs per
    // warp access
    h.heavy = (S >= 256 && 32ull * s_same >= near_pairs) ? 1u : 0u;
    // two elements share a key with chance >= kFarTimes / nb: buckets holding a
    // single key (many copies of it) are likely
    h.dup = (far && (uint64_t)far_same * nb >= kFarTimes * far_pairs) ? 1u : 0u;
    h.spec = 0;
    h.cand_cap = 0;
    h.spec_lo[0] = h.spec_lo[1] = 0;
    h.spec_len[0] = h.spec_len[1] = 0;
    if (nwin) {
      // bucket intervals and the sample ranks they hold, ordered and merged
      uint32_t blo[2], bhi[2], clo[2], chi[2];
#pragma unroll
      for (uint32_t w = 0; w < 2; ++w) {
        if (w >= nwin) break;
        blo[w] = wlo_open[w] ? 0u : s_sp[4 * w + 0];
        bhi[w] = whi_open[w] ? nb - 1u : s_sp[4 * w + 1];
        clo[w] = wlo_open[w] ? 0u : s_sp[4 * w + 2];
        chi[w] = whi_open[w] ? S : s_sp[4 * w + 3];
      }
      uint32_t ni = nwin;
      if (ni == 2) {
        if (blo[1] < blo[0]) {
          uint32_t t0 = blo[0]; blo[0] = blo[1]; blo[1] = t0;
          t0 = bhi[0]; bhi[0] = bhi[1]; bhi[1] = t0;
          t0 = clo[0]; clo[0] = clo[1]; clo[1] = t0;
          t0 = chi[0]; chi[0] = chi[1]; chi[1] = t0;
        }
        if (blo[1] <= bhi[0] + 1u) {
          bhi[0] = bhi[1] > bhi[0] ? bhi[1] : bhi[0];
          chi[0] = chi[1] > chi[0] ? chi[1] : chi[0];
          ni = 1;
        }
      }
      uint32_t pred = 0;  // samples inside the intervals
#pragma unroll
      for (uint32_t i = 0; i < 2; ++i)
        if (i < ni) pred += chi[i] - clo[i];
      // the expected candidates with half as much again, plus one partly
      // filled chunk per histogram warp, must fit the pool
      const float want = 1.5f * (float)n * (float)pred / (float)S +
                         (float)G * kCandWarps * kCandChunk;
      if (want <= (float)cand_cap * kCandChunk) {
        h.spec = ni;
        h.cand_cap = cand_cap;
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i)
          if (i < ni) {
            h.spec_lo[i] = blo[i];
            h.spec_len[i] = bhi[i] - blo[i] + 1u;
          }
      }
    }
    *hdr = h;
    ctrl->nb = nb;
    ctrl->spec_on = h.spec != 0 ? 1u : 0u;
  }
}

// ---------------------------------------------------------------------------
// keys by their sample rank
// ---------------------------------------------------------------------------
// The fine slices holding W sample ranks, and their samples.  k_slice: grid of
// front_ctas(S); every CTA finds the slices for itself from the counts and
// appends its samples in them to the slices' lists.  rank_keys, in the prologue
// of the kernel that follows, then takes the key of the wanted rank.
struct SliceWant {
  uint32_t rank[2];  // 0-based among the S samples
};
// samples of one list (values of 8 bits put 2048 samples into a fine slice).  A
// slice with more has no list but the counts of its samples in kLutIdx parts:
// doubles spread their span over every exponent, so that a slice is half a binade
// and holds up to a quarter of uniform values.
constexpr uint32_t kSliceBuf = 4096;
template <class K>
struct SliceOut {
  uint32_t at[2];                // list lengths so far (zero on entry, as all down to sub)
  uint32_t pad[2];
  unsigned long long lo_inv[2];  // slices of more than kSliceBuf samples: the
  unsigned long long hi[2];      // complement of the smallest and the largest
  uint32_t sub[2][kLutIdx];      // and their samples per part
  uint32_t cnt[2];               // samples in the slice
  uint32_t rank[2];              // the wanted rank inside the slice
  uint32_t shift, pad2;          // slices are 2^shift keys wide
  K base[2];                     // the slice's first key
  K buf[2][kSliceBuf];
};
constexpr uint32_t kSliceZeroWords = 12 + 2 * kLutIdx;  // words that are zero on entry
static_assert(offsetof(SliceOut<uint64_t>, sub) % 16 == 0 &&
                  offsetof(SliceOut<uint64_t>, cnt) == kSliceZeroWords * 4,
              "the counts are read in 16-byte vectors");
// a slice of 2^shift keys has parts of 2^part_shift(shift) keys
__device__ __forceinline__ uint32_t part_shift(uint32_t shift) {
  return shift > (uint32_t)kLutIdxBits ? shift - kLutIdxBits : 0u;
}

template <class K, int W>
__global__ void __launch_bounds__(1024)
    k_slice(const K *samples, uint32_t S, const K *spans,
            const uint32_t *fine_g, const __grid_constant__ SliceWant want,
            SliceOut<K> *out) {
  pdl_start();
  __shared__ uint32_t s_scan[32];
  __shared__ uint32_t s_slice[W], s_rank[W], s_cnt[W];
  const uint32_t tid = threadIdx.x, i = blockIdx.x * 1024 + tid;
  const uint4 c4 = __ldcg(reinterpret_cast<const uint4 *>(fine_g) + tid);
  const K k = i < S ? __ldcg(samples + i) : K(0);
  const SampleSpan<K> sp = sample_span<K>(spans, gridDim.x);
  if (tid < W) s_slice[tid] = s_rank[tid] = s_cnt[tid] = 0;
  const uint32_t fc[4] = {c4.x, c4.y, c4.z, c4.w};
  uint32_t all;
  uint32_t pre = block_excl_scan(fc[0] + fc[1] + fc[2] + fc[3], s_scan, &all);
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
#pragma unroll
    for (int w = 0; w < W; ++w)
      if (fc[q] && pre <= want.rank[w] && want.rank[w] < pre + fc[q]) {
        s_slice[w] = 4 * tid + q;
        s_rank[w] = want.rank[w] - pre;
        s_cnt[w] = fc[q];
      }
    pre += fc[q];
  }
  __syncthreads();
  const uint32_t j = (uint32_t)((k - sp.kmin) >> sp.shift);
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const bool in = i < S && j == s_slice[w];
    if (s_cnt[w] <= kSliceBuf) {
      if (in) {
        const uint32_t at = atomicAdd(&out->at[w], 1u);
        if (at < kSliceBuf) out->buf[w][at] = k;
      }
    } else if (__any_sync(0xffffffffu, in)) {
      K lo = in ? k : KeyMax<K>::v, hi = in ? k : K(0);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const K a = __shfl_xor_sync(0xffffffffu, lo, o), z = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = a < lo ? a : lo;
        hi = z > hi ? z : hi;
      }
      if ((tid & 31) == 0) {
        atomicMax(&out->lo_inv[w], (unsigned long long)~(uint64_t)lo);
        atomicMax(&out->hi[w], (unsigned long long)hi);
      }
      const K o = k - sp.kmin - ((K)s_slice[w] << sp.shift);
      const uint32_t part = in ? (uint32_t)(o >> part_shift(sp.shift)) : 0xFFFFFFFFu;
      const uint32_t peers = __match_any_sync(0xffffffffu, part);
      if (in && (tid & 31) == (uint32_t)__ffs(peers) - 1)
        atomicAdd(&out->sub[w][part], (uint32_t)__popc(peers));
    }
    if (i == 0) {
      out->rank[w] = s_rank[w];
      out->cnt[w] = s_cnt[w];
      out->base[w] = sp.kmin + ((K)s_slice[w] << sp.shift);
      out->shift = sp.shift;
    }
  }
}

// The keys of the wanted ranks of lists 0 .. W - 1, by the whole CTA (1024 threads;
// skip: a list that is not wanted).  Up to 256 samples are ranked by counting the
// samples before each (four threads per sample), more by a radix select.  A list of
// up to 1024 samples comes in one round of loads (with its unused end), through L1.
// A slice without a list is narrowed to the part that holds the rank, whose samples
// are gathered from all S, one reading for both lists; a part of more than
// kSliceBuf samples is narrowed again by counting.  (Taking the slice's first or
// last sample instead made the window up to a quarter of the vector, too many
// candidates: the 30 % quantile of 2^26 normal doubles 360 us a call, against 247 in the
// pipeline, now 149.)  keys: W * kSliceBuf keys of shared memory, 16-byte
// aligned, the caller's again afterwards.  same: the samples that hold the key.  One
// call per sh.
template <class K>
struct RankShared {
  K found[2];
  uint32_t same[2];
  uint32_t cnt[256], sel[2][3], scan[2][32], at[2];
};
template <int W, class K>
__device__ __forceinline__ void rank_keys(const SliceOut<K> *out, const K *samples, uint32_t S,
                                          const bool (&skip)[W], K *keys, RankShared<K> &sh,
                                          K (&found)[W], uint32_t (&same)[W]) {
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  uint32_t cnt[W], r[W], shift[W];
  K base[W], first[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    cnt[w] = out->cnt[w];
    r[w] = out->rank[w];
    shift[w] = out->shift;
    first[w] = skip[w] ? K(0) : out->buf[w][tid];
    base[w] = out->base[w];
  }
  // every sample: fn(key, whether there is one)
  auto each = [&](auto &&fn) {
    constexpr uint32_t U = 8;
    for (uint32_t i0 = 0; i0 < S; i0 += U * 1024) {
      K k[U];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) {
        const uint32_t i = i0 + 1024 * u + tid;
        k[u] = i < S ? __ldcg(samples + i) : K(0);
      }
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) fn(k[u], i0 + 1024 * u + tid < S);
    }
  };
  bool rank_it[W], gather = false;  // lists to rank; lists to gather first
  if (tid == 0) {  // (which alone writes same before the barrier ahead of the ranking)
#pragma unroll
    for (int w = 0; w < W; ++w) sh.same[w] = sh.at[w] = 0;
  }
#pragma unroll
  for (int w = 0; w < W; ++w) {
    rank_it[w] = !skip[w];
    if (skip[w]) continue;
    K *kw = keys + (size_t)w * kSliceBuf;
    if (cnt[w] <= kSliceBuf) {
      kw[tid] = first[w];
      for (uint32_t i = 1024 + tid; i < cnt[w]; i += 1024) kw[i] = out->buf[w][i];
      shift[w] = 0xFFFFFFFFu;  // nothing to gather
      continue;
    }
    if ((K)~out->lo_inv[w] == (K)out->hi[w]) {  // copies of one key
      if (tid == 0) {
        sh.found[w] = (K)out->hi[w];
        sh.same[w] = cnt[w];
      }
      rank_it[w] = false;
      continue;
    }
    uint32_t *hist = reinterpret_cast<uint32_t *>(kw);
    uint4 c4 = __ldcg(reinterpret_cast<const uint4 *>(out->sub[w]) + tid);
    for (;;) {
      const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w}, sub = part_shift(shift[w]);
      uint32_t all;
      uint32_t pre = block_excl_scan(c4.x + c4.y + c4.z + c4.w, sh.scan[w], &all);
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
        if (c[q] && pre <= r[w] && r[w] < pre + c[q]) {
          sh.sel[w][0] = 4 * tid + q;
          sh.sel[w][1] = r[w] - pre;
          sh.sel[w][2] = c[q];
        }
        pre += c[q];
      }
      __syncthreads();
      base[w] += (K)sh.sel[w][0] << sub;
      r[w] = sh.sel[w][1];
      cnt[w] = sh.sel[w][2];
      shift[w] = sub;
      if (cnt[w] <= kSliceBuf || sub == 0) break;
      fill_words(hist, kLutIdx, 0u);
      __syncthreads();  // (also: sel is read)
      const uint32_t next = part_shift(sub);
      each([&](K k, bool valid) {
        const K o = k - base[w];
        if (valid && k >= base[w] && (o >> sub) == 0) atomicAdd(&hist[(uint32_t)(o >> next)], 1u);
      });
      __syncthreads();
      c4 = reinterpret_cast<const uint4 *>(hist)[tid];
    }
    if (cnt[w] > kSliceBuf) {  // a part of one key
      if (tid == 0) {
        sh.found[w] = base[w];
        sh.same[w] = cnt[w];
      }
      rank_it[w] = false;
    } else {
      gather = true;
    }
  }
  if (gather) {
    __syncthreads();
    each([&](K k, bool valid) {
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const bool in = rank_it[w] && shift[w] != 0xFFFFFFFFu && valid && k >= base[w] &&
                        ((k - base[w]) >> shift[w]) == 0;
        const uint32_t m = __ballot_sync(0xffffffffu, in);
        if (!m) continue;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&sh.at[w], (uint32_t)__popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (in && at < kSliceBuf) keys[(size_t)w * kSliceBuf + at] = k;
      }
    });
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < W; ++w) {
    if (!rank_it[w]) continue;
    const K *kw = keys + (size_t)w * kSliceBuf;
    if (cnt[w] <= 256) {
      const uint32_t me = tid >> 2;
      const K mine = kw[me];
      uint32_t less = 0, eq = 0;
      if (me < cnt[w])
        for (uint32_t i = tid & 3; i < cnt[w]; i += 4) {
          const K o = kw[i];
          less += o < mine || (o == mine && i < me) ? 1u : 0u;
          eq += o == mine ? 1u : 0u;
        }
      less += __shfl_xor_sync(0xffffffffu, less, 1);
      less += __shfl_xor_sync(0xffffffffu, less, 2);
      eq += __shfl_xor_sync(0xffffffffu, eq, 1);
      eq += __shfl_xor_sync(0xffffffffu, eq, 2);
      if (me < cnt[w] && less == r[w] && (tid & 3) == 0) {
        sh.found[w] = mine;
        sh.same[w] = eq;
      }
    } else {
      const K k = cta_select_rank<K>(kw, cnt[w], r[w], sh.cnt, sh.sel[w]);
      uint32_t eq = 0;
      for (uint32_t i = tid; i < cnt[w]; i += 1024) eq += kw[i] == k ? 1u : 0u;
      eq = __reduce_add_sync(0xffffffffu, eq);
      if (lane == 0 && eq) atomicAdd(&sh.same[w], eq);
      if (tid == 0) sh.found[w] = k;
    }
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < W; ++w) {
    found[w] = sh.found[w];
    same[w] = sh.same[w];
  }
}

// Whether copies of a key that `same` of S samples hold are counted rather than kept
// as candidates: more than one key in 128.  (A window that kept the copies of its
// two end keys held up to the whole of a few-valued vector: of ten values in 2^26
// floats, the median took 264 us a call by a miss, now 87; of two values 267, now 87;
// 179 and 133 in the pipeline.)
__host__ __device__ constexpr bool popular(uint32_t same, uint32_t S) { return same * 128u > S; }

}  // namespace ggks
