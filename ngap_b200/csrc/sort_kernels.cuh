// Report compaction: sort of 64-bit report keys (offset << 32 | id, or the
// batched layout) followed by duplicate removal and conversion to the
// reference's packed form (id << 32 | offset). Replaces the host sort/unique of the reference
// (code/src/ngap/ngap.cu:1890-1932, order of compareResult ngap.cu:19-30).
//
// Small sets are sorted by one CTA (sort_unique_cta). Larger ones go through
// an LSD radix pipeline of 8-bit digits: per pass, digit counts of every tile
// of 2048 keys, a scan of each digit's counts over the tiles (one CTA per
// digit), and a stable scatter. Digits that cannot vary (bits above the
// largest offset, id and group) are skipped by the host. The key count is read
// from device memory (*d_n, clamped to cap), so the whole pipeline runs
// without a host round trip; grids stride over tiles. A pass reads the keys
// twice and writes them once; up to about 10 M keys they stay in L2. Measured
// on a B200, sort + unique of 1.5 M reports: 394 us with 4-bit digits (36
// kernels), 148 us with 8-bit digits (19).
#pragma once

#include <cstdint>

namespace ngap {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 2048 keys per tile
constexpr int kScanThreads = 1024;
constexpr int kDigits = 256;                          // values of a digit
constexpr int kDigitBits = 8;

__device__ __forceinline__ uint64_t dev_count(const unsigned long long* d_n, uint64_t cap) {
  uint64_t n = *d_n;
  return n < cap ? n : cap;
}

__device__ __forceinline__ uint32_t num_tiles(uint64_t n) {
  return (uint32_t)((n + kSortTile - 1) / kSortTile);
}

__device__ __forceinline__ uint32_t digit_of(uint64_t key, int shift) {
  return (uint32_t)(key >> shift) & (kDigits - 1);
}

// One count per key of a warp (d = kDigits: no key). High digits are often the
// same for a whole warp, which then adds once; otherwise shared-memory
// atomics, which beat __match_any_sync by far on mixed digits (1.5 M keys:
// radix_hist 15 us with it).
__device__ __forceinline__ void count_digit(uint32_t* cnt, uint32_t d, int lane) {
  const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
  if (__all_sync(0xffffffffu, d == d0)) {
    if (lane == 0 && d0 < kDigits) atomicAdd(&cnt[d0], 32u);
  } else if (d < kDigits) {
    atomicAdd(&cnt[d], 1u);
  }
}

// hist[d * ntiles + tile] = number of keys of the tile whose digit is d.
__global__ void __launch_bounds__(kSortThreads) radix_hist(const uint64_t* __restrict__ keys,
                                                           const unsigned long long* d_n,
                                                           uint64_t cap, int shift,
                                                           uint32_t* __restrict__ hist) {
  __shared__ uint32_t cnt[kDigits];
  static_assert(kSortThreads == kDigits, "one thread per digit");
  const uint64_t n = dev_count(d_n, cap);
  const uint32_t ntiles = num_tiles(n);
  const int lane = threadIdx.x & 31;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)tile * kSortTile + threadIdx.x;
    uint32_t d[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
      const uint64_t g = base + (uint64_t)k * kSortThreads;
      d[k] = g < n ? digit_of(keys[g], shift) : (uint32_t)kDigits;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; k++) count_digit(cnt, d[k], lane);
    __syncthreads();
    hist[(uint64_t)threadIdx.x * ntiles + tile] = cnt[threadIdx.x];
    __syncthreads();
  }
}

// CTA d: exclusive scan of digit d's counts over the tiles, in place; their sum
// to totals[d].
__global__ void __launch_bounds__(kSortThreads) radix_scan(uint32_t* __restrict__ hist,
                                                           const unsigned long long* d_n,
                                                           uint64_t cap,
                                                           uint32_t* __restrict__ totals) {
  __shared__ uint32_t wsum[kSortThreads / 32];
  const uint32_t ntiles = num_tiles(dev_count(d_n, cap));
  uint32_t* row = hist + (uint64_t)blockIdx.x * ntiles;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t run = 0;
  for (uint32_t i0 = 0; i0 < ntiles; i0 += kSortThreads) {
    const uint32_t i = i0 + (uint32_t)t;
    const uint32_t x = i < ntiles ? row[i] : 0u;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int w = 0; w < kSortThreads / 32; w++) {
      before += w < warp ? wsum[w] : 0u;
      all += wsum[w];
    }
    if (i < ntiles) row[i] = run + before + incl - x;
    run += all;
    __syncthreads();
  }
  if (t == 0) totals[blockIdx.x] = run;
}

// In-place exclusive scan of a[0 .. ntiles(*d_n)) with one block. Writes the
// total to *total.
__global__ void __launch_bounds__(kScanThreads) scan_exclusive_1block(uint32_t* a,
                                                                      const unsigned long long* d_n,
                                                                      uint64_t cap,
                                                                      unsigned long long* total) {
  __shared__ uint32_t part[kScanThreads];
  const uint32_t n = num_tiles(dev_count(d_n, cap));
  const uint32_t per = (n + kScanThreads - 1) / kScanThreads;
  const uint32_t b = min(threadIdx.x * per, n), e = min(b + per, n);
  uint32_t s = 0;
  for (uint32_t i = b; i < e; i++) s += a[i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < kScanThreads; o <<= 1) {  // Hillis-Steele inclusive scan
    uint32_t y = threadIdx.x >= (unsigned)o ? part[threadIdx.x - o] : 0u;
    __syncthreads();
    part[threadIdx.x] += y;
    __syncthreads();
  }
  uint32_t run = threadIdx.x > 0 ? part[threadIdx.x - 1] : 0u;
  for (uint32_t i = b; i < e; i++) {
    uint32_t x = a[i];
    a[i] = run;
    run += x;
  }
  if (n > 0 && threadIdx.x == kScanThreads - 1) *total = part[kScanThreads - 1];
}

// Stable ranks of one warp's 32 keys among the warp's earlier ones: cnt holds
// the warp's running count of each digit. Lanes without a key pass act = false.
template <class C>
__device__ __forceinline__ uint32_t warp_rank(C* cnt, uint32_t d, bool act, int lane) {
  unsigned peers = __ballot_sync(0xffffffffu, act);  // lanes with the same digit, bit by bit
#pragma unroll
  for (int b = 0; b < kDigitBits; b++) {
    const unsigned m = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    peers &= (d >> b) & 1u ? m : ~m;
  }
  const uint32_t r = act ? (uint32_t)cnt[d] + __popc(peers & ((1u << lane) - 1u)) : 0u;
  __syncwarp();
  if (act && __ffs(peers) - 1 == lane) cnt[d] = (C)(cnt[d] + __popc(peers));
  __syncwarp();
  return r;
}

// Stable scatter of one digit pass: hist = radix_scan's result, totals = keys
// per digit. Warp w of a CTA ranks the tile's keys [w, w + 1) * 256.
__global__ void __launch_bounds__(kSortThreads) radix_scatter(const uint64_t* __restrict__ in,
                                                              uint64_t* __restrict__ out,
                                                              const unsigned long long* d_n,
                                                              uint64_t cap, int shift,
                                                              const uint32_t* __restrict__ hist,
                                                              const uint32_t* __restrict__ totals) {
  constexpr int kWarps = kSortThreads / 32;
  __shared__ uint32_t cnt[kWarps][kDigits];
  __shared__ uint32_t wsum[kWarps];
  const uint64_t n = dev_count(d_n, cap);
  const uint32_t ntiles = num_tiles(n);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (blockIdx.x >= ntiles) return;
  uint32_t first;  // keys of smaller digits than t
  {
    const uint32_t x = totals[t];
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    first = incl - x;
    for (int w = 0; w < warp; w++) first += wsum[w];
  }
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    for (int w = 0; w < kWarps; w++) cnt[w][t] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)tile * kSortTile + (uint64_t)warp * (32 * kSortItems) + lane;
    uint64_t key[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) key[k] = base + 32 * k < n ? in[base + 32 * k] : 0ull;
#pragma unroll
    for (int k = 0; k < kSortItems; k++)
      rank[k] = warp_rank(cnt[warp], digit_of(key[k], shift), base + 32 * k < n, lane);
    __syncthreads();
    uint32_t run = first + hist[(uint64_t)t * ntiles + tile];
    for (int w = 0; w < kWarps; w++) {
      const uint32_t x = cnt[w][t];
      cnt[w][t] = run;
      run += x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++)
      if (base + 32 * k < n) out[cnt[warp][digit_of(key[k], shift)] + rank[k]] = key[k];
    __syncthreads();
  }
}

// The lane's keys of a tile and, per round of 32 consecutive keys of its warp,
// which of them differ from their predecessor (the first of a run).
struct TileRuns {
  uint64_t key[kSortItems];
  unsigned first[kSortItems];  // ballots
};

__device__ __forceinline__ uint32_t tile_runs(const uint64_t* __restrict__ keys, uint64_t n,
                                              uint32_t tile, int lane, int warp, TileRuns& r) {
  const uint64_t base = (uint64_t)tile * kSortTile + (uint64_t)warp * (32 * kSortItems) + lane;
  uint64_t before[kSortItems];
#pragma unroll
  for (int k = 0; k < kSortItems; k++) {
    const uint64_t g = base + 32 * k;
    r.key[k] = g < n ? keys[g] : 0ull;
    before[k] = g < n && g > 0 ? keys[g - 1] : 0ull;
  }
  uint32_t c = 0;
#pragma unroll
  for (int k = 0; k < kSortItems; k++) {
    const uint64_t g = base + 32 * k;
    r.first[k] = __ballot_sync(0xffffffffu, g < n && (g == 0 || r.key[k] != before[k]));
    c += __popc(r.first[k]);
  }
  return c;
}

// Per tile: number of keys that differ from their predecessor.
__global__ void __launch_bounds__(kSortThreads) unique_count(const uint64_t* __restrict__ keys,
                                                             const unsigned long long* d_n,
                                                             uint64_t cap,
                                                             uint32_t* __restrict__ cnt) {
  __shared__ uint32_t wsum[kSortThreads / 32];
  const uint64_t n = dev_count(d_n, cap);
  const uint32_t ntiles = num_tiles(n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    TileRuns r;
    const uint32_t c = tile_runs(keys, n, tile, lane, warp, r);
    if (lane == 0) wsum[warp] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t all = 0;
      for (int w = 0; w < kSortThreads / 32; w++) all += wsum[w];
      cnt[tile] = all;
    }
    __syncthreads();
  }
}

// Writes the first key of every run of equal keys, in order, in the reference
// encoding (id << 32 | offset). MODE 0: keys are offset << 32 | id. MODE 1
// (batched): keys are stream << sshift | offset << oshift | id; the stream
// index of each unique report goes to out_stream.
template <int MODE>
__global__ void __launch_bounds__(kSortThreads) unique_write(
    const uint64_t* __restrict__ keys, const unsigned long long* d_n, uint64_t cap,
    const uint32_t* __restrict__ offs, int oshift, int sshift, uint64_t* __restrict__ out,
    uint32_t* __restrict__ out_stream) {
  __shared__ uint32_t wsum[kSortThreads / 32];
  const uint64_t n = dev_count(d_n, cap);
  const uint32_t ntiles = num_tiles(n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    TileRuns r;
    const uint32_t c = tile_runs(keys, n, tile, lane, warp, r);
    if (lane == 0) wsum[warp] = c;
    __syncthreads();
    uint32_t pos = offs[tile];
    for (int w = 0; w < warp; w++) pos += wsum[w];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
      if ((r.first[k] >> lane) & 1u) {
        const uint32_t at = pos + __popc(r.first[k] & ((1u << lane) - 1u));
        const uint64_t key = r.key[k];
        if (MODE == 0) {
          out[at] = (key << 32) | (key >> 32);
        } else {
          const uint64_t id = key & ((1ull << oshift) - 1);
          const uint64_t off = (key >> oshift) & ((1ull << (sshift - oshift)) - 1);
          out[at] = (id << 32) | off;
          out_stream[at] = sshift < 64 ? (uint32_t)(key >> sshift) : 0u;
        }
      }
      pos += __popc(r.first[k]);
    }
    __syncthreads();
  }
}

// What the last kernel of a match leaves for the host in pinned memory: the
// engine's counters, and the first kHostReports unique reports (with their stream
// indices in batched matching), so that small results need no device copy. A
// device-to-host copy of 64 bytes costs a call 13 us on this machine, a 64-byte
// memset 3 us; these stores and the reset cost neither.
constexpr int kHostReports = 1024;
constexpr int kNumCounters = 32;
struct HostOut {
  unsigned long long* counters = nullptr;  // pinned, kNumCounters
  uint64_t* reports = nullptr;             // pinned, kHostReports
  uint32_t* streams = nullptr;             // pinned, kHostReports (batched)
  unsigned long long* d_counters = nullptr;  // copied out, then zeroed for the next match
};

// Copies the counters out and zeroes them: called by one warp, after a barrier
// that orders the CTA's own counter writes before it. (The end of the kernel
// makes the stores visible to the host; a system fence here only costs time.)
__device__ __forceinline__ void publish_counters(const HostOut& ho, int lane) {
  if (lane < kNumCounters) {
    ho.counters[lane] = __ldcg(ho.d_counters + lane);
    ho.d_counters[lane] = 0ull;
  }
}

__global__ void __launch_bounds__(32) publish_kernel(HostOut ho) { publish_counters(ho, threadIdx.x); }

// After the radix pipeline: the first reports and the counters, for the host.
__global__ void __launch_bounds__(kHostReports) publish_results(HostOut ho,
                                                                const unsigned long long* d_unique_n,
                                                                const uint64_t* __restrict__ out,
                                                                const uint32_t* __restrict__ streams) {
  const uint64_t n = *d_unique_n;
  if (threadIdx.x < n) {
    ho.reports[threadIdx.x] = out[threadIdx.x];
    if (streams) ho.streams[threadIdx.x] = streams[threadIdx.x];
  }
  __syncthreads();
  if (threadIdx.x < 32) publish_counters(ho, threadIdx.x);
}

// One CTA sorts and deduplicates: up to kBitonic keys with a bitonic network, up
// to kSmallSort with radix passes between two shared-memory buffers (only
// over the digits that vary), and up to `most`, where that is larger, with the same
// passes between d_in and tmp in global memory. It then writes the unique
// reports like unique_write. It stores in *radix_n the key count the radix
// pipeline still has to sort: 0 when the keys were handled here (the
// pipeline's kernels then find no tiles), n otherwise; launched from a graph, it
// also sets the condition of the conditional node that holds the pipeline.
// ho.counters != nullptr: it publishes when it handled the keys; otherwise it
// copies the counters out and leaves them to the pipeline.
constexpr int kSmallSort = 8192;
constexpr int kBitonic = 1024;
constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallSortSmem = 2 * kSmallSort * 8 + kSmallWarps * kDigits * 2;

// Exclusive scan of 256 values held by the first 256 threads (all threads of the
// CTA call it); wsum: kDigits words of scratch.
__device__ __forceinline__ uint32_t scan_digits(uint32_t x, uint32_t* wsum) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t f = incl - x;
  for (int w = 0; w < warp && w < kDigits / 32; w++) f += wsum[w];
  __syncthreads();
  return f;
}

// One stable pass over n keys, src -> dst (generic pointers), in tiles of
// kSmallSort keys. The counts of a single tile give the digits' first places;
// several tiles need a count of all keys first.
__device__ __forceinline__ void cta_radix_pass(const uint64_t* src, uint64_t* dst, uint64_t n,
                                               int shift, uint16_t (*cnt)[kDigits],
                                               uint32_t* first, uint32_t* wsum) {
  constexpr int kItems = kSmallSort / kSmallThreads;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool one = n <= (uint64_t)kSmallSort;
  if (!one) {
    if (t < kDigits) first[t] = 0;
    __syncthreads();
    for (uint64_t g0 = 0; g0 < n; g0 += kSmallThreads) {
      const uint64_t g = g0 + t;
      count_digit(first, g < n ? digit_of(src[g], shift) : (uint32_t)kDigits, lane);
    }
    __syncthreads();
    const uint32_t f = scan_digits(t < kDigits ? first[t] : 0u, wsum);
    if (t < kDigits) first[t] = f;
  }
  for (uint64_t g0 = 0; g0 < n; g0 += kSmallSort) {
    for (int i = t; i < kSmallWarps * kDigits / 4; i += kSmallThreads)
      reinterpret_cast<uint2*>(cnt)[i] = make_uint2(0u, 0u);
    __syncthreads();
    // each warp takes rows of 32 keys, as many as the tile's keys need
    const int rows = (int)((min(n - g0, (uint64_t)kSmallSort) + kSmallThreads - 1) / kSmallThreads);
    const uint64_t base = g0 + (uint64_t)warp * (32 * rows) + lane;
    uint64_t key[kItems];
    uint32_t rank[kItems];
#pragma unroll
    for (int k = 0; k < kItems; k++)
      key[k] = k < rows && base + 32 * k < n ? src[base + 32 * k] : 0ull;
#pragma unroll
    for (int k = 0; k < kItems; k++)
      if (k < rows)
        rank[k] = warp_rank(cnt[warp], digit_of(key[k], shift), base + 32 * k < n, lane);
    __syncthreads();
    uint32_t run = 0;
    if (t < kDigits) {  // each warp's keys of the digit come after those of the warps before it
      for (int w = 0; w < kSmallWarps; w++) {
        const uint32_t c = cnt[w][t];
        cnt[w][t] = (uint16_t)run;
        run += c;
      }
    }
    if (one) {
      const uint32_t f = scan_digits(run, wsum);
      if (t < kDigits) first[t] = f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; k++)
      if (k < rows && base + 32 * k < n) {
        const uint32_t d = digit_of(key[k], shift);
        dst[first[d] + cnt[warp][d] + rank[k]] = key[k];
      }
    __syncthreads();
    if (!one && t < kDigits) first[t] += run;
    __syncthreads();
  }
}

template <int MODE>
__global__ void __launch_bounds__(kSmallThreads) sort_unique_cta(
    uint64_t* keys, uint64_t* tmp, const unsigned long long* d_n, uint64_t cap,
    unsigned long long* radix_n, unsigned long long* d_unique_n, int oshift, int sshift,
    uint64_t* __restrict__ out, uint32_t* __restrict__ out_stream, cudaGraphConditionalHandle cond,
    int set_cond, uint64_t most, HostOut ho) {
  extern __shared__ __align__(16) uint64_t sk[];
  __shared__ uint32_t wsum[kDigits], first[kDigits];
  __shared__ unsigned long long s_vary;
  const uint64_t n = dev_count(d_n, cap);
  const bool big = n > most;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) {
    *radix_n = big ? n : 0ull;
    if (set_cond) cudaGraphSetConditional(cond, big ? 1u : 0u);  // graph launches only
  }
  if (big) {
    __syncthreads();
    if (ho.counters && t < kNumCounters) ho.counters[t] = __ldcg(ho.d_counters + t);
    return;
  }
  const uint64_t* src = sk;
  if (n <= (uint64_t)kBitonic) {
    const uint32_t nn = (uint32_t)n;
    uint32_t m = 1;
    while (m < nn) m <<= 1;
    uint64_t v = t < nn ? keys[t] : ~0ull;  // padding sorts last
    for (uint32_t k = 2; k <= m; k <<= 1) {
      for (uint32_t j = k >> 1; j > 0; j >>= 1) {  // partners of a warp exchange by shuffle
        uint64_t o;
        if (j < 32) {
          o = __shfl_xor_sync(0xffffffffu, v, j);
        } else {
          sk[t] = v;
          __syncthreads();
          o = sk[t ^ j];
          __syncthreads();
        }
        v = ((t & j) == 0) == ((t & k) == 0) ? min(v, o) : max(v, o);
      }
    }
    sk[t] = v;
    __syncthreads();
  } else {
    const bool shared = n <= (uint64_t)kSmallSort;
    uint64_t* a = shared ? sk : keys;
    uint64_t* b = shared ? sk + kSmallSort : tmp;
    uint16_t(*cnt)[kDigits] = reinterpret_cast<uint16_t(*)[kDigits]>(sk + 2 * kSmallSort);
    if (t == 0) s_vary = 0ull;
    __syncthreads();
    const uint64_t k0 = keys[0];
    unsigned long long vary = 0ull;
    for (uint64_t i = t; i < n; i += kSmallThreads) {
      const uint64_t k = keys[i];
      vary |= k ^ k0;
      if (shared) a[i] = k;
    }
    atomicOr(&s_vary, vary);
    __syncthreads();
    for (unsigned long long m = s_vary; m;) {  // the digits that vary
      const int shift = __ffsll((long long)m) - 1;
      cta_radix_pass(a, b, n, shift, cnt, first, wsum);
      m &= ~((unsigned long long)(kDigits - 1) << shift);
      uint64_t* x = a;
      a = b;
      b = x;
    }
    src = a;
  }
  // first key of every run, compacted in order: thread t owns [b, e)
  const uint64_t per = (n + kSmallThreads - 1) / kSmallThreads;
  const uint64_t b = min((uint64_t)t * per, n), e = min(b + per, n);
  uint32_t c = 0;
  for (uint64_t i = b; i < e; i++) c += (i == 0 || src[i] != src[i - 1]) ? 1u : 0u;
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t pos = incl - c;
  for (int i = 0; i < warp; i++) pos += wsum[i];
  for (uint64_t i = b; i < e; i++) {
    if (!(i == 0 || src[i] != src[i - 1])) continue;
    const uint64_t key = src[i];
    uint64_t rep;
    uint32_t stream = 0u;
    if (MODE == 0) {
      rep = (key << 32) | (key >> 32);
    } else {
      const uint64_t id = key & ((1ull << oshift) - 1);
      const uint64_t off = (key >> oshift) & ((1ull << (sshift - oshift)) - 1);
      rep = (id << 32) | off;
      stream = sshift < 64 ? (uint32_t)(key >> sshift) : 0u;
      out_stream[pos] = stream;
    }
    out[pos] = rep;
    if (ho.counters && pos < (uint32_t)kHostReports) {
      ho.reports[pos] = rep;
      if (MODE == 1) ho.streams[pos] = stream;
    }
    pos++;
  }
  if (t == kSmallThreads - 1) *d_unique_n = pos;
  if (ho.counters) {
    __syncthreads();
    if (t < 32) publish_counters(ho, t);
  }
}

}  // namespace ngap
