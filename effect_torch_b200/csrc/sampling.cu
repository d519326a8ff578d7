// Next-token sampling on the device: temperature softmax, top-k and top-p with the splitmix64 draw of
// crates/runtime/src/sampling.rs:35-42, 80-206 (the greedy case is argmax_kernel's).
//
// The reference orders candidates by (value descending, token ascending), keeps the first top_k, turns them into
// weights exp((value - max) / temperature), keeps the smallest prefix whose weight reaches top_p x total, and walks that
// prefix subtracting weights from draw = unit x total until it goes negative. Without top-k and top-p it walks the row in
// token order instead.
//
// One row is served by a cluster of 1 to 8 CTAs; every CTA keeps its slice of the logits in shared memory, so HBM (or L2,
// behind the head projection) is read once. Every candidate has a 52-bit sort key (order-preserving bits of the f32
// logit, then the inverted token). "The first n candidates", "the smallest prefix reaching a weight" and "the candidate
// where the walk goes negative" are one primitive: a histogram over 1024 bins of (max - value) / temperature, whose bins
// are in candidate order, finds the bin in which a running sum crosses its target; that bin's few hundred candidates are
// gathered into the first CTA, sorted by key and summed in order. A bin that holds more than the list (rows with few
// distinct values, or everything far below the maximum) is narrowed by 10 bits of the key at a time first. When top_k
// leaves few enough candidates the list holds all of them and decides everything, and only they are exponentiated; the bins
// they are in follow from the threads' largest candidates alone, and only threads whose largest is in them look again.
// The token-order walk is a prefix sum over the warps' slices and a second look at the one that holds the draw.
//
// What bounds it: at 32 rows x 128256 the logits are 16 MB (2.5 us of HBM); the rest is latency, half a dozen passes over
// shared memory with a cluster barrier (about a microsecond) between them. A single CTA per row that re-read the row for
// each of 7 radix digits per select, with f64 atomics on 256 bins, took 2192 us with top-k 40 and top-p 0.95; a histogram of all
// candidates, four-byte loads and a sorting network for any list 24.6; this takes 18.4 (one row 18.8 -> 14.3; 8 rows with top-p
// alone 45.1 -> 37.7). 64 registers: two CTAs per SM (at 128 and one CTA 32.6 us).
//
// Sums are f64 like the reference's but associated differently (histogram bins, scans), so a comparison of a running sum
// against the draw or the top-p threshold can come out differently only when the two are within about vocab x 2^-52 of
// each other, relative to the total weight.
#include <cooperative_groups.h>

#include <algorithm>

#include "chain.cuh"
#include "kernels.h"

namespace etc {

namespace {

namespace cg = cooperative_groups;

constexpr int kSampleThreads = 512;
constexpr int kSampleWarps = kSampleThreads / 32;
constexpr int kBins = 1024;           // also the digits of a narrowing step (10 bits of the key)
constexpr int kList = 1024;           // candidates that can be sorted
constexpr int kFewEnough = 200;       // top_k that the threads' largest candidates are counted for
constexpr int kRankSorted = 256;      // up to this many by counting (two barriers) instead of a network of them (36 for 256)
constexpr int kMaxSlice = 16384;      // logits a CTA keeps in shared memory (64 KB: two CTAs per SM)
constexpr int kMaxSampleCluster = 8;  // the portable cluster size
constexpr int kSliceTarget = 4096;    // a row is spread over more CTAs until a slice is this short

struct SampleArgs {
  const float* logits;
  int64_t vocab;
  double temperature, top_p;
  int64_t top_k;  // 0: no limit
  uint64_t seed, counter;
  const uint64_t* seeds;     // optional per-row keys (device); the scalars serve every row otherwise
  const uint64_t* counters;
  uint32_t* tokens;
  DeviceStatus* status;
  int slice;   // logits per CTA of the row's cluster
  int cached;  // the slice is kept in shared memory
};

__device__ __forceinline__ double random_unit(uint64_t seed, uint64_t counter) {
  uint64_t value = seed ^ (counter * 0x9e3779b97f4a7c15ull);
  value += 0x9e3779b97f4a7c15ull;
  value = (value ^ (value >> 30)) * 0xbf58476d1ce4e5b9ull;
  value = (value ^ (value >> 27)) * 0x94d049bb133111ebull;
  value ^= value >> 31;
  return (double)(value >> 11) * (1.0 / 9007199254740992.0);
}

// Larger logit -> larger key; among equal logits (0 and -0 are equal) the lower token has the larger key. Tokens are below 2^20.
__device__ __forceinline__ uint64_t sort_key(float v, uint32_t token) {
  const uint32_t u = __float_as_uint(__fadd_rn(v, 0.0f));
  const uint32_t ordered = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((uint64_t)ordered << 20) | (uint64_t)(0xFFFFFu - token);
}
__device__ __forceinline__ uint32_t key_token(uint64_t key) { return 0xFFFFFu - (uint32_t)(key & 0xFFFFFu); }
__device__ __forceinline__ float key_value(uint64_t key) {
  const uint32_t ordered = (uint32_t)(key >> 20);
  return __uint_as_float((ordered & 0x80000000u) ? (ordered ^ 0x80000000u) : ~ordered);
}

struct alignas(16) Shared {
  double weight[kBins];       // this CTA's bins; in the first CTA afterwards: inclusive sums over the row's bins
  double sum[kBins];
  uint32_t count[kBins];
  uint32_t total_count[kBins];  // first CTA: inclusive counts
  uint64_t key[kList];          // first CTA: gathered candidates, then sorted
  double cumulative[kList];
  double warp_sum[kSampleWarps];
  long long warp_bad[kSampleWarps];
  double slice_sum[kSampleWarps];  // token-order walk
  float best;
  long long bad;
  uint32_t listed;
  int crossing;  // bin or list position a search found
  // decisions of the first CTA that the others read
  struct Decision {
    int bin;              // -1: the running sum never gets there
    uint32_t in_bin, up_to;  // candidates in the bin, and up to and including it
    double before;        // running sum ahead of the bin
    double total;
    uint64_t picked;
    double at;            // running sum including `picked`
  } decision;
};

enum Crossing { kReaches = 0, kExceeds = 1 };  // running >= target (counts, top-p) or running > target (the draw)
__device__ __forceinline__ bool crosses(double running, double target, Crossing c) { return c == kReaches ? running >= target : running > target; }

// Which candidates a pass looks at, and in which bin each falls.
struct Scope {
  float best, per_unit;   // first level: bins of (max - value) * per_unit
  int bin = -1;           // >= 0: only that first-level bin, by `shift` bits of the key that match `prefix` above them
  int shift = 0;
  uint64_t prefix = 0, mask = 0, floor_key = 0;
  __device__ __forceinline__ int first_level(float v) const { return (int)fminf((best - v) * per_unit, (float)(kBins - 1)); }
  __device__ __forceinline__ bool whole() const { return bin < 0 && floor_key == 0; }  // every candidate, by first-level bins
  // -1: not in scope
  __device__ __forceinline__ int digit(float v, uint64_t key) const {
    if (key < floor_key) return -1;
    const int b = first_level(v);
    if (bin < 0) return b;
    if (b != bin || (key & mask) != prefix) return -1;
    return kBins - 1 - (int)((key >> shift) & (uint64_t)(kBins - 1));  // larger keys first
  }
};

struct Row {
  cg::cluster_group cluster;
  Shared& sh;
  Shared& first;     // the first CTA's
  const float* x;    // this CTA's slice
  int n;
  uint32_t token0;
  double mx, temperature;
  bool quads;        // x + n start on 16 bytes: a thread's candidates are groups of four
  float mine;        // the largest of this thread's candidates
  __device__ double weight_of(float v) const { return exp(((double)v - mx) / temperature); }

  // f(index, value) for each of this thread's candidates.
  template <typename F>
  __device__ __forceinline__ void each(F&& f) const {
    const int n4 = quads ? n / 4 : 0;
    for (int q = threadIdx.x; q < n4; q += kSampleThreads) {
      const float4 v = reinterpret_cast<const float4*>(x)[q];
      f(4 * q, v.x);
      f(4 * q + 1, v.y);
      f(4 * q + 2, v.z);
      f(4 * q + 3, v.w);
    }
    for (int i = 4 * n4 + threadIdx.x; i < n; i += kSampleThreads) f(i, x[i]);
  }

  // Inclusive sums of the cluster's bins, in the first CTA. WEIGHTED: of weights too. LARGEST: of each thread's largest
  // candidate only.
  template <bool WEIGHTED, bool LARGEST = false>
  __device__ void histogram(const Scope& scope) {
    for (int b = threadIdx.x; b < kBins; b += kSampleThreads) {
      sh.count[b] = 0u;
      if (WEIGHTED) sh.weight[b] = 0.0;
    }
    __syncthreads();
    if (LARGEST) {
      if (mine > -INFINITY) atomicAdd(&sh.count[scope.first_level(mine)], 1u);
    } else {
      each([&](int i, float v) {
        const int b = scope.whole() ? scope.first_level(v) : scope.digit(v, sort_key(v, token0 + (uint32_t)i));
        if (b < 0) return;
        atomicAdd(&sh.count[b], 1u);
        if (WEIGHTED) atomicAdd(&sh.weight[b], weight_of(v));
      });
    }
    cluster.sync();
    if (cluster.block_rank() == 0) {
      constexpr int PER = kBins / kSampleThreads;
      const int b0 = threadIdx.x * PER, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      uint32_t c[PER] = {};
      double w[PER] = {};
      static_assert(PER == 2 && kMaxSampleCluster % 4 == 0, "a pair of bins per thread");
      for (unsigned r0 = 0; r0 < cluster.num_blocks(); r0 += 4) {  // four peers' bins are requested before the first is added
        uint2 counts[4];
        double2 weights[4];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
          if (r0 + u < cluster.num_blocks()) {
            const Shared* peer = cluster.map_shared_rank(&sh, r0 + u);
            counts[u] = *reinterpret_cast<const uint2*>(peer->count + b0);
            if (WEIGHTED) weights[u] = *reinterpret_cast<const double2*>(peer->weight + b0);
          }
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
          if (r0 + u < cluster.num_blocks()) {
            c[0] += counts[u].x;
            c[1] += counts[u].y;
            if (WEIGHTED) { w[0] += weights[u].x; w[1] += weights[u].y; }
          }
      }
      // counts are exact in f64 too, so one scan over (count, weight) pairs
      uint32_t cs = 0;
      double ws = 0.0;
#pragma unroll
      for (int j = 0; j < PER; ++j) { c[j] = cs += c[j]; w[j] = ws += w[j]; }
      uint32_t ci = cs;
      double wi = ws;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t oc = __shfl_up_sync(0xffffffffu, ci, off);
        const double ow = __shfl_up_sync(0xffffffffu, wi, off);
        if (lane >= off) { ci += oc; wi += ow; }
      }
      if (lane == 31) { sh.warp_sum[warp] = wi; sh.warp_bad[warp] = ci; }
      __syncthreads();
      uint32_t ahead_c = ci - cs;
      double ahead_w = wi - ws;
      for (int k = 0; k < warp; ++k) { ahead_c += (uint32_t)sh.warp_bad[k]; ahead_w += sh.warp_sum[k]; }
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        sh.total_count[b0 + j] = ahead_c + c[j];
        sh.sum[b0 + j] = WEIGHTED ? ahead_w + w[j] : (double)(ahead_c + c[j]);
      }
      __syncthreads();
      if (threadIdx.x == 0) sh.decision.total = sh.sum[kBins - 1];
    }
  }

  // First CTA, after histogram(): the bin in which before + running sum crosses the target; the others learn it.
  __device__ void find_bin(double before, double target, Crossing c) {
    if (cluster.block_rank() == 0) {
      if (threadIdx.x == 0) sh.crossing = kBins;
      __syncthreads();
      for (int b = threadIdx.x; b < kBins; b += kSampleThreads) {
        const bool held = sh.total_count[b] != (b > 0 ? sh.total_count[b - 1] : 0u);
        if (held && crosses(before + sh.sum[b], target, c)) atomicMin(&sh.crossing, b);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        const int b = sh.crossing;
        Shared::Decision& d = sh.decision;
        d.bin = b < kBins ? b : -1;
        if (b < kBins) {
          d.up_to = sh.total_count[b];
          d.in_bin = sh.total_count[b] - (b > 0 ? sh.total_count[b - 1] : 0u);
          d.before = before + (b > 0 ? sh.sum[b - 1] : 0.0);
        }
        sh.listed = 0u;
      }
    }
    cluster.sync();
  }

  // Candidates of the bins [lo, hi] of the scope into the first CTA's list (the first kList of them; `listed` counts all).
  __device__ void collect(const Scope& scope, int lo, int hi) {
    const auto list = [&](uint64_t key) {
      const uint32_t at = atomicAdd(&first.listed, 1u);
      if (at < (uint32_t)kList) first.key[at] = key;
    };
    if (scope.whole() && lo == 0) {
      if (scope.first_level(mine) <= hi)  // (-infinity, of a thread without candidates, is in the last bin)
        each([&](int i, float v) {
          if (scope.first_level(v) <= hi) list(sort_key(v, token0 + (uint32_t)i));
        });
    } else {
      each([&](int i, float v) {
        const uint64_t key = sort_key(v, token0 + (uint32_t)i);
        const int b = scope.digit(v, key);
        if (b >= lo && b <= hi) list(key);
      });
    }
    cluster.sync();
  }

  // The first CTA sorts its list by descending key.
  __device__ void sort_list() {
    if (cluster.block_rank() != 0) return;
    const int m = min((int)sh.listed, kList);
    if (m <= kRankSorted) {  // no two keys are alike: a key's place is the number of larger ones
      const uint64_t mine_key = threadIdx.x < m ? sh.key[threadIdx.x] : 0ull;
      int place = 0;
      if (threadIdx.x < m) {
#pragma unroll 8
        for (int j = 0; j < m; ++j) place += sh.key[j] > mine_key;
      }
      __syncthreads();
      if (threadIdx.x < m) sh.key[place] = mine_key;
      __syncthreads();
      return;
    }
    int padded = 32;
    while (padded < m) padded <<= 1;
    for (int i = m + threadIdx.x; i < padded; i += kSampleThreads) sh.key[i] = 0ull;
    for (int size = 2; size <= padded; size <<= 1)
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        __syncthreads();
        for (int p = threadIdx.x; p < padded / 2; p += kSampleThreads) {
          const int i = 2 * p - (p & (stride - 1)), j = i + stride;
          const uint64_t a = sh.key[i], b = sh.key[j];
          if (((i & size) == 0) == (a < b)) { sh.key[i] = b; sh.key[j] = a; }
        }
      }
    __syncthreads();
  }

  // First CTA: inclusive sums of the first m listed candidates' weights (or of ones).
  __device__ void accumulate(int m, bool weighted) {
    constexpr int PER = kList / kSampleThreads;
    const int i0 = threadIdx.x * PER, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double w[PER], s = 0.0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      w[j] = s += i0 + j >= m ? 0.0 : (weighted ? weight_of(key_value(sh.key[i0 + j])) : 1.0);
    }
    double inclusive = s;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const double o = __shfl_up_sync(0xffffffffu, inclusive, off);
      if (lane >= off) inclusive += o;
    }
    if (lane == 31) sh.warp_sum[warp] = inclusive;
    __syncthreads();
    double ahead = inclusive - s;
    for (int k = 0; k < warp; ++k) ahead += sh.warp_sum[k];
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (i0 + j < kList) sh.cumulative[i0 + j] = ahead + w[j];
    __syncthreads();
  }

  // First CTA: position of the first of m listed candidates at which before + running sum crosses the target (m: none).
  __device__ int find_listed(int m, double before, double target, Crossing c) {
    if (threadIdx.x == 0) sh.crossing = m;
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += kSampleThreads)
      if (crosses(before + sh.cumulative[i], target, c)) atomicMin(&sh.crossing, i);
    __syncthreads();
    const int at = sh.crossing;
    __syncthreads();
    return at;
  }

  // The candidate of first-level bin decision.bin at which decision.before + running sum crosses the target, into
  // decision.picked / at. Rounding may leave the bin's own sum an ulp short of the target: then its last candidate.
  __device__ void resolve(Scope scope, bool weighted, double target, Crossing c) {
    int lo = first.decision.bin, hi = lo;
    double before = first.decision.before;
    uint32_t held = first.decision.in_bin;
    for (int level = 0; held > (uint32_t)kList; ++level) {
      scope.bin = level == 0 ? lo : scope.bin;
      scope.shift = max(0, 42 - 10 * level);
      if (weighted) histogram<true>(scope);
      else histogram<false>(scope);
      find_bin(before, target, c);
      lo = first.decision.bin;
      if (lo < 0) {  // rounding again: the scope's last digit that holds a candidate
        cluster.sync();  // every CTA has seen that there is none
        if (cluster.block_rank() == 0 && threadIdx.x == 0) {
          int b = kBins - 1;
          while (b > 0 && sh.total_count[b - 1] == sh.total_count[kBins - 1]) --b;
          sh.decision.bin = b;
          sh.decision.in_bin = sh.total_count[b] - (b > 0 ? sh.total_count[b - 1] : 0u);
          sh.decision.before = before + (b > 0 ? sh.sum[b - 1] : 0.0);
        }
        cluster.sync();
        lo = first.decision.bin;
      }
      hi = lo;
      before = first.decision.before;
      held = first.decision.in_bin;
      if (held > (uint32_t)kList) {
        scope.prefix |= (uint64_t)(kBins - 1 - lo) << scope.shift;
        scope.mask |= (uint64_t)(kBins - 1) << scope.shift;
      }
      cluster.sync();  // the decision is read before the next one is written
    }
    collect(scope, lo, hi);
    sort_list();
    if (cluster.block_rank() == 0) {
      const int m = min((int)sh.listed, kList);
      accumulate(m, weighted);
      const int at = min(find_listed(m, before, target, c), m - 1);
      if (threadIdx.x == 0) {
        // Nothing listed: the bin lies behind the cut at floor_key. The bins of a top-p draw are those of before the cut, and
        // their sum up to it can be an ulp short of the retained total, which was added up in another order; a draw between
        // the two has walked past every retained candidate, and the last one of those is the one at the cut.
        sh.decision.picked = m > 0 ? sh.key[at] : scope.floor_key;
        sh.decision.at = m > 0 ? before + sh.cumulative[at] : target;
      }
    }
    cluster.sync();
  }
};

// FILTERED: top-k or top-p (a kernel of its own, so that the walk in token order is not held to the other's registers).
template <bool FILTERED>
__global__ void __launch_bounds__(kSampleThreads, 2) sample_rows_kernel(SampleArgs a) {
  extern __shared__ __align__(16) float cache[];
  __shared__ Shared sh;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  const int64_t row = blockIdx.x / ranks;
  const int64_t begin = min(a.vocab, (int64_t)rank * a.slice), end = min(a.vocab, begin + a.slice);
  const int n = (int)(end - begin), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* source = a.logits + row * a.vocab + begin;
  // ---- every logit must be finite; the largest one anchors the exponentials
  float best = -INFINITY;
  long long bad = 0x7fffffffffffffffll;
  auto see = [&](int i, float v) {
    if (!isfinite(v)) bad = min(bad, (long long)(begin + i));
    best = fmaxf(best, v);
  };
  // in groups of four where the slice starts on 16 bytes, four of them in flight per thread
  const bool quads = (reinterpret_cast<uintptr_t>(source) & 15) == 0;
  const int n4 = quads ? n / 4 : 0;
  constexpr int IN_FLIGHT = 4;
  for (int q0 = threadIdx.x; q0 < n4; q0 += IN_FLIGHT * kSampleThreads) {
    float4 v[IN_FLIGHT];
#pragma unroll
    for (int u = 0; u < IN_FLIGHT; ++u)
      if (q0 + u * kSampleThreads < n4) v[u] = reinterpret_cast<const float4*>(source)[q0 + u * kSampleThreads];
#pragma unroll
    for (int u = 0; u < IN_FLIGHT; ++u) {
      const int q = q0 + u * kSampleThreads;
      if (q >= n4) break;
      if (a.cached) reinterpret_cast<float4*>(cache)[q] = v[u];
      see(4 * q, v[u].x);
      see(4 * q + 1, v[u].y);
      see(4 * q + 2, v[u].z);
      see(4 * q + 3, v[u].w);
    }
  }
  {
    int i = 4 * n4 + threadIdx.x;
    for (; i + 3 * kSampleThreads < n; i += 4 * kSampleThreads) {  // four loads in flight
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = source[i + u * kSampleThreads];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (a.cached) cache[i + u * kSampleThreads] = v[u];
        see(i + u * kSampleThreads, v[u]);
      }
    }
    for (; i < n; i += kSampleThreads) {
      const float v = source[i];
      if (a.cached) cache[i] = v;
      see(i, v);
    }
  }
  const float mine = best;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, off));
    bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, off));
  }
  if (lane == 0) { sh.warp_sum[warp] = (double)best; sh.warp_bad[warp] = bad; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 0; w < kSampleWarps; ++w) { best = fmaxf(best, (float)sh.warp_sum[w]); bad = min(bad, sh.warp_bad[w]); }
    sh.best = best;
    sh.bad = bad;
    sh.listed = 0u;
  }
  cluster.sync();
  best = -INFINITY;
  bad = 0x7fffffffffffffffll;
#pragma unroll
  for (int r = 0; r < kMaxSampleCluster; ++r)
    if (r < ranks) {
      const Shared* peer = cluster.map_shared_rank(&sh, r);
      best = fmaxf(best, peer->best);
      bad = min(bad, peer->bad);
    }
  if (bad != 0x7fffffffffffffffll) {  // the same answer in every CTA of the row
    if (rank == 0 && threadIdx.x == 0) {
      a.tokens[row] = 0u;
      if (atomicCAS(&a.status->code, kStatusNone, kStatusNonFiniteLogit) == kStatusNone) {
        a.status->value = bad;
        a.status->bound = a.vocab;
      }
    }
    cluster.sync();
    return;
  }
  Row r{cluster, sh, *cluster.map_shared_rank(&sh, 0), a.cached ? cache : source, n, (uint32_t)begin, (double)best, a.temperature, quads, mine};
  const double unit = random_unit(a.seeds ? a.seeds[row] : a.seed, a.counters ? a.counters[row] : a.counter);
  const bool has_top_k = FILTERED && a.top_k > 0 && a.top_k < a.vocab;

  if constexpr (!FILTERED) {
    // ---- walk in token order: every warp sums its part of the slice, then the one that holds the draw walks it
    const int part = (a.slice + kSampleWarps - 1) / kSampleWarps;
    const int lo = min(n, warp * part), hi = min(n, lo + part);
    double mine = 0.0;
    for (int i = lo + lane; i < hi; i += 32) mine += r.weight_of(r.x[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, off);
    if (lane == 0) sh.slice_sum[warp] = mine;
    cluster.sync();
    double ahead = 0.0, total = 0.0;
    for (int p = 0; p < ranks * kSampleWarps; ++p) {  // the same order in every warp
      if (p == rank * kSampleWarps + warp) ahead = total;
      total += cluster.map_shared_rank(&sh, p / kSampleWarps)->slice_sum[p % kSampleWarps];
    }
    const double draw = unit * total;
    const bool last = end == a.vocab && n > 0 && hi == n && lo < hi;  // the draw can reach the row's end by rounding only
    if (lo < hi && ahead <= draw && (draw < ahead + mine || last)) {
      double left = draw - ahead;
      int token = hi - 1;
      for (int i0 = lo; i0 < hi; i0 += 32) {
        double w = i0 + lane < hi ? r.weight_of(r.x[i0 + lane]) : 0.0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const double o = __shfl_up_sync(0xffffffffu, w, off);
          if (lane >= off) w += o;
        }
        const unsigned over = __ballot_sync(0xffffffffu, w > left);
        if (over) { token = min(hi - 1, i0 + __ffs(over) - 1); break; }
        left -= __shfl_sync(0xffffffffu, w, 31);
      }
      if (lane == 0) a.tokens[row] = (uint32_t)(begin + token);
    }
    cluster.sync();
    return;
  } else {

  // ---- filtered: candidates in (value descending, token ascending) order
  Scope scope;
  scope.best = best;
  scope.per_unit = fminf((float)(32.0 / a.temperature), 1e30f);  // bins of 1/32 in the logarithm of the weight, the last one open
  if (has_top_k) {
    // The list decides everything where it holds the first top_k candidates. They are in the bins up to the one at which a count
    // of the threads' largest candidates alone reaches top_k, and only the threads whose largest is there have any.
    const auto from_list = [&] {
      const int k = (int)a.top_k;
      r.sort_list();
      r.accumulate(k, true);
      int kept = k;
      double total = sh.cumulative[k - 1];
      if (a.top_p < 1.0) {
        const int at = r.find_listed(k, 0.0, a.top_p * total, kReaches);
        if (at < k) { kept = at + 1; total = sh.cumulative[at]; }  // otherwise every candidate stays
      }
      const int at = min(r.find_listed(kept, 0.0, unit * total, kExceeds), kept - 1);
      if (threadIdx.x == 0) a.tokens[row] = key_token(sh.key[at]);
    };
    // Not for lists that grow by it to more than is sorted by counting, or beyond kList, nor where few threads have candidates or the
    // bin is the open last one: against the histogram of all candidates alone, top-k 150 of 8192 tokens 0.8, of 50257 0.9, but
    // 450 of 8192 1.2, 700 1.25, 1000 of 50257 1.29, 320 of 4096 1.23, and 1.0 between.
    const int64_t holders = min((int64_t)ranks * kSampleThreads, a.vocab / 4);  // threads with candidates, of groups of four
    if (a.top_k <= kFewEnough && 3 * a.top_k <= holders) {
      r.histogram<false, true>(scope);
      r.find_bin(0.0, (double)a.top_k, kReaches);
      const int bin = r.first.decision.bin;
      if (bin >= 0 && (bin < kBins - 1 || a.vocab <= kList)) {  // the open last bin holds all that is far below the maximum
        r.collect(scope, 0, bin);
        const bool fits = r.first.listed <= (uint32_t)kList;
        cluster.barrier_arrive();  // the first CTA stays until the others have read that
        if (fits && rank == 0) from_list();
        cluster.barrier_wait();
        if (fits) return;
      }
    }
    r.histogram<false>(scope);
    r.find_bin(0.0, (double)a.top_k, kReaches);
    if (r.first.decision.up_to <= (uint32_t)kList) {
      r.collect(scope, 0, r.first.decision.bin);
      if (rank == 0) from_list();
      return;
    }
    r.resolve(scope, false, (double)a.top_k, kReaches);
    scope.floor_key = r.first.decision.picked;
    cluster.sync();
  }
  r.histogram<true>(scope);
  cluster.sync();  // the first CTA's total
  double total = r.first.decision.total;
  if (a.top_p < 1.0) {
    r.find_bin(0.0, a.top_p * total, kReaches);
    if (r.first.decision.bin >= 0) {
      const bool narrowed = r.first.decision.in_bin > (uint32_t)kList;
      r.resolve(scope, true, a.top_p * total, kReaches);
      scope.floor_key = r.first.decision.picked;
      total = r.first.decision.at;
      if (narrowed) r.histogram<true>(scope);  // the narrowing steps took the first-level sums' place
    }
    cluster.sync();
  }
  r.find_bin(0.0, unit * total, kExceeds);
  if (r.first.decision.bin < 0) {  // the walk never went negative: the last retained candidate, in the last bin that holds one
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) {
      int b = kBins - 1;
      while (b > 0 && sh.total_count[b - 1] == sh.total_count[kBins - 1]) --b;
      sh.decision.bin = b;
      sh.decision.in_bin = sh.total_count[b] - (b > 0 ? sh.total_count[b - 1] : 0u);
      sh.decision.before = b > 0 ? sh.sum[b - 1] : 0.0;
    }
    cluster.sync();
  }
  r.resolve(scope, true, unit * total, kExceeds);
  if (rank == 0 && threadIdx.x == 0) a.tokens[row] = key_token(sh.decision.picked);
  }
}

}  // namespace

cudaError_t launch_sample_rows(const float* logits, int64_t rows, int64_t vocab, double temperature, int64_t top_k, double top_p,
                               uint64_t seed, uint64_t counter, const uint64_t* seeds, const uint64_t* counters, uint32_t* tokens,
                               DeviceStatus* status, cudaStream_t stream) {
  if (rows == 0) return cudaSuccess;
  int ranks = 1;
  while (ranks < kMaxSampleCluster && (vocab + ranks - 1) / ranks > kSliceTarget) ranks *= 2;
  const int slice = (int)((vocab + ranks - 1) / ranks);
  SampleArgs a{logits, vocab, temperature, top_p, top_k, seed, counter, seeds, counters, tokens, status, slice, slice <= kMaxSlice};
  const bool filtered = (top_k > 0 && top_k < vocab) || top_p < 1.0;
  auto kernel = filtered ? sample_rows_kernel<true> : sample_rows_kernel<false>;
  const cudaError_t attr = opt_in_shared_memory(kernel, kMaxSlice * sizeof(float));
  if (attr != cudaSuccess) return attr;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)(rows * ranks));
  config.blockDim = dim3(kSampleThreads);
  config.dynamicSmemBytes = a.cached ? (size_t)slice * sizeof(float) : 0;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = (unsigned)ranks;
  attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, a);
}

}  // namespace etc
