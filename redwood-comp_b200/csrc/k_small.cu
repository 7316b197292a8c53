// The whole pipeline of a small cloud in one cooperative launch.
//
// A cloud of up to a few hundred thousand points does not fill the chip, and
// the chain of one kernel per step (k_keys.cu, k_tree.cu) costs it latency:
// 14 launches of 3 to 10 us each, whatever the size (85 us on the device and
// 45 us of launch calls at 3,001 points, 97 us at 307,200).  Here up to one
// block of 1,024 threads per SM keeps its share of the keys in shared memory,
// and the steps are separated by barriers over the grid (1.3 us each, 2.3 with
// stores to drain; none when one block takes the cloud).  A call with its wait,
// before and now, 32-bit keys: 2,000 points 100 and 43 us, 4,096 100 and 54,
// 20,000 100 and 59, 303,104 110 and 72, 600,000 126 and 88; 64-bit keys: 4,200
// points 123 and 57 us, 303,104 143 and 77, 400,000 155 and 83.  What is left is
// latency: eight barriers, and chains of dependent shared-memory and L2
// accesses in every step.
//
// Sort: one exchange instead of one per digit.  Every block gives one or two
// lists of 32 sampled keys; the samples' exact ranks yield a splitter per block; every block sends
// its keys to the blocks that own them (bucket regions filled through one
// atomic counter each) and sorts what it receives in shared memory by 8-bit
// digits, leaving out the digits that all its keys share.  Keys equal to a
// repeated splitter may go to any of the buckets it bounds, so duplicates do
// not fill one bucket.  A bucket that overflows all the same (the samples
// missed most of the keys) sends the cloud through a digit-by-digit sort over
// the grid in the same launch.
//
// Stages 3 to 7 are the same tile routines as in the general kernels
// (tree_tiles.cuh), with each block's tile sized by the cloud.
#include <algorithm>

#include "block_sort.cuh"
#include "internal.hpp"
#include "morton.cuh"
#include "tree_tiles.cuh"

namespace rwt {

constexpr int kSmThreads = 1024, kSmWarps = kSmThreads / 32;
constexpr int kSmSamples = 32;    // of a list: one per warp when they are ranked
constexpr int kSmEncode = 8;      // points per thread of a block's share
constexpr int kSmMaxBlocks = 256;
constexpr int kSmGroups = kSmThreads / kOctThreads;  // octree tiles at a time per block
static_assert(kSmGroups < kSortBarrier, "the groups use the named barriers below");
constexpr int kSmFill = 32;         // words between two bucket counters: a line each
constexpr int kSmTreeChunks = 128;  // chunks of 32 gaps per radix-tree tile, at most

template <typename K>
struct SmallCfg {
  static constexpr int kCap = 57344 / int(sizeof(K));  // keys of a block, sorted in place
  static constexpr int kKpt = kCap / kSortThreads;
  static constexpr size_t kSort = 2 * size_t(kCap) * sizeof(K) + 2 * size_t(kSortHist) * 4;
  static constexpr size_t kTree = AnsvCfg<K, kSmTreeChunks>::kSmem;
  static constexpr size_t kOct = kSmGroups * sizeof(OctTileShared<K>);
  static constexpr size_t kSmem = kSort > kTree ? (kSort > kOct ? kSort : kOct)
                                                : (kTree > kOct ? kTree : kOct);
};

struct SmallArgs {
  const float4* points;
  void *keys, *alt;
  // points, points per block, keys per bucket region, sample lists per block
  uint32_t n, chunk, cap, lists;
  float min_coord, range, inv_range;
  uint8_t *prefix_n, *hl, *hr;
  int32_t *lc, *parents, *edge_count, *edge_offset;
  OctOut o;
  bool leaves;
  // scratch
  // [0] arrivals, [1] arrivals before this launch, [2] a wait gave up, [3] launches
  // that sorted digit by digit
  uint32_t* sync;
  uint32_t spin_limit, missing;  // of the barriers: polls; arrivals that never come
  void *samples, *splitters, *first, *last, *region, *tmp;
  uint32_t *fill, *counts, *heads, *mat, *sums;
  uint32_t *far, *far_n, far_cap;
  DevStatus *status, *host_status;
};

struct SmallShared {
  DigitShared digit;
  uint32_t place[256];
  uint32_t warp[kSmWarps + 1];
  uint32_t hist[kSmMaxBlocks], off[kSmMaxBlocks];
  uint32_t diff[2];
  uint32_t dup, ok;
  unsigned long long gsum[kSmGroups][kOctThreads / 32];
  TreeTileShared tree;
};

// Sorts a block's c keys in `a` (with `b` as the other half); returns where
// they end.  Digits that all keys share are left out.  The keys are filled up
// to whole steps with the largest word, which stays behind them.
//
// A few thousand keys rarely share the first 24 bits of those in which they
// differ: with `bits` 24 only these are sorted by digits (three passes instead
// of four to eight, 2.1 us each), then every key of a run that shares them finds
// its place by counting the run's smaller keys: 64-bit keys, 3,001 points 20.0
// -> 9.0 us of sorting, 307,200 points 20.2 -> 10.1.  A run beyond kSortRun keys
// sends the block through all digits.
constexpr int kSortRun = 32;

template <typename K>
__device__ K* block_sort(K* a, K* b, int c, int bits, uint32_t* hist, uint32_t* next, SmallShared& sh) {
  constexpr int kBits = KeyTraits<K>::kCodeBits;
  if (c < 2) return a;
  const int steps = (c + kSortThreads - 1) / kSortThreads;
  if (threadIdx.x < 2) sh.diff[threadIdx.x] = 0;
  __syncthreads();
  K d = 0;
  const K k0 = a[0];
  for (int i = int(threadIdx.x); i < steps * kSortThreads; i += kSmThreads) {
    if (i < c) d |= a[i] ^ k0;
    else a[i] = K(~K(0));
  }
  const uint32_t lo = __reduce_or_sync(0xffffffffu, uint32_t(d));
  const uint32_t hi =
      sizeof(K) == 8 ? __reduce_or_sync(0xffffffffu, uint32_t(uint64_t(d) >> 32)) : 0u;
  if (lane_id() == 0) {
    if (lo) atomicOr(&sh.diff[0], lo);
    if (hi) atomicOr(&sh.diff[1], hi);
  }
  __syncthreads();
  const K all = sizeof(K) == 8 ? K(uint64_t(sh.diff[1]) << 32 | sh.diff[0]) : K(sh.diff[0]);
  const int low = max(KeyTraits<K>::kWordBits - KeyTraits<K>::clz(all) - bits, 0);
  for (int from = low;; from = 0) {
    for (int shift = from; shift < kBits && (all >> shift); shift += 8) {
      if (((all >> shift) & K(255)) == 0) continue;
      if (threadIdx.x < kSortThreads)
        block_digit_pass<K, SmallCfg<K>::kKpt>(a, b, steps, shift, hist, next, sh.digit);
      K* t = a;
      a = b;
      b = t;
      uint32_t* h = hist;
      hist = next;
      next = h;
    }
    __syncthreads();
    if (from == 0) return a;
    bool far = false;
    for (int i = int(threadIdx.x); i < c; i += kSmThreads) {
      const K k = a[i], p = k >> from;
      int less = 0, l = i - 1, r = i + 1;
      while (l >= 0 && i - l <= kSortRun && (a[l] >> from) == p) less += int(a[l--] <= k);
      while (r < c && r - i <= kSortRun && (a[r] >> from) == p) less += int(a[r++] < k);
      far |= i - l > kSortRun || r - i > kSortRun;
      b[l + 1 + less] = k;
    }
    if (!__syncthreads_or(int(far))) return b;
  }
}

__device__ __forceinline__ uint32_t small_hash(uint32_t x) {  // Wang-style integer mix
  x = (x ^ 61u) ^ (x >> 16);
  x *= 9u;
  x ^= x >> 4;
  x *= 0x27d4eb2du;
  return x ^ (x >> 15);
}

template <typename K, int LESS>
__global__ void __launch_bounds__(kSmThreads, 1) k_small(SmallArgs a) {
  using C = SmallCfg<K>;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SmallShared sh;
  __shared__ K s_spl[kSmMaxBlocks];
  K* sa = reinterpret_cast<K*>(smem);
  K* sb = sa + C::kCap;
  uint32_t* hist = reinterpret_cast<uint32_t*>(sb + C::kCap);
  uint32_t* next = hist + kSortHist;
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  const uint32_t P = gridDim.x, b = blockIdx.x;
  GridBarrier bar{a.sync, P + a.missing, ld_relaxed(a.sync + 1), a.spin_limit,
                  &sh.ok, a.sync + 2, a.status, a.host_status};
  if (ld_relaxed(a.sync + 2)) {  // an earlier wait gave up and nothing cleared the scratch since
    if (b == 0 && tid == 0)
      *reinterpret_cast<volatile int32_t*>(&a.host_status->err) = RW_ERR_TIMEOUT;
    return;
  }
  if (b == 0) {
    for (uint32_t i = uint32_t(tid); i < P; i += kSmThreads) a.fill[i * kSmFill] = 0;
    for (uint32_t i = uint32_t(tid); i < (a.n + kOctTile - 1) / kOctTile; i += kSmThreads)
      a.sums[i] = 0;
    if (tid == 0) {
      *a.status = DevStatus{0, 0, 0, 0};
      *a.far_n = 0;
    }
  }
  K* keys = static_cast<K*>(a.keys);
  K* alt = static_cast<K*>(a.alt);

  // ---- stage 1: the block's share of the points ----
  const uint32_t p0 = min(b * a.chunk, a.n);
  const int mine = int(min(a.n - p0, a.chunk));
#pragma unroll
  for (int h = 0; h < kSmEncode; h += 4) {
    float4 p[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = tid + (h + q) * kSmThreads;
      if (i < mine) p[q] = __ldcs(a.points + p0 + i);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = tid + (h + q) * kSmThreads;
      if (i < mine) {
        const K k = a.inv_range != 0.0f
                        ? encode<K, true>(p[q].x, p[q].y, p[q].z, a.min_coord, a.range, a.inv_range)
                        : encode<K, false>(p[q].x, p[q].y, p[q].z, a.min_coord, a.range);
        sa[i] = k;
        keys[p0 + i] = k;
      }
    }
  }
  for (int i = tid; i < kSortHist / 4; i += kSmThreads)
    reinterpret_cast<uint4*>(hist)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();

  // ---- stage 2 ----
  // 30-bit codes of a large cloud have such runs wherever it is dense: 899,000
  // mixture points took 138 us with 24 bits and take 118 with all (uniform ones
  // 117 and 119; up to 2^18 points 24 bits gain 2 us in both)
  const int bits = sizeof(K) == 4 && a.n > (1u << 18) ? KeyTraits<K>::kCodeBits : 24;
  K* sorted = nullptr;  // this block's run of the sorted keys, in shared memory
  int c = mine;
  uint32_t base = p0;  // its place among all
  if (P == 1) {
    sorted = block_sort<K>(sa, sb, c, bits, hist, next, sh);
  } else {
    K* samples = static_cast<K*>(a.samples);
    K* splitters = static_cast<K*>(a.splitters);
    const int R = int(a.lists);
    if (warp < R) {
      // one key of each of 32 strata of the share (of 64, the second list the
      // other half), sorted within the warp; a share without a key stands for
      // the largest one
      const int t = warp * kSmSamples + lane, strata = R * kSmSamples;
      const uint32_t lo = uint32_t(uint64_t(mine) * t / strata),
                     hi = uint32_t(uint64_t(mine) * (t + 1) / strata);
      static_assert(kSmSamples == 32, "a lane per sample");
      K k = mine == 0 ? K(~K(0)) : sa[hi > lo ? lo + small_hash(p0 + lo) % (hi - lo) : lo];
#pragma unroll
      for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
        for (int st = size >> 1; st > 0; st >>= 1) {
          const K other = __shfl_xor_sync(0xffffffffu, k, st);
          const bool up = (lane & size) == 0, low = (lane & st) == 0;
          k = (low == up) == (other < k) ? other : k;
        }
      samples[(int(b) * R + warp) * kSmSamples + lane] = k;
    }
    if (!bar.sync()) return;
    const int nl = int(P) * R;  // lists
    constexpr int kPitch = kSmSamples + 1;  // a list's samples: lanes in different banks
    K* ss = sa + mine;  // behind the keys (small_takes: there is room)
    for (int i = tid; i < nl * kSmSamples; i += kSmThreads)
      ss[i / kSmSamples * kPitch + i % kSmSamples] = samples[i];
    __syncthreads();
    for (int own = int(b) * R; own < int(b + 1) * R; ++own) {
      // the exact rank of this warp's sample among all, ties in their order:
      // a search in every list; every (32 R)-th sample is a splitter
      static_assert(kSmSamples == kSmWarps, "a warp ranks one sample of a list");
      const K my = ss[own * kPitch + warp];
      uint32_t r = 0;
      for (int j = lane; j < nl; j += 32) {
        const K* q = ss + j * kPitch;
        if (j == own) {
          r += uint32_t(warp);
        } else {
          // keys of list j below my sample, or not above it if j comes first
          uint32_t at = 0;
#pragma unroll
          for (int st = kSmSamples / 2; st > 0; st >>= 1) {
            const K x = q[at + st - 1];
            if (x < my || (j < own && x == my)) at += st;
          }
          const K x = q[at];
          r += at + uint32_t(x < my || (j < own && x == my));
        }
      }
      r = warp_sum(r);
      if (lane == 0 && r && r % uint32_t(kSmSamples * R) == 0)
        splitters[r / uint32_t(kSmSamples * R) - 1] = my;
    }
    if (!bar.sync()) return;
    const int nspl = int(P) - 1;
    for (int i = tid; i < int(P); i += kSmThreads) {
      if (i < nspl) s_spl[i] = splitters[i];
      sh.hist[i] = 0;
    }
    __syncthreads();
    uint32_t slot[kSmEncode];  // bucket << 16 | rank among the block's keys of that bucket
    static_assert(kSmEncode * kSmThreads <= 65536, "16-bit ranks");
#pragma unroll
    for (int q = 0; q < kSmEncode; ++q) {
      const int i = tid + q * kSmThreads;
      if (i < mine) {
        const K k = sa[i];
        int lo = 0, hi = nspl;  // splitters below k
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s_spl[mid] < k) lo = mid + 1;
          else hi = mid;
        }
        uint32_t bk = uint32_t(lo);
        if (lo < nspl && s_spl[lo] == k) {
          // splitters [lo, hi) equal k: any of the buckets lo .. hi may take it
          int at = lo + 1;
          hi = nspl;
          while (at < hi) {
            const int mid = (at + hi) >> 1;
            if (s_spl[mid] == k) at = mid + 1;
            else hi = mid;
          }
          bk += small_hash(p0 + uint32_t(i)) % uint32_t(hi - lo + 1);
        }
        slot[q] = bk << 16 | atomicAdd(&sh.hist[bk], 1u);
      }
    }
    __syncthreads();
    for (int i = tid; i < int(P); i += kSmThreads)
      sh.off[i] = sh.hist[i] ? atomicAdd(a.fill + i * kSmFill, sh.hist[i]) : 0u;
    __syncthreads();
    K* region = static_cast<K*>(a.region);
#pragma unroll
    for (int q = 0; q < kSmEncode; ++q) {
      const int i = tid + q * kSmThreads;
      if (i < mine) {
        const uint32_t bk = slot[q] >> 16, at = sh.off[bk] + (slot[q] & 0xffffu);
        if (at < a.cap) region[size_t(bk) * a.cap + at] = sa[i];
      }
    }
    if (!bar.sync()) return;
    uint32_t f = 0, before = 0, over = 0;
    if (tid < int(P)) {
      f = a.fill[tid * kSmFill];
      over = f > a.cap;
      before = tid < int(b) ? f : 0u;
    }
    static_assert(kSmMaxBlocks <= kSmThreads, "a thread per block");
    if (!__syncthreads_or(int(over))) {
      uint32_t total;
      block_exclusive_scan<kSmThreads>(before, sh.warp, &total);
      base = total;
      if (tid == int(b)) sh.off[0] = f;
      __syncthreads();
      c = int(sh.off[0]);
      const K* mineq = region + size_t(b) * a.cap;
      for (int i = tid; i < c; i += kSmThreads) sa[i] = mineq[i];
      __syncthreads();
      sorted = block_sort<K>(sa, sb, c, bits, hist, next, sh);
    } else {
      // digit by digit over the grid: every block ranks its share, the counts
      // of all blocks give its keys' places
      K* tmp = static_cast<K*>(a.tmp);
      if (b == 0 && tid == 0) ++a.sync[3];
      for (int shift = 0; shift < KeyTraits<K>::kCodeBits; shift += 8) {
        const int steps = (c + kSortThreads - 1) / kSortThreads;
        for (int i = c + tid; i < steps * kSortThreads; i += kSmThreads) sa[i] = K(~K(0));
        __syncthreads();
        if (tid < kSortThreads)
          block_digit_pass<K, SmallCfg<K>::kKpt>(sa, sb, steps, shift, hist, next, sh.digit);
        __syncthreads();
        uint32_t* h = hist;
        hist = next;
        next = h;
        // (the filling counts in the last digit: its end is c)
        if (tid < 256)
          a.mat[b * 256 + tid] = (tid < 255 ? sh.digit.start[tid + 1] : uint32_t(c)) - sh.digit.start[tid];
        if (!bar.sync()) return;
        uint32_t tot = 0, prior = 0;
        if (tid < 256)
          for (uint32_t j = 0; j < P; ++j) {
            const uint32_t v = a.mat[j * 256 + tid];
            prior += j < b ? v : 0u;
            tot += v;
          }
        uint32_t all;
        const uint32_t ex = block_exclusive_scan<kSmThreads>(tot, sh.warp, &all);
        if (tid < 256) sh.place[tid] = ex + prior - sh.digit.start[tid];
        __syncthreads();
        for (int i = tid; i < c; i += kSmThreads)
          tmp[sh.place[uint32_t(sb[i] >> shift) & 255u] + uint32_t(i)] = sb[i];
        if (!bar.sync()) return;
        for (int i = tid; i < c; i += kSmThreads) sa[i] = tmp[p0 + i];
        __syncthreads();
      }
      sorted = sa;
    }
  }

  // ---- stage 3 ----
  for (int i = tid; i < c; i += kSmThreads) alt[base + i] = sorted[i];
  const int per = (c + kSmThreads - 1) / kSmThreads;  // consecutive keys per thread
  const int i0 = min(tid * per, c), i1 = min(i0 + per, c);
  uint32_t hm = 0;  // which of them differ from the key before (the block's first: taken as such)
  for (int i = i0; i < i1; ++i)
    hm |= uint32_t(i == 0 || sorted[i] != sorted[i - 1]) << (i - i0);
  uint32_t heads;
  uint32_t pos = block_exclusive_scan<kSmThreads>(uint32_t(__popc(hm)), sh.warp, &heads);
  uint32_t u = heads;
  if (P > 1) {
    K* first = static_cast<K*>(a.first);
    K* last = static_cast<K*>(a.last);
    if (tid == 0) {
      a.heads[b] = heads;
      sh.dup = 0;
      first[b] = c ? sorted[0] : K(0);
      last[b] = c ? sorted[c - 1] : K(0);
      a.counts[b] = uint32_t(c);
    }
    if (!bar.sync()) return;
    uint32_t h = 0;
    if (tid < int(P)) {
      // loaded together; an empty block before this one is rare
      const uint32_t ct = a.counts[tid], ht = a.heads[tid], cb = tid ? a.counts[tid - 1] : 1u;
      const K ft = first[tid];
      K lb = tid ? last[tid - 1] : K(~K(0));
      if (cb == 0) {
        int before = tid - 2;
        while (before >= 0 && a.counts[before] == 0) --before;
        lb = before >= 0 ? last[before] : K(~K(0));
      }
      if (ct) {
        h = ht - uint32_t(lb == ft);
        if (lb == ft && tid == int(b)) sh.dup = 1;
      }
    }
    const uint32_t ex = block_exclusive_scan<kSmThreads>(h, sh.warp, &u);
    if (tid == int(b)) sh.off[0] = ex;
    __syncthreads();
    pos += sh.off[0];
    if (sh.dup) {  // the block's first key is not the first of its value
      if (tid == 0) hm &= ~1u;
      else --pos;
    }
  }
  for (int i = i0; i < i1; ++i)
    if ((hm >> (i - i0)) & 1u) keys[pos++] = sorted[i];
  if (b == 0 && tid == 0) a.status->n_unique = u;
  if (!bar.sync()) return;

  auto finish = [&](uint32_t m) {  // block 0, one thread: the host's copy of the counts
    if (P > 1) st_relaxed(a.sync + 1, bar.target);
    volatile DevStatus* hs = a.host_status;
    hs->n_unique = u;
    hs->n_octree_nodes = m;
    hs->err = *reinterpret_cast<volatile int32_t*>(&a.status->err);
    hs->err_site = *reinterpret_cast<volatile uint32_t*>(&a.status->err_site);
  };
  if (u < 3) {
    if (b == 0 && tid == 0) {
      a.status->err = RW_ERR_DEGENERATE;
      finish(0);
    }
    return;
  }

  // ---- stages 4 and 5 ----
  const int n = int(u - 1);
  {
    const int total = (n + 31) / 32, cpb = (total + int(P) - 1) / int(P);
    const int end = min((int(b) + 1) * cpb, total);
    for (int ch = int(b) * cpb; ch < end; ch += kSmTreeChunks) {
      tree_tile<K, true, LESS, kSmThreads, kSmTreeChunks, true, false>(
          smem, sh.tree, keys, n, ch * 32, min(kSmTreeChunks, end - ch), &a.status->err,
          a.prefix_n, a.hl, a.hr, a.lc, a.parents, a.edge_count, a.sums);
      __syncthreads();  // the next tile reuses the shared arrays
    }
  }
  if (!bar.sync()) return;

  const int group = tid / kOctThreads, gt = tid % kOctThreads;
  auto gsync = [group] {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(kOctThreads) : "memory");
  };
  // sum over the group's threads (every thread gets it)
  auto group_sum = [&](unsigned long long v) {
    v = warp_sum(v);
    gsync();  // the words' last readers are done
    if (lane == 0) sh.gsum[group][gt >> 5] = v;
    gsync();
    unsigned long long t = 0;
#pragma unroll
    for (int w = 0; w < kOctThreads / 32; ++w) t += sh.gsum[group][w];
    return t;
  };
  const int tiles = (n + int(kOctTile) - 1) / int(kOctTile);
  // ---- stages 6 and 7: offsets, rows, links inside a tile ----
  uint32_t m = 0;
  OctTileShared<K>* osh = reinterpret_cast<OctTileShared<K>*>(smem) + group;
  // (tiles go to the blocks in turn, so that few tiles spread over all SMs)
  for (int t = group * int(P) + int(b); t < tiles; t += int(P) * kSmGroups) {
    unsigned long long v = 0;  // all tiles' rows << 32 | those of the tiles before (below 2^32)
    for (int j = gt; j < tiles; j += kOctThreads) {
      const unsigned long long x = a.sums[j];
      v += x << 32 | (j < t ? x : 0ull);
    }
    v = group_sum(v);
    m = uint32_t(v >> 32);
    const bool fits = uint64_t(m) + 1 <= a.o.capacity;
    if (t == 0 && gt == 0) {
      a.status->n_octree_nodes = m;
      if (!fits) atomicCAS(reinterpret_cast<int*>(&a.status->err), 0, RW_ERR_CAPACITY);
    }
    const OctSeg os{0, a.o.capacity, m, n, true, fits};
    octree_tile<K, true>(*osh, gsync, gt, keys, a.prefix_n, a.parents, a.edge_count,
                         a.edge_offset, os, 0, t * int(kOctTile), [&] { return uint32_t(v); },
                         a.min_coord, a.range, a.o, a.far, a.far_cap, a.far_n);
    gsync();
  }
  if (!bar.sync()) return;

  // ---- links that leave their tile, and the leaves ----
  octree_far_links<K>(keys, a.prefix_n, a.parents, a.edge_count, a.edge_offset,
                      SegTable{1u, a.n, nullptr}, TileMap{uint32_t(tiles), nullptr},
                      &a.status->n_unique, &a.status->n_octree_nodes, &a.status->err, a.o, a.far,
                      a.far_cap, a.far_n);
  if (a.leaves) {
    if (!bar.sync()) return;
    leaf_claim<K>(keys, a.prefix_n, a.hl, a.hr, a.lc, a.parents, a.edge_count, a.edge_offset,
                  a.o.children, &a.status->n_unique, a.o.capacity);
    if (!bar.sync()) return;
    leaf_write(a.lc, a.o.children, &a.status->n_unique, &a.status->n_octree_nodes, a.o.capacity);
  }
  if (b == 0 && tid == 0) finish(m);  // (tile 0 is this thread's)
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

namespace {

// Blocks for n points: one up to where several with their barriers cost the
// same (4,096 points in one block 54 us, 4,200 in three 58), then a block per
// kSmShare points, at most one per SM.
constexpr uint32_t kSmAlone = 4096, kSmShare = 2048;

uint32_t small_blocks(uint32_t n, int sms) {
  if (n <= kSmAlone) return 1;
  return std::min({div_up(n, kSmShare), uint32_t(sms), uint32_t(kSmMaxBlocks)});
}

// Keys of a bucket region: three times the mean and a little, at most what a
// block sorts.
uint32_t small_cap(uint32_t n, uint32_t blocks, int key_bits) {
  const uint32_t most = key_bits == 32 ? SmallCfg<uint32_t>::kCap : SmallCfg<uint64_t>::kCap;
  return std::min(most, 3 * div_up(n, blocks) + 512);
}

// Sample lists per block; 0: the cloud is too large.  A bucket between two
// splitters with 32 samples each holds a mass of standard deviation 0.18 means
// and more than 2.4 means once in 10^7, one with 64 samples 0.125 and more than
// 1.9 once in 10^7.
uint32_t small_lists(uint32_t n, uint32_t blocks, int key_bits) {
  const uint32_t share = div_up(n, blocks), cap = small_cap(n, blocks, key_bits);
  if (share > uint32_t(kSmEncode * kSmThreads)) return 0;
  if (blocks == 1 || 12 * share <= 5 * cap) return 1;
  // (64 samples of every block fit behind a share's keys)
  const uint32_t room = 2u * (key_bits == 32 ? SmallCfg<uint32_t>::kCap : SmallCfg<uint64_t>::kCap);
  return 19 * share <= 10 * cap && share + blocks * 2u * (kSmSamples + 1) <= room ? 2 : 0;
}

template <typename K, int LESS>
cudaError_t small_t(const Bufs& b, SmallArgs a, uint32_t blocks, cudaStream_t s) {
  a.inv_range = pow2_reciprocal(b.range);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = blocks;
  cfg.blockDim = kSmThreads;
  cfg.dynamicSmemBytes = SmallCfg<K>::kSmem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_small<K, LESS>, a);
}

template <typename K>
cudaError_t small_ready(int* per_sm) {
  cudaError_t e = cudaFuncSetAttribute(k_small<K, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(SmallCfg<K>::kSmem));
  if (e == cudaSuccess && sizeof(K) == 4)
    e = cudaFuncSetAttribute(k_small<K, sizeof(K) == 4>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(SmallCfg<K>::kSmem));
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_small<K, 0>, kSmThreads,
                                                      SmallCfg<K>::kSmem);
  return e;
}

}  // namespace

uint32_t small_alone() { return kSmAlone; }

uint32_t small_limit(int key_bits) { return key_bits == 32 ? kSmallLimit32 : kSmallLimit64; }

bool small_takes(uint32_t n, int key_bits, int sms) {
  if (n > small_limit(key_bits)) return false;
  return small_lists(n, small_blocks(n, sms), key_bits) != 0;
}

cudaError_t small_prepare(int key_bits, bool* usable) {
  int per_sm = 0;
  const cudaError_t e =
      key_bits == 32 ? small_ready<uint32_t>(&per_sm) : small_ready<uint64_t>(&per_sm);
  *usable = e == cudaSuccess && per_sm >= 1;
  return e;
}

namespace {
struct SmallLayout {
  size_t samples, splitters, first, last, fill, counts, heads, mat, sums, region, bytes;
};

SmallLayout small_layout(uint32_t n_cap, int key_bits, int sms) {
  const uint32_t n = std::min(n_cap, small_limit(key_bits));
  const size_t ks = key_bits == 32 ? 4 : 8, P = small_blocks(n, sms);
  // blocks * (3 * share + 512) keys, for every cloud of up to n points
  const size_t region = P == 1 ? 0 : 3 * size_t(n) + 515 * P;
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  SmallLayout l{};
  size_t o = 0;
  auto take = [&](size_t bytes) { const size_t at = o; o += up(bytes); return at; };
  l.samples = take(P * 2 * kSmSamples * ks);
  l.splitters = take(P * ks);
  l.first = take(P * ks);
  l.last = take(P * ks);
  l.fill = take(P * 4 * kSmFill);
  l.counts = take(P * 4);
  l.heads = take(P * 4);
  l.mat = take(P * 256 * 4);
  l.sums = take(size_t(div_up(n, kOctTile)) * 4);
  l.region = take(region * ks);
  l.bytes = o;
  return l;
}
}  // namespace

size_t small_scratch_bytes(uint32_t n_cap, int key_bits, int sms) {
  return small_layout(n_cap, key_bits, sms).bytes;
}

cudaError_t launch_small(const Bufs& b, const Scratch& sc, uint32_t n, uint32_t n_cap,
                         uint32_t oct_capacity, bool geometric, bool leaves, char* scratch,
                         uint32_t* sync, DevStatus* host_status, cudaStream_t s) {
  const SmallLayout l = small_layout(n_cap, b.key_bits, sc.num_sms);
  const uint32_t blocks = small_blocks(n, sc.num_sms);
  SmallArgs a{};
  a.points = b.points;
  a.keys = b.keys;
  a.alt = b.alt;
  a.n = n;
  a.chunk = div_up(n, blocks);
  a.cap = small_cap(n, blocks, b.key_bits);
  a.lists = small_lists(n, blocks, b.key_bits);
  if (!small_takes(n, b.key_bits, sc.num_sms) || n > n_cap) return cudaErrorInvalidValue;
  a.min_coord = b.min_coord;
  a.range = b.range;
  a.prefix_n = b.prefix_n;
  a.hl = b.hl;
  a.hr = b.hr;
  a.lc = b.lc;
  a.parents = b.parents;
  a.edge_count = b.edge_count;
  a.edge_offset = b.edge_offset;
  a.o = OctOut{b.children, b.corner, b.cell_size, b.node_mask, b.leaf_mask, nullptr, oct_capacity};
  a.leaves = leaves;
  a.sync = sync;
  a.samples = scratch + l.samples;
  a.splitters = scratch + l.splitters;
  a.first = scratch + l.first;
  a.last = scratch + l.last;
  a.fill = reinterpret_cast<uint32_t*>(scratch + l.fill);
  a.counts = reinterpret_cast<uint32_t*>(scratch + l.counts);
  a.heads = reinterpret_cast<uint32_t*>(scratch + l.heads);
  a.mat = reinterpret_cast<uint32_t*>(scratch + l.mat);
  a.sums = reinterpret_cast<uint32_t*>(scratch + l.sums);
  a.region = scratch + l.region;
  a.tmp = b.tmp;
  a.far = sc.tree_far;
  a.far_cap = sc.tree_far_cap;
  a.far_n = sc.tile_ctr + kCtrLinks;
  a.status = sc.status;
  a.host_status = host_status;
  a.spin_limit = sc.spin_limit;
  a.missing = sc.missing;
  if (a.missing && blocks == 1) return cudaErrorInvalidValue;  // nothing waits
  if (b.key_bits == 64) return small_t<uint64_t, 0>(b, a, blocks, s);
  return geometric ? small_t<uint32_t, 1>(b, a, blocks, s) : small_t<uint32_t, 0>(b, a, blocks, s);
}

}  // namespace rwt
