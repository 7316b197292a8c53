// The end of the 64-bit sort: the keys come sorted by their top bits only.
//
// A 63-bit code takes eight 8-bit passes, but a few million points rarely share
// their first 32 bits (40 bits for more than kSplitPoints points): the passes
// over the low bits (37 us each at 5,000,011 points) are left out, and every
// key of a run that shares its top bits finds its place by counting the run's
// smaller keys (k_sort_fix).  The clouds that this is for have runs of a few
// keys (uniform) or a few tens (mixtures of sigma 4 and more in a box of 1,024).
//
// Two other kinds of keys go to k_sort_rest, one launch behind:
//   - Segments in which keys mostly share their top bits, as samples taken in
//     stage 1 tell (dense_sample, k_keys.cu): the passes leave such a segment
//     alone, and it is sorted by the digits in which its keys differ, as the
//     passes would without leaving low bits out, in one launch.
//   - Runs of more than kFixRun keys among sparse ones: each is sorted by itself,
//     by the digits left out, by one block.
#include <algorithm>

#include "binning.cuh"
#include "internal.hpp"
#include "morton.cuh"

namespace rwt {

constexpr int kFixThreads = 256;
constexpr int kFixRun = 256;  // keys of a run, at most; the halo of a tile
constexpr int kFixTile = int(kUniqueTile);
constexpr int kFixWin = kFixTile + 2 * kFixRun;

// One tile of 4,096 keys per block, with a halo of kFixRun keys on either side
// inside the segment, so that every run that touches the tile is in the
// window, whole.  Also counts the tile's heads (keys with no equal key before
// them) for stage 3, whose counting pass over the keys it replaces.  Each key
// is read and written once.  A warp takes 32 keys at a time, and a group without
// any that share their top bits (nearly all of them) is stored as it is; the
// others find their run's ends in the window's flags ("same top bits as the key
// before", a bit each).  The window comes by one bulk copy: 25.4 us at 5,000,011
// points, where plain loads took 27.8 and gathering the sorted tile in a second
// buffer 26.1; with the runs' ends from the flags 21.7 (80 MB: 3.7 TB/s), the empty
// launch of k_sort_rest included.  The last of two waves of tiles is what is left.
// Where it is dense, a block's time is what counts: 2,000,000 points in a cube of
// side 24 (runs of 36) took 381 us in all when each key walked its run from
// neighbour to neighbour, 269 now; with 1 % of them in a cube of side 4 447 and 248.
template <typename K>
__global__ void __launch_bounds__(kFixThreads, 6)
    k_sort_fix(const K* __restrict__ in, K* __restrict__ out, uint32_t top, SegTable seg,
               TileMap map, uint32_t* __restrict__ heads, const uint32_t* __restrict__ dense,
               uint2* __restrict__ runs, uint32_t* __restrict__ runs_n, uint32_t runs_cap,
               DevStatus* __restrict__ st) {
  pdl_enter();
  __shared__ __align__(16) K s_raw[kFixWin + 2];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_warp[kFixThreads / 32], s_flag[kFixWin / 32 + 1];
  uint32_t first;
  const uint32_t c = tile_segment(seg, map, blockIdx.x, &first);
  if (dense[c]) return;  // the passes have left it to k_sort_rest
  const uint32_t sb = seg_begin(seg, c), se = sb + seg_size(seg, c);
  const uint32_t t0 = sb + (blockIdx.x - first) * uint32_t(kFixTile);
  const uint32_t t1 = min(t0 + uint32_t(kFixTile), se);
  const uint32_t lo = t0 - min(uint32_t(kFixRun), t0 - sb);
  const uint32_t hi = min(t1 + uint32_t(kFixRun), se);
  const int m = int(hi - lo), a0 = int(t0 - lo), a1 = int(t1 - lo);
  constexpr int kWarps = kFixThreads / 32;
  // the window, sorted by the top bits: a full one by a bulk copy from the
  // 16-byte boundary at or below it, with the last key by itself where that is
  // one key early
  static_assert(kFixWin * sizeof(K) % 16 == 0, "bulk copies move 16-byte units");
  const bool full = m == kFixWin;
  const int early = full ? int((reinterpret_cast<uintptr_t>(in + lo) & 15u) / sizeof(K)) : 0;
  K* s = s_raw + early;
  if (full) {
    if (threadIdx.x == 0) bulk_barrier_init(&s_bar);
    __syncthreads();
    if (threadIdx.x == 0) {
      bulk_load(s_raw, in + lo - early, uint32_t(kFixWin * sizeof(K)), &s_bar);
      if (early) s_raw[kFixWin] = in[lo + kFixWin - 1];
    }
    const bool landed = bulk_wait(&s_bar, kSpinLimit);
    if (__syncthreads_or(!landed)) {  // the whole block gives up together
      // report, and let the copy land before the block's shared memory goes
      if (threadIdx.x == 0) report_error(st, RW_ERR_TIMEOUT, kSiteSort);
      bulk_wait(&s_bar, kSpinLimit);
      return;
    }
  } else {
    for (int i = int(threadIdx.x); i < m; i += kFixThreads) s[i] = in[lo + uint32_t(i)];
  }
  __syncthreads();
  // equal top bits: the upper words and the bits of `top` in the lower one
  static_assert(sizeof(K) == 8, "the bits left out lie in the lower word");
  auto same = [top](K x, K y) {
    return uint32_t(x >> 32) == uint32_t(y >> 32) && ((uint32_t(x) ^ uint32_t(y)) & top) == 0;
  };
  // bit i of the flags: key i shares its top bits with the key before it
  const int lane = int(lane_id()), warp = int(threadIdx.x >> 5);
  const int groups = (m + 31) / 32;
  for (int g = warp; g < groups; g += kWarps) {
    const int i = 32 * g + lane;
    const uint32_t w = __ballot_sync(0xffffffffu, i > 0 && i < m && same(s[max(i - 1, 0)], s[i]));
    if (lane == 0) s_flag[g] = w;
  }
  if (threadIdx.x == 0) s_flag[groups] = 0;
  __syncthreads();
  auto flag = [&](int i) { return i < m && ((s_flag[i >> 5] >> (i & 31)) & 1u); };
  // a key of the halo matters only if its run reaches into the tile
  const int g0 = flag(a0) ? 0 : a0 / 32, g1 = flag(a1) ? groups : (a1 + 31) / 32;
  const uint32_t upto = (2u << lane) - 1u;  // the lanes up to this one
  uint32_t count = 0;
#pragma unroll 2
  for (int g = g0 + warp; g < g1; g += kWarps) {
    const uint32_t word = s_flag[g], next = s_flag[g + 1];
    const int i = 32 * g + lane;
    const uint32_t either = word | word >> 1 | next << 31;  // same as the key before or after
    if (i >= m) continue;
    const K k = s[i];
    int at = i;
    bool head = true;
    if ((either >> lane) & 1u) {
      // the run [l, r), at most nine words of flags to either side
      int l, r, q = g;
      uint32_t z = ~word & upto;
      while (!z && q > g - 9) z = ~s_flag[--q];
      l = z ? 32 * q + 31 - __clz(z) : 32 * q;
      z = ~word & ~upto;
      q = g;
      while (!z && q < g + 9) z = ~s_flag[++q];
      r = z ? 32 * q + __ffs(z) - 1 : 32 * q + 32;
      if (i < a0 ? r <= a0 : i >= a1 && l >= a1) continue;
      if (r - l > kFixRun) {
        // every key of a longer run that reaches into the tile sees that it is
        // longer (257 of its keys are in the window); the tile where it starts
        // enters it in the list
        if (l == i && i >= a0 && i < a1) {
          const uint32_t e = atomicAdd(runs_n, 1u);
          if (e < runs_cap) runs[e] = make_uint2(lo + uint32_t(i), blockIdx.x);
        }
        continue;
      }
      // (with the ends known, and the same for all lanes of a run, the loads of the
      // loop are in flight together)
      const uint32_t* w = reinterpret_cast<const uint32_t*>(s);  // the lower words
      const uint32_t kw = uint32_t(k);
      int less = 0, most = 0;
#pragma unroll 8
      for (int j = l; j < r; ++j) {
        const uint32_t x = w[2 * j];
        less += int(x < kw);
        most += int(x <= kw);
      }
      if (most - less > 1) {  // copies: in the order in which they stand
        const int first_copy = less;
        for (int j = l; j < i; ++j) less += int(w[2 * j] == kw);
        head = less == first_copy;
      }
      at = l + less;
    }
    if (at >= a0 && at < a1) {
      out[lo + uint32_t(at)] = k;
      count += uint32_t(head);
    }
  }
  count = warp_sum(count);
  if (lane_id() == 0) s_warp[threadIdx.x >> 5] = count;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kFixThreads / 32; ++w) t += s_warp[w];
    heads[blockIdx.x] = t;
  }
}

// Tiles of 4,096 keys; a tile's ranking goes by ballots where its first digit
// holds a quarter of the segment's keys (in a dense segment the top digits are
// skewed, which serialises the atomics), and a digit that all keys share is left
// out.
constexpr int kRestThreads = 256, kRestKpt = 16, kRestBlocks = 4;
constexpr int kRestTile = kRestThreads * kRestKpt;
constexpr int kRestDigits = 8, kRestHistTiles = 4;
static_assert(kRestTile == int(kUniqueTile) && kRestTile == kFixTile, "stage 3's tiles");
// zero, histogram, which digits, passes (one more for a copy), heads
enum : int { kPhaseZero = 0, kPhaseHist = 1, kPhasePlan = 2, kPhasePass = 3,
             kPhaseHeads = kPhasePass + kRestDigits + 1, kPhases };
static_assert(kRestWords >= kRestTickets + 2 * kPhases, "counters of the phases");

struct RestArgs {
  const void* keys;
  void *tmp, *alt;
  SegTable seg;
  TileMap map;
  const uint32_t* dense;
  uint32_t *heads, *desc, *hist, *ctr;
  uint32_t* digits;  // [segments]: the digits that differ, a bit each
  const uint2* runs;
  uint32_t runs_cap, top;
  int low;
  uint32_t spin_limit, missing;
  DevStatus* status;
};

// One run of keys [r0, r1) with equal top bits, out of order in tmp: sorted by the
// digits of its low bits (stable passes by one block, tmp -> alt -> tmp ..), and
// its heads added to their tiles'.
template <typename K>
__device__ __forceinline__ void sort_run(const RestArgs& a, unsigned char* smem, uint32_t* s_base,
                                         uint32_t r0, uint32_t r1, uint32_t sb, uint32_t first) {
  using C = BinCfg<K, 8, kRestThreads, kRestKpt, kRankMixed>;
  const int tid = int(threadIdx.x);
  uint32_t* s_cnt = s_base + 256;
  uint32_t* s_warp = s_base + 512;
  K* buf[2] = {static_cast<K*>(a.tmp), static_cast<K*>(a.alt)};
  const int digits = (a.low + 7) / 8;
  for (int q = 0; q < digits; ++q) {
    const K* src = buf[q & 1];
    K* dst = buf[~q & 1];
    s_cnt[tid] = 0;
    __syncthreads();
    for (uint32_t t = r0 + uint32_t(tid); t < r1; t += 8 * kRestThreads) {
      uint32_t d[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t i = t + uint32_t(j) * kRestThreads;
        d[j] = i < r1 ? uint32_t(src[i] >> (8 * q)) & 255u : 256u;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (d[j] < 256u) atomicAdd(&s_cnt[d[j]], 1u);
    }
    __syncthreads();
    digit_exclusive_scan<8, kRestThreads>(s_cnt, s_base, s_warp);
    for (uint32_t t = r0; t < r1; t += uint32_t(kRestTile)) {
      bin_zero<K, 8, kRestThreads, kRestKpt, kRankMixed>(smem);
      __syncthreads();
      bin_tile<K, 8, kRestThreads, kRestKpt, kRankMixed, 8>(
          smem, src, dst, t, r1, a.seg.total, 8 * q, 255u, false, 0u, [](uint32_t, uint32_t) {},
          [&](uint32_t d, uint32_t count) {
            const uint32_t at = s_base[d];
            s_base[d] = at + count;
            return r0 + at;
          });
      __syncthreads();
    }
  }
  const K* src = buf[digits & 1];
  K* alt = buf[1];
  // 32 keys at a time that lie in one tile of stage 3
  const uint32_t g0 = (r0 - sb) & ~31u;
  for (uint32_t g = g0 + uint32_t(tid); g < ((r1 - sb + 31u) & ~31u); g += kRestThreads) {
    const uint32_t i = sb + g;
    bool head = false;
    if (i >= r0 && i < r1) {
      const K k = src[i];
      head = i == r0 || src[i - 1] != k;
      if (src != alt) alt[i] = k;
    }
    const uint32_t m = __ballot_sync(0xffffffffu, head);
    if (m && lane_id() == 0) atomicAdd(a.heads + first + g / uint32_t(kFixTile), uint32_t(__popc(m)));
  }
  __syncthreads();
  static_assert(C::TILE == kRestTile, "bin_tile's tile");
}

// What the passes and k_sort_fix have left: the listed runs, then the dense
// segments' keys -> alt by all digits, with their head counts.
//
// The steps of a dense segment (zero, histogram, passes, heads) are phases
// of jobs that blocks take by ticket; a block that has a job of a phase waits
// until every job of the phase before is done, and a tile's look-back for the
// tiles before it.  Both wait only for jobs with earlier tickets, whose blocks are
// running, so the launch needs no more blocks than happen to run.  Waits are
// bounded (RW_ERR_TIMEOUT).
//
// Whole calls, 64-bit keys in a cube of side 2 (all dense), with eight onesweep
// passes, with the sorted top bits first and then everything again, and now:
// 2,000,000 points 310, 1,629 and 295 us, 5,000,011 points 545, 2,332 and 579;
// 256 clouds of 30,000 points 872 us, 23.8 ms and 808 us.  Four blocks per SM with
// 64 registers: with three and 80 5,000,011 points took 544 us, but 2,000,000
// (488 tiles, then more than a wave) 316.
template <typename K>
__global__ void __launch_bounds__(kRestThreads, kRestBlocks) k_sort_rest(const RestArgs a) {
  pdl_enter();
  const uint32_t listed = min(a.ctr[kRestRuns], a.runs_cap), dense_n = a.ctr[kRestDense];
  if (listed == 0 && dense_n == 0) return;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t s_base[512 + kRestThreads / 32 + 1], s_job, s_end;
  const int tid = int(threadIdx.x);
  K* const keys = static_cast<K*>(const_cast<void*>(a.keys));
  K* const tmp = static_cast<K*>(a.tmp);
  K* const alt = static_cast<K*>(a.alt);

  for (uint32_t e = blockIdx.x; e < listed; e += gridDim.x) {
    const uint2 run = a.runs[e];
    uint32_t first;
    const uint32_t c = tile_segment(a.seg, a.map, run.y, &first);
    const uint32_t sb = seg_begin(a.seg, c), se = sb + seg_size(a.seg, c);
    // the run's end: 256 probes 16 keys apart at a time, then key by key
    const K k = tmp[run.x];
    auto same = [&](uint32_t i) {
      const K x = tmp[i];
      return uint32_t(x >> 32) == uint32_t(k >> 32) && ((uint32_t(x) ^ uint32_t(k)) & a.top) == 0;
    };
    uint32_t from = run.x;
    for (;; from += 16 * kRestThreads) {
      const uint32_t i = from + 16 * uint32_t(tid);
      if (tid == 0) s_end = ~0u;
      __syncthreads();
      if (i >= se || !same(i)) atomicMin(&s_end, i);
      __syncthreads();
      if (s_end != ~0u) break;
      __syncthreads();
    }
    const uint32_t beyond = s_end;  // not of the run, the key 16 before it is
    __syncthreads();
    if (tid == 0) s_end = min(beyond, se);
    __syncthreads();
    if (tid < 16) {
      const uint32_t i = beyond - 16 + uint32_t(tid);
      if (i >= se || !same(i)) atomicMin(&s_end, i);
    }
    __syncthreads();
    const uint32_t end = s_end;
    sort_run<K>(a, smem, s_base, run.x, end, sb, first);
  }
  if (dense_n == 0) return;

  const uint32_t tiles = a.map.n_tiles;
  uint32_t* tickets = a.ctr + kRestTickets;
  uint32_t* done = tickets + kPhases;
  auto jobs_of = [&](int ph) {
    return ph == kPhaseHist   ? (tiles + kRestHistTiles - 1) / kRestHistTiles
           : ph == kPhasePlan ? a.seg.count
                              : tiles;
  };
  // waits until all jobs of a phase are done (block-uniform: false if it gave up)
  auto wait = [&](int ph) {
    __syncthreads();  // the last wait's answer has been read
    if (tid == 0) {
      s_end = 1u;
      for (uint32_t spin = 0; ld_acquire(done + ph) != jobs_of(ph) + a.missing;) {
        if (++spin > a.spin_limit || device_failed(a.status)) {
          report_error(a.status, RW_ERR_TIMEOUT, kSiteSort);
          s_end = 0u;
          break;
        }
        backoff(spin);
      }
    }
    __syncthreads();
    return s_end != 0u;
  };
  // passes over a segment in which `digits` of its digits differ: in place an even
  // number (the last one a copy), so that the first leaves the keys alone
  auto passes_of = [&](uint32_t digits) {
    return keys == alt ? (digits + 1u) & ~1u : max(digits, 1u);
  };
  auto histogram = [&](uint32_t job) {
    // digit counts of four tiles, added to their segments'
    uint32_t* h = reinterpret_cast<uint32_t*>(smem);
    uint32_t cur = ~0u;
    auto flush = [&] {
      __syncthreads();
      for (int i = tid; i < kRestDigits * 256; i += kRestThreads) {
        const uint32_t v = h[i];
        if (v) atomicAdd(a.hist + size_t(cur) * kRestDigits * 256 + uint32_t(i), v);
      }
      __syncthreads();
    };
    for (uint32_t t = job * kRestHistTiles; t < min((job + 1) * kRestHistTiles, tiles); ++t) {
      uint32_t first;
      const uint32_t c = tile_segment(a.seg, a.map, t, &first);
      if (!a.dense[c]) continue;
      if (c != cur) {
        if (cur != ~0u) flush();
        for (int i = tid; i < kRestDigits * 256; i += kRestThreads) h[i] = 0;
        __syncthreads();
        cur = c;
      }
      const uint32_t sb = seg_begin(a.seg, c), t0 = sb + (t - first) * uint32_t(kRestTile);
      const uint32_t t1 = min(t0 + uint32_t(kRestTile), sb + seg_size(a.seg, c));
      for (uint32_t r = t0 + (uint32_t(tid) & ~31u); r < t1; r += 4 * kRestThreads) {
        K k[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t i = r + uint32_t(j) * kRestThreads + lane_id();
          k[j] = i < t1 ? keys[i] : K(0);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t i0 = r + uint32_t(j) * kRestThreads;
          if (i0 + 32u <= t1) {
            // the upper digits are often the whole warp's
            const uint32_t up = uint32_t(k[j] >> 32);
            const uint32_t diff = __reduce_or_sync(0xffffffffu, up) ^
                                  __reduce_and_sync(0xffffffffu, up);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              atomicAdd(&h[256 * q + int(uint32_t(k[j] >> (8 * q)) & 255u)], 1u);
              uint32_t* hu = &h[256 * (q + 4) + int((up >> (8 * q)) & 255u)];
              if ((diff >> (8 * q)) & 255u) atomicAdd(hu, 1u);
              else if (lane_id() == 0) atomicAdd(hu, 32u);
            }
          } else if (i0 + lane_id() < t1) {
#pragma unroll
            for (int q = 0; q < kRestDigits; ++q)
              atomicAdd(&h[256 * q + int(uint32_t(k[j] >> (8 * q)) & 255u)], 1u);
          }
        }
      }
    }
    if (cur != ~0u) flush();
  };
  auto pass = [&](uint32_t j, uint32_t job, uint32_t c, uint32_t first, uint32_t sb, uint32_t n) {
    const uint32_t mask = a.digits[c], digits = uint32_t(__popc(mask)), steps = passes_of(digits);
    if (j >= steps) return;
    // the last pass ends in alt
    const K* src = j == 0 ? keys : ((steps - j) & 1u) ? tmp : alt;
    K* dst = ((steps - j) & 1u) ? alt : tmp;
    const uint32_t t0 = sb + (job - first) * uint32_t(kRestTile);
    // two sets of descriptor rows: a pass clears what the next one uses
    uint32_t* desc = a.desc + size_t(j & 1u) * tiles * 256;
    a.desc[(size_t(~j & 1u) * tiles + job) * 256 + uint32_t(tid)] = 0;
    if (j >= digits) {
      const uint32_t t1 = min(t0 + uint32_t(kRestTile), sb + n);
      for (uint32_t i = t0 + uint32_t(tid); i < t1; i += kRestThreads) dst[i] = src[i];
      return;
    }
    uint32_t rest = mask;
    for (uint32_t q = 0; q < j; ++q) rest &= rest - 1u;
    const int p = __ffs(rest) - 1;
    const uint32_t* dh = a.hist + (size_t(c) * kRestDigits + size_t(p)) * 256;
    const bool ballots = dh[uint32_t(src[t0] >> (8 * p)) & 255u] > n / 4u;
    const bool head = job == first;
    if (head) {  // where the segment's digits begin
      s_base[256 + tid] = dh[tid];
      __syncthreads();
      digit_exclusive_scan<8, kRestThreads>(s_base + 256, s_base, s_base + 512);
    }
    bin_zero<K, 8, kRestThreads, kRestKpt, kRankMixed>(smem);
    __syncthreads();
    uint32_t* drow = desc + size_t(job) * 256;
    bin_tile<K, 8, kRestThreads, kRestKpt, kRankMixed, 8>(
        smem, src, dst, t0, sb + n, a.seg.total, 8 * p, 255u, ballots, 0u,
        [&](uint32_t d, uint32_t count) {
          if (!head) st_relaxed(drow + d, kFlagAgg | (count << 2));
        },
        [&](uint32_t d, uint32_t count) {
          const uint32_t excl = head ? sb + s_base[d]
                                     : look_back<256>(desc, d, int(job), int(first), a.spin_limit,
                                                      a.status);
          st_relaxed(drow + d, kFlagInc | ((excl + count) << 2));
          return excl;
        });
  };
  uint32_t passes = 0;
  for (int ph = 0, before = -1; ph < kPhases; ++ph) {
    if (ph >= kPhasePass && ph < kPhaseHeads && uint32_t(ph - kPhasePass) >= passes) continue;
    const uint32_t jobs = jobs_of(ph);
    bool waited = before < 0;
    for (;;) {
      __syncthreads();  // the last job is finished with the shared memory
      if (tid == 0) s_job = atomicAdd(tickets + ph, 1u);
      __syncthreads();
      const uint32_t job = s_job;
      if (job >= jobs) break;
      if (!waited && !wait(before)) return;
      waited = true;
      if (ph == kPhaseHist) {
        histogram(job);
      } else if (ph == kPhasePlan) {
        const uint32_t n = seg_size(a.seg, job);
        if (a.dense[job]) {
          uint32_t mask = 0;
#pragma unroll
          for (int q = 0; q < kRestDigits; ++q) {
            const uint32_t v = a.hist[(size_t(job) * kRestDigits + size_t(q)) * 256 + size_t(tid)];
            mask |= uint32_t(!__syncthreads_or(v == n)) << q;
          }
          if (tid == 0) {
            a.digits[job] = mask;
            atomicMax(a.ctr + kRestPasses, passes_of(uint32_t(__popc(mask))));
          }
        }
      } else {
        uint32_t first;
        const uint32_t c = tile_segment(a.seg, a.map, job, &first);
        if (a.dense[c]) {
          const uint32_t sb = seg_begin(a.seg, c), n = seg_size(a.seg, c);
          if (ph == kPhaseZero) {
            a.desc[size_t(job) * 256 + size_t(tid)] = 0;
            a.desc[(size_t(tiles) + job) * 256 + size_t(tid)] = 0;
            if (job == first)
              for (int i = tid; i < kRestDigits * 256; i += kRestThreads)
                a.hist[size_t(c) * kRestDigits * 256 + size_t(i)] = 0;
          } else if (ph == kPhaseHeads) {
            const uint32_t t0 = sb + (job - first) * uint32_t(kRestTile);
            const uint32_t t1 = min(t0 + uint32_t(kRestTile), sb + n);
            uint32_t count = 0, sum;
            for (uint32_t i = t0 + uint32_t(tid); i < t1; i += kRestThreads)
              count += uint32_t(i == sb || alt[i] != alt[i - 1]);
            block_exclusive_scan<kRestThreads>(count, s_base, &sum);
            if (tid == 0) a.heads[job] = sum;
          } else {
            pass(uint32_t(ph - kPhasePass), job, c, first, sb, n);
          }
        }
      }
      __syncthreads();
      if (tid == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(done + ph) : "memory");
    }
    if (ph == kPhasePlan) {  // the most passes of any segment
      if (!waited && !wait(before)) return;
      if (!wait(ph)) return;
      passes = ld_relaxed(a.ctr + kRestPasses);
    }
    before = ph;
  }
}

namespace {

template <typename K>
cudaError_t fix_t(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s) {
  constexpr size_t smem = BinCfg<K, 8, kRestThreads, kRestKpt, kRankMixed>::kSmem;
  // six blocks need nearly all of the SM's shared memory
  cudaError_t e = cudaFuncSetAttribute(k_sort_fix<K>,
                                       cudaFuncAttributePreferredSharedMemoryCarveout,
                                       int(cudaSharedmemCarveoutMaxShared));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sort_rest<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(smem));
  if (e != cudaSuccess) return e;
  const uint32_t tiles = pl.unique_map.n_tiles;
  if (!tiles) return cudaSuccess;
  // two sets of rows in the descriptors of the passes, which are done
  if (2ull * tiles > uint64_t(sc.passes) * sc.sort_rows) return cudaErrorInvalidValue;
  const int low = sorted_low_bits(sc);  // at most 32
  const uint32_t top = low < 32 ? ~0u << low : 0u;
  uint2* runs = reinterpret_cast<uint2*>(sc.rest + size_t(pl.seg.count) * kRestDigits * 256);
  const uint32_t cap = rest_runs(pl.seg.total);
  uint32_t* digits = reinterpret_cast<uint32_t*>(runs + cap);
  launch_pdl(k_sort_fix<K>, tiles, kFixThreads, 0, s, static_cast<const K*>(b.tmp),
             static_cast<K*>(b.alt), top, pl.seg, pl.unique_map, sc.unique_desc,
             static_cast<const uint32_t*>(sc.dense), runs, sc.rest_ctr + kRestRuns, cap,
             sc.status);
  RestArgs a{b.keys,   b.tmp,       b.alt,   pl.seg, pl.unique_map, sc.dense, sc.unique_desc,
             sc.sort_desc, sc.rest, sc.rest_ctr, digits, runs, cap, top, low, sc.spin_limit,
             sc.missing, sc.status};
  launch_pdl(k_sort_rest<K>, std::min(tiles, uint32_t(sc.num_sms) * kRestBlocks), kRestThreads,
             smem, s, a);
  return cudaGetLastError();
}

}  // namespace

size_t rest_words(uint32_t segments, uint32_t n) {
  return size_t(segments) * (kRestDigits * 256 + 1) + 2 * size_t(rest_runs(n));
}

cudaError_t launch_sort_finish(const Bufs& b, const Scratch& sc, const Plan& pl,
                               cudaStream_t s) {
  if (!sc.low_bits) return cudaSuccess;
  return fix_t<uint64_t>(b, sc, pl, s);
}

}  // namespace rwt
