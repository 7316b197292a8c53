// The end of the 64-bit sort: the keys come sorted by their top bits only.
//
// A 63-bit code takes eight 8-bit passes, but a few million points rarely share
// their first 32 bits (40 bits for more than kSplitPoints points): the passes
// over the low bits (37 us each at 5,000,011 points) are left out, and every
// key of a run that shares its top bits finds its place by counting the run's
// smaller keys (k_sort_fix).  The clouds that this is for have runs of a few
// keys (uniform) or a few tens (mixtures of sigma 4 and more in a box of 1,024;
// the densest places, edges of the box that points were clamped to, grow with
// the cloud to about 130 keys at 2^21 points, hence the line there).  A run
// beyond kFixRun keys that is not in order sets its cloud's flag, and
// k_sort_long, launched behind in any case, sorts the flagged clouds by all
// digits from the unsorted keys.
#include <algorithm>

#include "block_sort.cuh"
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
// is read and written once.  A warp takes 32 keys at a time whose flags "same
// top bits as the key before" are one ballot, and a group without any (nearly
// all of them) is stored as it is; the window comes by one bulk copy: 25.4 us
// at 5,000,011 points (80 MB: 3.2 TB/s), where plain loads took 27.8, looking at
// both neighbours key by key 33.6 and gathering the sorted tile in a second
// buffer 26.1.  The last of two waves of tiles is what is left.
template <typename K>
__global__ void __launch_bounds__(kFixThreads, 6)
    k_sort_fix(const K* __restrict__ in, K* __restrict__ out, uint32_t top, SegTable seg,
               TileMap map,
               uint32_t* __restrict__ heads, uint32_t* __restrict__ long_run,
               DevStatus* __restrict__ st) {
  pdl_enter();
  __shared__ __align__(16) K s_raw[kFixWin + 2];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_warp[kFixThreads / 32];
  uint32_t first;
  const uint32_t c = tile_segment(seg, map, blockIdx.x, &first);
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
  bool far = false;
  uint32_t count = 0;
  // key i, which shares its top bits with a neighbour
  auto place = [&](int i, K k) {
    // a key of the halo matters only if its run reaches into the tile
    if (i < a0 ? !same(s[a0], k) : i >= a1 && !same(s[a1 - 1], k)) return;
    int at = i, l = i - 1, r = i + 1, less = 0;
    bool head = true;
    for (K x; l >= 0 && i - l <= kFixRun && same(x = s[l], k); --l) {
      less += int(uint32_t(x) <= uint32_t(k));
      head &= uint32_t(x) != uint32_t(k);
    }
    for (K x; r < m && r - i <= kFixRun && same(x = s[r], k); ++r)
      less += int(uint32_t(x) < uint32_t(k));
    if (r - l - 1 <= kFixRun) {
      at = l + 1 + less;
    } else if (i > 0 && same(s[i - 1], k)) {
      // every key of a longer run that reaches into the tile sees that it is
      // longer (257 of its keys are in the window): the run stays as it is,
      // which is right if it is in order (copies of one key, say)
      far |= s[i - 1] > k;
      head = s[i - 1] != k;
    }
    if (at >= a0 && at < a1) {
      out[lo + uint32_t(at)] = k;
      count += uint32_t(head);
    }
  };
  if (full) {
    static_assert(kFixRun == kFixThreads, "a halo key per thread");
    const int lane = int(lane_id()), i0 = kFixRun + int(threadIdx.x >> 5) * (kFixTile / kWarps) + lane;
    constexpr int kGroups = kFixTile / kWarps / 32;
    K k = s[i0];
    uint32_t flags = __ballot_sync(0xffffffffu, same(s[i0 - 1], k));
    K* o = out + lo + uint32_t(i0);
#pragma unroll 4
    for (int q = 0; q < kGroups; ++q) {
      const int i = i0 + 32 * q;
      const K nk = s[i + 32];
      const uint32_t nf = __ballot_sync(0xffffffffu, same(s[i + 31], nk));
      const uint32_t either = flags | flags >> 1 | nf << 31;  // same as the key before or after
      if (either == 0) {
        o[32 * q] = k;
        ++count;
      } else if ((either >> lane) & 1u) {
        place(i, k);
      } else {
        o[32 * q] = k;
        ++count;
      }
      k = nk;
      flags = nf;
    }
    if (same(s[a0 - 1], s[a0])) place(int(threadIdx.x), s[threadIdx.x]);
    if (same(s[a1 - 1], s[a1])) place(a1 + int(threadIdx.x), s[a1 + int(threadIdx.x)]);
  } else {
    for (int i = int(threadIdx.x); i < m; i += kFixThreads) place(i, s[i]);
  }
  count = warp_sum(count);
  if (lane_id() == 0) s_warp[threadIdx.x >> 5] = count;
  const bool any = __syncthreads_or(int(far)) != 0;
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kFixThreads / 32; ++w) t += s_warp[w];
    heads[blockIdx.x] = t;
    if (any) long_run[c] = 1u;
  }
}

constexpr int kLongThreads = 1024, kLongKpt = 7;
constexpr int kLongTile = kLongKpt * kSortThreads;

template <typename K>
constexpr size_t long_smem() {
  return 2 * size_t(kLongTile) * sizeof(K) + 2 * size_t(kSortHist) * 4;
}

struct LongArgs {
  const void* keys;
  void *tmp, *alt;
  SegTable seg;
  TileMap map;  // stage 3's tiles
  uint32_t *heads, *long_run, *mat, *sync;
  DevStatus* status;
};

// Sorts the flagged segments by all their digits, keys -> alt, and counts
// their heads: a cooperative launch of up to one block per SM, each block a
// share of the segment, two barriers per digit.  It is for correctness, not
// for speed (about four times the time of the onesweep passes); with no flag
// set it costs its launch.
template <typename K>
__global__ void __launch_bounds__(kLongThreads, 1) k_sort_long(LongArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  K* sa = reinterpret_cast<K*>(smem);
  K* sb = sa + kLongTile;
  uint32_t* hist = reinterpret_cast<uint32_t*>(sb + kLongTile);
  uint32_t* next = hist + kSortHist;
  __shared__ DigitShared sd;
  __shared__ uint32_t s_cnt[256], s_off[256], s_warp[kLongThreads / 32 + 1], s_ok;
  const int tid = int(threadIdx.x);
  bool mine = false;
  for (uint32_t c = uint32_t(tid); c < a.seg.count; c += kLongThreads) mine |= a.long_run[c] != 0;
  if (!__syncthreads_or(int(mine))) return;  // the whole grid: the flags are final
  const uint32_t P = gridDim.x, b = blockIdx.x;
  GridBarrier bar{a.sync, P, 0u, &s_ok, a.sync + 1, a.status, nullptr};
  for (int i = tid; i < 2 * kSortHist / 4; i += kLongThreads)
    reinterpret_cast<uint4*>(hist)[i] = make_uint4(0, 0, 0, 0);
  for (uint32_t c = 0; c < a.seg.count; ++c) {
    if (!a.long_run[c]) continue;
    const uint32_t s0 = seg_begin(a.seg, c), n = seg_size(a.seg, c);
    const uint32_t share = (n + P - 1) / P;
    const uint32_t p0 = min(b * share, n), p1 = min(p0 + share, n);
    constexpr int kDigits = int(sizeof(K));
    static_assert(kDigits % 2 == 0, "the last pass ends in alt");
    for (int q = 0; q < kDigits; ++q) {
      const K* src = static_cast<const K*>(q == 0 ? a.keys : (q & 1) ? a.tmp : a.alt) + s0;
      K* dst = static_cast<K*>((q & 1) ? a.alt : a.tmp) + s0;
      const int shift = 8 * q;
      if (tid < 256) s_cnt[tid] = 0;
      __syncthreads();
      for (uint32_t i = p0 + uint32_t(tid); i < p1; i += kLongThreads)
        atomicAdd(&s_cnt[uint32_t(src[i] >> shift) & 255u], 1u);
      __syncthreads();
      if (tid < 256) a.mat[b * 256 + uint32_t(tid)] = s_cnt[tid];
      if (!bar.sync()) return;
      uint32_t tot = 0, prior = 0, all;
      if (tid < 256)
        for (uint32_t j = 0; j < P; ++j) {
          const uint32_t v = a.mat[j * 256 + uint32_t(tid)];
          prior += j < b ? v : 0u;
          tot += v;
        }
      const uint32_t ex = block_exclusive_scan<kLongThreads>(tot, s_warp, &all);
      if (tid < 256) s_off[tid] = ex + prior;
      for (uint32_t t = p0; t < p1; t += kLongTile) {
        const int cnt = int(min(uint32_t(kLongTile), p1 - t));
        const int steps = (cnt + kSortThreads - 1) / kSortThreads;
        for (int i = tid; i < steps * kSortThreads; i += kLongThreads)
          sa[i] = i < cnt ? src[t + uint32_t(i)] : K(~K(0));
        __syncthreads();
        if (tid < kSortThreads)
          block_digit_pass<K, kLongKpt>(sa, sb, steps, shift, hist, next, sd);
        uint32_t* h = hist;
        hist = next;
        next = h;
        __syncthreads();
        for (int i = tid; i < cnt; i += kLongThreads) {
          const K k = sb[i];
          const uint32_t g = uint32_t(k >> shift) & 255u;
          dst[s_off[g] + uint32_t(i) - sd.start[g]] = k;
        }
        __syncthreads();
        // (the filling counts in the last digit: its end is cnt)
        if (tid < 256) s_off[tid] += (tid < 255 ? sd.start[tid + 1] : uint32_t(cnt)) - sd.start[tid];
      }
      if (!bar.sync()) return;
    }
    // stage 3's counts
    const K* sorted = static_cast<const K*>(a.alt) + s0;
    const uint32_t f0 = a.map.toff ? a.map.toff[c] : 0u;
    const uint32_t tiles = (n + uint32_t(kFixTile) - 1) / uint32_t(kFixTile);
    for (uint32_t t = b; t < tiles; t += P) {
      uint32_t count = 0, sum;
      const uint32_t e = min((t + 1) * uint32_t(kFixTile), n);
      for (uint32_t i = t * uint32_t(kFixTile) + uint32_t(tid); i < e; i += kLongThreads)
        count += uint32_t(i == 0 || sorted[i] != sorted[i - 1]);
      block_exclusive_scan<kLongThreads>(count, s_warp, &sum);
      if (tid == 0) a.heads[f0 + t] = sum;
    }
  }
}

namespace {

template <typename K>
cudaError_t fix_t(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s) {
  // six blocks need nearly all of the SM's shared memory
  cudaError_t e = cudaFuncSetAttribute(k_sort_fix<K>,
                                       cudaFuncAttributePreferredSharedMemoryCarveout,
                                       int(cudaSharedmemCarveoutMaxShared));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sort_long<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(long_smem<K>()));
  if (e != cudaSuccess) return e;
  if (!pl.unique_map.n_tiles) return cudaSuccess;
  const int low = sorted_low_bits(sc);  // at most 32
  const uint32_t top = low < 32 ? ~0u << low : 0u;
  launch_pdl(k_sort_fix<K>, pl.unique_map.n_tiles, kFixThreads, 0, s,
             static_cast<const K*>(b.tmp), static_cast<K*>(b.alt), top, pl.seg, pl.unique_map,
             sc.unique_desc, sc.long_run, sc.status);
  LongArgs a{b.keys, b.tmp, b.alt, pl.seg, pl.unique_map, sc.unique_desc, sc.long_run,
             sc.sort_desc, sc.tile_ctr + kCtrLong, sc.status};
  // the passes' descriptors are free by now: a row of digit counts per block
  const uint64_t rows = uint64_t(sc.passes) * sc.sort_rows;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = uint32_t(std::min<uint64_t>(rows, uint64_t(sc.num_sms)));
  cfg.blockDim = kLongThreads;
  cfg.dynamicSmemBytes = long_smem<K>();
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_sort_long<K>, a);
}

}  // namespace

cudaError_t launch_sort_finish(const Bufs& b, const Scratch& sc, const Plan& pl,
                               cudaStream_t s) {
  if (!sc.low_bits) return cudaSuccess;
  return fix_t<uint64_t>(b, sc, pl, s);
}

}  // namespace rwt
