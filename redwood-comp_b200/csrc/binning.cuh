// One tile of a onesweep pass, shared by the passes (k_keys.cu) and the kernel
// that sorts what they leave (k_sortfix.cu).
#pragma once

#include "rank.cuh"

namespace rwt {

// Descriptors a look-back reads per round trip.
constexpr int kLookback = 8;

template <typename K, int D, int THREADS, int KPT, int RANK>
struct BinCfg {
  static constexpr int RADIX = 1 << D;
  static constexpr int NW = THREADS / 32;
  static constexpr int TILE = THREADS * KPT;
  static constexpr size_t kKeysBytes = size_t(TILE) * sizeof(K);
  // one set of counters per warp; the unordered scheme has one per block
  static constexpr size_t kHistBytes = size_t(RANK == kRankUnordered ? 1 : NW) * RADIX * 4;
  // the two-array scheme keeps a match-mask array beside the counters; the
  // half-warp scheme has two words per digit and warp (one per half-warp)
  static constexpr size_t kMatchBytes =
      (RANK == kRankAtomicOr || RANK == kRankHalfPacked || RANK == kRankMixed) ? kHistBytes : 0;
  static constexpr size_t kSmem =
      kKeysBytes + kHistBytes + kMatchBytes + 3 * size_t(RADIX) * 4 + 64 * 4;
  static_assert(kSmem <= 227 * 1024, "onesweep variant exceeds shared memory per CTA");
};

// Sets a tile's counters to zero (before bin_tile, with a barrier between).
template <typename K, int D, int THREADS, int KPT, int RANK>
__device__ __forceinline__ void bin_zero(unsigned char* smem) {
  using C = BinCfg<K, D, THREADS, KPT, RANK>;
  static_assert(C::RADIX % 4 == 0 && C::kKeysBytes % 16 == 0, "16-byte zeroing");
  const uint4 z = make_uint4(0, 0, 0, 0);
  constexpr int kWords =
      (RANK == kRankAtomicOr || RANK == kRankHalfPacked || RANK == kRankMixed ? 2 : 1) *
      (RANK == kRankUnordered ? 1 : C::NW) * C::RADIX;
  uint4* h = reinterpret_cast<uint4*>(smem + C::kKeysBytes);
  for (int i = int(threadIdx.x); i < kWords / 4; i += THREADS) h[i] = z;
}

// The exclusive prefix of digit d for the tile of descriptor row `row`: the
// decoupled look-back, kLookback descriptors per round trip.  first_row is
// never published but as inclusive, so rows are read clamped to it and the
// walk stops there at the latest.
template <int RADIX>
__device__ __forceinline__ uint32_t look_back(const uint32_t* desc, uint32_t d, int row,
                                              int first_row, uint32_t spin_limit,
                                              DevStatus* st) {
  uint32_t excl = 0;
  int k = row - 1;
  uint32_t spin = 0;
  while (true) {
    uint32_t v[kLookback];
#pragma unroll
    for (int q = 0; q < kLookback; ++q)
      v[q] = ld_relaxed(desc + size_t(max(k - q, first_row)) * RADIX + d);
    int used = 0;
    bool done = false;
#pragma unroll
    for (int q = 0; q < kLookback; ++q) {
      const uint32_t f = v[q] & kFlagMask;
      if (done || f == 0 || used != q) break;
      excl += v[q] >> 2;
      ++used;
      done = f == kFlagInc;
    }
    if (done) break;
    if (used) {
      k -= used;
      spin = 0;
      continue;
    }
    if (++spin > spin_limit || device_failed(st)) {
      report_error(st, RW_ERR_TIMEOUT, kSiteSort);
      break;
    }
    backoff(spin);
  }
  return excl;
}

// Stable counting sort of the tile [base, base + TILE) of keys that end at n by
// the digit (key >> shift) & dmask, into out at the digits' prefixes: publish(d,
// count) as soon as the tile's counts are known, then prefix(d, count) gives
// the place of the tile's first key of digit d.  `off` (block-uniform): the
// tile is not wanted; tested once the keys are on their way.  BB, ballots: see
// warp_rank.  The caller synchronises before the shared memory is used again.
template <typename K, int D, int THREADS, int KPT, int RANK, int BB, typename Publish,
          typename Prefix>
__device__ __forceinline__ void bin_tile(unsigned char* smem, const K* in, K* out, uint32_t base,
                                         uint32_t n, uint32_t total, int shift, uint32_t dmask,
                                         bool ballots, uint32_t off, const Publish& publish,
                                         const Prefix& prefix) {
  using C = BinCfg<K, D, THREADS, KPT, RANK>;
  constexpr int RADIX = C::RADIX, NW = C::NW, TILE = C::TILE;
  K* s_keys = reinterpret_cast<K*>(smem);
  uint32_t* s_hist = reinterpret_cast<uint32_t*>(smem + C::kKeysBytes);
  uint32_t* s_match = s_hist + NW * RADIX;  // only with kRankAtomicOr / kRankMixed
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + C::kKeysBytes + C::kHistBytes +
                                                C::kMatchBytes);
  uint32_t* s_start = s_cnt + RADIX;
  uint32_t* s_gofs = s_start + RADIX;
  uint32_t* s_misc = s_gofs + RADIX;  // [0] the caller's, [1..] warp scan scratch
  const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const bool full = base + TILE <= n;

  // load: warp w owns [w*32*KPT, (w+1)*32*KPT) of the tile, 32 keys per step
  // (half-warp scheme: half h of warp w owns [w*32*KPT + h*16*KPT, +16*KPT),
  // 16 keys per step)
  K keys[KPT];
  uint32_t rank2[RankPack<KPT>::kRegs];  // packed warp ranks
  uint32_t rank16[(KPT + 1) / 2];        // unordered: the block's ranks
  const uint32_t wbase = base + warp * 32u * KPT + lane;
  const uint32_t hbase = base + warp * 32u * KPT + (lane >> 4) * 16u * KPT + (lane & 15u);
  uint32_t* wh = s_hist + warp * RADIX;
  uint32_t* wm = s_match + warp * RADIX;
  uint32_t* wp = s_hist + warp * 2u * RADIX;  // half-warp scheme: [2 RADIX] per warp
  if (sizeof(K) == 8 && off) return;
  if (RANK == kRankUnordered) {
    // any order within a digit will do, so ranks come straight from the
    // block's counters: one shared atomic per key instead of four accesses, a
    // shuffle and two population counts (16.8M 32-bit keys 71.7 -> 55.5 us,
    // 5,000,011 64-bit keys 36.8 -> 30.7)
    static_assert(TILE <= 65536, "16-bit ranks");
    if (full) {
#pragma unroll
      for (int i = 0; i < KPT; ++i) keys[i] = in[wbase + 32u * i];
    } else {
#pragma unroll
      for (int i = 0; i < KPT; ++i) keys[i] = wbase + 32u * i < n ? in[wbase + 32u * i] : K(0);
    }
    if (full) {
#pragma unroll
      for (int i = 0; i < KPT; ++i) {
        const uint32_t dig = uint32_t(keys[i] >> shift) & dmask;
        const uint32_t r = atomicAdd(&s_hist[dig], 1u);
        if (i % 2 == 0) rank16[i / 2] = r;
        else rank16[i / 2] |= r << 16;
      }
    } else {
#pragma unroll
      for (int i = 0; i < KPT; ++i) {
        const uint32_t dig = uint32_t(keys[i] >> shift) & dmask;
        const uint32_t r = wbase + 32u * i < n ? atomicAdd(&s_hist[dig], 1u) : 0u;
        if (i % 2 == 0) rank16[i / 2] = r;
        else rank16[i / 2] |= r << 16;
      }
    }
  } else if (RANK == kRankHalfPacked) {
    if (full) {
#pragma unroll
      for (int i = 0; i < KPT; ++i) keys[i] = in[hbase + 16u * i];
      half_rank<D, KPT, true>(keys, rank2, shift, hbase, n, wp, dmask);
    } else {
#pragma unroll
      for (int i = 0; i < KPT; ++i) {
        const uint32_t idx = hbase + 16u * i;
        keys[i] = idx < n ? in[idx] : K(0);
      }
      half_rank<D, KPT, false>(keys, rank2, shift, hbase, n, wp, dmask);
    }
  } else if (RANK == kRankMixed) {
      if (full) {
#pragma unroll
      for (int i = 0; i < KPT; ++i) keys[i] = in[wbase + 32u * i];
      warp_rank<D, KPT, kRankMixed, true, BB>(keys, rank2, shift, wbase, n, wh, wm, KPT, ballots,
                                              dmask);
    } else {
#pragma unroll
      for (int i = 0; i < KPT; ++i) {
        const uint32_t idx = wbase + 32u * i;
        keys[i] = idx < n ? in[idx] : K(0);
      }
      warp_rank<D, KPT, kRankMixed, false, BB>(keys, rank2, shift, wbase, n, wh, wm, KPT,
                                               ballots, dmask);
    }
  } else if (full) {
#pragma unroll
    for (int i = 0; i < KPT; ++i) keys[i] = in[wbase + 32u * i];
    warp_rank<D, KPT, RANK, true, BB>(keys, rank2, shift, wbase, n, wh, wm, KPT, false, dmask);
  } else {
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      const uint32_t idx = wbase + 32u * i;
      keys[i] = idx < n ? in[idx] : K(0);
    }
    warp_rank<D, KPT, RANK, false, BB>(keys, rank2, shift, wbase, n, wh, wm, KPT, false, dmask);
  }
  __syncthreads();

  // per digit: exclusive scan over warps (half-warps) and publish the tile
  // aggregate
  if (RANK == kRankHalfPacked) {
    // lane pairs own a digit: the even lane its half-warp-0 words, the odd
    // lane its half-warp-1 words (consecutive addresses, no bank conflicts);
    // units run in the order (warp, half), the partner's count by a shuffle
    static_assert((2 * RADIX) % 32 == 0 && THREADS % 32 == 0, "whole warps per pass");
    for (int x = tid; x < 2 * RADIX; x += THREADS) {
      const uint32_t h = uint32_t(x) & 1u;
      uint32_t run = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        uint32_t* p = s_hist + w * 2 * RADIX + x;
        const uint32_t mine = *p >> 16;
        const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
        *p = run + (h ? other : 0u);
        run += mine + other;
      }
      if (!h) {
        s_cnt[x >> 1] = run;
        publish(uint32_t(x >> 1), run);
      }
    }
  } else {
    for (int d = tid; d < RADIX; d += THREADS) {
      uint32_t run = 0;
      if (RANK == kRankUnordered) {
        run = s_hist[d];
      } else {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          const uint32_t c = s_hist[w * RADIX + d];
          s_hist[w * RADIX + d] = run;
          run += c;
        }
      }
      s_cnt[d] = run;
      publish(uint32_t(d), run);
    }
  }
  __syncthreads();
  digit_exclusive_scan<D, THREADS>(s_cnt, s_start, s_misc + 1);
  __syncthreads();
  // fold the digit starts into the per-warp offsets once per tile, so that
  // placing a key below reads one shared-memory word instead of two
  if (RANK == kRankHalfPacked) {
    for (int i = tid; i < 2 * NW * RADIX; i += THREADS)
      s_hist[i] += s_start[(i >> 1) & (RADIX - 1)];
  } else if (RANK != kRankUnordered) {
    for (int i = tid; i < NW * RADIX; i += THREADS) s_hist[i] += s_start[i & (RADIX - 1)];
  }
  if (RANK != kRankUnordered) __syncthreads();

  // reorder the tile by digit in shared memory first: it needs only the
  // tile's own counts, and gives the predecessors time to publish their
  // inclusive prefixes before the look-back below reads them
  if (RANK == kRankUnordered) {
    if (full) {
#pragma unroll
      for (int i = 0; i < KPT; ++i) {
        const uint32_t dig = uint32_t(keys[i] >> shift) & dmask;
        s_keys[s_start[dig] + ((rank16[i / 2] >> (16 * (i % 2))) & 0xffffu)] = keys[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < KPT; ++i)
        if (wbase + 32u * i < n) {
          const uint32_t dig = uint32_t(keys[i] >> shift) & dmask;
          s_keys[s_start[dig] + ((rank16[i / 2] >> (16 * (i % 2))) & 0xffffu)] = keys[i];
        }
    }
  } else if (RANK == kRankHalfPacked) {
    if (full) half_place<D, KPT, true>(keys, rank2, shift, hbase, n, wp, s_keys, dmask);
    else half_place<D, KPT, false>(keys, rank2, shift, hbase, n, wp, s_keys, dmask);
  } else if (full) {
    warp_place<D, KPT, true>(keys, rank2, shift, wbase, n, wh, s_keys, KPT, dmask);
  } else {
    warp_place<D, KPT, false>(keys, rank2, shift, wbase, n, wh, s_keys, KPT, dmask);
  }

  for (int d = tid; d < RADIX; d += THREADS)
    s_gofs[d] = prefix(uint32_t(d), s_cnt[d]) - s_start[d];
  __syncthreads();

  // write runs of equal digits to their global positions (a destination is
  // out of range only if a look-back gave up)
  if (full) {
#pragma unroll 4
    for (int i = 0; i < KPT; ++i) {
      const uint32_t p = tid + uint32_t(i) * THREADS;
      const K k = s_keys[p];
      const uint32_t dst = s_gofs[uint32_t(k >> shift) & dmask] + p;
      if (dst < total) out[dst] = k;
    }
  } else {
    const uint32_t tile_n = n - base;
    for (uint32_t p = tid; p < tile_n; p += THREADS) {
      const K k = s_keys[p];
      const uint32_t dst = s_gofs[uint32_t(k >> shift) & dmask] + p;
      if (dst < total) out[dst] = k;
    }
  }
}

}  // namespace rwt
