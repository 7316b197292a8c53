// Stage 1 (Morton encode) and stage 2 (onesweep LSD radix sort).
//
// Stage 1 follows apps/tree/cuda/01_morton.cu:8-19 (per-point
// xyz_to_morton32); in the fused pipeline it also builds the sort's digit
// histograms for every pass while the keys are in registers, which removes the
// reference's separate k_GlobalHistogram read of the keys
// (cu_dispatcher.cu:82-170).
//
// Stage 2 replaces k_GlobalHistogram / k_Scan / 4 x k_DigitBinningPass
// (cu_dispatcher.cu:82-468,528-591) with a onesweep sort designed for 148 SMs:
// one CTA per tile (grid = number of tiles, not 16), tiles handed out by an
// atomic ticket so that every look-back waits only on tiles already running,
// per-warp stable ranking (shared-memory atomic-OR peer masks by default;
// ballot multi-split and match.any in the variant menu; the first pass of keys
// alone need not be stable and ranks by the block's counters), the tile reordered by
// digit in shared memory, and a per-digit decoupled look-back.  Digit width is
// 8, 10 or 11 bits; 32-bit keys take 4, 3 or 3 passes, 64-bit keys 4 or 5 (the
// low bits are put in order afterwards, k_sortfix.cu), 7 or 6.  The
// default 32-bit variant (384 threads x 24 keys) runs three blocks per SM.
#include <algorithm>

#include "binning.cuh"
#include "internal.hpp"
#include "morton.cuh"

namespace rwt {

// ---------------------------------------------------------------------------
// stage 1
// ---------------------------------------------------------------------------

// Digit of pass p of the sort: its lowest bit and its mask.  CODES: the keys are
// codes that stage 1 has just made, else a caller's, of which every bit of the
// word may be set.  30-bit codes with 8-bit digits take 8, 8, 7 and 7 bits instead
// of a word's 8, 8, 8 and 8: the top six bits (a quarter of the box per axis) of a
// clustered cloud put many lanes of a warp on one counter, the top seven half as
// many (16.8M mixture points, last two passes 163.8 -> 155.5 us; uniform ones
// 133.9 -> 134.7).
template <typename K, int D, bool CODES>
__host__ __device__ constexpr int pass_shift(int p) {
  return CODES && sizeof(K) == 4 && D == 8 && p == 3 ? 23 : p * D;
}
template <typename K, int D, bool CODES>
__host__ __device__ constexpr uint32_t pass_mask(int p) {
  return CODES && sizeof(K) == 4 && D == 8 && p == 2 ? 0x7fu : (1u << D) - 1u;
}

// Keys that share their top bits are counted against one another at the end of a
// sort that leaves low bits out (k_sort_fix), in time proportional to their
// number.  Segments where a key shares them with kDenseRun - 1 others on average
// take all digits instead: of 2,000,000 points, runs of 36 keys take 269 us by
// counting and 293 by all digits, runs of 9 keys 238 and 293.  That is decided from samples, which blocks of stage
// 1 take beside their others (in a block of k_sort_init they were 10 us that all
// waited for): of S keys, S^2 / 2 * r / n pairs share their top bits when a key's
// run has r keys on average.  The keys are those at random places, not every
// (n / S)-th: neighbours in the input may be neighbours in space.  Sorted either
// way the result is the same; a sample that misses costs time only.
constexpr int kDenseMost = 1024;  // samples of a block
constexpr uint32_t kDenseRun = 48, kDenseFrom = 4096;

// Enough for about 50 pairs at the line, in as little of the block's time as may be:
// a batch of 1,000 clouds of 6,000 points takes 502 us without samples, 528 with
// 1,024 of each cloud and 514 with 256 (256 clouds of 30,000: 558, 577, 574).
__device__ __forceinline__ uint32_t dense_samples_log2(uint32_t n) {
  return n <= (1u << 15) ? 8u : n <= (1u << 17) ? 9u : 10u;
}
__host__ __device__ __forceinline__ uint32_t dense_blocks(uint32_t segments) {
  return segments == 1 ? 4u : 1u;  // per segment
}
__device__ __forceinline__ bool is_dense(uint32_t pairs, uint32_t n, uint32_t segments) {
  const unsigned long long all = 1ull << (2u * dense_samples_log2(n) - 1u);
  return n > kDenseFrom && pairs > 2 &&
         pairs * (unsigned long long)n > kDenseRun * all * dense_blocks(segments);
}

// One block's samples: the pairs among them of n keys, which key(i) gives without
// their low bits, added to *pairs.
template <typename KeyAt>
__device__ __forceinline__ void dense_sample(uint32_t n, const KeyAt& key, uint32_t* pairs) {
  // a slot: the top bits (41 at most) << 20 | how many samples had them
  __shared__ unsigned long long s_slot[2 * kDenseMost];
  if (n <= kDenseFrom) return;
  const uint32_t log2s = dense_samples_log2(n), slots = 2u << log2s;
  const int each = int((1u << log2s) / 256u);  // a thread's samples
  uint64_t k[kDenseMost / 256];
#pragma unroll
  for (int q = 0; q < kDenseMost / 256; ++q) {
    if (q >= each) break;
    uint32_t x = (blockIdx.x * kDenseMost + 256u * q + threadIdx.x) * 0x9e3779b9u + n;
    x = (x ^ (x >> 16)) * 0x85ebca6bu;  // murmur3's finisher
    x = (x ^ (x >> 13)) * 0xc2b2ae35u;
    k[q] = key(__umulhi(x ^ (x >> 16), n));
  }
  for (uint32_t i = threadIdx.x; i < slots; i += 256) s_slot[i] = 0;
  __syncthreads();
  uint32_t found = 0;
#pragma unroll
  for (int q = 0; q < kDenseMost / 256; ++q) {
    if (q >= each) break;
    const unsigned long long top = (unsigned long long)k[q] << 20;
    uint32_t at = uint32_t((k[q] * 0x9e3779b97f4a7c15ull) >> (63u - log2s));
    for (uint32_t probe = 0; probe < slots; ++probe, at = (at + 1) & (slots - 1u)) {
      unsigned long long old = s_slot[at];
      if (old == 0) old = atomicCAS(&s_slot[at], 0ull, top | 1ull);
      if (old == 0) break;
      if ((old ^ top) >> 20 == 0) {
        found += atomicAdd(reinterpret_cast<uint32_t*>(&s_slot[at]), 1u) & 0xfffffu;
        break;
      }
    }
  }
  found = warp_sum(found);
  if (lane_id() == 0 && found) atomicAdd(pairs, found);
}

// Points are walked in tiles of kPointTile that never straddle two segments;
// each CTA takes a contiguous run of tiles, so with HIST its shared-memory
// histograms are flushed to the segment's global ones only when the segment
// changes.  ghist: [segments][passes][RADIX].
// LOW: the low bits that the sort's passes leave out; then the first blocks
// (dense_blocks per segment) take samples, if pairs [segments] is given.
template <typename K, int D, int LOW, bool HIST, bool ENCODE, bool POW2>
__global__ void __launch_bounds__(256)
    k_keys_pass(const float4* __restrict__ pts, K* __restrict__ keys, SegTable seg,
                TileMap map, uint32_t tiles_per_cta, float min_coord, float range,
                float inv_range, uint32_t* __restrict__ ghist,
                const uint32_t* __restrict__ gate, uint32_t* __restrict__ pairs) {
  pdl_enter();
  if (gate && *gate == 0) return;  // a gated sort that is not needed this run
  uint32_t block = blockIdx.x;
  if constexpr (HIST && LOW > 0) {
    const uint32_t per = pairs ? dense_blocks(seg.count) : 0u;
    if (block < per * seg.count) {
      const uint32_t c = block / per, sb = seg_begin(seg, c);
      dense_sample(seg_size(seg, c), [&](uint32_t i) -> uint64_t {
        if constexpr (ENCODE) {
          const float4 p = pts[sb + i];
          return encode<K, POW2>(p.x, p.y, p.z, min_coord, range, inv_range) >> LOW;
        } else {
          return keys[sb + i] >> LOW;
        }
      }, pairs + c);
      return;
    }
    block -= per * seg.count;
  }
  constexpr int RADIX = 1 << D;
  // the sort's passes: ceil(sorted bits / D), as the storage computes them
  constexpr int P = (KeyTraits<K>::kCodeBits - LOW + D - 1) / D;
  extern __shared__ uint32_t s_hist[];  // [P][RADIX] when HIST
  const int nh = P * RADIX;
  if (HIST) {
    for (int i = threadIdx.x; i < nh; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
  }
  const uint32_t t0 = block * tiles_per_cta;
  const uint32_t t1 = min(t0 + tiles_per_cta, map.n_tiles);
  uint32_t cur = 0xffffffffu;
  auto flush = [&](uint32_t c) {
    __syncthreads();
    uint32_t* g = ghist + size_t(c) * nh;
    for (int i = threadIdx.x; i < nh; i += blockDim.x) {
      const uint32_t v = s_hist[i];
      if (v) atomicAdd(&g[i], v);
      s_hist[i] = 0;
    }
    __syncthreads();
  };
  for (uint32_t t = t0; t < t1; ++t) {
    uint32_t first;
    const uint32_t c = tile_segment(seg, map, t, &first);
    if (HIST && c != cur && cur != 0xffffffffu) flush(cur);
    cur = c;
    const uint32_t sb = seg_begin(seg, c);
    const uint32_t lo = sb + (t - first) * kPointTile;
    const uint32_t hi = min(lo + kPointTile, sb + seg_size(seg, c));
    auto count = [&](K k) {
      if (HIST) {
#pragma unroll
        for (int ps = 0; ps < P; ++ps)
          atomicAdd(&s_hist[ps * RADIX + int((k >> (LOW + pass_shift<K, D, ENCODE>(ps))) &
                                             K(pass_mask<K, D, ENCODE>(ps)))], 1u);
      }
    };
    if (hi - lo == kPointTile) {
      // full tile: four loads in flight per thread before any is used
      static_assert(kPointTile % (4 * 256) == 0, "whole rounds of four points per thread");
      for (uint32_t i = lo + threadIdx.x; i < hi; i += 4 * 256) {
        K k[4];
        if (ENCODE) {
          float4 p[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) p[u] = __ldcs(pts + i + 256u * u);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            k[u] = encode<K, POW2>(p[u].x, p[u].y, p[u].z, min_coord, range, inv_range);
            keys[i + 256u * u] = k[u];
          }
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) k[u] = keys[i + 256u * u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) count(k[u]);
      }
    } else {
      for (uint32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        K k;
        if (ENCODE) {
          const float4 p = __ldcs(pts + i);
          k = encode<K, POW2>(p.x, p.y, p.z, min_coord, range, inv_range);
          keys[i] = k;
        } else {
          k = keys[i];
        }
        count(k);
      }
    }
  }
  if (HIST && cur != 0xffffffffu) flush(cur);
}

// One block per (segment, pass): exclusive scan of the segment's digit
// histogram, stored as the inclusive descriptor of the virtual tile before the
// segment's first tile.  Values are absolute positions (segment start added).
// Descriptor rows of a pass: segment c's init row is toff[c] + c, its tile j
// uses row toff[c] + c + 1 + j.
// For the top pass it also sets skew[c] when the digits are skewed: the
// chance that two keys share a digit, sum over digits of (count / n)^2, above
// 2^-skew_log2 (many lanes of a warp on one digit then serialise the
// atomic-OR ranking, which the ballot ranking does not).
// DENSE: it also decides which segments are dense, by the pairs that stage 1's
// samples found (all: every one is).
template <int D, bool DENSE>
__global__ void __launch_bounds__(256)
    k_sort_init(const uint32_t* __restrict__ ghist, uint32_t* __restrict__ desc,
                SegTable seg, TileMap map, int passes, uint32_t rows_per_pass,
                const uint32_t* __restrict__ gate, uint32_t* __restrict__ skew, int skew_log2,
                uint32_t* __restrict__ dense, uint32_t* __restrict__ dense_n, bool all) {
  pdl_enter();
  if (gate && *gate == 0) return;
  constexpr int RADIX = 1 << D;
  constexpr int R = (RADIX + 255) / 256;
  static_assert(R * 256 >= RADIX, "every digit needs an offset");
  __shared__ uint32_t s_warp[9];
  const uint32_t c = blockIdx.x / passes;
  const int pass = int(blockIdx.x % passes);
  if (map.toff && map.toff[c + 1] == map.toff[c]) return;  // no tile in this map
  if (DENSE && dense && pass == 0 && threadIdx.x == 0 &&
      (all || is_dense(dense[seg.count + c], seg_size(seg, c), seg.count))) {
    dense[c] = 1u;
    atomicAdd(dense_n, 1u);
  }
  const uint32_t* h = ghist + (size_t(c) * passes + pass) * RADIX;
  const uint32_t init_row = (map.toff ? map.toff[c] : 0u) + c;
  uint32_t* row0 = desc + (size_t(pass) * rows_per_pass + init_row) * RADIX;
  uint32_t v[R];
  uint32_t local = 0;
  const int first = threadIdx.x * R;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    v[r] = first + r < RADIX ? h[first + r] : 0u;
    local += v[r];
  }
  uint32_t total;
  uint32_t run = seg_begin(seg, c) + block_exclusive_scan<256>(local, s_warp, &total);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (first + r < RADIX) row0[first + r] = kFlagInc | (run << 2);
    run += v[r];
  }
  if (skew && pass == passes - 1) {  // block-uniform
    __shared__ unsigned long long s_sq[8];
    unsigned long long sq = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) sq += (unsigned long long)v[r] * v[r];
    sq = warp_sum(sq);
    if (lane_id() == 0) s_sq[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long all = 0;
      for (int w = 0; w < 8; ++w) all += s_sq[w];
      skew[c] = (all << skew_log2) > (unsigned long long)total * total ? 1u : 0u;
    }
  }
}

// ---------------------------------------------------------------------------
// stage 2: one onesweep pass
// ---------------------------------------------------------------------------


// One onesweep pass over `n` keys: digit `shift`..`shift+D-1`, stable.
// desc: [(tiles + 1) x RADIX] descriptors, row 0 prefilled with the global
// exclusive digit offsets (k_sort_init), rows 1.. zero.
// PERSIST: a CTA takes tiles by ticket until they run out (a grid of at most
// one wave), instead of one tile per CTA.  Used when the pass is gated, so
// that a pass that is not needed costs one short wave of CTAs.  A CTA holds a
// ticket only while it runs, so every look-back still waits only on running
// tiles, whatever the grid.
// skip (64-bit keys): [segments] those that the pass leaves alone.
template <typename K, int D, int THREADS, int KPT, int RANK, int MINB, bool PERSIST, int BB = D>
__global__ void __launch_bounds__(THREADS, MINB)
    k_binning(const K* __restrict__ in, K* __restrict__ out, SegTable seg, TileMap map,
              int shift, uint32_t dmask, uint32_t* __restrict__ desc,
              uint32_t* __restrict__ tile_ctr, DevStatus* __restrict__ st,
              uint32_t spin_limit, const uint32_t* __restrict__ gate,
              const uint32_t* __restrict__ skew, const uint32_t* __restrict__ skip) {
  pdl_enter();
  if (gate && *gate == 0) return;  // every tile of the pass returns: no look-back waits
  using C = BinCfg<K, D, THREADS, KPT, RANK>;
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* s_tile = reinterpret_cast<uint32_t*>(smem + C::kSmem - 64 * 4);
  uint32_t off = 0;
  if (sizeof(K) == 8 && skip && !map.toff) off = skip[0];
  for (;;) {
    if (threadIdx.x == 0) *s_tile = atomicAdd(tile_ctr, 1u);
    bin_zero<K, D, THREADS, KPT, RANK>(smem);
    __syncthreads();
    const uint32_t tile = *s_tile;
    if (PERSIST && tile >= map.n_tiles) break;  // block-uniform
    if (sizeof(K) == 8 && off) return;
    uint32_t first_tile;
    const uint32_t segc = tile_segment(seg, map, tile, &first_tile);
    const uint32_t base = seg_begin(seg, segc) + (tile - first_tile) * C::TILE;
    const uint32_t n = seg_begin(seg, segc) + seg_size(seg, segc);  // end of the segment
    const int row = int(tile + segc + 1);         // this tile's descriptor row
    const int init_row = int(first_tile + segc);  // the segment's inclusive row
    uint32_t* drow = desc + size_t(row) * C::RADIX;
    uint32_t seg_off = 0;
    if (sizeof(K) == 8 && skip && map.toff) seg_off = skip[segc];
    // this segment's digits decide the ranking scheme (block-uniform)
    const bool ballots = RANK == kRankMixed && skew != nullptr && skew[segc] != 0u;
    bin_tile<K, D, THREADS, KPT, RANK, BB>(
        smem, in, out, base, n, seg.total, shift, dmask, ballots, seg_off,
        [&](uint32_t d, uint32_t count) { st_relaxed(drow + d, kFlagAgg | (count << 2)); },
        [&](uint32_t d, uint32_t count) {
          const uint32_t excl = look_back<C::RADIX>(desc, d, row, init_row, spin_limit, st);
          st_relaxed(drow + d, kFlagInc | ((excl + count) << 2));
          return excl;
        });
    if (!PERSIST) break;
    __syncthreads();  // the next tile reuses every shared array
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

namespace {

template <typename K, int D, int LOW>
cudaError_t keys_t(const Bufs& b, const Scratch& sc, const Plan& pl, bool encode,
                   bool hist, cudaStream_t s) {
  const uint32_t tiles = pl.point_map.n_tiles;
  if (tiles == 0) return cudaSuccess;
  const uint32_t ctas = std::max(1u, std::min<uint32_t>(tiles, uint32_t(sc.num_sms) * 8));
  const uint32_t per = div_up(tiles, ctas);
  const uint32_t grid = div_up(tiles, per);
  if (hist && (sc.passes != (KeyTraits<K>::kCodeBits - LOW + D - 1) / D || sc.codes != encode))
    return cudaErrorInvalidValue;
  constexpr int kWordLow = LOW ? LOW + 1 : 0;  // the top bit belongs to a digit of a word
  const size_t smem = hist ? size_t(sc.passes) * (1u << D) * 4 : 0;
  K* keys = static_cast<K*>(b.keys);
  const float inv = pow2_reciprocal(b.range);
  const uint32_t samples = LOW ? dense_blocks(pl.seg.count) * pl.seg.count : 0u;
#define RWT_KEYS_LAUNCH(H, E)                                                        \
  do {                                                                               \
    constexpr int kLow = E ? LOW : kWordLow;                                         \
    auto kern = inv != 0.0f ? k_keys_pass<K, D, kLow, H, E, true>                    \
                            : k_keys_pass<K, D, kLow, H, E, false>;                  \
    if (smem > 48 * 1024)                                                            \
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)); \
    launch_pdl(kern, grid + (H ? samples : 0u), 256, smem, s, b.points, keys, pl.seg,       \
               pl.point_map, per, b.min_coord, b.range, inv, sc.ghist, sc.gate,             \
               samples ? sc.dense + pl.seg.count : static_cast<uint32_t*>(nullptr));        \
  } while (0)
  if (encode && hist) RWT_KEYS_LAUNCH(true, true);
  else if (encode) RWT_KEYS_LAUNCH(false, true);
  else RWT_KEYS_LAUNCH(true, false);
#undef RWT_KEYS_LAUNCH
  return cudaGetLastError();
}

// probe_spins != 0: the bounded-wait test hook (launch_sort_lookback_probe).
// RANK kRankMixed: atomic-OR ranking for the passes over full digits; the
// top pass ranks a segment by ballots over the code's remaining bits when
// k_sort_init found its top digits skewed (sum of squared digit frequencies
// above 1/32 for 32-bit keys, 1/64 for 64-bit keys, where the two schemes
// measured even), else by atomic OR.
template <typename K, int D, int THREADS, int KPT, int RANK, int MINB>
cudaError_t passes_t(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s,
                     cudaEvent_t* marks, uint32_t probe_spins) {
  // with low bits left out the passes end in tmp (launch_sort_finish goes on to alt)
  const int low = sorted_low_bits(sc), P = sc.passes;
  constexpr int kFull = (KeyTraits<K>::kCodeBits + D - 1) / D;
  constexpr int RB = RANK == kRankMixed ? kRankAtomicOr : RANK;  // passes 0 .. P-2
  constexpr int RT = RANK;                                       // pass P-1
  // bits of a code's top digit (left out bits are chosen so that it is a full one;
  // so is a word's)
  constexpr int TB = RANK == kRankMixed && !(sizeof(K) == 8 && D == 8)
                         ? KeyTraits<K>::kCodeBits - pass_shift<K, D, true>(kFull - 1)
                         : D;
  static_assert((63 - kSplitLow32) % 8 == 0 && (63 - kSplitLow40) % 8 == 0, "full digits");
  const auto shift = [&](int p) {
    return low + (sc.codes ? pass_shift<K, D, true>(p) : pass_shift<K, D, false>(p));
  };
  const auto mask = [&](int p) {
    return sc.codes ? pass_mask<K, D, true>(p) : pass_mask<K, D, false>(p);
  };
  constexpr int kSkewLog2 = sizeof(K) == 4 ? 5 : 6;
  uint32_t* skew = RANK == kRankMixed ? sc.skew : nullptr;
  using C = BinCfg<K, D, THREADS, KPT, RB>;
  using CT = BinCfg<K, D, THREADS, KPT, RT>;
  // a gated sort (a fallback that may not be needed) runs persistent passes
  const bool persist = sc.gate != nullptr && !probe_spins;
  auto kern = persist ? k_binning<K, D, THREADS, KPT, RB, MINB, true>
                      : k_binning<K, D, THREADS, KPT, RB, MINB, false>;
  auto kern_top = persist ? k_binning<K, D, THREADS, KPT, RT, MINB, true, TB>
                          : k_binning<K, D, THREADS, KPT, RT, MINB, false, TB>;
  if (!sc.codes)
    kern_top = persist ? k_binning<K, D, THREADS, KPT, RT, MINB, true, D>
                       : k_binning<K, D, THREADS, KPT, RT, MINB, false, D>;
  // the first pass need not be stable (a gated sort, which rarely runs, keeps to
  // the other kernel, and so do the wider digits)
  using CF = BinCfg<K, D, THREADS, KPT, D == 8 ? kRankUnordered : RB>;
  auto kern_first = kern;
  size_t smem_first = C::kSmem;
  if constexpr (D == 8) {
    if (!persist && !probe_spins) {
      kern_first = k_binning<K, D, THREADS, KPT, kRankUnordered, MINB, false>;
      smem_first = CF::kSmem;
    }
  }
  const uint32_t tiles = pl.sort_map.n_tiles;
  if (tiles + pl.seg.count > sc.sort_rows ||
      P != (KeyTraits<K>::kCodeBits - low + D - 1) / D || P > kMaxPasses ||
      (low != 0) != (sizeof(K) == 8 && D == 8))
    return cudaErrorInvalidValue;
  // (the first of several passes would overwrite keys that are sorted in place)
  const bool rest = low != 0 && !probe_spins;
  launch_pdl(k_sort_init<D, sizeof(K) == 8 && D == 8>, pl.seg.count * sc.passes, 256, 0, s,
             sc.ghist, sc.sort_desc, pl.seg, pl.sort_map, sc.passes, sc.sort_rows, sc.gate, skew,
             kSkewLog2, rest ? sc.dense : static_cast<uint32_t*>(nullptr),
             sc.rest_ctr + kRestDense, b.keys == b.alt);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (marks) cudaEventRecord(marks[0], s);
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(C::kSmem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern_top, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(CT::kSmem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern_first, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(smem_first));
  if (e != cudaSuccess) return e;
  K* keys = static_cast<K*>(b.keys);
  K* alt = static_cast<K*>(b.alt);
  K* tmp = static_cast<K*>(b.tmp);
  if (probe_spins) {
    // pass 0 with the tile ticket starting at 1: tile 0 never runs, so its
    // descriptor row stays unpublished and every other tile's look-back runs
    // into its spin limit; tiles 1 .. tiles-1 are launched (all in range)
    if (tiles < 2 || pl.seg.count != 1) return cudaErrorInvalidValue;
    e = cudaMemsetAsync(sc.tile_ctr + kCtrSortBase, 0x01, 1, s);
    if (e != cudaSuccess) return e;
    launch_pdl(kern, tiles - 1, THREADS, C::kSmem, s, static_cast<const K*>(keys), alt, pl.seg,
               pl.sort_map, low, uint32_t(C::RADIX - 1), sc.sort_desc, sc.tile_ctr + kCtrSortBase,
               sc.status,
               probe_spins, static_cast<const uint32_t*>(nullptr),
               static_cast<const uint32_t*>(nullptr), static_cast<const uint32_t*>(nullptr));
    return cudaGetLastError();
  }
  const K* src = keys;
  const uint32_t grid =
      persist ? std::min<uint32_t>(tiles, uint32_t(sc.num_sms) * uint32_t(MINB)) : tiles;
  for (int p = 0; p < P; ++p) {
    K* dst = ((P - 1 - p) % 2 == 0) == (low == 0) ? alt : tmp;
    if (tiles)
      launch_pdl(p == P - 1 ? kern_top : p == 0 ? kern_first : kern, grid, THREADS,
                 p == P - 1 ? CT::kSmem : p == 0 ? smem_first : C::kSmem, s, src, dst, pl.seg,
                 pl.sort_map, shift(p), mask(p),
                 sc.sort_desc + size_t(p) * sc.sort_rows * C::RADIX,
                 sc.tile_ctr + kCtrSortBase + p, sc.status, sc.spin_limit, sc.gate,
                 static_cast<const uint32_t*>(p == P - 1 ? skew : nullptr),
                 static_cast<const uint32_t*>(rest ? sc.dense : nullptr));
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (marks) cudaEventRecord(marks[1 + p], s);
    src = dst;
  }
  return cudaSuccess;
}

using PassFn = cudaError_t (*)(const Bufs&, const Scratch&, const Plan&, cudaStream_t,
                               cudaEvent_t*, uint32_t);

struct SortVariant {
  int key_bits, radix_bits, threads, kpt, rank;
  PassFn fn;
};

// The menu the autotuner chooses from (entry 0 of each key/digit width is
// the default).
const SortVariant kVariants[] = {
    {32, 8, 384, 24, kRankAtomicOr, passes_t<uint32_t, 8, 384, 24, kRankAtomicOr, 3>},
    {32, 8, 384, 24, kRankMixed, passes_t<uint32_t, 8, 384, 24, kRankMixed, 3>},
    {32, 8, 384, 24, kRankHalfPacked, passes_t<uint32_t, 8, 384, 24, kRankHalfPacked, 3>},
    {32, 8, 512, 16, kRankHalfPacked, passes_t<uint32_t, 8, 512, 16, kRankHalfPacked, 2>},
    {32, 8, 256, 24, kRankHalfPacked, passes_t<uint32_t, 8, 256, 24, kRankHalfPacked, 4>},
    {32, 8, 512, 24, kRankHalfPacked, passes_t<uint32_t, 8, 512, 24, kRankHalfPacked, 2>},
    {32, 8, 512, 16, kRankAtomicOr, passes_t<uint32_t, 8, 512, 16, kRankAtomicOr, 2>},
    {32, 8, 384, 16, kRankAtomicOr, passes_t<uint32_t, 8, 384, 16, kRankAtomicOr, 2>},
    {32, 8, 256, 16, kRankAtomicOr, passes_t<uint32_t, 8, 256, 16, kRankAtomicOr, 3>},
    {32, 8, 256, 24, kRankAtomicOr, passes_t<uint32_t, 8, 256, 24, kRankAtomicOr, 2>},
    {32, 8, 512, 24, kRankAtomicOr, passes_t<uint32_t, 8, 512, 24, kRankAtomicOr, 1>},
    {32, 8, 256, 16, kRankBallot, passes_t<uint32_t, 8, 256, 16, kRankBallot, 3>},
    {32, 8, 512, 16, kRankBallot, passes_t<uint32_t, 8, 512, 16, kRankBallot, 1>},
    {32, 8, 384, 16, kRankMatchAny, passes_t<uint32_t, 8, 384, 16, kRankMatchAny, 2>},
    {32, 8, 512, 16, kRankBallot, passes_t<uint32_t, 8, 512, 16, kRankBallot, 2>},
    {32, 8, 384, 16, kRankBallot, passes_t<uint32_t, 8, 384, 16, kRankBallot, 2>},
    {32, 8, 256, 32, kRankBallot, passes_t<uint32_t, 8, 256, 32, kRankBallot, 2>},
    {32, 8, 512, 16, kRankMatchAny, passes_t<uint32_t, 8, 512, 16, kRankMatchAny, 2>},
    {32, 8, 1024, 16, kRankAtomicOr, passes_t<uint32_t, 8, 1024, 16, kRankAtomicOr, 1>},
    {32, 8, 1024, 8, kRankAtomicOr, passes_t<uint32_t, 8, 1024, 8, kRankAtomicOr, 1>},
    {32, 10, 256, 24, kRankAtomicOr, passes_t<uint32_t, 10, 256, 24, kRankAtomicOr, 2>},
    {32, 10, 256, 16, kRankAtomicOr, passes_t<uint32_t, 10, 256, 16, kRankAtomicOr, 2>},
    {32, 10, 256, 24, kRankBallot, passes_t<uint32_t, 10, 256, 24, kRankBallot, 3>},
    {32, 10, 384, 16, kRankBallot, passes_t<uint32_t, 10, 384, 16, kRankBallot, 2>},
    {32, 10, 512, 16, kRankBallot, passes_t<uint32_t, 10, 512, 16, kRankBallot, 2>},
    {32, 10, 256, 24, kRankMatchAny, passes_t<uint32_t, 10, 256, 24, kRankMatchAny, 3>},
    {32, 10, 256, 24, kRankHalfPacked, passes_t<uint32_t, 10, 256, 24, kRankHalfPacked, 2>},
    {32, 11, 512, 16, kRankBallot, passes_t<uint32_t, 11, 512, 16, kRankBallot, 1>},
    {32, 11, 256, 16, kRankAtomicOr, passes_t<uint32_t, 11, 256, 16, kRankAtomicOr, 1>},
    {32, 11, 256, 24, kRankAtomicOr, passes_t<uint32_t, 11, 256, 24, kRankAtomicOr, 1>},
    {32, 11, 256, 24, kRankBallot, passes_t<uint32_t, 11, 256, 24, kRankBallot, 1>},
    {32, 11, 256, 16, kRankBallot, passes_t<uint32_t, 11, 256, 16, kRankBallot, 2>},
    {32, 11, 384, 16, kRankBallot, passes_t<uint32_t, 11, 384, 16, kRankBallot, 1>},
    {64, 8, 384, 16, kRankAtomicOr, passes_t<uint64_t, 8, 384, 16, kRankAtomicOr, 2>},
    {64, 8, 384, 16, kRankMixed, passes_t<uint64_t, 8, 384, 16, kRankMixed, 2>},
    {64, 8, 384, 16, kRankHalfPacked, passes_t<uint64_t, 8, 384, 16, kRankHalfPacked, 2>},
    {64, 8, 256, 16, kRankHalfPacked, passes_t<uint64_t, 8, 256, 16, kRankHalfPacked, 3>},
    {64, 8, 256, 16, kRankAtomicOr, passes_t<uint64_t, 8, 256, 16, kRankAtomicOr, 2>},
    {64, 8, 256, 12, kRankAtomicOr, passes_t<uint64_t, 8, 256, 12, kRankAtomicOr, 3>},
    {64, 8, 256, 16, kRankBallot, passes_t<uint64_t, 8, 256, 16, kRankBallot, 2>},
    {64, 10, 256, 16, kRankAtomicOr, passes_t<uint64_t, 10, 256, 16, kRankAtomicOr, 2>},
    {64, 10, 256, 16, kRankBallot, passes_t<uint64_t, 10, 256, 16, kRankBallot, 2>},
    {64, 11, 384, 16, kRankBallot, passes_t<uint64_t, 11, 384, 16, kRankBallot, 1>},
    {64, 11, 256, 16, kRankAtomicOr, passes_t<uint64_t, 11, 256, 16, kRankAtomicOr, 1>},
    {64, 11, 256, 12, kRankAtomicOr, passes_t<uint64_t, 11, 256, 12, kRankAtomicOr, 1>},
    {64, 11, 256, 16, kRankBallot, passes_t<uint64_t, 11, 256, 16, kRankBallot, 1>},
};
constexpr int kNumVariants = int(sizeof(kVariants) / sizeof(kVariants[0]));

}  // namespace

// Smallest tile of any variant for this key/digit width: sizes the descriptors.
uint32_t sort_tile_for(int key_bits, int radix_bits) {
  uint32_t t = 0xffffffffu;
  for (const auto& v : kVariants)
    if (v.key_bits == key_bits && v.radix_bits == radix_bits)
      t = std::min<uint32_t>(t, uint32_t(v.threads * v.kpt));
  return t;
}

uint32_t sort_variant_tile(int idx) {
  if (idx < 0 || idx >= kNumVariants) return 0;
  return uint32_t(kVariants[idx].threads * kVariants[idx].kpt);
}

int sort_variant_count() { return kNumVariants; }

int sort_variant_info(int idx, int* key_bits, int* radix_bits, int* threads, int* kpt,
                      int* rank) {
  if (idx < 0 || idx >= kNumVariants) return -1;
  const auto& v = kVariants[idx];
  *key_bits = v.key_bits;
  *radix_bits = v.radix_bits;
  *threads = v.threads;
  *kpt = v.kpt;
  *rank = v.rank;
  return 0;
}

int default_sort_variant(int key_bits, int radix_bits) {
  for (int i = 0; i < kNumVariants; ++i)
    if (kVariants[i].key_bits == key_bits && kVariants[i].radix_bits == radix_bits) return i;
  return -1;
}

cudaError_t launch_keys(const Bufs& b, const Scratch& sc, const Plan& pl, bool encode,
                        bool hist, cudaStream_t s) {
  if (b.key_bits == 32) {
    if (sc.radix_bits == 8) return keys_t<uint32_t, 8, 0>(b, sc, pl, encode, hist, s);
    if (sc.radix_bits == 10) return keys_t<uint32_t, 10, 0>(b, sc, pl, encode, hist, s);
    return keys_t<uint32_t, 11, 0>(b, sc, pl, encode, hist, s);
  }
  if (sc.radix_bits == 8)
    return sc.low_bits == kSplitLow32
               ? keys_t<uint64_t, 8, kSplitLow32>(b, sc, pl, encode, hist, s)
               : keys_t<uint64_t, 8, kSplitLow40>(b, sc, pl, encode, hist, s);
  if (sc.radix_bits == 10) return keys_t<uint64_t, 10, 0>(b, sc, pl, encode, hist, s);
  return keys_t<uint64_t, 11, 0>(b, sc, pl, encode, hist, s);
}

cudaError_t launch_sort_passes(const Bufs& b, const Scratch& sc, const Plan& pl,
                               cudaStream_t s, cudaEvent_t* marks) {
  const int v = sc.sort_variant;
  if (v < 0 || v >= kNumVariants || kVariants[v].key_bits != b.key_bits ||
      kVariants[v].radix_bits != sc.radix_bits)
    return cudaErrorInvalidValue;
  return kVariants[v].fn(b, sc, pl, s, marks, 0u);
}

cudaError_t launch_sort_lookback_probe(const Bufs& b, const Scratch& sc, const Plan& pl,
                                       uint32_t spin_limit, cudaStream_t s) {
  const int v = sc.sort_variant;
  if (v < 0 || v >= kNumVariants || kVariants[v].key_bits != b.key_bits ||
      kVariants[v].radix_bits != sc.radix_bits || spin_limit == 0)
    return cudaErrorInvalidValue;
  cudaError_t e = launch_keys(b, sc, pl, false, true, s);
  if (e != cudaSuccess) return e;
  return kVariants[v].fn(b, sc, pl, s, nullptr, spin_limit);
}

}  // namespace rwt
