// Stages 3-7: unique compaction, Karras radix tree, edge count, exclusive
// scan, octree.
//
// Stage 3 replaces k_FindDups + host std::partial_sum + k_MoveDups
// (apps/tree/cuda/03_unique.cu, cu_dispatcher.cu:597-627) with three
// launches: per-tile head counts, one block scanning the tile counts, then a
// compaction of every tile at its scanned offset.
//
// Stage 4 builds the nodes of process_radix_tree_i (apps/tree/host/
// func_brt.hpp:45-138) from nearest smaller values: the radix tree is the
// Cartesian tree of the gap deltas, so each gap's node follows from the
// nearest strictly smaller gap on either side (k_radix_tree; the few gaps
// whose answer lies beyond the tile's window are searched for in the keys by
// the block at its end).  Node 0
// keeps the reference's own range [0, n_brt-1] (coop_root_split, write_root);
// nodes i >= 1 are the true Karras nodes and each names its children once, so
// the parent writes are deterministic.
//
// The fused form computes stages 4 and 5 in one pass: the edge count of node i
// needs prefix_n[parent[i]], and the parent's prefix length is the larger of
// the two boundary deltas of i's key range (the parent splits at one end of
// it; when that split is the global minimum the parent is the root, whose
// prefix_n the reference computes over [0, n_brt-1]).
//
// Stage 6 run alone is a reduce, a one-block scan of the tile sums and a
// write.  In the fused pipeline its first two steps run on the octree's tiles
// and the octree kernel scans its own tile's counts on that prefix, writing
// the offsets as it uses them.
//
// Stage 7 follows process_oct_node (func_octree.hpp:28-112) in one pass per
// tile of nodes (k_octree): every row is written once, complete, with the
// links whose target row lies in the tile merged in shared memory; the links
// that leave the tile are applied afterwards with atomicMax/atomicOr
// (k_octree_far_links).  Sequential ascending-i execution leaves in every
// child slot the largest value written (node i writes only values in
// [off[i], off[i]+cnt[i]) and these ranges grow with i), and the node mask is
// an OR, so the result is the reference's sequential one.
#include <algorithm>

#include "internal.hpp"
#include "morton.cuh"
#include "tree_tiles.cuh"

namespace rwt {

// ---------------------------------------------------------------------------
// stage 3: unique
// ---------------------------------------------------------------------------

// Exclusive scan of per-tile values E[0, tiles) in place (E[tiles] = total),
// one block; then each segment's total (its tiles per the tile map) into
// seg_total.  Between the per-tile count and the per-tile write launches of
// stages 3 and 6.
__global__ void __launch_bounds__(1024)
    k_tile_scan(uint32_t* __restrict__ E, uint32_t tiles, SegTable seg, TileMap map,
                uint32_t* __restrict__ seg_total) {
  pdl_enter();
  // Rounds of up to 1,024 x 4 J tiles, a contiguous slice of 128 q per warp: a
  // lane takes four consecutive tiles at a time as a vector and adds them up, so
  // that a warp scan serves 128 tiles, then one warp scans the 32 warp sums.
  // One block: its shuffles are what counts (J scans of single words for every
  // warp, whether it had tiles or not: unique and edge scan of
  // 16.8M points 60.8 -> 56.7 us, of 5M 64-bit keys 31.6 -> 26.4)
  constexpr int J = 4;
  __shared__ uint32_t s_warp[33];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const bool vec = (reinterpret_cast<uintptr_t>(E) & 15u) == 0;
  uint32_t carry = 0;
  for (uint32_t c0 = 0; c0 < tiles; c0 += 4096u * J) {
    const uint32_t q = min(uint32_t(J), (tiles - c0 + 4095u) / 4096u);
    const uint32_t wb = c0 + warp * 128u * q + 4u * lane;
    uint4 v[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const uint32_t i = wb + 128u * j;
      v[j] = make_uint4(0, 0, 0, 0);
      if (uint32_t(j) < q) {
        if (vec && i + 4u <= tiles) {
          v[j] = *reinterpret_cast<const uint4*>(E + i);
        } else {
          if (i < tiles) v[j].x = E[i];
          if (i + 1u < tiles) v[j].y = E[i + 1u];
          if (i + 2u < tiles) v[j].z = E[i + 2u];
          if (i + 3u < tiles) v[j].w = E[i + 3u];
        }
      }
    }
    uint32_t run = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      if (uint32_t(j) < q) {
        const uint4 x = v[j];
        const uint32_t sum = x.x + x.y + x.z + x.w;
        const uint32_t inc = warp_inclusive_scan(sum);
        const uint32_t at = run + inc - sum;  // exclusive within the warp's slice
        v[j] = make_uint4(at, at + x.x, at + x.x + x.y, at + x.x + x.y + x.z);
        run += __shfl_sync(0xffffffffu, inc, 31);
      }
    }
    if (lane == 0) s_warp[warp] = run;
    __syncthreads();
    if (warp == 0) {
      const uint32_t w = s_warp[lane];
      const uint32_t wi = warp_inclusive_scan(w);
      s_warp[lane] = wi - w;
      if (lane == 31) s_warp[32] = wi;
    }
    __syncthreads();
    const uint32_t wofs = carry + s_warp[warp];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const uint32_t i = wb + 128u * j;
      if (uint32_t(j) < q) {
        const uint4 x = make_uint4(wofs + v[j].x, wofs + v[j].y, wofs + v[j].z, wofs + v[j].w);
        if (vec && i + 4u <= tiles) {
          *reinterpret_cast<uint4*>(E + i) = x;
        } else {
          if (i < tiles) E[i] = x.x;
          if (i + 1u < tiles) E[i + 1u] = x.y;
          if (i + 2u < tiles) E[i + 2u] = x.z;
          if (i + 3u < tiles) E[i + 3u] = x.w;
        }
      }
    }
    carry += s_warp[32];
    __syncthreads();  // s_warp is reused by the next round
  }
  if (threadIdx.x == 0) E[tiles] = carry;
  __syncthreads();
  for (uint32_t sg = threadIdx.x; sg < seg.count; sg += 1024) {
    const uint32_t t0 = map.toff ? map.toff[sg] : 0u;
    const uint32_t t1 = map.toff ? map.toff[sg + 1] : tiles;
    seg_total[sg] = (t1 < tiles ? E[t1] : carry) - (t0 < tiles ? E[t0] : carry);
  }
}

// Stage 3 in three launches without a serial chain between tiles: (1) every
// tile counts its heads (a key is a head when it differs from its left
// neighbour in the segment, or starts the segment) into E[tile]; (2) one block
// turns E into its exclusive scan (E[tiles] = total) and writes each
// segment's n_unique; (3) every tile compacts its heads to segment begin +
// E[tile] - E[first tile of the segment].  Same result as
// cu_dispatcher.cu:597-627 (a std::unique over the sorted keys).
template <typename K>
__device__ __forceinline__ uint32_t tile_heads(const K* __restrict__ sorted, uint32_t sb,
                                               uint32_t n, uint32_t wbase,
                                               K (&keys)[kUniqueKpt],
                                               uint32_t (&heads)[kUniqueKpt]) {
  const uint32_t lane = lane_id();
  // every load first, so that all of them are in flight together
#pragma unroll
  for (int i = 0; i < kUniqueKpt; ++i) {
    const uint32_t idx = wbase + 32u * i + lane;
    keys[i] = idx < n ? sorted[idx] : K(0);
  }
  const K before = (lane == 0 && wbase > sb && wbase - 1 < n) ? sorted[wbase - 1] : K(0);
  K carry = K(0);
  uint32_t count = 0;
#pragma unroll
  for (int i = 0; i < kUniqueKpt; ++i) {
    const uint32_t idx = wbase + 32u * i + lane;
    const K k = keys[i];
    K left = __shfl_up_sync(0xffffffffu, k, 1);
    if (lane == 0) {
      if (i == 0)
        left = (wbase > sb && wbase - 1 < n) ? before : K(~k);
      else
        left = carry;
    }
    carry = __shfl_sync(0xffffffffu, k, 31);
    const bool head = idx < n && (idx == sb || k != left);
    heads[i] = __ballot_sync(0xffffffffu, head);
    count += __popc(heads[i]);
  }
  return count;
}

// The same head flags for a warp whose 32 * kUniqueKpt keys are all in the
// segment and start on a 16-byte boundary: vector j of lane l holds keys
// wbase + (32 j + l) V + [0, V) (V keys per 16 bytes); hm[j] bit e flags key e
// of that vector.
template <typename K>
struct UniqueVec {
  static constexpr int V = 16 / int(sizeof(K));
  static constexpr int NVEC = int(kUniqueKpt) / V;
};

template <typename K>
__device__ __forceinline__ bool unique_vec_ok(const K* sorted, uint32_t wbase, uint32_t n) {
  return wbase + 32u * kUniqueKpt <= n &&
         (reinterpret_cast<uintptr_t>(sorted + wbase) & 15u) == 0;
}

template <typename K>
__device__ __forceinline__ uint32_t tile_heads_vec(const K* __restrict__ sorted, uint32_t sb,
                                                   uint32_t wbase, K (&keys)[kUniqueKpt],
                                                   uint32_t (&hm)[UniqueVec<K>::NVEC]) {
  constexpr int V = UniqueVec<K>::V, NVEC = UniqueVec<K>::NVEC;
  const uint32_t lane = lane_id();
#pragma unroll
  for (int j = 0; j < NVEC; ++j) {
    const uint4 x = *reinterpret_cast<const uint4*>(sorted + wbase + (32u * j + lane) * V);
    const K* xk = reinterpret_cast<const K*>(&x);
#pragma unroll
    for (int e = 0; e < V; ++e) keys[j * V + e] = xk[e];
  }
  const K before = (lane == 0 && wbase > sb) ? sorted[wbase - 1] : K(0);
  K carry = K(0);
  uint32_t count = 0;
#pragma unroll
  for (int j = 0; j < NVEC; ++j) {
    const K last = keys[j * V + V - 1];
    K up = __shfl_up_sync(0xffffffffu, last, 1);
    if (lane == 0) up = j == 0 ? (wbase > sb ? before : K(~keys[0])) : carry;
    carry = __shfl_sync(0xffffffffu, last, 31);
    uint32_t m = 0;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const K prev = e == 0 ? up : keys[j * V + e - 1];
      const uint32_t idx = wbase + (32u * j + lane) * V + e;
      m |= uint32_t(idx == sb || keys[j * V + e] != prev) << e;
    }
    hm[j] = m;
    count += __popc(m);
  }
  return count;
}

template <typename K>
__global__ void __launch_bounds__(kUniqueThreads)
    k_unique_count(const K* __restrict__ sorted, SegTable seg, TileMap map,
                   uint32_t* __restrict__ E) {
  pdl_enter();
  constexpr int NW = kUniqueThreads / 32;
  __shared__ uint32_t s_warp[NW];
  const uint32_t tile = blockIdx.x, lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t first;
  const uint32_t c = tile_segment(seg, map, tile, &first);
  const uint32_t sb = seg_begin(seg, c);
  const uint32_t n = sb + seg_size(seg, c);
  const uint32_t wbase = sb + (tile - first) * kUniqueTile + warp * 32u * kUniqueKpt;
  K keys[kUniqueKpt];
  uint32_t count;
  if (unique_vec_ok(sorted, wbase, n)) {
    uint32_t hm[UniqueVec<K>::NVEC];
    count = warp_sum(tile_heads_vec(sorted, sb, wbase, keys, hm));
  } else {
    uint32_t heads[kUniqueKpt];
    count = tile_heads(sorted, sb, n, wbase, keys, heads);
  }
  if (lane == 0) s_warp[warp] = count;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < NW; ++w) t += s_warp[w];
    E[tile] = t;
  }
}

template <typename K>
__global__ void __launch_bounds__(kUniqueThreads)
    k_unique_write(const K* __restrict__ sorted, K* __restrict__ out, SegTable seg, TileMap map,
                   const uint32_t* __restrict__ E) {
  pdl_enter();
  constexpr int NW = kUniqueThreads / 32;
  __shared__ uint32_t s_warp[NW];
  const uint32_t tile = blockIdx.x, lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t first;
  const uint32_t c = tile_segment(seg, map, tile, &first);
  const uint32_t sb = seg_begin(seg, c);
  const uint32_t n = sb + seg_size(seg, c);
  const uint32_t wbase = sb + (tile - first) * kUniqueTile + warp * 32u * kUniqueKpt;
  K keys[kUniqueKpt];
  constexpr int V = UniqueVec<K>::V, NVEC = UniqueVec<K>::NVEC;
  const bool vec = unique_vec_ok(sorted, wbase, n);
  uint32_t heads[kUniqueKpt];  // scalar path: ballots; vector path: hm[j] in heads[j]
  uint32_t count;
  if (vec) {
    uint32_t hm[NVEC];
    count = warp_sum(tile_heads_vec(sorted, sb, wbase, keys, hm));
#pragma unroll
    for (int j = 0; j < NVEC; ++j) heads[j] = hm[j];
  } else {
    count = tile_heads(sorted, sb, n, wbase, keys, heads);
  }
  if (lane == 0) s_warp[warp] = count;
  __syncthreads();
  if (warp == 0) {
    const uint32_t cw = lane < NW ? s_warp[lane] : 0u;
    const uint32_t inc = warp_inclusive_scan(cw);
    if (lane < NW) s_warp[lane] = inc - cw;
  }
  __syncthreads();
  uint32_t pos = sb + (E[tile] - E[first]) + s_warp[warp];
  if (vec) {
#pragma unroll
    for (int j = 0; j < NVEC; ++j) {
      const uint32_t c = uint32_t(__popc(heads[j]));
      const uint32_t inc = warp_inclusive_scan(c);
      uint32_t dst = pos + inc - c;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        if (((heads[j] >> e) & 1u) && dst < n) out[dst] = keys[j * V + e];
        dst += (heads[j] >> e) & 1u;
      }
      pos += __shfl_sync(0xffffffffu, inc, 31);
    }
  } else {
#pragma unroll
    for (int i = 0; i < kUniqueKpt; ++i) {
      const uint32_t dst = pos + __popc(heads[i] & lanemask_lt());
      if (((heads[i] >> lane) & 1u) && dst < n) out[dst] = keys[i];
      pos += __popc(heads[i]);
    }
  }
}

// ---------------------------------------------------------------------------
// stage 4: Karras radix tree node (func_brt.hpp:45-138)
// ---------------------------------------------------------------------------

template <typename K, bool EDGES, int LESS>
// 8 blocks (64 warps) per SM with 32-bit keys; the shared memory holds 5 with
// 64-bit ones, which then need no more than 48 registers (77.6 against 81.0 us at
// 5,000,011 points with 32)
__global__ void __launch_bounds__(kTreeThreads, sizeof(K) == 4 ? 8 : 5)
    k_radix_tree(const K* __restrict__ codes_all, SegTable seg, TileMap map,
                 const uint32_t* __restrict__ n_unique, int32_t* __restrict__ seg_err,
                 uint8_t* __restrict__ prefix_n, uint8_t* __restrict__ hl,
                 uint8_t* __restrict__ hr, int32_t* __restrict__ lc,
                 int32_t* __restrict__ parents, int32_t* __restrict__ edge_count,
                 TileMap nodes, uint32_t* __restrict__ sums) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TreeTileShared sh;
  uint32_t first;
  const uint32_t c = tile_segment(seg, map, blockIdx.x, &first);
  const uint32_t nu = *reinterpret_cast<const volatile uint32_t*>(n_unique + c);
  if (nu < 3 || nu == RW_COUNT_UNSET || nu > seg_size(seg, c)) {
    if (blockIdx.x == first && threadIdx.x == 0) seg_error(seg_err, c, RW_ERR_DEGENERATE);
    return;
  }
  const uint32_t sb = seg_begin(seg, c);
  const int n = int(nu - 1);  // gaps (= nodes); keys are [0, n]
  const int g0 = int(blockIdx.x - first) * int(kTreeTile);
  if (g0 >= n) return;
  tree_tile<K, EDGES, LESS, kTreeThreads, kTreeTile / 32, false, true>(
      smem_raw, sh, codes_all + sb, n, g0, 0, seg_err + c, prefix_n + sb, hl + sb, hr + sb,
      lc + sb, parents + sb, EDGES ? edge_count + sb : nullptr,
      EDGES ? sums + (nodes.toff ? nodes.toff[c] : 0u) : nullptr);
}

// ---------------------------------------------------------------------------
// stage 5: edge count (func_edge.hpp:9-16, 05_edge_count.cu:16-29)
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256)
    k_edge_count(const uint8_t* __restrict__ prefix_n, const int32_t* __restrict__ parents,
                 int32_t* __restrict__ ec, SegTable seg, TileMap map,
                 const uint32_t* __restrict__ n_unique) {
  pdl_enter();
  uint32_t first;
  const uint32_t c = tile_segment(seg, map, blockIdx.x, &first);
  const uint32_t nu = n_unique[c];
  if (nu < 3 || nu == RW_COUNT_UNSET || nu > seg_size(seg, c)) return;
  const int n = int(nu - 1);
  const uint32_t sb = seg_begin(seg, c);
  const int base = int(blockIdx.x - first) * kOctTile;
  for (int q = 0; q < kOctNpt; ++q) {
    const int i = base + q * kOctThreads + int(threadIdx.x);
    if (i >= n) break;
    const int p = parents[sb + i];
    // parents[] holds node indices in [0, n) after stage 4; anything else is a
    // caller error and reads node 0 instead of leaving the buffer
    ec[sb + i] = prefix_n[sb + i] / 3 - prefix_n[sb + (uint32_t(p) < uint32_t(n) ? p : 0)] / 3;
  }
}

// ---------------------------------------------------------------------------
// stage 6: exclusive scan of the edge counts
// ---------------------------------------------------------------------------

// Stage 6 in three launches (no serial chain between tiles): (1) every tile
// sums its edge counts into E[tile]; (2) one block scans E (E[tiles] = total)
// and writes each segment's node count; (3) every tile writes its exclusive
// offsets from E[tile] - E[the segment's first tile].
// Tiles past a segment's nodes (the tile map is sized by points) count zero.
__device__ __forceinline__ bool scan_tile(const SegTable& seg, const TileMap& map,
                                          const uint32_t* n_unique, uint32_t tile,
                                          uint32_t* c, uint32_t* firstt, uint32_t* n,
                                          uint32_t* j) {
  *c = tile_segment(seg, map, tile, firstt);
  const uint32_t nu = *reinterpret_cast<const volatile uint32_t*>(n_unique + *c);
  const bool valid = nu >= 3 && nu != RW_COUNT_UNSET && nu <= seg_size(seg, *c);
  *n = valid ? nu - 1 : 0;
  *j = tile - *firstt;
  return *j < (*n + kScanTile - 1) / kScanTile;
}

__device__ __forceinline__ void scan_load(const int32_t* ec, uint32_t first, uint32_t n,
                                          bool vec, int32_t (&v)[kScanKpt]) {
  if (vec) {
#pragma unroll
    for (int q = 0; q < kScanKpt / 4; ++q) {
      const int4 x = reinterpret_cast<const int4*>(ec + first)[q];
      v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int q = 0; q < kScanKpt; ++q) v[q] = first + q < n ? ec[first + q] : 0;
  }
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_reduce(const int32_t* __restrict__ ec_all, SegTable seg, TileMap map,
                  const uint32_t* __restrict__ n_unique, uint32_t* __restrict__ E) {
  pdl_enter();
  constexpr int NW = kScanThreads / 32;
  __shared__ uint32_t s_warp[NW];
  const uint32_t tile = blockIdx.x;
  uint32_t c, firstt, n, j;
  uint32_t local = 0;
  if (scan_tile(seg, map, n_unique, tile, &c, &firstt, &n, &j)) {
    const uint32_t sb = seg_begin(seg, c);
    const uint32_t first = j * kScanTile + threadIdx.x * kScanKpt;
    int32_t v[kScanKpt];
    scan_load(ec_all + sb, first, n, first + kScanKpt <= n && (sb & 3u) == 0, v);
#pragma unroll
    for (int q = 0; q < kScanKpt; ++q) local += uint32_t(v[q]);
  }
  local = warp_sum(local);
  if (lane_id() == 0) s_warp[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < NW; ++w) t += s_warp[w];
    E[tile] = t;
  }
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_write(const int32_t* __restrict__ ec_all, int32_t* __restrict__ off_all,
                 SegTable seg, TileMap map, const uint32_t* __restrict__ n_unique,
                 const uint32_t* __restrict__ E) {
  pdl_enter();
  __shared__ uint32_t s_warp[kScanThreads / 32 + 1];
  const uint32_t tile = blockIdx.x;
  uint32_t c, firstt, n, j;
  if (!scan_tile(seg, map, n_unique, tile, &c, &firstt, &n, &j)) return;  // whole CTA
  const uint32_t sb = seg_begin(seg, c);
  const uint32_t first = j * kScanTile + threadIdx.x * kScanKpt;
  const bool vec = first + kScanKpt <= n && (sb & 3u) == 0;
  int32_t v[kScanKpt];
  scan_load(ec_all + sb, first, n, vec, v);
  uint32_t local = 0;
#pragma unroll
  for (int q = 0; q < kScanKpt; ++q) local += uint32_t(v[q]);
  uint32_t total;
  uint32_t run = (E[tile] - E[firstt]) +
                 block_exclusive_scan<kScanThreads>(local, s_warp, &total);
  int32_t* off = off_all + sb;
  if (vec) {
#pragma unroll
    for (int q = 0; q < kScanKpt / 4; ++q) {
      int4 x;
      x.x = int32_t(run); run += uint32_t(v[4 * q]);
      x.y = int32_t(run); run += uint32_t(v[4 * q + 1]);
      x.z = int32_t(run); run += uint32_t(v[4 * q + 2]);
      x.w = int32_t(run); run += uint32_t(v[4 * q + 3]);
      reinterpret_cast<int4*>(off + first)[q] = x;
    }
  } else {
#pragma unroll
    for (int q = 0; q < kScanKpt; ++q) {
      if (first + q < n) off[first + q] = int32_t(run);
      run += uint32_t(v[q]);
    }
  }
}

// ---------------------------------------------------------------------------
// stage 7: octree rows and links (func_octree.hpp:28-112)
// ---------------------------------------------------------------------------

template <typename K, bool OFFS>
__global__ void // 8 blocks per SM with 32-bit keys (32 registers, all of the shared memory); 7
// fit with 64-bit keys, but 6 with 40 registers are faster: 74.1 against 82.7 us
// at 5,000,011 points
__launch_bounds__(kOctThreads, sizeof(K) == 4 ? 8 : 6)
    k_octree(const K* __restrict__ codes_all, const uint8_t* __restrict__ prefix_all,
             const int32_t* __restrict__ parents_all, const int32_t* __restrict__ ec_all,
             int32_t* __restrict__ off_all, const uint32_t* __restrict__ tile_prefix,
             SegTable seg, TileMap map, const uint32_t* __restrict__ n_unique,
             const uint32_t* __restrict__ n_octree, int32_t* __restrict__ seg_err,
             float min_coord, float range, OctOut o, uint32_t* __restrict__ far,
             uint32_t far_cap, uint32_t* __restrict__ far_n) {
  pdl_enter();
  __shared__ OctTileShared<K> sh;
  uint32_t first;
  const uint32_t c = tile_segment(seg, map, blockIdx.x, &first);
  const OctSeg os = oct_segment(seg, o, n_unique, n_octree, seg_err, c,
                                blockIdx.x == first && threadIdx.x == 0);
  // with OFFS a too small octree still gets its edge offsets (stage 6's
  // output), as when stage 6 runs on its own
  if (OFFS ? !os.counts : !os.ok) return;
  const int tile0 = int(blockIdx.x - first) * int(kOctTile);
  if (tile0 >= os.n) return;
  const uint32_t sb = seg_begin(seg, c);
  octree_tile<K, OFFS>(
      sh, [] { __syncthreads(); }, int(threadIdx.x), codes_all + sb, prefix_all + sb,
      parents_all + sb, ec_all + sb, off_all + sb, os, c, tile0,
      [&] { return tile_prefix[blockIdx.x] - tile_prefix[first]; }, min_coord, range, o, far,
      far_cap, far_n);
}

template <typename K>
__global__ void __launch_bounds__(256)
    k_octree_far_links(const K* __restrict__ codes_all, const uint8_t* __restrict__ prefix_all,
                       const int32_t* __restrict__ parents_all,
                       const int32_t* __restrict__ ec_all, const int32_t* __restrict__ off_all,
                       SegTable seg, TileMap map, const uint32_t* __restrict__ n_unique,
                       const uint32_t* __restrict__ n_octree, int32_t* __restrict__ seg_err,
                       OctOut o, const uint32_t* __restrict__ far, uint32_t far_cap,
                       const uint32_t* __restrict__ far_n) {
  pdl_enter();
  octree_far_links<K>(codes_all, prefix_all, parents_all, ec_all, off_all, seg, map, n_unique,
                      n_octree, seg_err, o, far, far_cap, far_n);
}

// ---------------------------------------------------------------------------
// options outside the reference contract (rw_tree_im_storage_set_options)
// ---------------------------------------------------------------------------

template <typename K>
__global__ void __launch_bounds__(256)
    k_leaf_claim(const K* __restrict__ codes, const uint8_t* __restrict__ pn,
                 const uint8_t* __restrict__ hl, const uint8_t* __restrict__ hr,
                 const int32_t* __restrict__ lc, const int32_t* __restrict__ par,
                 const int32_t* __restrict__ ec, const int32_t* __restrict__ off,
                 int32_t* __restrict__ children, const uint32_t* __restrict__ n_unique,
                 uint32_t rows) {
  pdl_enter();
  leaf_claim<K>(codes, pn, hl, hr, lc, par, ec, off, children, n_unique, rows);
}

__global__ void __launch_bounds__(256)
    k_leaf_write(const int32_t* __restrict__ lc, int32_t* __restrict__ children,
                 const uint32_t* __restrict__ n_unique, const uint32_t* __restrict__ n_octree,
                 uint32_t rows) {
  pdl_enter();
  leaf_write(lc, children, n_unique, n_octree, rows);
}

// ---------------------------------------------------------------------------
// counts and errors to and from the host
// ---------------------------------------------------------------------------

// Kernels in the chain of programmatic launches instead of 16-byte copies, which
// would end it and wait for a copy engine (2,000,003 points, the stages called one by
// one: 349 -> 289 us; a batch of 256 clouds 707 -> 689); host memory is pinned.
__global__ void k_status_in(DevStatus* __restrict__ st, uint32_t n_unique, uint32_t n_octree,
                            uint32_t* __restrict__ far_n) {
  pdl_enter();
  *st = DevStatus{n_unique, n_octree, 0, 0};
  *far_n = 0;
}

__global__ void __launch_bounds__(256)
    k_words_out(const uint32_t* a, const uint32_t* b, const uint32_t* c, uint32_t count,
                const DevStatus* __restrict__ st, uint32_t* host) {
  pdl_enter();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += gridDim.x * blockDim.x) {
    host[i] = a[i];
    host[count + i] = b[i];
    host[2 * count + i] = c[i];
  }
  if (blockIdx.x == 0 && threadIdx.x < sizeof(DevStatus) / 4)
    host[3 * count + threadIdx.x] = reinterpret_cast<const uint32_t*>(st)[threadIdx.x];
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

namespace {


template <typename K>
cudaError_t unique_t(const Bufs& b, const Scratch& sc, const Plan& pl, bool counted,
                     cudaStream_t s) {
  const uint32_t tiles = pl.unique_map.n_tiles;
  if (!tiles) return cudaSuccess;
  const K* sorted = static_cast<const K*>(b.alt);
  if (!counted)
    launch_pdl(k_unique_count<K>, tiles, kUniqueThreads, 0, s, sorted, pl.seg, pl.unique_map,
               sc.unique_desc);
  launch_pdl(k_tile_scan, 1, 1024, 0, s, sc.unique_desc, tiles, pl.seg, pl.unique_map, pl.n_unique);
  launch_pdl(k_unique_write<K>, tiles, kUniqueThreads, 0, s, sorted, static_cast<K*>(b.keys), pl.seg,
                                                     pl.unique_map, sc.unique_desc);
  return cudaGetLastError();
}

template <typename K, bool EDGES, int LESS>
cudaError_t tree_t(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s) {
  const uint32_t tiles = pl.tree_map.n_tiles;
  if (!tiles) return cudaSuccess;
  constexpr size_t smem = AnsvCfg<K, kTreeTile / 32>::kSmem;
  const auto kern = k_radix_tree<K, EDGES, LESS>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  // eight blocks of 32-bit keys need nearly all of the SM's shared memory
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                             int(cudaSharedmemCarveoutMaxShared));
  if (e != cudaSuccess) return e;
  launch_pdl(kern, tiles, kTreeThreads, smem, s, static_cast<const K*>(b.keys), pl.seg,
             pl.tree_map, pl.n_unique, pl.seg_err, b.prefix_n, b.hl, b.hr, b.lc, b.parents,
             EDGES ? b.edge_count : static_cast<int32_t*>(nullptr), pl.node_map,
             EDGES ? sc.scan_desc : static_cast<uint32_t*>(nullptr));
  return cudaGetLastError();
}

template <typename K>
cudaError_t octree_t(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s,
                     cudaEvent_t* marks, bool fused_offsets) {
  OctOut o{b.children, b.corner, b.cell_size, b.node_mask, b.leaf_mask, pl.oct_off,
           pl.oct_capacity};
  const K* codes = static_cast<const K*>(b.keys);
  const uint32_t tiles = pl.node_map.n_tiles;
  uint32_t* far_n = sc.tile_ctr + kCtrLinks;
  // (*far_n is zero: the fused pipeline clears every counter when it starts,
  // stage 7 run alone brings its counts with launch_status_in)
  // eight blocks of 32-bit keys need nearly all of the SM's shared memory
  cudaError_t e = cudaFuncSetAttribute(fused_offsets ? k_octree<K, true> : k_octree<K, false>,
                                       cudaFuncAttributePreferredSharedMemoryCarveout,
                                       int(cudaSharedmemCarveoutMaxShared));
  if (e != cudaSuccess) return e;
  if (tiles) {
    if (fused_offsets)
      launch_pdl(k_octree<K, true>, tiles, kOctThreads, 0, s, 
          codes, b.prefix_n, b.parents, b.edge_count, b.edge_offset, sc.scan_desc, pl.seg,
          pl.node_map, pl.n_unique, pl.n_octree, pl.seg_err, b.min_coord, b.range, o,
          sc.tree_far, sc.tree_far_cap, far_n);
    else
      launch_pdl(k_octree<K, false>, tiles, kOctThreads, 0, s, 
          codes, b.prefix_n, b.parents, b.edge_count, b.edge_offset, nullptr, pl.seg,
          pl.node_map, pl.n_unique, pl.n_octree, pl.seg_err, b.min_coord, b.range, o,
          sc.tree_far, sc.tree_far_cap, far_n);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (marks) cudaEventRecord(marks[0], s);
  if (tiles)
    launch_pdl(k_octree_far_links<K>, std::max(1, sc.num_sms * 8), 256, 0, s, 
        codes, b.prefix_n, b.parents, b.edge_count, b.edge_offset, pl.seg, pl.node_map,
        pl.n_unique, pl.n_octree, pl.seg_err, o, sc.tree_far, sc.tree_far_cap, far_n);
  e = cudaGetLastError();
  if (e == cudaSuccess && marks) cudaEventRecord(marks[1], s);
  return e;
}

}  // namespace

cudaError_t launch_unique(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s,
                          bool counted) {
  return b.key_bits == 32 ? unique_t<uint32_t>(b, sc, pl, counted, s)
                          : unique_t<uint64_t>(b, sc, pl, counted, s);
}

namespace {
template <typename K>
cudaError_t leaf_links_t(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s) {
  const K* codes = static_cast<const K*>(b.keys);
  const int grid = std::max(1, sc.num_sms * 8);
  launch_pdl(k_leaf_claim<K>, grid, 256, 0, s, codes, b.prefix_n, b.hl, b.hr, b.lc, b.parents,
             b.edge_count, b.edge_offset, b.children, pl.n_unique, pl.oct_capacity);
  launch_pdl(k_leaf_write, grid, 256, 0, s, b.lc, b.children, pl.n_unique, pl.n_octree,
             pl.oct_capacity);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_leaf_links(const Bufs& b, const Scratch& sc, const Plan& pl,
                              cudaStream_t s) {
  if (pl.seg.count != 1) return cudaErrorInvalidValue;
  return b.key_bits == 32 ? leaf_links_t<uint32_t>(b, sc, pl, s)
                          : leaf_links_t<uint64_t>(b, sc, pl, s);
}

cudaError_t launch_unique_raw(const void* sorted, void* out, uint32_t n, int key_bits,
                              uint32_t* counts, DevStatus* status, int num_sms,
                              cudaStream_t s) {
  Bufs b;
  b.key_bits = key_bits;
  b.alt = const_cast<void*>(sorted);
  b.keys = out;
  Scratch sc;
  sc.num_sms = num_sms;
  sc.unique_desc = counts;
  sc.status = status;
  const Plan pl = single_plan(n, 0, status, 0);
  return launch_unique(b, sc, pl, s);
}

cudaError_t launch_radix_tree(const Bufs& b, const Scratch& sc, const Plan& pl, bool edges,
                              bool geometric, cudaStream_t s) {
  // 64-bit codes fill their word but for the sign bit: their clz - 1 is exact
  if (b.key_bits == 64)
    return edges ? tree_t<uint64_t, true, 0>(b, sc, pl, s) : tree_t<uint64_t, false, 0>(b, sc, pl, s);
  if (geometric)
    return edges ? tree_t<uint32_t, true, 1>(b, sc, pl, s) : tree_t<uint32_t, false, 1>(b, sc, pl, s);
  return edges ? tree_t<uint32_t, true, 0>(b, sc, pl, s) : tree_t<uint32_t, false, 0>(b, sc, pl, s);
}

cudaError_t launch_edge_count(const Bufs& b, const Scratch& sc, const Plan& pl,
                              cudaStream_t s) {
  (void)sc;
  if (!pl.node_map.n_tiles) return cudaSuccess;
  launch_pdl(k_edge_count, pl.node_map.n_tiles, kOctThreads, 0, s, 
      b.prefix_n, b.parents, b.edge_count, pl.seg, pl.node_map, pl.n_unique);
  return cudaGetLastError();
}

cudaError_t launch_edge_scan(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s) {
  const uint32_t tiles = pl.scan_map.n_tiles;
  if (!tiles) return cudaSuccess;
  launch_pdl(k_scan_reduce, tiles, kScanThreads, 0, s, b.edge_count, pl.seg, pl.scan_map, pl.n_unique,
                                               sc.scan_desc);
  launch_pdl(k_tile_scan, 1, 1024, 0, s, sc.scan_desc, tiles, pl.seg, pl.scan_map, pl.n_octree);
  launch_pdl(k_scan_write, tiles, kScanThreads, 0, s, b.edge_count, b.edge_offset, pl.seg,
                                              pl.scan_map, pl.n_unique, sc.scan_desc);
  return cudaGetLastError();
}

cudaError_t launch_edge_sums(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s) {
  const uint32_t tiles = pl.node_map.n_tiles;
  if (!tiles) return cudaSuccess;
  launch_pdl(k_tile_scan, 1, 1024, 0, s, sc.scan_desc, tiles, pl.seg, pl.node_map, pl.n_octree);
  return cudaGetLastError();
}

cudaError_t launch_octree(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s,
                          cudaEvent_t* marks, bool fused_offsets) {
  return b.key_bits == 32 ? octree_t<uint32_t>(b, sc, pl, s, marks, fused_offsets)
                          : octree_t<uint64_t>(b, sc, pl, s, marks, fused_offsets);
}

cudaError_t launch_status_in(const Scratch& sc, uint32_t n_unique, uint32_t n_octree,
                             cudaStream_t s) {
  launch_pdl(k_status_in, 1, 1, 0, s, sc.status, n_unique, n_octree, sc.tile_ctr + kCtrLinks);
  return cudaGetLastError();
}

cudaError_t launch_status_out(const DevStatus* status, DevStatus* host, cudaStream_t s) {
  launch_pdl(k_words_out, 1, 32, 0, s, nullptr, nullptr, nullptr, 0u, status,
             reinterpret_cast<uint32_t*>(host));
  return cudaGetLastError();
}

cudaError_t launch_results_out(const Plan& pl, const DevStatus* status, uint32_t* host,
                               cudaStream_t s) {
  launch_pdl(k_words_out, std::min(32u, div_up(pl.seg.count, 256)), 256, 0, s, pl.n_unique,
             pl.n_octree, reinterpret_cast<const uint32_t*>(pl.seg_err), pl.seg.count, status, host);
  return cudaGetLastError();
}

Plan single_plan(uint32_t n, uint32_t oct_capacity, DevStatus* status, uint32_t sort_tile) {
  Plan pl;
  pl.seg = SegTable{1u, n, nullptr};
  pl.point_map = TileMap{div_up(n, kPointTile), nullptr};
  pl.sort_map = TileMap{sort_tile ? div_up(n, sort_tile) : 0u, nullptr};
  pl.unique_map = TileMap{div_up(n, kUniqueTile), nullptr};
  pl.tree_map = TileMap{div_up(n, kTreeTile), nullptr};
  pl.scan_map = TileMap{div_up(n, kScanTile), nullptr};
  pl.node_map = TileMap{div_up(n, kOctTile), nullptr};
  pl.n_unique = &status->n_unique;
  pl.n_octree = &status->n_octree_nodes;
  pl.seg_err = &status->err;
  pl.oct_off = nullptr;
  pl.oct_capacity = oct_capacity;
  return pl;
}

}  // namespace rwt
