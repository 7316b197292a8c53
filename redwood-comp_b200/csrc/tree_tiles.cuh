// Device code of stages 4 to 7 over one tile of radix-tree gaps or nodes, shared
// by the kernels that launch a block per tile (k_tree.cu) and the one that
// keeps a whole small cloud on the chip (k_small.cu).
#pragma once

#include "internal.hpp"
#include "morton.cuh"

namespace rwt {

// Highest set bit of x, -1 for 0.
__device__ __forceinline__ int highest_bit(uint32_t x) {
  int r;
  asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}
// x / 3 for 0 <= x < 256.
__device__ __forceinline__ int third(int x) { return (x * 171) >> 9; }

// ---------------------------------------------------------------------------
// stage 4: radix-tree nodes (func_brt.hpp:45-138)
// ---------------------------------------------------------------------------

// delta(a, b) > d, for codes whose top bit is clear (the reference asserts it,
// func_brt.hpp:30-31): clz(a ^ b) - 1 > d  <=>  a ^ b < 2^(W - 2 - d).  `lim`
// is that bound (0 when d >= W - 1: never true).
template <typename K>
__device__ __forceinline__ K delta_limit(int d) {
  constexpr int W = KeyTraits<K>::kWordBits;
  return (d >= 0 && d <= W - 2) ? (K(1) << (W - 2 - d)) : K(0);
}

// Writes node 0 (the reference's root over [0, n - 1], func_brt.hpp:80-138),
// which splits at gamma: prefix_n / leaf flags / left_child, parents[0] = 0
// and a zero for each internal child of the true root of [0, n] (sequential
// execution on a zeroed buffer leaves exactly those entries 0, and no other
// node names them).
template <typename K, int LESS>
__device__ __forceinline__ void write_root(const K* __restrict__ codes, int n, int dnode,
                                           int gamma, uint8_t* prefix_n, uint8_t* hl,
                                           uint8_t* hr, int32_t* lc, int32_t* parents) {
  prefix_n[0] = uint8_t(dnode - LESS);
  hl[0] = gamma == 0;
  hr[0] = gamma + 1 == n - 1;
  lc[0] = gamma;
  parents[0] = 0;
  const int gamma_true = delta(codes[n - 1], codes[n]) < dnode ? n - 1 : gamma;
  if (gamma_true > 0) parents[gamma_true] = 0;
  if (gamma_true + 1 < n) parents[gamma_true + 1] = 0;
}

__device__ __forceinline__ void seg_error(int32_t* seg_err, uint32_t c, int32_t code) {
  atomicCAS(reinterpret_cast<int*>(seg_err + c), 0, code);
}

// ---- stages 4 (+5) from nearest smaller values ----------------------------
//
// With D[k] = delta(key k, key k+1) for the n gaps k in [0, n), the binary
// radix tree of the keys is the Cartesian tree of D: the node that splits at
// gap g covers keys [L+1, R], where L < g and R > g are the nearest gaps with
// D strictly smaller than D[g] (-1 and n when there are none); its prefix
// length is D[g]; its parent splits at whichever of L, R has the larger D; and
// its Karras index (the one process_radix_tree_i gives it, func_brt.hpp:45-138)
// is R when it is its parent's left child and L+1 when it is the right child.
// Every node's outputs follow without a search: left_child = g, leaf flags
// g == L+1 and g+1 == R, the internal children's parent links, and the edge
// count from the parent's prefix max(D[L], D[R]).  The root (L = -1, R = n)
// is node 0, which keeps the reference's own range [0, n-1] (write_root above).
//
// L and R per gap: in chunks of 32 gaps (one per lane) a bit-serial warp
// comparison of E = D + 1 (0 marks the walls at -1 and n) gives every lane
// the lanes with a smaller value, hence the nearest smaller in the chunk, and
// every value v the last / first position in the chunk below v.  Across the
// tile and a halo of kAnsvHalo chunks on either side, per-value bitmasks of
// the chunks whose minimum lies below v find the nearest such chunk in one
// clz / ffs, and its summary gives the answer; a gap whose nearest smaller
// lies beyond the halo (a node near the top of the tree) goes to a list in
// shared memory that the block resolves at its end with warp-cooperative
// searches of the keys.
constexpr int kAnsvHalo = 8;             // chunks per side
constexpr int kAnsvNone = -0x7fffffff;     // "no smaller gap found to the left"
constexpr int kAnsvNoneR = 0x7fffffff;     // "none to the right"

// Last / first position in a chunk of 32 E values (4-byte aligned) whose
// value is below e; the caller knows there is one.
__device__ __forceinline__ int chunk_last_below(const uint8_t* ce, int e) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(ce);
  const uint32_t ev = 0x01010101u * uint32_t(e);
  for (int q = 7; q > 0; --q) {
    const uint32_t below = __vcmpltu4(w[q], ev);  // 0xff in each byte below e
    if (below) return 4 * q + (31 - __clz(below)) / 8;
  }
  return (31 - __clz(__vcmpltu4(w[0], ev))) / 8;
}

__device__ __forceinline__ int chunk_first_below(const uint8_t* ce, int e) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(ce);
  const uint32_t ev = 0x01010101u * uint32_t(e);
  for (int q = 0; q < 7; ++q) {
    const uint32_t below = __vcmpltu4(w[q], ev);
    if (below) return 4 * q + (__ffs(below) - 1) / 8;
  }
  return 28 + (__ffs(__vcmpltu4(w[7], ev)) - 1) / 8;
}

// TCH: the most chunks of 32 gaps that a tile has.
template <typename K, int TCH>
struct AnsvCfg {
  static constexpr int NV = sizeof(K) == 4 ? 32 : 64;  // values of E
  static constexpr int VB = sizeof(K) == 4 ? 5 : 6;    // bits of E
  static constexpr int kChunks = TCH + 2 * kAnsvHalo;  // chunks per window
  static constexpr int kWin = kChunks * 32;            // gaps per window
  static constexpr int kRow = TCH + 1;  // padded: lane v and chunk c in different banks
  static constexpr size_t kKeyBytes = (size_t(kWin) + 1) * sizeof(K);
  static constexpr int MW = (kChunks + 31) / 32;  // mask words per value
  static constexpr size_t kSmem = kKeyBytes + size_t(NV) * MW * 4 + 4 * size_t(TCH) * 32 +
                                  size_t(kWin) + 2 * size_t(NV) * kRow + size_t(kChunks);
};

// Warp-cooperative search for the nearest smaller gaps of gap g beyond any
// window, both sides in lockstep: 32 probes per side and round (doubling
// distances, then 32-ary refinement), the two sides' loads issued together,
// so the pair costs about as many dependent loads as the longer side.
// Left: pred(a) = delta(key a, key g) > D is true from some a_min up to g;
// *first_key = a_min (the node's first key).  Right: pred(b) = delta(key g+1,
// key b) > D is true from g+1 up to some b_max <= n; *last_key = b_max.
template <typename K>
__device__ void coop_node_keys(const K* __restrict__ codes, int n, int g, int D,
                               int* first_key, int* last_key) {
  const uint32_t lane = lane_id();
  const K cl = codes[g], cr = codes[g + 1], lim = delta_limit<K>(D);
  const int pl = lane < 31 ? g - (1 << lane) : -1;
  const long long pr = lane < 31 ? (long long)g + 1 + (1ll << lane) : (long long)n + 1;
  const bool fl = pl >= 0 && (codes[pl] ^ cl) < lim;
  const bool fr = pr <= n && (codes[int(pr)] ^ cr) < lim;
  const int jl = __ffs(__ballot_sync(0xffffffffu, !fl)) - 1;  // a false probe exists
  const int jr = __ffs(__ballot_sync(0xffffffffu, !fr)) - 1;
  int llo = max(jl < 31 ? g - (1 << jl) : -1, -1);                // pred(llo) false
  int lhi = jl == 0 ? g : g - (1 << (jl - 1));                    // pred(lhi) true
  int rhi = jr < 31 ? int(min((long long)g + 1 + (1ll << jr), (long long)n + 1)) : n + 1;
  int rlo = jr == 0 ? g + 1 : g + 1 + (1 << (jr - 1));            // pred(rlo) true
  while (lhi - llo > 1 || rhi - rlo > 1) {
    const bool la = lhi - llo > 1, ra = rhi - rlo > 1;  // warp-uniform
    const int ls = la ? (lhi - llo + 31) / 32 : 0, rs = ra ? (rhi - rlo + 31) / 32 : 0;
    const int lq = llo + (int(lane) + 1) * ls, rq = rlo + (int(lane) + 1) * rs;
    const bool lin = la && lane < 31 && lq < lhi, rin = ra && lane < 31 && rq < rhi;
    const bool lt = lin && (codes[lq] ^ cl) < lim;
    const bool rt = rin && (codes[rq] ^ cr) < lim;
    const uint32_t mlt = __ballot_sync(0xffffffffu, lt), mli = __ballot_sync(0xffffffffu, lin);
    const uint32_t mrf = __ballot_sync(0xffffffffu, rin && !rt),
                   mri = __ballot_sync(0xffffffffu, rin);
    if (la) {
      if (mlt) {
        const int ft = __ffs(mlt) - 1;
        lhi = llo + (ft + 1) * ls;
        llo = ft > 0 ? llo + ft * ls : llo;
      } else {
        llo = llo + (32 - __clz(mli)) * ls;  // the last probe in range is false
      }
    }
    if (ra) {
      if (mrf) {
        const int ff = __ffs(mrf) - 1;
        rhi = rlo + (ff + 1) * rs;
        rlo = ff > 0 ? rlo + ff * rs : rlo;
      } else {
        rlo = rlo + (32 - __clz(mri)) * rs;  // every probe in range is true
      }
    }
  }
  *first_key = lhi;
  *last_key = rlo;
}

// Last b in [0, n - 1) with delta(key 0, key b) > D, for a D with delta(key 0,
// key n - 1) = D (so key n - 1 does not qualify): where node 0 splits.  One
// warp, 32 probes a round (doubling distances, then 32-ary refinement).
template <typename K>
__device__ int coop_root_split(const K* __restrict__ codes, int n, int D) {
  const int lane = int(lane_id());
  const K c0 = codes[0], lim = delta_limit<K>(D);
  const int pd = lane < 31 ? (1 << lane) : 0x7fffffff;
  const bool t = pd < n - 1 && (codes[pd] ^ c0) < lim;
  const int j = __ffs(__ballot_sync(0xffffffffu, !t)) - 1;  // lane 31 never holds
  int lo = j == 0 ? 0 : 1 << (j - 1);                       // holds
  int hi = j < 31 ? min(1 << j, n - 1) : n - 1;             // does not
  while (hi - lo > 1) {
    const int st = (hi - lo + 31) / 32, q = lo + (lane + 1) * st;
    const bool in = lane < 31 && q < hi;
    const uint32_t f = __ballot_sync(0xffffffffu, in && !((codes[q] ^ c0) < lim));
    const uint32_t mi = __ballot_sync(0xffffffffu, in);
    if (f) {
      const int ff = __ffs(f) - 1;
      hi = lo + (ff + 1) * st;
      lo += ff * st;
    } else {
      lo += (32 - __clz(mi)) * st;  // every probe in range holds
    }
  }
  return lo;
}

// Writes the node that splits at gap g, given its nearest smaller gaps L, R
// (see the ANSV comment below); the root (L = -1, R = n) is skipped.
// dl, dr: D of gaps L and R (-1 for the walls at -1 and n).  LESS (0 or 1) is
// taken off every prefix length that is written or counted
// (RW_TREE_OPT_GEOMETRIC_DELTA: the tree's shape depends only on comparisons
// between deltas, so the clz - 2 tree is the clz - 1 tree with every prefix,
// at least 1 for distinct 30-bit keys, lowered by one).
// Returns the node's index; *count gets its edge count (0 without EDGES).
template <bool EDGES, int LESS>
__device__ __forceinline__ int write_gap_node_d(int g, int D, int L, int R, int dl, int dr,
                                                int root_true_delta, int root_prefix,
                                                uint8_t* pn, uint8_t* l8, uint8_t* r8,
                                                int32_t* lcs, int32_t* par, int32_t* ec,
                                                int* count) {
  const int i = dr > dl ? R : L + 1;  // left child of R's node, else right child of L's
  const bool leaf_l = g == L + 1, leaf_r = g + 1 == R;
  // The kernel is bound by its integer instructions: 32-bit byte offsets from
  // the arrays' starts (below 2^32: i < 2^30) and thirds by one multiplication
  // took 16.8M points from 187.7 to 179.6 us, the mixture from 126.6 to 121.4.
  const uint32_t u = uint32_t(i), g4 = 4u * uint32_t(g);
  auto word = [](int32_t* p, uint32_t bytes) {
    return reinterpret_cast<int32_t*>(reinterpret_cast<char*>(p) + bytes);
  };
  pn[u] = uint8_t(D - LESS);
  l8[u] = leaf_l;
  r8[u] = leaf_r;
  *word(lcs, 4u * u) = g;
  if (!leaf_l) *word(par, g4) = i;
  if (!leaf_r) *word(par, g4 + 4u) = i;
  *count = 0;
  if (EDGES) {
    const int pd = max(dl, dr);
    const int pp = pd == root_true_delta ? root_prefix : pd;
    *count = third(D - LESS) - third(pp - LESS);
    *word(ec, 4u * u) = *count;
  }
  return i;
}

// Octree tiles that the nodes of a radix-tree tile of up to 4,096 gaps can lie in
// (a tile of k_small starts anywhere).
constexpr int kTreeSums = 4096 / int(kOctTile) + 1;

// The shared words of a tile besides the arrays in dynamic shared memory.
struct TreeTileShared {
  uint32_t far[kTreeFarPerTile];  // the tile's gaps left to phase D
  uint32_t far_n, pend_n;
  int sum[kTreeSums];  // edge counts of the nodes [g0, ..) by octree tile
  alignas(8) uint64_t bar;
};

// Stage 4 (and 5 with EDGES) for the gaps [g0, g0 + 32 tch) of a cloud whose n
// gaps lie between codes[0 .. n], by a block of NT threads.  DYN: tch is a run
// time number up to TCH, else it is TCH.  BULK: the keys may come by a bulk
// copy (not in a kernel that wrote them itself: the copy engine would need a
// proxy fence).  `err` takes the first error.  The tile that starts at 0 also
// writes node 0.  With EDGES the counts of every kOctTile nodes are also added
// up in sums (zero before): stage 6's reduction, which as a kernel of its own
// read every count again (16.8M uniform points, 32-bit keys: tree and scan 205.1
// -> 198.5 us; gathering the nodes in shared memory to write and sum them in
// order took more instructions than it saved, 203.4).
template <typename K, bool EDGES, int LESS, int NT, int TCH, bool DYN, bool BULK>
__device__ __forceinline__ void tree_tile(unsigned char* smem_raw, TreeTileShared& sh,
                                          const K* __restrict__ codes, int n, int g0,
                                          int tch_arg, int32_t* err, uint8_t* __restrict__ pn,
                                          uint8_t* __restrict__ l8, uint8_t* __restrict__ r8,
                                          int32_t* __restrict__ lcs, int32_t* __restrict__ par,
                                          int32_t* __restrict__ ec,
                                          uint32_t* __restrict__ sums) {
  using C = AnsvCfg<K, TCH>;
  constexpr int NV = C::NV, VB = C::VB, NW = NT / 32, JN = DYN ? 1 : 2;
  static_assert(kTreeFarPerTile >= 2 * uint32_t(NV), "far gaps of a tile: NV per side");
  const int tch = DYN ? tch_arg : TCH;
  const int chunks = tch + 2 * kAnsvHalo, win = chunks * 32;
  // positions inside a chunk are kept as lane indices (0xff: none)
  K* s_key = reinterpret_cast<K*>(smem_raw);                                // [win + 1]
  uint32_t* s_mask = reinterpret_cast<uint32_t*>(smem_raw + C::kKeyBytes);  // [NV][MW]
  // the tile's gaps left to phase C: tile index | in-chunk left << 16 |
  // in-chunk right << 24 (lane indices, 0xff: none)
  uint32_t* s_pend = s_mask + NV * C::MW;                                   // [32 TCH]
  uint8_t* s_e = reinterpret_cast<uint8_t*>(s_pend + 32 * TCH);             // [win]
  // summaries of the tile's chunks only (a halo chunk is scanned when asked)
  uint8_t* s_last = s_e + C::kWin;                                          // [NV][kRow]
  uint8_t* s_first = s_last + NV * C::kRow;                                 // [NV][kRow]
  uint8_t* s_cmin = s_first + NV * C::kRow;                                 // [chunks]
  const int wlo = g0 - kAnsvHalo * 32;  // first gap of the window

  int root_true_delta = 0, root_prefix = 0;
  if (EDGES) {
    root_true_delta = delta(codes[0], codes[n]);
    root_prefix = delta(codes[0], codes[n - 1]);
  }
  // node 0, the reference's range [0, n - 1], by the last warp: as one thread's
  // binary search it was a chain of about 2 log2(n) dependent loads that the
  // whole first block waited for (16.5 us for the kernel at 3,001 points, two
  // blocks); 32 probes a round need at most 6
  auto root_node = [&] {
    const int d0 = delta(codes[0], codes[n - 1]);
    const int gamma = coop_root_split<K>(codes, n, d0);
    if (lane_id() == 0) {
      write_root<K, LESS>(codes, n, d0, gamma, pn, l8, r8, lcs, par);
      if (EDGES) ec[0] = 0;
    }
  };
  if (!DYN && g0 == 0 && threadIdx.x >= NT - 32) root_node();

  // read after the barriers below
  if (threadIdx.x == 0) sh.far_n = sh.pend_n = 0;
  if (EDGES && threadIdx.x < kTreeSums) sh.sum[threadIdx.x] = 0;
  const int t0 = g0 / int(kOctTile);  // the octree tile of sh.sum[0]

  // the window's keys [wlo, wlo + kAnsvWin]: one bulk copy when the window
  // lies inside the keys and starts on a 16-byte boundary (every interior
  // tile of a plain run), else key by key; outside [0, n] the first and the last
  // key go on with their top bit changing from each key to the next, so that
  // the gaps there come out as E = 0 without a check, whatever the keys (16.8M
  // 32-bit keys 179.6 -> 173.8 us together with highest_bit)
  static_assert((size_t(C::kWin) * sizeof(K)) % 16 == 0, "bulk copies move 16-byte units");
  const bool bulk = BULK && wlo >= 0 && wlo + win <= n &&
                    (reinterpret_cast<uintptr_t>(codes + wlo) & 15u) == 0;
  if (bulk) {
    if (threadIdx.x == 0) bulk_barrier_init(&sh.bar);
    __syncthreads();
    if (threadIdx.x == 0) {
      bulk_load(s_key, codes + wlo, uint32_t(win * sizeof(K)), &sh.bar);
      s_key[win] = codes[wlo + win];
    }
    const bool landed = bulk_wait(&sh.bar, kSpinLimit);
    if (__syncthreads_or(!landed)) {  // the whole block gives up together
      // report, and let the copy land before the block's shared memory goes
      if (threadIdx.x == 0) atomicCAS(reinterpret_cast<int*>(err), 0, RW_ERR_TIMEOUT);
      bulk_wait(&sh.bar, kSpinLimit);
      return;
    }
  } else {
    for (int j = threadIdx.x; j <= win; j += NT) {
      const int k = wlo + j;
      const int out = k < 0 ? -k : k > n ? k - n : 0;  // how far outside
      s_key[j] = codes[min(max(k, 0), n)] ^ K(out & 1) << (8 * sizeof(K) - 1);
    }
  }
  __syncthreads();

  // phase A: per chunk, E, the nearest smaller inside the chunk, and the
  // chunk's summaries (last / first position with E below each value).  A gap
  // of the tile whose nearest smaller gaps on both sides lie in its own chunk
  // (about four in five on uniform keys) writes its node here, with the D of
  // both from its neighbours' lanes; the others go to the list of phase C.
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  static_assert(C::kKeyBytes % 4 == 0, "the masks follow the keys");
  // the halo chunks need only E and their minimum: a lookup that ends in one
  // scans its 32 values (phase C)
  static_assert(2 * kAnsvHalo % NW == 0 || NW > 2 * kAnsvHalo, "whole rounds of halo chunks");
  for (int hc = int(warp); hc < 2 * kAnsvHalo; hc += NW) {
    const int ch = hc < kAnsvHalo ? hc : hc + tch;
    const int w = ch * 32 + int(lane);
    const int e = KeyTraits<K>::clz(s_key[w] ^ s_key[w + 1]);
    s_e[w] = uint8_t(e);
    const uint32_t cmin = __reduce_min_sync(0xffffffffu, uint32_t(e));
    if (lane == 0) s_cmin[ch] = uint8_t(cmin);
  }
  // the tile's chunks two at a time per warp, so that their ballot chains
  // interleave (one at a time where a warp has few)
  static_assert(DYN || TCH % (JN * NW) == 0, "whole groups of chunks per warp");
  // lane v's threshold bits as masks (all ones where v has the bit), the same
  // for every chunk: kept in registers, since the kernel is bound by its
  // integer instructions
  uint32_t mlane[VB];
#pragma unroll
  for (int bt = 0; bt < VB; ++bt) mlane[bt] = 0u - ((lane >> bt) & 1u);
  int acc = 0;  // edge counts of this lane's nodes
  for (int ch0 = kAnsvHalo + int(warp); ch0 < kAnsvHalo + tch; ch0 += JN * NW) {
    int e[JN];
#pragma unroll
    for (int j = 0; j < JN; ++j) {
      const int ch = ch0 + j * NW;
      const int w = ch * 32 + int(lane);  // window index of this lane's gap
      // distinct keys whose top bit is clear: E = delta + 1 = clz of the xor,
      // at least 1 for a real gap, so 0 marks walls only
      e[j] = KeyTraits<K>::clz(s_key[w] ^ s_key[w + 1]);
      s_e[w] = uint8_t(e[j]);
      const uint32_t cmin = __reduce_min_sync(0xffffffffu, uint32_t(e[j]));
      if (lane == 0) s_cmin[ch] = uint8_t(cmin);
    }
    // bit-serial comparison of every lane's E against v = lane (and lane + 32
    // for 64-bit keys): lane v ends with the lanes whose E is below v; the
    // lanes below my own value are then lane e's result
    // (branch-free: with m = all ones where v has the bit, a lane stays equal
    // while its bit matches, eq &= ~(B ^ m), and falls below where v has the
    // bit and it has not, lt |= eq & ~B & m)
    uint32_t lt0[JN], eq0[JN];  // below v = lane
    uint32_t lt1[JN], eq1[JN];  // below v = lane + 32
#pragma unroll
    for (int j = 0; j < JN; ++j) {
      lt0[j] = lt1[j] = 0;
      eq0[j] = eq1[j] = 0xffffffffu;
    }
#pragma unroll
    for (int bt = VB - 1; bt >= 0; --bt) {
      uint32_t B[JN];
#pragma unroll
      for (int j = 0; j < JN; ++j) B[j] = __ballot_sync(0xffffffffu, (e[j] >> bt) & 1);
      // v = lane + 32 has bit 5 set and lane's bits below it
      const uint32_t m0 = mlane[bt], m1 = bt == 5 ? 0xffffffffu : mlane[bt];
#pragma unroll
      for (int j = 0; j < JN; ++j) {
        lt0[j] |= eq0[j] & ~B[j] & m0;
        eq0[j] &= ~(B[j] ^ m0);
        if (NV > 32) {
          lt1[j] |= eq1[j] & ~B[j] & m1;
          eq1[j] &= ~(B[j] ^ m1);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < JN; ++j) {
      const int ch = ch0 + j * NW;
      // (the shuffles take the lane index modulo 32)
      const uint32_t from0 = __shfl_sync(0xffffffffu, lt0[j], e[j]);
      const uint32_t from1 = NV > 32 ? __shfl_sync(0xffffffffu, lt1[j], e[j]) : 0u;
      const uint32_t lt = (NV > 32 && e[j] >= 32) ? from1 : from0;
      {
        const int tg = (ch - kAnsvHalo) * 32 + int(lane);
        // lt never holds the lane itself; clz(0) = 32 and ffs(0) = 0 give -1
        const uint32_t lm = lt & lanemask_lt(), rm = lt & ~lm;
        // (the one instruction is the faster form with the 64-bit kernel's
        // registers only: 75.1 against 76.0 us, 32-bit 176.2 against 173.8)
        const int lp = NV > 32 ? highest_bit(lm) : 31 - __clz(lm);
        const int rp = __ffs(rm) - 1;
        // E of the two nearest smaller lanes (a wall lane past the last gap
        // has E = 0, so D = -1 there as for the wall at n)
        const int el = __shfl_sync(0xffffffffu, e[j], lp);
        const int er = __shfl_sync(0xffffffffu, e[j], rp);
        const int g = g0 + tg;
        const bool here = lm && rm;  // (no lane lies below a wall)
        int count = 0;
        if (here)
          write_gap_node_d<EDGES, LESS>(g, e[j] - 1, g - int(lane) + lp, g - int(lane) + rp,
                                        el - 1, er - 1, root_true_delta, root_prefix, pn, l8, r8,
                                        lcs, par, ec, &count);
        if (EDGES) {
          // a chunk's own nodes lie in the chunk, so in one octree tile, and
          // the chunks of a round in the same one (a sum kept over the rounds
          // would need a register more than eight blocks leave: 194 us)
          static_assert(JN == 1 || (JN * NW * 32) <= int(kOctTile), "a round in one octree tile");
          acc += count;
          if (j == JN - 1) {
            acc = __reduce_add_sync(0xffffffffu, acc);
            if (lane == 0) atomicAdd(&sh.sum[(g0 + (ch - kAnsvHalo) * 32) / int(kOctTile) - t0], acc);
            acc = 0;
          }
        }
        const uint32_t pm = __ballot_sync(0xffffffffu, e[j] != 0 && !here);
        if (pm) {
          uint32_t at = 0;
          if (lane == uint32_t(__ffs(pm) - 1)) at = atomicAdd(&sh.pend_n, uint32_t(__popc(pm)));
          at = __shfl_sync(0xffffffffu, at, __ffs(pm) - 1) + __popc(pm & lanemask_lt());
          if (e[j] != 0 && !here)
            s_pend[at] = uint32_t(tg) | uint32_t(lp & 0xff) << 16 | uint32_t(rp & 0xff) << 24;
        }
      }
      // an empty mask gives 0xff (none) by itself: 31 - clz(0) = ffs(0) - 1 = -1
      const int tc = ch - kAnsvHalo;  // the chunk's column among the tile's
      s_last[int(lane) * C::kRow + tc] = uint8_t(highest_bit(lt0[j]));
      s_first[int(lane) * C::kRow + tc] = uint8_t(__ffs(lt0[j]) - 1);
      if (NV > 32) {
        s_last[(int(lane) + 32) * C::kRow + tc] = uint8_t(highest_bit(lt1[j]));
        s_first[(int(lane) + 32) * C::kRow + tc] = uint8_t(__ffs(lt1[j]) - 1);
      }
    }
  }
  __syncthreads();

  // phase B: for every value v, a bitmask of the window's chunks whose
  // minimum lies below v (bit c of word c / 32)
  for (int v = int(warp); v < NV; v += NW) {
#pragma unroll
    for (int wd = 0; wd < C::MW; ++wd) {
      const int cidx = wd * 32 + int(lane);
      const uint32_t bits = __ballot_sync(0xffffffffu, cidx < chunks && int(s_cmin[cidx]) < v);
      if (lane == 0) s_mask[v * C::MW + wd] = bits;
    }
  }
  __syncthreads();

  // phase C: every gap of the list writes its node; a gap whose nearest
  // smaller gap lies beyond the window goes to the far-search list
  const int wend = wlo + win - 1;  // last gap of the window
  auto d_at = [&](int p) -> int {       // D of gap p in [0, n)
    return (p >= wlo && p <= wend) ? int(s_e[p - wlo]) - 1 : delta(codes[p], codes[p + 1]);
  };
  // writes the node that splits at gap g, given its nearest smaller gaps L and
  // R (-1 and n for the walls; the root is skipped), and adds its count (to
  // registers for the octree tiles t0 and t0 + 1, the tile's own but for the
  // largest of k_small)
  int sum0 = 0, sum1 = 0;
  auto put = [&](int g, int D, int L, int R, const auto& d_of) {
    if (L < 0 && R >= n) return;
    int count;
    const int i = write_gap_node_d<EDGES, LESS>(
        g, D, L, R, L >= 0 ? d_of(L) : -1, R < n ? d_of(R) : -1, root_true_delta, root_prefix, pn,
        l8, r8, lcs, par, ec, &count);
    if (EDGES) {
      const int t = i / int(kOctTile) - t0;
      if (t == 0) sum0 += count;
      else if (t == 1) sum1 += count;
      else if (count) atomicAdd(sums + t0 + t, uint32_t(count));
    }
  };
  const int np = int(sh.pend_n);
  for (int q = int(threadIdx.x); q < np; q += NT) {
    const uint32_t pw = s_pend[q];
    const int tg = int(pw & 0xffffu), lp = int((pw >> 16) & 0xffu), rp = int(pw >> 24);
    const int g = g0 + tg;
    const int ch = kAnsvHalo + tg / 32;
    const int e = s_e[g - wlo];
    // not inside its own chunk: the nearest chunk on that side whose minimum
    // is below e holds the answer in its summary
    const int cb = wlo + ch * 32;  // first gap of this chunk
    int L = lp != 0xff ? cb + lp : kAnsvNone;
    if (L == kAnsvNone) {
      for (int wd = (ch - 1) >> 5; wd >= 0; --wd) {
        uint32_t bits = s_mask[e * C::MW + wd];
        if (wd == (ch - 1) >> 5) bits &= 0xffffffffu >> (31 - ((ch - 1) & 31));
        if (bits) {
          const int c2 = wd * 32 + 31 - __clz(bits);
          L = wlo + c2 * 32 + (c2 >= kAnsvHalo ? int(s_last[e * C::kRow + c2 - kAnsvHalo])
                                               : chunk_last_below(s_e + c2 * 32, e));
          break;
        }
      }
    }
    int R = rp != 0xff ? cb + rp : kAnsvNoneR;
    if (R == kAnsvNoneR) {
      for (int wd = (ch + 1) >> 5; wd < C::MW; ++wd) {
        uint32_t bits = s_mask[e * C::MW + wd];
        if (wd == (ch + 1) >> 5) bits &= 0xffffffffu << ((ch + 1) & 31);
        if (bits) {
          const int c2 = wd * 32 + __ffs(bits) - 1;
          R = wlo + c2 * 32 +
              (c2 < kAnsvHalo + tch ? int(s_first[e * C::kRow + c2 - kAnsvHalo])
                                                : chunk_first_below(s_e + c2 * 32, e));
          break;
        }
      }
    }
    if (L == kAnsvNone || R == kAnsvNoneR) {
      // resolved by this block below.  The list cannot overflow: two gaps
      // whose nearest smaller gap on the left lies beyond the window never
      // share a value (if a < b did, every gap between them would be at least
      // that value, so the keys a+1 .. b would all have the bit at which keys
      // a and a+1 first differ set, while gap b needs key b to have it clear),
      // so the tile holds at most NV such gaps, and NV more on the right
      const uint32_t local = atomicAdd(&sh.far_n, 1u);
      if (local < kTreeFarPerTile) sh.far[local] = uint32_t(g);
      else atomicCAS(reinterpret_cast<int*>(err), 0, RW_ERR_CAPACITY);  // not reachable, see above
      continue;
    }
    put(g, e - 1, max(L, -1), min(R, n), d_at);
  }
  __syncthreads();

  // phase D: the tile's gaps whose nearest smaller gap lies beyond the
  // window, one warp per gap (the warp-cooperative search of the keys in
  // global memory); their latency overlaps the other resident blocks' work
  // (with DYN node 0 too: the other blocks wait for this one at a barrier)
  if (DYN && g0 == 0 && warp == uint32_t(NW - 1)) root_node();
  const uint32_t nf = min(sh.far_n, kTreeFarPerTile);
  auto d_glob = [&](int p) -> int { return delta(codes[p], codes[p + 1]); };
  for (uint32_t f = warp; f < nf; f += NW) {
    const int g = int(sh.far[f]);
    const int D = delta(codes[g], codes[g + 1]);
    int first_key, last_key;
    coop_node_keys<K>(codes, n, g, D, &first_key, &last_key);
    if (lane == 0) put(g, D, first_key - 1, last_key, d_glob);
  }
  if (EDGES) {
    sum0 = __reduce_add_sync(0xffffffffu, sum0);
    sum1 = __reduce_add_sync(0xffffffffu, sum1);
    if (lane == 0) {
      if (sum0) atomicAdd(&sh.sum[0], sum0);
      if (sum1) atomicAdd(&sh.sum[1], sum1);
    }
    __syncthreads();
    if (threadIdx.x < kTreeSums && sh.sum[threadIdx.x])
      atomicAdd(sums + t0 + threadIdx.x, uint32_t(sh.sum[threadIdx.x]));
  }
}

// ---------------------------------------------------------------------------
// stage 7: octree rows and links (func_octree.hpp:28-112)
// ---------------------------------------------------------------------------

struct OctOut {
  int32_t* children;
  float4* corner;
  float* cell_size;
  int32_t* node_mask;
  int32_t* leaf_mask;
  const uint32_t* oct_off;  // [segments + 1] row offsets; null with one segment
  uint32_t capacity;        // rows with one segment
};

struct OctSeg {
  uint32_t row0, cap, m;
  int n;        // radix-tree nodes
  bool counts;  // the counts are valid (the edge offsets can be made)
  bool ok;      // ... and the octree fits its rows
};

// The segment's octree rows and counts; reports a too small octree.
__device__ __forceinline__ OctSeg oct_segment(const SegTable& seg, const OctOut& o,
                                              const uint32_t* n_unique,
                                              const uint32_t* n_octree, int32_t* seg_err,
                                              uint32_t c, bool report) {
  OctSeg r{};
  // (both loads go out together)
  const uint32_t nu = *reinterpret_cast<const volatile uint32_t*>(n_unique + c);
  const uint32_t m = *reinterpret_cast<const volatile uint32_t*>(n_octree + c);
  r.ok = nu >= 3 && nu != RW_COUNT_UNSET && nu <= seg_size(seg, c);
  if (!r.ok) return r;
  r.n = int(nu - 1);
  r.m = m;
  r.row0 = o.oct_off ? o.oct_off[c] : 0u;
  r.cap = o.oct_off ? o.oct_off[c + 1] - o.oct_off[c] : o.capacity;
  r.counts = true;
  if (uint64_t(r.m) + 1 > r.cap) {
    if (report) seg_error(seg_err, c, RW_ERR_CAPACITY);
    r.ok = false;
  }
  return r;
}

// Nearest ancestor of node c that owns rows: parents are followed while the
// count is zero, at most 31 steps as in the reference (func_octree.hpp:80-92).
// Returns -1 when a parent index is outside [0, n).
__device__ __forceinline__ int link_parent(const int32_t* __restrict__ parents,
                                           const int32_t* __restrict__ ec, int c, int n) {
  int rp = parents[c];
  if (uint32_t(rp) >= uint32_t(n)) return -1;
  int counter = 0;
  while (ec[rp] == 0) {
    rp = parents[rp];
    if (uint32_t(rp) >= uint32_t(n)) return -1;
    if (++counter > 30) break;
  }
  return rp;
}

// The link of node c (count cnt > 0) into the global rows: child slot of the
// chain's top row (level prefix_n[c] / 3 - cnt + 1) in row offset[rp]
// (func_octree.hpp:94-102).  The reference overwrites in ascending node
// order; the value off[c] + cnt - 1 grows with c, so the maximum is the last
// write.
template <typename K>
__device__ __forceinline__ void link_global(const K* __restrict__ codes,
                                            const uint8_t* __restrict__ prefix_n,
                                            const int32_t* __restrict__ off, int c, int cnt,
                                            int rp, const OctSeg& os, const OctOut& o) {
  constexpr int B = KeyTraits<K>::kCodeBits;
  const int oct_parent = off[rp];
  const int top = prefix_n[c] / 3 - cnt + 1;
  const int slot = int((codes[c] >> (B - 3 * top)) & K(7));
  if (uint32_t(oct_parent) < os.cap) {
    const size_t r = size_t(os.row0) + uint32_t(oct_parent);
    atomicMax(o.children + 8 * r + slot, off[c] + cnt - 1);
    atomicOr(o.node_mask + r, 1 << slot);
  }
}

// A far link (16 bytes): segment, node, kind << 30 | counter << 3 | slot,
// link value.  kFarFromParent: the walk starts at parents[node] (node = the
// linking node); kFarFromStep: node is the last ancestor reached inside the
// tile, count 0, the walk continues at parents[node] with counter + 1;
// kFarFinal: node is the ancestor whose row takes the link.  kFarLocal is
// used inside k_octree only.
constexpr uint32_t kFarFromParent = 0, kFarFromStep = 1, kFarFinal = 2, kFarLocal = 3;

// Stage 7 in one pass over a tile of radix-tree nodes (func_octree.hpp:28-112).
//
// Rows [off[i], off[i] + cnt[i]) belong to node i (i >= 1); the offsets are
// an exclusive scan of non-negative counts, so a tile of nodes owns one
// contiguous run of rows, and the owner of row p is the last node whose
// first row is <= p.  Row off+k sits at level L - k (L = prefix_n[i] / 3);
// for k > 0 its one child is the chain row off+k-1 (func_octree.hpp:56-78).
// A row with k = 0 gets its children only from links: the chain's top row
// p = off[c] + cnt[c] - 1 of node c is named in row off[rp] of c's nearest
// ancestor rp that owns rows (func_octree.hpp:80-111).  When rp lies in the
// tile and owns rows, that row is a k = 0 row of the tile: the link is
// merged in shared memory and every row is written once, complete.  Other
// links go to the far list (node, segment), applied after this kernel with
// global atomics; a list that overflows makes the far kernel apply every
// link again (the atomics are idempotent).
//
// A thread loads four consecutive nodes as vectors and names itself the owner
// of their rows in shared memory; then threads take the tile's rows in turn
// (row r by thread r mod threads), so that every lane has a row.  The kernel is
// bound by its instructions: with four nodes 256 apart per thread, a scan per
// group of them and a binary search over the tile's first rows for each row's
// owner it executed 156M of them instead of 146M and took 183.9 instead of 170.0
// us at 16.8M uniform points (5,000,011 64-bit keys: 75.7, then 71.8).  Corners
// decoded by multiplications (decode) and one expansion of the child slots for
// first and later rows of a chain alike: 164.0 us (64-bit keys 69.7).
//
// Node 0 owns no row; tile 0 writes the root initialisation when there is
// no octree row at all (07_octree.cu:188-198) and clears the spare row m
// that a link may name.
//
// With OFFS the offsets are not read but made here (stage 6's write folded
// into stage 7): tile_prefix holds the exclusive scan of every tile's count
// sum (tree_tile, k_tile_scan), the block scans its tile's counts on top
// of it and writes them to off_all.
template <typename K>
struct OctTileShared {
  // k = 0 row of each node: child slot values relative to the tile's first
  // row, plus one (0: no child; the nonzero slots are the node mask)
  uint4 child[kOctTile];  // 8 x u16
  alignas(16) K code[kOctTile];
  // first row of each node relative to the tile's first row (a tile's rows
  // number at most kTile times the largest count, 21 levels; 0xffff past the
  // tile's nodes); [kOctTile]: end of the tile's rows
  alignas(8) uint16_t off[kOctTile + 4];
  // per node: (count class << 12) | tile-relative parent (0xfff: outside);
  // class 0: count 0, 1: count > 0, 2: count < 0
  alignas(8) uint16_t node[kOctTile];
  uint16_t owner[kOctTile];  // of the first rows
  alignas(4) uint8_t level[kOctTile];  // prefix_n / 3
  uint32_t wsum[kOctThreads / 32];
};

// The tile of nodes from tile0 on, of a segment os (number c) whose arrays are
// given, by kOctThreads threads (tid) that sync() synchronises.  first_row():
// the tile's first row, with OFFS.
template <typename K, bool OFFS, typename Sync, typename FirstRow>
__device__ __forceinline__ void octree_tile(
    OctTileShared<K>& sh, const Sync& sync, int tid, const K* __restrict__ codes,
    const uint8_t* __restrict__ prefix_n, const int32_t* __restrict__ parents,
    const int32_t* __restrict__ ec, int32_t* __restrict__ off, const OctSeg& os, uint32_t c,
    int tile0, const FirstRow& first_row, float min_coord, float range, const OctOut& o,
    uint32_t* __restrict__ far, uint32_t far_cap, uint32_t* __restrict__ far_n) {
  constexpr int B = KeyTraits<K>::kCodeBits;
  constexpr int kTile = int(kOctTile);
  constexpr int kRowCap = kTile;  // rows whose owner is kept
  static_assert(kTile < 0xfff && (kTile & (kTile - 1)) == 0, "12-bit parents, 2^k tile");
  static_assert(kTile == 4 * kOctThreads, "four nodes per thread");
  const int n = os.n;
  const uint32_t m = os.m;
  const int tile_end = min(tile0 + kTile, n);

  // thread tid: nodes tile0 + 4 tid + q, q < 4, as vectors; a tile that ends
  // early or starts off a 16-byte boundary (a cloud of a batch) goes through
  // shared memory, in the place of the child slots
  static_assert(kOctNpt == 4, "four nodes per thread");
  auto low = [](const void* p) { return uint32_t(reinterpret_cast<uintptr_t>(p)); };
  const bool vec = tile_end == tile0 + kTile && (low(prefix_n + tile0) & 3u) == 0 &&
                   ((low(ec + tile0) | low(parents + tile0) | low(off + tile0) |
                     low(codes + tile0)) & 15u) == 0;
  const uint32_t base = OFFS ? first_row() : 0u;
  const int root_level = prefix_n[0] / 3;
  const int n0 = 4 * tid;  // the thread's first node in the tile
  int* tmp = reinterpret_cast<int*>(sh.child);
  int4 e4, p4, o4 = make_int4(0, 0, 0, 0);
  if (vec) {
    e4 = reinterpret_cast<const int4*>(ec + tile0)[tid];
    p4 = reinterpret_cast<const int4*>(parents + tile0)[tid];
    if (!OFFS) o4 = reinterpret_cast<const int4*>(off + tile0)[tid];
    const uint32_t pre = reinterpret_cast<const uint32_t*>(prefix_n + tile0)[tid];
    constexpr int kCodeVecs = int(sizeof(K)) / 4;  // of 16 bytes
#pragma unroll
    for (int q = 0; q < kCodeVecs; ++q)
      reinterpret_cast<uint4*>(sh.code)[tid * kCodeVecs + q] =
          reinterpret_cast<const uint4*>(codes + tile0)[tid * kCodeVecs + q];
    *reinterpret_cast<uint32_t*>(sh.level + n0) =
        uint32_t(third(pre & 255u)) | uint32_t(third(pre >> 8 & 255u)) << 8 |
        uint32_t(third(pre >> 16 & 255u)) << 16 | uint32_t(third(pre >> 24)) << 24;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int t = tid + q * kOctThreads;
      const int i = tile0 + t;
      const bool valid = i < tile_end;
      tmp[t] = valid ? ec[i] : 0;
      tmp[kTile + t] = valid ? parents[i] : -1;
      if (!OFFS) tmp[2 * kTile + t] = valid ? off[i] : 0;
      sh.code[t] = valid ? codes[i] : K(0);
      sh.level[t] = valid ? uint8_t(third(prefix_n[i])) : uint8_t(0);
    }
    sync();
    e4 = reinterpret_cast<const int4*>(tmp)[tid];
    p4 = reinterpret_cast<const int4*>(tmp + kTile)[tid];
    if (!OFFS) o4 = reinterpret_cast<const int4*>(tmp + 2 * kTile)[tid];
    sync();
  }
  const int ev[4] = {e4.x, e4.y, e4.z, e4.w}, pa[4] = {p4.x, p4.y, p4.z, p4.w};
  int ov[4] = {o4.x, o4.y, o4.z, o4.w};
  uint32_t word[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t pr = uint32_t(pa[q] - tile0) < uint32_t(tile_end - tile0)
                            ? uint32_t(pa[q] - tile0) : 0xfffu;
    word[q] = (ev[q] == 0 ? 0u : ev[q] > 0 ? 1u : 2u) << 12 | pr;
  }
  *reinterpret_cast<uint2*>(sh.node + n0) =
      make_uint2(word[0] | word[1] << 16, word[2] | word[3] << 16);
  uint32_t rows_end = 0;
  int rbase = 0;  // the tile's first row
  if (OFFS) {
    // exclusive scan of the counts in node order, as stage 6 computes it
    const uint32_t lane = lane_id(), warp = uint32_t(tid) >> 5;
    const uint32_t sum = uint32_t(ev[0]) + uint32_t(ev[1]) + uint32_t(ev[2]) + uint32_t(ev[3]);
    const uint32_t inc = warp_inclusive_scan(sum);
    if (lane == 31) sh.wsum[warp] = inc;
    sync();
    uint32_t run = base + inc - sum;
    rows_end = base;
#pragma unroll
    for (int w = 0; w < kOctThreads / 32; ++w) {
      const uint32_t x = sh.wsum[w];
      run += uint32_t(w) < warp ? x : 0u;
      rows_end += x;
    }
    rbase = int(base);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      ov[q] = int32_t(run);
      run += uint32_t(ev[q]);
    }
    if (vec) {
      reinterpret_cast<int4*>(off + tile0)[tid] = make_int4(ov[0], ov[1], ov[2], ov[3]);
    } else {
      reinterpret_cast<int4*>(tmp)[tid] = make_int4(ov[0], ov[1], ov[2], ov[3]);
      sync();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = tid + q * kOctThreads;
        if (tile0 + t < tile_end) off[tile0 + t] = tmp[t];
      }
      sync();
    }
  } else {
    rbase = off[tile0];
    rows_end = uint32_t(tile_end < n ? off[tile_end] : int(m));
  }
  if (!os.ok) return;  // the whole block: no octree row is written
  // relative rows kept in [0, 0xfffe] (offsets made by stage 6 stay far inside);
  // the entry behind the tile's last node is the end of its rows, 0xffff follows
  auto rel16 = [&](int v) -> uint32_t { return uint32_t(min(max(v - rbase, 0), 0xfffe)); };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    sh.child[tid + q * kOctThreads] = make_uint4(0, 0, 0, 0);
    const int i = tile0 + n0 + q;
    word[q] = i < tile_end ? rel16(ov[q]) : i == tile_end ? rel16(int(rows_end)) : 0xffffu;
    // the rows' owner
    if (i < tile_end) {
      const int r = int(word[q]);
      for (int k = 0; k < min(ev[q], 32) && r + k < kRowCap; ++k) sh.owner[r + k] = uint16_t(n0 + q);
    }
  }
  *reinterpret_cast<uint2*>(sh.off + n0) =
      make_uint2(word[0] | word[1] << 16, word[2] | word[3] << 16);
  if (tid == 0) {
    sh.off[kTile] = uint16_t(rel16(int(rows_end)));
    if (tile0 == 0) {
      const size_t rm = size_t(os.row0) + m;
      int4* row = reinterpret_cast<int4*>(o.children + 8 * rm);
      row[0] = make_int4(0, 0, 0, 0);
      row[1] = make_int4(0, 0, 0, 0);
      o.node_mask[rm] = 0;
      o.leaf_mask[rm] = 0;
      if (m == 0) {
        const K pre = codes[0] >> (B - 3 * root_level);
        o.corner[os.row0] = decode<K>(K(pre << (B - 3 * root_level)), min_coord, range);
        o.cell_size[os.row0] = range;
      }
    }
  }
  sync();

  const int rend = min(rbase + int(sh.off[kTile]), int(m));  // rows [rbase, rend)
  auto owner_of = [&](int r) -> int {  // last node whose first row is <= rbase + r
    if (r < kRowCap) return int(sh.owner[r] & (kTile - 1));
    int t = 0;
#pragma unroll
    for (int step = kTile / 2; step >= 1; step >>= 1)
      if (int(sh.off[t + step]) <= r) t += step;
    return t;
  };

  // links, from the chain top rows; the walk of link_parent over the tile's
  // counts and parents.  A walk that leaves the tile, ends on a node without
  // rows or gives up, and a value that does not fit 16 bits, go to the far
  // list with the walk's state (FarLink), where k_octree_far_links finishes
  // the walk in global memory and merges with atomics.  Several links may
  // name one slot (the reference keeps the last, the largest value): the
  // 16-bit maximum is taken with compare-and-swap on the slot's word.
  for (int r = tid; rbase + r < rend; r += kOctThreads) {
    const int p = rbase + r;
    const int t = owner_of(r);
    if (r != int(sh.off[t + 1]) - 1) continue;  // not the top row of its chain
    const int level = int(sh.level[t]) - (r - int(sh.off[t]));  // the top row's level
    const int slot = int((sh.code[t] >> (B - 3 * level)) & K(7));
    int rp = int(sh.node[t] & 0xfffu), counter = 0, x = t;
    uint32_t kind = kFarFromParent;
    if (rp != 0xfff) {
      for (;;) {
        const uint32_t w = sh.node[rp];
        if (w >> 12) {
          kind = (w >> 12) == 1 ? kFarLocal : kFarFinal;
          break;
        }
        const int nx = int(w & 0xfffu);
        if (nx == 0xfff) {  // the parent lies outside the tile
          kind = kFarFromStep;
          x = rp;
          break;
        }
        rp = nx;
        if (++counter > 30) {
          kind = kFarFinal;
          break;
        }
      }
    }
    if (kind == kFarLocal) {
      bool done = false;
      if (r < 0xffff) {
        uint32_t* wp = reinterpret_cast<uint32_t*>(&sh.child[rp]) + (slot >> 1);
        const int sh = 16 * (slot & 1);
        const uint32_t rel = uint32_t(r) + 1u;  // the link value is p itself
        uint32_t cur = *reinterpret_cast<volatile uint32_t*>(wp);
        for (int tries = 0; tries < 64 && !done; ++tries) {  // each failure is another's success
          if (((cur >> sh) & 0xffffu) >= rel) {
            done = true;
          } else {
            const uint32_t nv = (cur & ~(0xffffu << sh)) | (rel << sh);
            const uint32_t prev = atomicCAS(wp, cur, nv);
            done = prev == cur;
            cur = prev;
          }
        }
      }
      if (done) continue;
      kind = kFarFinal;
    }
    const uint32_t at = atomicAdd(far_n, 1u);
    if (at < far_cap) {
      const int node = kind == kFarFinal ? tile0 + rp : tile0 + x;
      reinterpret_cast<uint4*>(far)[at] =
          make_uint4(c, uint32_t(node), kind << 30 | uint32_t(counter) << 3 | uint32_t(slot),
                     uint32_t(p));
    }
  }
  sync();

  // rows
  for (int r = tid; rbase + r < rend; r += kOctThreads) {
    const int p = rbase + r;
    const int t = owner_of(r);
    const size_t rp = size_t(os.row0) + uint32_t(p);
    const int k = r - int(sh.off[t]);
    const int level = int(sh.level[t]) - k;
    const K code = sh.code[t];
    const K pre = code >> (B - 3 * level);
    o.corner[rp] = decode<K>(K(pre << (B - 3 * level)), min_coord, range);
    // range / 2^s, s = level - root_level in [0, 21]: the product with the
    // exact reciprocal 2^-s is the same correctly rounded value
    o.cell_size[rp] =
        __fmul_rn(range, __uint_as_float(uint32_t(127 - (level - root_level)) << 23));
    int4* row = reinterpret_cast<int4*>(o.children + 8 * rp);
    // the children as slots of 16 bits, relative to the tile's first row, plus one
    uint4 a;
    if (k == 0) {
      a = sh.child[t];
    } else {  // the chain's row before this one
      const uint32_t slot = uint32_t(code >> (B - 3 * (level + 1))) & 7u;
      const uint32_t w = uint32_t(r) << (16 * (slot & 1u));
      a = make_uint4(slot >> 1 == 0 ? w : 0u, slot >> 1 == 1 ? w : 0u, slot >> 1 == 2 ? w : 0u,
                     slot >> 1 == 3 ? w : 0u);
    }
    const uint32_t wv[4] = {a.x, a.y, a.z, a.w};
    int32_t child[8];
    uint32_t mask = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t v = (wv[q >> 1] >> (16 * (q & 1))) & 0xffffu;
      child[q] = v ? int32_t(v) - 1 + rbase : 0;
      mask |= uint32_t(v != 0) << q;
    }
    row[0] = make_int4(child[0], child[1], child[2], child[3]);
    row[1] = make_int4(child[4], child[5], child[6], child[7]);
    o.node_mask[rp] = int32_t(mask);
    o.leaf_mask[rp] = 0;
  }
}

// Links that k_octree left to the far list, with global atomics; when the
// list overflowed, every node's link again (blocks stride over all tiles).
template <typename K>
__device__ __forceinline__ void octree_far_links(
    const K* __restrict__ codes_all, const uint8_t* __restrict__ prefix_all,
    const int32_t* __restrict__ parents_all, const int32_t* __restrict__ ec_all,
    const int32_t* __restrict__ off_all, const SegTable& seg, const TileMap& map,
    const uint32_t* __restrict__ n_unique, const uint32_t* __restrict__ n_octree,
    int32_t* __restrict__ seg_err, const OctOut& o, const uint32_t* __restrict__ far,
    uint32_t far_cap, const uint32_t* __restrict__ far_n) {
  const uint32_t count = *far_n;
  if (count <= far_cap) {
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < count;
         w += gridDim.x * blockDim.x) {
      // the walk is a chain of dependent loads: every step loads the count,
      // the parent and the offset of its node together, and the first step
      // goes out with the segment's counts (k_octree wrote only nodes of the
      // segment, in [0, n), into the list)
      const uint4 f = reinterpret_cast<const uint4*>(far)[w];
      const uint32_t c = f.x, kind = f.z >> 30, slot = f.z & 7u;
      const uint32_t sb = seg_begin(seg, c);
      const int32_t* parents = parents_all + sb;
      const int32_t* ec = ec_all + sb;
      const int32_t* off = off_all + sb;
      int rp = int(f.y);
      const int first = kind != kFarFinal ? parents[rp] : rp;
      const OctSeg os = oct_segment(seg, o, n_unique, n_octree, seg_err, c, false);
      if (!os.ok) continue;
      const int n = os.n;
      int oct_parent;
      if (kind != kFarFinal) {  // the rest of link_parent's walk
        int counter = int((f.z >> 3) & 31u);
        rp = first;
        if (uint32_t(rp) >= uint32_t(n)) continue;
        bool stop = kind == kFarFromStep && ++counter > 30;
        int cnt = ec[rp], par = parents[rp];
        oct_parent = off[rp];
        while (!stop && cnt == 0) {
          rp = par;
          if (uint32_t(rp) >= uint32_t(n)) break;
          stop = ++counter > 30;
          cnt = ec[rp];
          par = parents[rp];
          oct_parent = off[rp];
        }
        if (uint32_t(rp) >= uint32_t(n)) continue;
      } else {
        oct_parent = off[rp];
      }
      if (uint32_t(oct_parent) < os.cap) {
        const size_t r = size_t(os.row0) + uint32_t(oct_parent);
        atomicMax(o.children + 8 * r + slot, int32_t(f.w));
        atomicOr(o.node_mask + r, 1 << slot);
      }
    }
    return;
  }
  for (uint32_t tile = blockIdx.x; tile < map.n_tiles; tile += gridDim.x) {
    uint32_t first;
    const uint32_t c = tile_segment(seg, map, tile, &first);
    const OctSeg os = oct_segment(seg, o, n_unique, n_octree, seg_err, c, false);
    if (!os.ok) continue;
    const uint32_t sb = seg_begin(seg, c);
    const int32_t* ec = ec_all + sb;
    const int base = int(tile - first) * int(kOctTile);
    for (int q = int(threadIdx.x); q < int(kOctTile); q += int(blockDim.x)) {
      const int i = base + q;
      if (i >= os.n) break;
      if (i == 0) continue;
      const int cnt = ec[i];
      if (cnt <= 0) continue;
      const int rp = link_parent(parents_all + sb, ec, i, os.n);
      if (rp < 0) continue;
      link_global<K>(codes_all + sb, prefix_all + sb, off_all + sb, i, cnt, rp, os, o);
    }
  }
}

// ---------------------------------------------------------------------------
// leaf links (rw_tree_im_storage_set_options)
// ---------------------------------------------------------------------------

// RW_TREE_OPT_LINK_LEAVES: process_link_leaf (func_octree.hpp:114-163) for
// every radix-tree node, as if run in ascending order after stage 7.  Leaf
// `side` of node i goes to slot (leaf code at level prefix_n[i]/3 + 1) & 7 of
// the bottom octree row of the nearest ancestor-or-self with octree rows.
// The walk stops after 31 steps (the reference CPU walk has no bound and
// never ends at a root without rows; its CUDA left-leaf walk stops there),
// and a negative level shift (32-bit keys, prefix_n = 30) is taken modulo
// the word width, as an x86 build of the reference does.
//
// Pass 1: every writer claims its slot with atomicMin of -(2 i + side) - 2,
// so the slot ends holding the claim of the last writer in sequential order
// (claims are negative, the rows' node links are not).  set_leaf also clears
// the slot's bit of the leaf mask, which stage 7 has left at zero.
//
// What a node and a step of its walk need is loaded together, and one walk
// serves both of its leaves; pass 2 goes over the slots, not over the nodes and
// their walks once more (1,000,003 points, both options, in one launch: 159.6 ->
// 144.7 us).
template <typename K>
__device__ __forceinline__ void leaf_claim(const K* __restrict__ codes, const uint8_t* __restrict__ pn,
                 const uint8_t* __restrict__ hl, const uint8_t* __restrict__ hr,
                 const int32_t* __restrict__ lc, const int32_t* __restrict__ par,
                 const int32_t* __restrict__ ec, const int32_t* __restrict__ off,
                 int32_t* __restrict__ children, const uint32_t* __restrict__ n_unique,
                 uint32_t rows) {
  constexpr int B = KeyTraits<K>::kCodeBits, W = KeyTraits<K>::kWordBits;
  const uint32_t nu = *n_unique;
  if (nu < 3 || nu == RW_COUNT_UNSET) return;
  const int n = int(nu - 1);
  for (int i = int(blockIdx.x * blockDim.x + threadIdx.x); i < n; i += int(gridDim.x * blockDim.x)) {
    const uint32_t sides = uint32_t(hl[i] != 0) | uint32_t(hr[i] != 0) << 1;
    const int gap = lc[i], level = third(pn[i]) + 1;
    int count = ec[i], up = par[i], bottom = off[i];
    if (!sides) continue;
    for (int step = 0; step < 31 && count == 0; ++step) {
      const int rt = uint32_t(up) < uint32_t(n) ? up : 0;
      count = ec[rt];
      up = par[rt];
      bottom = off[rt];
    }
    if (uint32_t(bottom) >= rows) continue;
#pragma unroll
    for (int side = 0; side < 2; ++side)
      if ((sides >> side) & 1u) {
        const int leaf = min(max(gap + side, 0), n);  // keys are [0, n]
        const uint32_t which = uint32_t(codes[leaf] >> ((B - 3 * level) & (W - 1))) & 7u;
        atomicMin(children + size_t(bottom) * 8 + which, int(-(int64_t(2 * i + side) + 2)));
      }
  }
}

// Pass 2: every claim that survived becomes its node's leaf index.  Rows up to
// the spare one behind the last can hold claims.
__device__ __forceinline__ void leaf_write(const int32_t* __restrict__ lc,
                                           int32_t* __restrict__ children,
                                           const uint32_t* __restrict__ n_unique,
                                           const uint32_t* __restrict__ n_octree, uint32_t rows) {
  const uint32_t nu = *n_unique, m = *n_octree;
  if (nu < 3 || nu == RW_COUNT_UNSET) return;
  const int n = int(nu - 1);
  const uint64_t vecs = 2 * min(uint64_t(m) + 1, uint64_t(rows));
  for (uint64_t j = blockIdx.x * blockDim.x + threadIdx.x; j < vecs; j += gridDim.x * blockDim.x) {
    const int4 v = reinterpret_cast<const int4*>(children)[j];
    if ((v.x | v.y | v.z | v.w) >= 0) continue;
    const int c[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c[q] < 0) {
        const int claim = -(c[q] + 2), i = claim >> 1;  // 2 i + side
        if (uint32_t(i) < uint32_t(n)) children[4 * j + q] = min(max(lc[i] + (claim & 1), 0), n);
      }
  }
}

}  // namespace rwt
