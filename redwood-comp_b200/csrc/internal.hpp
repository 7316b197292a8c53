// Host-side internals shared by the kernel translation units and the C ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "common.cuh"
#include "rw_tree.h"

// Scratch for one pipeline instance (the reference's cuda::ImStorage,
// apps/tree/cuda/im_storage.cuh:10-42, with the look-back state this design
// needs).  The "zero region" is the part of it that is cleared before every run of the
// general chain of kernels.
struct rw_tree_im_storage {
  uint32_t n_cap = 0;   // largest n_input this scratch serves
  int32_t key_bits = 32;
  int device = 0;
  int num_sms = 148;

  // sort configuration (radix bits, passes, tile) fixed at creation
  int radix_bits = 8;
  int passes = 4;
  int low_bits = 0;          // bits that the passes leave out (sort_low_bits)
  int sort_variant = 0;      // index into the onesweep variant menu (k_keys.cu)
  uint32_t sort_tile = 0;
  uint32_t sort_tiles = 0;  // tiles per pass at n_cap

  void* d_tmp_keys = nullptr;  // [n_cap] ping-pong buffer of the sort
  uint32_t* d_rest_ctr = nullptr;   // [kRestWords] (64-bit keys)
  uint32_t* d_rest = nullptr;       // [rest_words], not zeroed (64-bit keys)
  uint32_t* d_tree_far = nullptr;  // far links of the octree
  uint32_t tree_far_cap = 0;       // entries (16 bytes each)

  // zero region
  void* d_zero = nullptr;
  size_t zero_bytes = 0;
  uint32_t* d_ghist = nullptr;      // [passes][radix]
  uint32_t* d_skew = nullptr;       // [1]: the top sort pass's digits are skewed
  uint32_t* d_dense = nullptr;      // [2]: Scratch::dense
  uint32_t* d_sort_desc = nullptr;  // [passes][sort_tiles + 1][radix]
  uint32_t* d_unique_desc = nullptr;
  uint32_t* d_scan_desc = nullptr;
  uint32_t* d_tile_ctr = nullptr;   // [kCounters]
  rwt::DevStatus* d_status = nullptr;
  size_t sort_zero_off = 0, sort_zero_bytes = 0;  // ghist + sort_desc

  rwt::DevStatus* h_status = nullptr;  // pinned mirror

  // scratch of the one-launch pipeline of small clouds (inside d_tmp_keys, which
  // no cloud of that size fills); null when the device cannot hold its blocks
  char* d_small = nullptr;

  // optional learned-CDF sort for stage 2 (32-bit keys); not owned
  rw_tree_learned* learned = nullptr;
  int32_t learned_mode = 0;
  rw_tree_learned_stats learned_stats{};

  // RW_TREE_OPT_* bits (0: the reference's own behaviour)
  int32_t options = 0;
};

namespace rwt {

enum : int { kCtrUnique = 0, kCtrScan = 1, kCtrTree = 2, kCtrLinks = 3, kCtrSortBase = 4,
             kMaxPasses = 8, kCtrSortClassStride = kMaxPasses, kMaxSortClasses = 4, kCtrSmall = 48, kCounters = 64 };

// Tile sizes of the kernels (points or nodes per tile).
constexpr uint32_t kPointTile = 4096;  // Morton / histogram
constexpr uint32_t kUniqueThreads = 256, kUniqueKpt = 16;
constexpr uint32_t kUniqueTile = kUniqueThreads * kUniqueKpt;
constexpr uint32_t kScanThreads = 256, kScanKpt = 16;
constexpr uint32_t kScanTile = kScanThreads * kScanKpt;
constexpr int kTreeThreads = 256;
constexpr uint32_t kTreeTile = 2048;  // radix-tree nodes (key gaps) per tile
constexpr int kOctThreads = 256, kOctNpt = 4;
constexpr uint32_t kOctTile = kOctThreads * kOctNpt;

// 64-bit keys with 8-bit digits: the passes leave out the low bits, which
// k_sort_fix puts in order (k_sortfix.cu).  Four passes over the top 32 bits of
// the 63, five over the top 40 for scratch of more points, where runs of equal
// top bits get long.  A caller's keys may have the top bit of the word set as
// well: one bit more is then left out (sorted_low_bits).
constexpr int kSplitLow32 = 31, kSplitLow40 = 23;
constexpr uint32_t kSplitPoints = 1u << 21;
inline int sort_low_bits(int key_bits, int radix_bits, uint32_t largest) {
  if (key_bits != 64 || radix_bits != 8) return 0;
  return largest <= kSplitPoints ? kSplitLow32 : kSplitLow40;
}
// k_sort_rest's counters: dense segments, listed runs, passes over dense segments,
// then tickets and jobs done of each of its phases; a listed run has more than 256 keys.
enum : int { kRestDense = 0, kRestRuns = 1, kRestPasses = 2, kRestTickets = 3, kRestWords = 32 };
inline uint32_t rest_runs(uint32_t n) { return n / 257u + 1u; }
size_t rest_words(uint32_t segments, uint32_t n);
inline int sort_pass_count(int key_bits, int radix_bits, uint32_t largest) {
  const int bits = (key_bits == 32 ? 30 : 63) - sort_low_bits(key_bits, radix_bits, largest);
  return (bits + radix_bits - 1) / radix_bits;
}

// Boundary MLP of the learned sort: kMlpIn -> kMlpHidden -> kMlpHidden -> 1.
constexpr int kMlpIn = 16, kMlpHidden = 64;
constexpr int kMlpParams = kMlpHidden * kMlpIn + kMlpHidden + kMlpHidden * kMlpHidden +
                           kMlpHidden + kMlpHidden + 1;

inline uint32_t div_up(uint64_t a, uint64_t b) { return uint32_t((a + b - 1) / b); }

// A count either known on the host (value) or produced on the device (ptr).
struct Count {
  const uint32_t* ptr;
  uint32_t value;
};

// Device buffers of one pipeline run: one AppData, or a batch of clouds
// stored back to back (octree rows at per-cloud row offsets).
struct Bufs {
  int key_bits = 32;
  float min_coord = 0.0f, range = 1024.0f;
  const float4* points = nullptr;
  void* keys = nullptr;
  void* alt = nullptr;
  void* tmp = nullptr;  // ping-pong buffer of the sort
  uint8_t* prefix_n = nullptr;
  uint8_t* hl = nullptr;
  uint8_t* hr = nullptr;
  int32_t* lc = nullptr;
  int32_t* parents = nullptr;
  int32_t* edge_count = nullptr;
  int32_t* edge_offset = nullptr;
  int32_t* children = nullptr;
  float4* corner = nullptr;
  float* cell_size = nullptr;
  int32_t* node_mask = nullptr;
  int32_t* leaf_mask = nullptr;
};

// Scratch: histograms, descriptors, tickets, status.
struct Scratch {
  int num_sms = 148;
  int radix_bits = 8;
  int passes = 4;
  int sort_variant = 0;
  uint32_t* ghist = nullptr;      // [segments][passes][radix]
  // [segments]: 1 when the segment's top-pass digits are skewed enough that
  // ballots rank them faster than shared-memory atomics (k_sort_init sets it,
  // the kRankMixed variants read it)
  uint32_t* skew = nullptr;
  // low bits that the passes leave to launch_sort_finish (0: none), and
  // [segments]: 1 when the segment is dense and the passes leave it alone, then
  // [segments]: pairs of its samples with equal top bits (k_keys.cu)
  int low_bits = 0;
  uint32_t* dense = nullptr;
  uint32_t* rest_ctr = nullptr;  // [kRestWords], zeroed
  uint32_t* rest = nullptr;      // [rest_words]
  // the keys are codes that stage 1 makes in the same chain, whose top bits are
  // clear; else a caller's, which are sorted by the whole word
  bool codes = false;
  uint32_t* sort_desc = nullptr;  // [passes][sort_rows][radix]
  uint32_t sort_rows = 0;         // rows per pass: sort tiles + segments
  uint32_t* unique_desc = nullptr;
  uint32_t* scan_desc = nullptr;
  uint32_t* tile_ctr = nullptr;
  DevStatus* status = nullptr;
  // polls of a look-back wait before it gives up with RW_ERR_TIMEOUT
  uint32_t spin_limit = kSpinLimit;
  // arrivals or jobs that the bounded waits of k_small and k_sort_rest wait for in
  // vain (rw_tree_wait_probe)
  uint32_t missing = 0;
  // when set, the sort's kernels (digit histograms, set-up, passes) do their
  // work only if *gate != 0, read on the device: a fallback sort enqueued
  // ahead of the decision that needs it
  const uint32_t* gate = nullptr;
  // tree_far_cap entries of 16 bytes: the octree's far links
  uint32_t* tree_far = nullptr;
  uint32_t tree_far_cap = 0;
};

inline int sorted_low_bits(const Scratch& sc) {
  return sc.low_bits && !sc.codes ? sc.low_bits + 1 : sc.low_bits;
}

// Entries of the radix tree's far-search list per tile: the gaps of a tile
// with no smaller gap inside its window have strictly decreasing (left side)
// or increasing (right side) prefix lengths, so there are at most 64 per side.
constexpr uint32_t kTreeFarPerTile = 128;

// Segments and the tile map of every kernel, plus per-segment results.
struct Plan {
  SegTable seg{};
  TileMap point_map{}, sort_map{}, unique_map{}, tree_map{}, scan_map{}, node_map{};
  uint32_t* n_unique = nullptr;  // [segments]
  uint32_t* n_octree = nullptr;  // [segments]
  int32_t* seg_err = nullptr;    // [segments] first error of each segment
  const uint32_t* oct_off = nullptr;  // [segments + 1] octree row offsets
  uint32_t oct_capacity = 0;          // rows when there is one segment
};

// ---- onesweep variant menu (k_keys.cu) --------------------------------------
uint32_t sort_tile_for(int key_bits, int radix_bits);
uint32_t sort_variant_tile(int idx);
int sort_variant_count();
int sort_variant_info(int idx, int* key_bits, int* radix_bits, int* threads, int* kpt,
                      int* rank);
int default_sort_variant(int key_bits, int radix_bits);

// ---- launchers (each returns the launch's cudaError_t) --------------------
// Stage 1 (encode) and/or the sort's digit histograms (hist).
cudaError_t launch_keys(const Bufs& b, const Scratch& sc, const Plan& pl, bool encode,
                        bool hist, cudaStream_t s);
// Init rows + every pass; `marks`, when given, gets one event after the init
// kernel and one after each pass (profiling only).
cudaError_t launch_sort_passes(const Bufs& b, const Scratch& sc, const Plan& pl,
                               cudaStream_t s, cudaEvent_t* marks = nullptr);
// After the passes of every segment, when they leave bits out (low_bits): the
// order within runs of equal top bits, the dense segments, and stage 3's counts
// per tile (launch_unique's `counted`).
cudaError_t launch_sort_finish(const Bufs& b, const Scratch& sc, const Plan& pl,
                               cudaStream_t s);
// The onesweep sort of keys[0, n) into out on `im`'s scratch, with every
// kernel gated on *gate (see Scratch::gate); `clear` zeroes the scratch's
// zero region first (not needed when a pipeline cleared it and has not used
// it since).  For the learned sort's device-decided fallback.
int sort_enqueue_gated(rw_tree_im_storage* im, const void* keys, void* out, uint32_t n,
                       const uint32_t* gate, bool clear, cudaStream_t s);

// The learned-CDF sort of keys[0, n) into sorted, enqueued without any host
// wait: the bucket sort and a gated onesweep fallback on fallback_im (needed)
// are both enqueued and the plan's overflow word picks one on the device.
// The plan is copied to pinned host memory; learned_last_stats reads it once
// the stream has passed this sort.
int learned_sort_enqueue(rw_tree_learned* L, const uint32_t* keys, uint32_t* sorted, uint32_t n,
                         int32_t mode, rw_tree_im_storage* fallback_im, bool clear_fallback,
                         cudaStream_t s);
void learned_last_stats(const rw_tree_learned* L, rw_tree_learned_stats* out);
uint32_t learned_capacity(const rw_tree_learned* L);  // n_max it was created for

// Test hook of the bounded look-back wait: the digit histograms of b.keys,
// then pass 0 of the sort into b.alt with tile 0 left out, so that every
// other tile's look-back waits on a row nothing publishes and gives up after
// spin_limit polls (RW_ERR_TIMEOUT in the status word).  Needs >= 2 tiles.
cudaError_t launch_sort_lookback_probe(const Bufs& b, const Scratch& sc, const Plan& pl,
                                       uint32_t spin_limit, cudaStream_t s);
// counted: the tiles' head counts are in sc.unique_desc already.
cudaError_t launch_unique(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s,
                          bool counted = false);
// The unique kernels on caller-given scratch: `counts` holds one word per
// kUniqueTile keys plus one and, like *status, must be zero.
cudaError_t launch_unique_raw(const void* sorted, void* out, uint32_t n, int key_bits,
                              uint32_t* counts, DevStatus* status, int num_sms,
                              cudaStream_t s);
// Stage 4 alone (edges = false) or stages 4 and 5 in one pass (edges = true);
// geometric: every prefix length lowered by one (RW_TREE_OPT_GEOMETRIC_DELTA,
// 32-bit keys).
cudaError_t launch_radix_tree(const Bufs& b, const Scratch& sc, const Plan& pl, bool edges,
                              bool geometric, cudaStream_t s);
cudaError_t launch_edge_count(const Bufs& b, const Scratch& sc, const Plan& pl,
                              cudaStream_t s);
cudaError_t launch_edge_scan(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s);
// The scan of the octree tiles' count sums that stages 4 and 5 in one pass left
// in sc.scan_desc (zero before them), and the octree row counts.  launch_octree
// with fused_offsets then makes and writes the offsets itself.
cudaError_t launch_edge_sums(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s);
cudaError_t launch_octree(const Bufs& b, const Scratch& sc, const Plan& pl, cudaStream_t s,
                          cudaEvent_t* marks = nullptr, bool fused_offsets = false);

// Device status := the given counts, no error, no far links (before a stage that
// runs alone); device status -> pinned host memory; a batch's counts, errors and
// status -> pinned host memory (3 x segments words, then the status).
cudaError_t launch_status_in(const Scratch& sc, uint32_t n_unique, uint32_t n_octree,
                             cudaStream_t s);
cudaError_t launch_status_out(const DevStatus* status, DevStatus* host, cudaStream_t s);
cudaError_t launch_results_out(const Plan& pl, const DevStatus* status, uint32_t* host,
                               cudaStream_t s);

// The leaf links after stage 7 (RW_TREE_OPT_LINK_LEAVES), single cloud only.
cudaError_t launch_leaf_links(const Bufs& b, const Scratch& sc, const Plan& pl,
                              cudaStream_t s);

// ---- a small cloud's whole pipeline in one launch (k_small.cu) ----------------
// It takes clouds up to these sizes, where a bucket still has room for 1.9
// shares of 148 blocks; it is faster than the general chain of kernels up to
// there (a call with 1,000,003 points 123 against 138 us, 32-bit keys; 549,000
// points 100 against 129 us, 64-bit keys).
constexpr uint32_t kSmallLimit32 = 1100000, kSmallLimit64 = 550000;
// Sets the kernels up on the current device; *usable: a block of them fits an SM.
cudaError_t small_prepare(int key_bits, bool* usable);
uint32_t small_limit(int key_bits);
uint32_t small_alone();  // points of the largest cloud that one block takes
bool small_takes(uint32_t n, int key_bits, int sms);
size_t small_scratch_bytes(uint32_t n_cap, int key_bits, int sms);
// All seven stages for n points: `scratch` of small_scratch_bytes(n_cap),
// `sync` four zeroed words that only these launches and a clear change.  The
// counts and the first error go to sc.status and, at the end, to host_status
// (pinned).
cudaError_t launch_small(const Bufs& b, const Scratch& sc, uint32_t n, uint32_t n_cap,
                         uint32_t oct_capacity, bool geometric, bool leaves, char* scratch,
                         uint32_t* sync, DevStatus* host_status, cudaStream_t s);

// Text returned by rw_tree_last_error (this thread).
void set_last_error(const std::string& msg);

// One-segment plan for n points (tile maps computed arithmetically); counts
// and errors go to `status`.
Plan single_plan(uint32_t n, uint32_t oct_capacity, DevStatus* status, uint32_t sort_tile);

}  // namespace rwt
