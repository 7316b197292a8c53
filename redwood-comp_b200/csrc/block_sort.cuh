// Building blocks of kernels that sort in a block's shared memory and whose
// blocks wait for one another (cooperative launches only).
#pragma once

#include "internal.hpp"
#include "rank.cuh"

namespace rwt {

// Barrier over the grid's blocks, which all run (cooperative launch): arrivals
// only ever grow, the host never resets them between launches.  Bounded: a
// block whose wait runs out takes kGaveUp off the arrivals, unless the last one
// has come by then, reports RW_ERR_TIMEOUT, marks the scratch (until it is cleared)
// and leaves.  Either every block passes a barrier or, from that moment, none
// does: no block can go on and report success for work that another has left.
struct GridBarrier {
  static constexpr uint32_t kGaveUp = 0x40000000u;  // far more than arrivals
  uint32_t* word;
  uint32_t blocks, target, limit;
  uint32_t* s_ok;       // shared: whether the last wait ended in time
  uint32_t* gave_up;    // set when one did not
  DevStatus* status;    // gets the error
  DevStatus* host_status;  // and the host's copy of it (may be null)
  __device__ __forceinline__ bool sync() {
    __syncthreads();
    if (blocks == 1) return true;
    target += blocks;
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(word) : "memory");
      bool ok = false;
      for (uint32_t spin = 0;;) {
        const uint32_t v = ld_acquire(word);
        const int32_t past = int32_t(v - target);
        ok = past >= 0;
        if (ok || past < -int32_t(kGaveUp / 2)) break;
        if (++spin < limit) backoff(spin);
        else if (atomicCAS(word, v, v - kGaveUp) == v) break;  // else look again
      }
      *s_ok = ok;
      if (!ok) {
        st_relaxed(gave_up, 1u);
        report_error(status, RW_ERR_TIMEOUT, kSiteGrid);
        if (host_status) *reinterpret_cast<volatile int32_t*>(&host_status->err) = RW_ERR_TIMEOUT;
      }
    }
    __syncthreads();
    return *s_ok != 0;
  }
};

// The local sort runs on half of the block's warps: below a few thousand keys
// its time is instructions per thread (ranking 32 keys, scanning the 512
// half-warp counters of every warp), so fewer warps with more keys each are
// faster (32 warps with 3 steps of 32 keys took 2.3 us a pass at 3,001 keys).
constexpr int kSortWarps = 16, kSortThreads = kSortWarps * 32;
constexpr int kSortHist = kSortWarps * 512;  // words: two per digit and warp
constexpr int kSortBarrier = 5;              // the named barrier of these warps

__device__ __forceinline__ void sort_sync() {
  asm volatile("bar.sync %0, %1;" ::"n"(kSortBarrier), "n"(kSortThreads) : "memory");
}

struct DigitShared {
  uint32_t start[256];  // first place of each digit after a pass
  uint32_t warp[kSortWarps];
};

// Stable pass over one 8-bit digit of `steps` x 512 keys, from `a` to `b`, by
// kSortThreads threads; leaves the digits' first places in sh.start.  A
// half-warp owns 16 * steps consecutive keys and ranks 16 a step in one word
// per digit (half_rank, rank.cuh: count << 16 | peer mask).  hist is zero on
// entry, `next` is left zero for the next pass.  At most KPT steps.
template <typename K, int KPT>
__device__ __forceinline__ void block_digit_pass(const K* a, K* b, int steps, int shift,
                                                 uint32_t* hist, uint32_t* next,
                                                 DigitShared& sh) {
  const int tid = int(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const uint32_t l16 = uint32_t(lane) & 15u, lt16 = (1u << l16) - 1u;
  uint32_t* wp = hist + warp * 512 + (lane >> 4);
  const int first = (2 * warp + (lane >> 4)) * 16 * steps + int(l16);
  uint32_t rank2[RankPack<KPT>::kRegs];
#pragma unroll
  for (int i = 0; i < KPT; ++i) {
    if (i >= steps) break;
    uint32_t* w = wp + 2 * (uint32_t(a[first + 16 * i] >> shift) & 255u);
    atomicOr(w, 1u << l16);
    __syncwarp();
    const uint32_t word = *w, peers = word & 0xffffu, cnt = word >> 16;
    const uint32_t below = uint32_t(__popc(peers & lt16));
    __syncwarp();
    if ((peers >> l16) == 1u) *w = (cnt + below + 1u) << 16;  // the highest peer
    RankPack<KPT>::set(rank2, i, cnt + below);
    __syncwarp();
  }
  sort_sync();
  // the counts in the order (digit, warp, half): thread (digit tid / 2, half
  // tid % 2 of the warps), so one scan over the threads gives every place
  constexpr int Q = kSortWarps / 2;
  const int d = tid >> 1, w0 = (tid & 1) * Q;
  uint2 v[Q];
  uint32_t sum = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    v[q] = *reinterpret_cast<const uint2*>(hist + (w0 + q) * 512 + 2 * d);
    v[q].x >>= 16;
    v[q].y >>= 16;
    sum += v[q].x + v[q].y;
  }
#pragma unroll
  for (int q = 0; q < kSortHist / 4 / kSortThreads; ++q)
    reinterpret_cast<uint4*>(next)[q * kSortThreads + tid] = make_uint4(0, 0, 0, 0);
  const uint32_t inc = warp_inclusive_scan(sum);
  if (lane == 31) sh.warp[warp] = inc;
  sort_sync();
  uint32_t run = inc - sum;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) run += w < warp ? sh.warp[w] : 0u;
  if ((tid & 1) == 0) sh.start[d] = run;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint2 o = make_uint2(run, run + v[q].x);
    *reinterpret_cast<uint2*>(hist + (w0 + q) * 512 + 2 * d) = o;
    run = o.y + v[q].y;
  }
  sort_sync();
#pragma unroll
  for (int i = 0; i < KPT; ++i) {
    if (i >= steps) break;
    const K k = a[first + 16 * i];
    b[wp[2 * (uint32_t(k >> shift) & 255u)] + RankPack<KPT>::get(rank2, i)] = k;
  }
  sort_sync();
}

}  // namespace rwt
