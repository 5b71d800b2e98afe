// pos_stage.cuh — ranking and re-layout of a split tile by source positions,
// shared by the split (split_index.cuh) and the batched split tiles (batch.cu).
//
// A tile stays in shared memory as loaded.  Ranking takes one shared-memory
// atomic per element: the old value of the (warp, bucket) counter is the
// element's rank among its warp's elements of the bucket.  What is re-laid out
// in bucket order is only the 16-bit source position; the write-out fetches key
// and value from there.
//
// Atomics of one warp instruction on one counter, and of successive
// instructions, have returned in lane and program order wherever it was
// looked at, but nothing promises that, so the write-out checks it: positions
// must ascend within every bucket's run.  A tile that fails is ranked again by
// peer groups (exact, slow) and written over.
//
// The counters are 16 bits, cnt16[warp * buckets + b], an even number of
// buckets; between rank() and place() the caller turns them into each warp's
// first slot of the bucket.  Callers put barriers between the steps.
#pragma once

#include "common.cuh"

namespace edpp {

// From here on a tile's ranking shows in the split's time where a warp's lanes share
// one counter (2^26 pairs, 90% of the keys in one bucket, against ranking by peer
// groups: 256 buckets 450 us against 492, 512 503 against 448).
constexpr int kJoinBuckets = 512;

// kJoin: used with kJoinBuckets buckets and more.
template <int NT, int TILE, bool kJoin = false> struct PosStage {
  static constexpr int kWarps = NT / 32;
  static constexpr int kSeg = TILE / kWarps;  // a warp's contiguous part of the tile
  static constexpr int kIters = kSeg / 32;

  __device__ __forceinline__ static int position(int it) {
    return static_cast<int>(threadIdx.x >> 5) * kSeg + it * 32 + static_cast<int>(threadIdx.x & 31);
  }

  // br[it] = bucket | rank << 16 of this lane's elements; bucket_at(position).
  template <typename F>
  __device__ __forceinline__ static void rank(uint16_t *cnt16, int buckets, int count, F bucket_at,
                                              uint32_t (&br)[kIters]) {
    // two counters per 32-bit word
    uint32_t *words =
        reinterpret_cast<uint32_t *>(cnt16) + (threadIdx.x >> 5) * (static_cast<unsigned>(buckets) >> 1);
#pragma unroll
    for (int it = 0; it < kIters; ++it) {
      const int pos = position(it);
      br[it] = pos < count ? static_cast<uint32_t>(bucket_at(pos)) : 0u;
    }
    // Keys already in bucket order put a whole warp on one counter, 32 atomics
    // in a row: where a warp's first and last element share a bucket, a step of
    // one bucket takes one atomic (split of 2^27 sorted pairs, 256 / 512 buckets
    // 0.885 / 0.969 -> 0.582 / 0.647 ms; uniform keys 0 to 1% slower for the test).
    const int lane = threadIdx.x & 31;
    const int first = position(0) - lane, last = min(first + kSeg, count) - 1;
    if (last >= first && bucket_at(first) == bucket_at(last)) {
      const uint32_t b = static_cast<uint32_t>(bucket_at(first)), shb = (b & 1u) * 16u;
      if (kJoin && buckets >= kJoinBuckets && rank_joined(words, count, b, br)) return;
#pragma unroll
      for (int it = 0; it < kIters; ++it) {
        const bool valid = position(it) < count;
        const unsigned mine = __ballot_sync(0xffffffffu, valid && br[it] == b);
        if (mine == 0xffffffffu) {
          uint32_t old = 0;
          if (lane == 0) old = atomicAdd(&words[b >> 1], 32u << shb);
          old = (__shfl_sync(0xffffffffu, old, 0) >> shb) & 0xffffu;
          br[it] |= (old + lane) << 16;
        } else if (valid) {
          const uint32_t sh = (br[it] & 1u) * 16u;
          br[it] |= ((atomicAdd(&words[br[it] >> 1], 1u << sh) >> sh) & 0xffffu) << 16;
        }
      }
      return;
    }
#pragma unroll
    for (int it = 0; it < kIters; ++it) {
      const uint32_t sh = (br[it] & 1u) * 16u;
      if (position(it) < count)
        br[it] |= ((atomicAdd(&words[br[it] >> 1], 1u << sh) >> sh) & 0xffffu) << 16;
    }
  }

  // Ranks of a warp that has much of bucket b, but not all of it in a row: in every
  // step the lanes of b take one atomic by their lowest, beside the other lanes' own,
  // and share its old value once all steps' atomics are out.  2^26 pairs with 90% of
  // the keys in one of 512 / 1024 buckets, in random order: 503 / 628 us with an
  // atomic for each, 387 / 560 so.  False: br as before.
  __device__ __forceinline__ static bool rank_joined(uint32_t *words, int count, uint32_t b,
                                                     uint32_t (&br)[kIters]) {
    // one step tells: all of b, or few of it
    const unsigned some = __ballot_sync(0xffffffffu, position(kIters / 2) < count && br[kIters / 2] == b);
    if (some == 0xffffffffu || __popc(some) < 8) return false;
    auto lower = [] {  // read at each use: held, it costs a register that the KO split lacks
      unsigned lt;
      asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
      return lt;
    };
#pragma unroll
    for (int it = 0; it < kIters; ++it) {
      const bool valid = position(it) < count, in = valid && br[it] == b;
      const unsigned mine = __ballot_sync(0xffffffffu, in);
      const uint32_t sh = (br[it] & 1u) * 16u;
      if (valid && !(in && (mine & lower()))) {
        const uint32_t old = atomicAdd(&words[br[it] >> 1], (in ? __popc(mine) : 1u) << sh);
        br[it] |= ((old >> sh) & 0xffffu) << 16;
      }
    }
#pragma unroll
    for (int it = 0; it < kIters; ++it) {
      const bool in = position(it) < count && (br[it] & 0xffffu) == b;
      const unsigned mine = __ballot_sync(0xffffffffu, in);
      const uint32_t first = __shfl_sync(0xffffffffu, br[it], __ffs(mine) - 1);
      if (in) br[it] = first + (static_cast<uint32_t>(__popc(mine & lower())) << 16);
    }
    return true;
  }

  __device__ __forceinline__ static void place(const uint16_t *cnt16, int buckets, int count,
                                               const uint32_t (&br)[kIters], uint16_t *s_pos) {
    const uint16_t *mine = cnt16 + (threadIdx.x >> 5) * buckets;
#pragma unroll
    for (int it = 0; it < kIters; ++it) {
      const int pos = position(it);
      if (pos < count) s_pos[mine[br[it] & 0xffffu] + (br[it] >> 16)] = static_cast<uint16_t>(pos);
    }
  }

  // Exact slots, instead of place(): the lanes of a bucket count their lower
  // peers, step by step in input order, advancing the warp's slot of the bucket.
  template <typename F>
  __device__ __forceinline__ static void place_exact(uint16_t *cnt16, int buckets, int count,
                                                     F bucket_at, uint16_t *s_pos) {
    uint16_t *mine = cnt16 + (threadIdx.x >> 5) * buckets;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    for (int it = 0; it < kIters; ++it) {
      const int pos = position(it);
      const bool valid = pos < count;
      const int b = valid ? bucket_at(pos) : 0;
      const unsigned vmask = __ballot_sync(0xffffffffu, valid);
      const unsigned peers = match_low_bits(static_cast<unsigned>(b), 31 - __clz(buckets), vmask);
      const int before = valid ? mine[b] : 0;
      __syncwarp();
      if (valid && (peers & lt) == 0u) mine[b] = static_cast<uint16_t>(before + __popc(peers));
      __syncwarp();
      if (valid) s_pos[before + __popc(peers & lt)] = static_cast<uint16_t>(pos);
    }
  }

  // store(slot, bucket, load(position)) for every slot, consecutive threads on
  // consecutive slots; bucket_of(element).  True when a position is out of order.
  template <int UNROLL, typename L, typename B, typename S>
  __device__ __forceinline__ static bool write_out(const uint16_t *s_pos, int count, L load,
                                                   B bucket_of, S store) {
    const int lane = threadIdx.x & 31;
    bool bad = false;
#pragma unroll UNROLL
    for (int s0 = 0; s0 < TILE; s0 += NT) {
      const int s = s0 + static_cast<int>(threadIdx.x);
      const bool valid = s < count;
      const int pos = valid ? s_pos[s] : 0;
      const auto e = load(pos);
      const int b = bucket_of(e);
      const int mine = b * TILE + pos;  // ascends from slot to slot
      int before = __shfl_up_sync(0xffffffffu, mine, 1);
      if (lane == 0 && valid) {
        const int q = s > 0 ? s_pos[s - 1] : 0;
        before = s > 0 ? bucket_of(load(q)) * TILE + q : -1;
      }
      bad |= valid && before >= mine;
      if (valid) store(s, b, e);
    }
    return bad;
  }
};

}  // namespace edpp
