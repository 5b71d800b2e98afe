// split_index.cuh — split scatter that stages source positions (split.cu).
//
// Ranking, re-layout and write-out as pos_stage.cuh describes them.
//
// Bound by the shared-memory pipe: 27 wavefronts per 32 pairs at 256 buckets
// (the returning atomic 8, the random reads of key and value 7, the position
// store and the slot lookup 3 each) against 34 for per-warp lane masks with
// the pairs themselves re-laid out, and nothing in the ranking waits for the
// step before.  Scatter alone, 2^28 pairs, 256 buckets: 1.30 -> 1.00 ms; whole
// splits at index_buckets() in split.cu.  512 and 1024 buckets ranked by a
// leader table before: 1.85 -> 1.51 and 2.57 -> 2.19 ms.
#pragma once

#include "pos_stage.cuh"

namespace edpp {
namespace {

constexpr int kIndexThreads = 512;
// tile | positions | counters of 16 bits per (warp, bucket) | totals | run starts
template <int LAYOUT, int TILE> size_t index_smem_bytes(int buckets) {
  return static_cast<size_t>(TILE) * (LAYOUT == EDPP_KO ? 4 : 8) + 2 * static_cast<size_t>(TILE) +
         round_up(static_cast<size_t>(kIndexThreads / 32) * buckets * 2, 16) +
         8 * static_cast<size_t>(buckets);
}

// Blocks per SM: three where shared memory holds them (40 registers), else two.
// 2^28 keys, 64 / 256 buckets, two against three: 0.989 -> 0.872, 1.090 -> 1.009
// ms.  The fused form has one or two blocks per SM to run anyway.
template <int LAYOUT, int TILE, bool kFused> constexpr int index_blocks() {
  return !kFused && (LAYOUT == EDPP_KO || TILE < 8192) ? 3 : 2;
}

template <int LAYOUT, int TILE, bool kFused>
__global__ void __launch_bounds__(kIndexThreads, index_blocks<LAYOUT, TILE, kFused>())
    split_index_kernel(const int32_t *__restrict__ keys_in, int32_t *__restrict__ keys_out,
                       const int32_t *__restrict__ vals_in, int32_t *__restrict__ vals_out,
                       int64_t n, int buckets, int shift, int64_t tiles,
                       const int32_t *__restrict__ his, bool tma, bool exact, uint64_t timeout_ns,
                       unsigned *fault, FusedArgs fused) {
  using C = PosStage<kIndexThreads, TILE, !kFused && TILE == 8192>;
  constexpr int THREADS = kIndexThreads;
  extern __shared__ __align__(128) unsigned char smem[];
  int32_t *s_keys = reinterpret_cast<int32_t *>(smem);
  int32_t *s_vals = s_keys + TILE;                 // SOA only
  int2 *s_pairs = reinterpret_cast<int2 *>(smem);  // AOS only
  uint16_t *s_pos = reinterpret_cast<uint16_t *>(smem + TILE * (LAYOUT == EDPP_KO ? 4 : 8));
  uint16_t *cnt16 = s_pos + TILE;
  int32_t *toff = reinterpret_cast<int32_t *>(
      reinterpret_cast<unsigned char *>(cnt16) + round_up(static_cast<size_t>(C::kWarps) * buckets * 2, 16));
  int32_t *gofs = toff + buckets;
  __shared__ alignas(8) uint64_t bar;
  __shared__ int32_t s_wsum[32];

  const int64_t t = blockIdx.x;
  const int64_t base = t * TILE;
  const int count = static_cast<int>(min64(TILE, n - base));
  const unsigned mask = static_cast<unsigned>(buckets - 1);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;

  // -- load the tile (bulk copies for the 16-byte-aligned prefix) --
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  uint32_t bulk_elems = 0;
  if (tma) bulk_elems = (LAYOUT == EDPP_KVS_AOS) ? (count & ~1) : (count & ~3);
  if (tid == 0 && bulk_elems) {
    mbar_arrive_expect_tx(&bar, bulk_elems * (LAYOUT == EDPP_KO ? 4 : 8));
    if (LAYOUT == EDPP_KVS_AOS) {
      tma_load_1d(s_pairs, keys_in + 2 * base, bulk_elems * 8, &bar);
    } else {
      tma_load_1d(s_keys, keys_in + base, bulk_elems * 4, &bar);
      if (LAYOUT == EDPP_KVS_SOA) tma_load_1d(s_vals, vals_in + base, bulk_elems * 4, &bar);
    }
  }
  // As in split_scatter_kernel; pairs in one array gain 1-2% (2^28, 8 / 256
  // buckets 1.288 / 1.338 -> 1.271 / 1.314 ms), the other layouts nothing.
  const int64_t ahead = base + static_cast<int64_t>(kGb300Sms) * TILE;
  if (!kFused && LAYOUT == EDPP_KVS_AOS && tid == 32 && tma && ahead + TILE <= n) {
    l2_prefetch(keys_in + 2 * ahead, TILE * 8);
  }
  for (int i = static_cast<int>(bulk_elems) + tid; i < count; i += THREADS) {
    if (LAYOUT == EDPP_KVS_AOS) {
      s_pairs[i] = make_int2(keys_in[2 * (base + i)], keys_in[2 * (base + i) + 1]);
    } else {
      s_keys[i] = keys_in[base + i];
      if (LAYOUT == EDPP_KVS_SOA) s_vals[i] = vals_in[base + i];
    }
  }
  for (int i = tid; i < C::kWarps * buckets / 2; i += THREADS)
    reinterpret_cast<uint32_t *>(cnt16)[i] = 0u;
  const int per = (buckets + THREADS - 1) / THREADS;
  const int b_lo = min(buckets, tid * per), b_hi = min(buckets, b_lo + per);
  constexpr int kHisPre = 2;  // 512 threads serve up to 1024 buckets
  int32_t his_pre[kHisPre];
#pragma unroll
  for (int k = 0; k < kHisPre; ++k)
    his_pre[k] = !kFused && b_lo + k < b_hi
                     ? __ldg(his + static_cast<int64_t>(b_lo + k) * tiles + t) : 0;
  if (bulk_elems) {
    if (!mbar_wait_bounded(&bar, 0, timeout_ns, fault)) return;
  }
  __syncthreads();
  // an element: {key, value}, or the key alone
  auto load = [&](int pos) {
    if constexpr (LAYOUT == EDPP_KVS_AOS) return s_pairs[pos];
    else if constexpr (LAYOUT == EDPP_KVS_SOA) return make_int2(s_keys[pos], s_vals[pos]);
    else return make_int2(s_keys[pos], 0);
  };
  auto bucket_of = [&](int2 e) {
    return static_cast<int>((static_cast<unsigned>(e.x) >> shift) & mask);
  };
  auto bucket_at = [&](int pos) {
    return bucket_of(make_int2(LAYOUT == EDPP_KVS_AOS ? s_pairs[pos].x : s_keys[pos], 0));
  };
  uint32_t br[C::kIters];
  C::rank(cnt16, buckets, count, bucket_at, br);
  __syncthreads();

  // -- per bucket: tile count, tile offset, then each warp's first slot
  // (cnt16[w][b] becomes the tile slot of warp w's first element of bucket b) --
  int32_t my_total = 0;
  for (int b = b_lo; b < b_hi; ++b) {
    int32_t tot = 0;
#pragma unroll 8
    for (int ww = 0; ww < C::kWarps; ++ww) tot += cnt16[ww * buckets + b];
    toff[b] = tot;
    my_total += tot;
  }
  int32_t incl = my_total;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += y;
  }
  if (lane == 31) s_wsum[w] = incl;
  __syncthreads();
  int32_t run = incl - my_total;
#pragma unroll
  for (int k = 0; k < C::kWarps; ++k)
    if (k < w) run += s_wsum[k];
  if (kFused) {
    // the position area is free until the re-layout
    if (!fused_starts<THREADS>(fused, static_cast<int>(t), static_cast<int>(tiles), buckets, toff,
                               gofs, reinterpret_cast<int32_t *>(s_pos), timeout_ns, fault))
      return;
#pragma unroll
    for (int k = 0; k < kHisPre; ++k) his_pre[k] = b_lo + k < b_hi ? gofs[b_lo + k] : 0;
  }
#pragma unroll
  for (int k = 0; k < kHisPre; ++k) {
    const int b = b_lo + k;
    if (b < b_hi) {
      gofs[b] = his_pre[k] - run;  // output index of a slot of this run, minus the slot
#pragma unroll 8
      for (int ww = 0; ww < C::kWarps; ++ww) {
        const int32_t c = cnt16[ww * buckets + b];
        cnt16[ww * buckets + b] = static_cast<uint16_t>(run);
        run += c;
      }
    }
  }
  __syncthreads();

  // -- re-lay out and write --
  auto store = [&](int slot, int b, int2 e) {
    const int64_t o = static_cast<int64_t>(gofs[b]) + slot;
    if (LAYOUT == EDPP_KVS_AOS) {
      reinterpret_cast<int2 *>(keys_out)[o] = e;
    } else {
      keys_out[o] = e.x;
      if (LAYOUT == EDPP_KVS_SOA) vals_out[o] = e.y;
    }
  };
  // 8192 pairs, 256 buckets: four elements in flight per thread 1.243, two 1.210
  // ms at 2^28; the other forms prefer four (6144 pairs 1.013 against 1.054 with
  // one)
  constexpr int kUnroll = LAYOUT == EDPP_KVS_SOA && TILE == 8192 ? 2 : 4;
  bool bad = exact;
  if (!exact) {
    C::place(cnt16, buckets, count, br, s_pos);
    __syncthreads();
    bad = C::template write_out<kUnroll>(s_pos, count, load, bucket_of, store);
  }
  if (__syncthreads_or(bad)) {
    C::place_exact(cnt16, buckets, count, bucket_at, s_pos);
    __syncthreads();
    C::template write_out<1>(s_pos, count, load, bucket_of, store);
  }
}

}  // namespace
}  // namespace edpp
