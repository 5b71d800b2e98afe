// gather_tiled.cu — gather of int32 payloads by tile-local windows:
// out[i] = in[loc[i]], same results as the windowed passes of
// gather_scatter.cu (and of the reference's gatherImpl.cpp:38-53) for every
// pass count.
//
// On a random permutation of 2^28 int32 a direct sweep is bound by DRAM random
// access (64-96 bytes pulled per 4-byte element).  Random reads inside a
// window of in[] that stays in L2 run at 225-260 G elements/s instead (2^28
// reads: 1.04 ms in windows of 2^16 to 2^20 elements, 1.13 ms at 2^22, 1.18 ms
// at 2^24, then 2.4 ms at 2^25, where the window no longer fits half of L2).
// So the requests are grouped by window, but only inside tiles of kTile
// consecutive i, which keeps every request of a tile in the tile's own
// stretch of the workspace:
//
//   group    one block per tile: loc grouped by window in shared memory and
//            written back as one run per window; slots[i] = where i's request
//            went in its tile; offs[w][tile] = where window w's run starts
//   fetch    window by window over all tiles: each run's indices are replaced
//            by in[index], read at random inside the one L2-resident window
//   restore  one block per tile: out[i] = the tile's value at slots[i], read
//            at random from shared memory
//
// A tile whose requests lie close together is gathered by the group kernel itself,
// with empty runs for the others (see kNear).
//
// Nothing is counted or claimed globally and the values need no second
// grouping on the way back, since a tile's values never leave the tile:
// 32 bytes per element (group 4 + 6, fetch 4 + 4 + 4, restore 6 + 4), against
// 72 for two partition levels out and two back.  Measured on permutations:
// 2^28 4.19 -> 2.06 ms (group 0.53, fetch 1.16, restore 0.37), 2^26 1.08 ->
// 0.54 ms.
#include <mutex>

#include "common.cuh"
#include "gather_scatter.h"

namespace edpp {
namespace {

constexpr int kTile = 8192;
constexpr int kThreads = 512;
constexpr int kPer = kTile / kThreads;  // 16 elements per thread, 4 vectors of 4
constexpr int kMaxWin = 128;
constexpr int kL2WinLog = 22;           // 16 MB windows: see the rates above
constexpr uint32_t kNoSlot = 0xffffu;   // an index outside [0, n): out[i] keeps its value
constexpr int kFetchThreads = 256;
constexpr int kFetchRuns = 4;           // tiles per warp
constexpr int kFetchTiles = kFetchThreads / 32 * kFetchRuns;

// A tile is read directly if its requests span at most kNear elements (one 32-byte
// sector per request: from DRAM that costs no more than the tiled way), if three
// quarters of its vectors lie within a 128-byte line each, or, in a large array, if the
// tile and one request of every 16th tile around it span at most kNearAll (a quarter of
// L2, for all tiles in flight): grouping gains nothing there.  2^26 requests, us, direct
// sweep / all tiles grouped / so: identity 129 / 673 / 170, rows of 4096 in random order
// 131 / 634 / 172, random within 4 MB 263 / 888 / 337, one address 90 / 922 / 119; a
// random permutation 999 / 524 / 524.  (The rest over the direct sweep is the other two
// kernels finding nothing to do.  A transpose, 275 / 683 / 700, looks random to a tile.)
constexpr uint32_t kNear = 8 * kTile, kNearAll = 1u << 23;
constexpr int64_t kNearAllFrom = 1 << 24;  // requests

// Windows of 2^log_w elements: 64 of them (runs of 128 requests, 512 bytes)
// while they fit L2 comfortably, then more windows up to kMaxWin, then larger
// ones.
struct GatherPlan {
  int log_w = 0, nwin = 1;
  int64_t tiles = 0, stride = 0;  // stride: tiles rounded up, the row length of offs
};

GatherPlan gather_plan(int64_t n) {
  GatherPlan p;
  p.log_w = 10;
  while (p.log_w < kL2WinLog && (n >> p.log_w) > kMaxWin / 2) ++p.log_w;
  while (((n - 1) >> p.log_w) >= kMaxWin) ++p.log_w;
  p.nwin = static_cast<int>(((n - 1) >> p.log_w) + 1);
  p.tiles = (n + kTile - 1) / kTile;
  p.stride = static_cast<int64_t>(round_up(static_cast<size_t>(p.tiles), kFetchTiles));
  return p;
}

struct GatherLayout {
  size_t buf, slots, offs, bytes;
};

GatherLayout gather_layout(const GatherPlan &p) {
  GatherLayout L{};
  const size_t elems = static_cast<size_t>(p.tiles) * kTile;
  L.buf = 0;
  L.slots = L.buf + 4 * elems;
  L.offs = L.slots + 2 * elems;
  L.bytes = L.offs + round_up(2 * static_cast<size_t>(p.stride) * (p.nwin + 1), 256);
  return L;
}

// Bound by the shared-memory pipe (one rank atomic, one offset lookup, one
// staging store per element, each ~3.5 wavefronts per warp at 64 windows) and
// by DRAM about equally.  Three blocks per SM (40 registers, a few spills)
// against two: the gather of 2^28 2.06 against 2.11 ms.
__global__ void __launch_bounds__(kThreads, 3)
    gather_group_kernel(const int32_t *__restrict__ loc, int64_t n, int log_w, int nwin,
                        int64_t stride, int32_t *__restrict__ buf, uint16_t *__restrict__ slots,
                        uint16_t *__restrict__ offs, bool vec, const int32_t *__restrict__ in,
                        int32_t *__restrict__ out, bool vec_out, bool near) {
  __shared__ alignas(16) int32_t stage[kTile];
  __shared__ uint32_t scnt[kMaxWin], soff[kMaxWin];
  __shared__ uint32_t s_total;
  __shared__ uint32_t s_lo[kThreads / 32], s_hi[kThreads / 32], s_tight[kThreads / 32];
  __shared__ bool s_maybe;
  const int t = threadIdx.x, lane = t & 31;
  const int64_t tile = blockIdx.x, base = tile * kTile;
  const uint32_t un = static_cast<uint32_t>(n);
  if (t < kMaxWin) scnt[t] = 0;
  if (tile + 1 == gridDim.x) {  // the rows of offs end in empty runs
    const int pad = static_cast<int>(stride - tile - 1);
    for (int i = t; i < pad * (nwin + 1); i += kThreads)
      offs[(i / pad) * stride + tile + 1 + i % pad] = 0;
  }
  int32_t l[kPer];
#pragma unroll
  for (int k = 0; k < kPer / 4; ++k) {
    const int64_t i = base + (k * kThreads + t) * 4;
    int4 q = make_int4(-1, -1, -1, -1);
    if (vec && i + 3 < n) {
      q = __ldcs(reinterpret_cast<const int4 *>(loc + i));
    } else {
      if (i + 0 < n) q.x = loc[i + 0];
      if (i + 1 < n) q.y = loc[i + 1];
      if (i + 2 < n) q.z = loc[i + 2];
      if (i + 3 < n) q.w = loc[i + 3];
    }
    l[4 * k] = q.x, l[4 * k + 1] = q.y, l[4 * k + 2] = q.z, l[4 * k + 3] = q.w;
  }
  // How near its requests lie: the first warp's first vectors tell a random tile apart,
  // all of them decide.
  uint32_t lo = ~0u, hi = 0, tight = 0;
  auto widen = [&](int k) {  // by a vector; tight: vectors whose requests lie within a line
    uint32_t a = ~0u, b = 0;
#pragma unroll
    for (int e = 4 * k; e < 4 * k + 4; ++e) {
      const uint32_t u = static_cast<uint32_t>(l[e]);
      if (u < un) a = min(a, u), b = max(b, u);
    }
    lo = min(lo, a), hi = max(hi, b);
    tight += __popc(__ballot_sync(0xffffffffu, b < a + 32 || b < a));
  };
  auto join = [&](uint32_t a, uint32_t b) {
    lo = __reduce_min_sync(0xffffffffu, a);
    hi = __reduce_max_sync(0xffffffffu, b);
  };
  const uint32_t near_all = n > kNearAllFrom ? kNearAll : kNear;
  if (t < 32) {
    widen(0);
    join(lo, hi);
    if (t == 0) s_maybe = near && (tight >= 16 || hi < lo || hi - lo < near_all);
  }
  __syncthreads();
  if (s_maybe) {
    tight = 0;
#pragma unroll
    for (int k = 0; k < kPer / 4; ++k) widen(k);
    join(lo, hi);
    if (lane == 0) s_lo[t >> 5] = lo, s_hi[t >> 5] = hi, s_tight[t >> 5] = tight;
    __syncthreads();
    constexpr int kWarps = kThreads / 32;
    join(s_lo[lane & (kWarps - 1)], s_hi[lane & (kWarps - 1)]);
    tight = __reduce_add_sync(0xffffffffu, lane < kWarps ? s_tight[lane] : 0u);
    bool direct = tight >= kThreads / 4 * 3 * (kPer / 4) || hi < lo || hi - lo < kNear;
    if (!direct && n > kNearAllFrom) {
      const int64_t j = base + (lane - 16) * (16ll * kTile) + 64 * lane;
      const uint32_t u = static_cast<uint32_t>(j >= 0 && j < n ? loc[j] : -1);
      join(u < un ? min(lo, u) : lo, u < un ? max(hi, u) : hi);
      direct = hi - lo < kNearAll;
    }
    if (direct) {
      for (int w = t; w <= nwin; w += kThreads) offs[w * stride + tile] = 0;
#pragma unroll
      for (int k = 0; k < kPer / 4; ++k) {
        const int64_t i = base + (k * kThreads + t) * 4;
        int32_t v[4];
        bool all = vec_out;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const bool ok = static_cast<uint32_t>(l[4 * k + q]) < un;
          all = all && ok;
          v[q] = ok ? in[l[4 * k + q]] : 0;
        }
        if (all) {
          __stcs(reinterpret_cast<int4 *>(out + i), make_int4(v[0], v[1], v[2], v[3]));
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (static_cast<uint32_t>(l[4 * k + q]) < un) out[i + q] = v[q];
        }
      }
      return;
    }
  }
  uint32_t rk[kPer / 2];  // two 16-bit ranks per register
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    uint32_t r = 0;
    if (static_cast<uint32_t>(l[e]) < un) r = atomicAdd(&scnt[l[e] >> log_w], 1u);
    if (e & 1) rk[e >> 1] |= r << 16;
    else rk[e >> 1] = r;
  }
  __syncthreads();
  if (t < 32) {  // exclusive scan of the window counts, 4 per lane
    uint32_t c[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c[k] = scnt[4 * t + k];
      s += c[k];
    }
    uint32_t incl = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
      if (t >= d) incl += y;
    }
    uint32_t run = incl - s;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int w = 4 * t + k;
      soff[w] = run;
      if (w <= nwin) offs[w * stride + tile] = static_cast<uint16_t>(run);
      run += c[k];
    }
    if (t == 31) {
      s_total = incl;
      if (nwin == kMaxWin) offs[nwin * stride + tile] = static_cast<uint16_t>(incl);
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kPer / 4; ++k) {
    uint32_t sl[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = 4 * k + q;
      sl[q] = kNoSlot;
      if (static_cast<uint32_t>(l[e]) < un) {
        sl[q] = soff[l[e] >> log_w] + ((rk[e >> 1] >> ((e & 1) * 16)) & 0xffffu);
        stage[sl[q]] = l[e];
      }
    }
    __stcs(reinterpret_cast<uint2 *>(slots + base) + k * kThreads + t,
           make_uint2(sl[0] | sl[1] << 16, sl[2] | sl[3] << 16));
  }
  __syncthreads();
  const int nv = static_cast<int>((s_total + 3) >> 2);
  int4 *dst = reinterpret_cast<int4 *>(buf + base);
  for (int v = t; v < nv; v += kThreads) __stcs(dst + v, reinterpret_cast<const int4 *>(stage)[v]);
}

// Blocks in window order, so the whole GPU reads one or two windows of in[] at
// a time; a warp takes the runs of kFetchRuns tiles as one list.  Bound by the
// L1's tag lookups, one per clock and SM for random reads (0.8 measured); the
// streamed side carries evict-first hints so the window stays in L2, and the
// random reads go past L1 (whole gather of 2^28: 2.064 -> 2.040 ms; with
// L1::no_allocate 2.115).
__global__ void __launch_bounds__(kFetchThreads, 6)
    gather_fetch_kernel(const int32_t *__restrict__ in, int64_t stride, unsigned groups,
                        const uint16_t *__restrict__ offs, int32_t *buf) {
  const unsigned w = blockIdx.x / groups, g = blockIdx.x - w * groups;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t t0 = static_cast<int64_t>(g) * kFetchTiles + wid * kFetchRuns;
  const ushort4 s = *reinterpret_cast<const ushort4 *>(offs + w * stride + t0);
  const ushort4 e = *reinterpret_cast<const ushort4 *>(offs + (w + 1) * stride + t0);
  const uint32_t p1 = e.x - s.x, p2 = p1 + (e.y - s.y), p3 = p2 + (e.z - s.z),
                 total = p3 + (e.w - s.w);
  const uint32_t b0 = static_cast<uint32_t>(t0) * kTile + s.x;
  const uint32_t b1 = static_cast<uint32_t>(t0 + 1) * kTile + s.y - p1;
  const uint32_t b2 = static_cast<uint32_t>(t0 + 2) * kTile + s.z - p2;
  const uint32_t b3 = static_cast<uint32_t>(t0 + 3) * kTile + s.w - p3;
  constexpr int U = 8;
  for (uint32_t e0 = lane; e0 < total; e0 += 32 * U) {
    uint32_t a[U];
    int32_t v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t j = e0 + 32 * u;
      a[u] = j + (j < p2 ? (j < p1 ? b0 : b1) : (j < p3 ? b2 : b3));
      v[u] = j < total ? __ldcs(buf + a[u]) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e0 + 32 * u < total) v[u] = __ldcg(in + v[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e0 + 32 * u < total) __stcs(buf + a[u], v[u]);
  }
}

// The tile's values by one bulk copy, then one random shared-memory read per
// element.  Bound by DRAM.
__global__ void __launch_bounds__(kThreads, 3)
    gather_restore_kernel(const int32_t *__restrict__ buf, const uint16_t *__restrict__ slots,
                          const uint16_t *__restrict__ totals, int64_t n, int32_t *__restrict__ out,
                          bool vec_out, uint64_t timeout_ns, unsigned *fault) {
  __shared__ alignas(128) int32_t val[kTile];
  __shared__ alignas(8) uint64_t bar;
  const int t = threadIdx.x;
  const int64_t tile = blockIdx.x, base = tile * kTile;
  const uint32_t bytes = (static_cast<uint32_t>(totals[tile]) * 4u + 15u) & ~15u;
  if (t == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    if (bytes) {
      mbar_arrive_expect_tx(&bar, bytes);
      tma_load_1d(val, buf + base, bytes, &bar);
    }
  }
  uint2 s[kPer / 4];
#pragma unroll
  for (int k = 0; k < kPer / 4; ++k)
    s[k] = __ldcs(reinterpret_cast<const uint2 *>(slots + base) + k * kThreads + t);
  __syncthreads();
  if (!bytes) return;
  if (!mbar_wait_bounded(&bar, 0, timeout_ns, fault)) return;
#pragma unroll
  for (int k = 0; k < kPer / 4; ++k) {
    const uint32_t sl[4] = {s[k].x & 0xffffu, s[k].x >> 16, s[k].y & 0xffffu, s[k].y >> 16};
    const int64_t i = base + (k * kThreads + t) * 4;
    int32_t v[4];
    bool all = vec_out;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      all = all && sl[q] != kNoSlot;
      v[q] = sl[q] != kNoSlot ? val[sl[q]] : 0;
    }
    if (all) {
      __stcs(reinterpret_cast<int4 *>(out + i), make_int4(v[0], v[1], v[2], v[3]));
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (sl[q] != kNoSlot) out[i + q] = v[q];
    }
  }
}

}  // namespace

size_t gather_tiled_bytes(int64_t n) { return gather_layout(gather_plan(n)).bytes; }

int gather_tiled(const int32_t *in, int32_t *out, int64_t n, const int32_t *loc, void *ws,
                 size_t ws_bytes, cudaStream_t st) {
  const GatherPlan p = gather_plan(n);
  const GatherLayout L = gather_layout(p);
  if (!ws || ws_bytes < L.bytes) return EDPP_ENOMEM;
  unsigned *fault = fault_word();
  if (!fault) return EDPP_ECUDA;
  char *w = static_cast<char *>(ws);
  auto *buf = reinterpret_cast<int32_t *>(w + L.buf);
  auto *slots = reinterpret_cast<uint16_t *>(w + L.slots);
  auto *offs = reinterpret_cast<uint16_t *>(w + L.offs);
  const unsigned tiles = static_cast<unsigned>(p.tiles);
  // a tile read directly is written while others still read: not in place
  auto apart = [n](const int32_t *a, const int32_t *b) { return a + n <= b || b + n <= a; };
  const bool near = apart(in, out) && apart(loc, out);
  gather_group_kernel<<<tiles, kThreads, 0, st>>>(loc, n, p.log_w, p.nwin, p.stride, buf, slots,
                                                  offs, aligned16(loc), in, out, aligned16(out),
                                                  near);
  const unsigned groups = static_cast<unsigned>(p.stride / kFetchTiles);
  gather_fetch_kernel<<<static_cast<unsigned>(p.nwin) * groups, kFetchThreads, 0, st>>>(
      in, p.stride, groups, offs, buf);
  gather_restore_kernel<<<tiles, kThreads, 0, st>>>(buf, slots, offs + p.nwin * p.stride, n, out,
                                                    aligned16(out), kDefaultWaitNs, fault);
  return launch_status();
}

}  // namespace edpp
