// scan_pipe.cu — the pipelined one-launch scan: reduce-then-scan with the tile
// held in shared memory between its two reads.
//
// A persistent grid of one block per SM walks the input in waves of G tiles
// (G = blocks); block b owns tile b of every wave.  Each block is a pipeline
// of warp roles over a ring of tile buffers:
//
//   load     one warp brings tiles in by TMA bulk copies as buffers empty
//   reduce   three warps, a tile each in turn, sum a landed tile and publish
//            the sum as one {flag, value} word, running ahead of the scan
//   prefix   four warps, a wave each in turn, read the wave's G words, add up
//            those before their own tile and the wave's total, and hand the
//            tile's exclusive prefix to the scan warps
//   scan     two groups of eight warps, a tile each in turn, scan it in
//            registers (the buffer is free again as soon as it is read), wait
//            for the prefix, and store
//
// Each element is read from DRAM once and written once, and no tile waits for
// another tile's prefix: a wave's words depend only on loads, so several waves
// are in flight per block.  In the look-back scan a block holds one tile from
// load to store and spends 40% of that time waiting for predecessors
// (5.8 of 14 us); the chunked reduce-then-scan reads every slice twice, the
// second time from L2, with one tile per block in flight.
// The sum of the earlier waves passes from prefix warp to prefix warp (in f64
// for f32 sums), so the summation order is fixed: repeated runs agree bit for
// bit.  Reading the words with one prefix warp bounded the kernel at one L2
// round trip per wave (2^30 int32 1.77 ms).
//
// Bound by DRAM.  Measured (ms, look-back form before): 2^30 int32 2.00 -> 1.30
// (6.6 TB/s), 2^30 f32 2.14 -> 1.25, 2^28 int64 1.04 -> 0.68, 2^24 int32 0.045
// -> 0.035 (launch, first loads and last stores).
//
// Launched cooperatively, since a wave's words come from all blocks.  Every
// wait is bounded; a wait that runs out raises EDPP_FAULT_TIMEOUT (or _TMA),
// sets the call's abort flag, and every role runs to its end without further
// waits or stores.
#include <algorithm>
#include <mutex>

#include "batch_plan.h"
#include "scan_pipe.h"
#include "scan_tile.cuh"

namespace edpp {
namespace {

// Two groups of eight scan warps take alternate tiles of 16 KB (four 16-byte
// chunks per thread), so one group's barrier and shuffle latency is covered by
// the other.  Measured at 2^30 int32 / 2^30 f32 / 2^28 int64 (ms): one group
// with 32 KB tiles 1.417 / 1.433 / 0.788, one with 16 KB 1.388 / 1.342 /
// 0.815, two with 16 KB 1.299 / 1.245 / 0.679, two with 8 KB 1.777 / 1.973 /
// 1.030 (the prefix warps' round trips per byte bound that one).
constexpr int kGroups = 2, kScanWarps = 8, kChunks = 4;
constexpr int kReduceWarps = 3, kPrefixWarps = 4;
constexpr int kScanThreads = 32 * kScanWarps;
constexpr int kThreads = kGroups * kScanThreads + 32 * (kReduceWarps + 1 + kPrefixWarps);
constexpr int kTileBytes = kScanThreads * kChunks * 16;
constexpr int kStages = 12;      // 192 KB of tile buffers per block
constexpr int kMaxBlocks = 256;  // words a prefix warp reads per wave: 8 per lane
constexpr size_t kHeader = 256;
constexpr uint32_t kFlagTail = kFlagIncl, kFlagHead = kFlagAgg;  // of a published tile sum
static_assert(kStages % kReduceWarps == 0 && kStages % kGroups == 0,
              "a buffer always has the same reduce warp and scan group");

// Sums across tiles: f32 in f64 (one warp's work), the rest in their own type.
template <typename T> struct Wide { using type = T; };
template <> struct Wide<float> { using type = double; };

struct PipeShared {
  uint64_t full[kStages];       // a tile landed
  uint64_t empty[kStages];      // its reduce warp and the scan warps have read it
  uint64_t ready[2 * kStages];  // its prefix is in pre[]
  uint64_t carried[kPrefixWarps];  // the sum of all earlier waves is in carry[]
  int abort;
};

// Wait for phase `parity` of bar: false once the block's abort flag is up or
// the limit runs out (which raises both flags).  The whole warp calls it and
// gets one answer.
__device__ __forceinline__ bool pipe_wait(uint64_t *bar, uint32_t parity, volatile int *s_abort,
                                          uint64_t timeout_ns, unsigned *fault,
                                          unsigned *abort_flag) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    const uint64_t t0 = globaltimer_ns();
    while (!(ok = mbar_try_wait(bar, parity))) {
      if (*s_abort) break;
      if (globaltimer_ns() - t0 > timeout_ns) {
        raise_fault(fault, EDPP_FAULT_TMA);
        atomicOr(abort_flag, 1u);
        *s_abort = 1;
        break;
      }
    }
  }
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ void scan_group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kScanThreads) : "memory");
}

// Where a tile lies.  head: its prefix starts from zero (kSegmented only).
struct TileAt {
  int64_t base;
  int32_t count, head;
};

// One array cut into tiles.  The sum of tile `withheld` is never published (the
// bounded-wait self-test; -1 otherwise).
template <typename T> struct ArrayTiles {
  static constexpr bool kSegmented = false;
  int64_t n, num_tiles, withheld;
  __device__ __forceinline__ TileAt at(int64_t tile) const {
    constexpr int kTile = kTileBytes / sizeof(T);
    return {tile * kTile, static_cast<int32_t>(min64(kTile, n - tile * kTile)), 0};
  }
};

// The scan tiles of a batch: tile i is a task's tile of its segment, and every
// segment's first tile is a head.  A task outside the plan's tables, or of a
// segment off 16-byte alignment (the tables of another plan: a bulk copy would
// fault there), is recorded and counts no elements.
struct TaskTiles {
  static constexpr bool kSegmented = true;
  const DevSeg *segs;
  const DevTask *tasks;
  int num_segs;
  int64_t num_tiles;
  unsigned *fault;
  __device__ __forceinline__ TileAt at(int64_t tile) const {
    constexpr int kTile = kTileBytes / 4;
    const DevTask t = tasks[tile];
    bool ok = t.seg >= 0 && t.seg < num_segs;
    DevSeg seg{};
    if (ok) seg = segs[t.seg];
    ok = ok && t.tile >= 0 && t.tile < seg.tiles && (seg.off & 3) == 0;
    if (!ok) raise_fault(fault, EDPP_FAULT_PLAN);
    if (!ok) return {0, 0, 1};
    const int64_t off = static_cast<int64_t>(t.tile) * kTile;
    return {seg.off + off, static_cast<int32_t>(min64(kTile, seg.len - off)), t.tile == 0};
  }
};

// Bit i set for the words i of this lane group that are at most `last`.
__device__ __forceinline__ uint32_t up_to(int last) {
  return last < 0 ? 0u : last >= 31 ? 0xffffffffu : (2u << last) - 1u;
}

template <typename T, bool kInclusive, typename Tiles>
__global__ void __launch_bounds__(kThreads, 1)
    scan_pipe_kernel(const T *in, T *out, Tiles tiles, LookbackState<T> st, unsigned *abort_flag,
                     uint64_t timeout_ns, unsigned *fault) {
  constexpr bool kSegmented = Tiles::kSegmented;
  const int64_t num_tiles = tiles.num_tiles;
  constexpr int E = Chunk<T>::E;
  constexpr int CH = kChunks, kTile = kTileBytes / sizeof(T), stages = kStages;
  using W = typename Wide<T>::type;
  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ PipeShared sh;
  __shared__ T pre[2 * kStages];
  __shared__ W carry[kPrefixWarps];
  __shared__ TileAt meta[kSegmented ? kStages : 1];  // of the tile in each buffer
  __shared__ T tot[kGroups][2][kScanWarps * CH];  // [group][alternating][row k][warp]
  const int lane = threadIdx.x & 31;
  // scan warps count within their group; the other roles follow the groups
  const int group = min(static_cast<int>(threadIdx.x) / kScanThreads, kGroups - 1);
  const int tid = threadIdx.x - group * kScanThreads, warp = tid >> 5;
  const int64_t G = gridDim.x, b = blockIdx.x;
  const int64_t steps = b < num_tiles ? (num_tiles - b + G - 1) / G : 0;
  volatile int *s_abort = &sh.abort;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1 + kScanWarps);
      mbar_init(&sh.ready[2 * s], 1);
      mbar_init(&sh.ready[2 * s + 1], 1);
    }
    for (int q = 0; q < kPrefixWarps; ++q) mbar_init(&sh.carried[q], 1);
    sh.abort = 0;
    fence_mbar_init();
  }
  __syncthreads();
  auto buf = [&](int s) { return reinterpret_cast<T *>(ring + static_cast<size_t>(s) * kTile * sizeof(T)); };
  auto wait = [&](uint64_t *bar, uint32_t parity) {
    return pipe_wait(bar, parity, s_abort, timeout_ns, fault, abort_flag);
  };

  if (warp < kScanWarps) {
    // ---- scan ----
    bool dead = false;
    int s = group, p = group;  // ring positions of the tile and of its prefix
    uint32_t sp = 0, pp = 0, half = 0;
    for (int64_t i = group; i < steps; i += kGroups, half ^= 1u) {
      if (!dead) dead = !wait(&sh.full[s], sp);
      const TileAt where = kSegmented ? meta[s] : tiles.at(i * G + b);
      const int64_t base = where.base;
      const int count = where.count;
      Chunk<T> c[CH];
      T incl[CH];
      const uint4 *src = reinterpret_cast<const uint4 *>(buf(s)) + tid;
#pragma unroll
      for (int k = 0; k < CH; ++k) c[k].raw = src[k * kScanThreads];
#pragma unroll
      for (int k = 0; k < CH; ++k) {
#pragma unroll
        for (int e = 1; e < E; ++e) c[k].e[e] = op_add(c[k].e[e - 1], c[k].e[e]);
        incl[k] = c[k].e[E - 1];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.empty[s]);  // the tile is in registers
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
        for (int k = 0; k < CH; ++k) {
          const T y = shfl_up(incl[k], d);
          if (lane >= d) incl[k] = op_add(incl[k], y);
        }
      }
      T *tw = tot[group][half];
      T wex[CH];  // exclusive over the lanes of the warp
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const T ex = shfl_up(incl[k], 1);
        wex[k] = lane == 0 ? zero_of<T>() : ex;
        if (lane == 31) tw[k * kScanWarps + warp] = incl[k];
      }
      // the only barrier of a step: tot[] alternates, so the next step's
      // totals land in the other half
      scan_group_sync(group);
      // every warp scans the NT warp totals for itself, PER consecutive ones
      // per lane
      constexpr int NT = kScanWarps * CH;
      constexpr int PER = NT >= 32 ? NT / 32 : 1;
      T x[PER], xs = zero_of<T>();
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        x[q] = lane * PER + q < NT ? tw[lane * PER + q] : zero_of<T>();
        xs = op_add(xs, x[q]);
      }
      const T xi = warp_incl_scan(xs, lane);
      const T xe = shfl_up(xi, 1);
      T run = lane == 0 ? zero_of<T>() : xe;
      T xp[PER];
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        xp[q] = run;
        run = op_add(run, x[q]);
      }
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int j = k * kScanWarps + warp;
        T v = zero_of<T>();
#pragma unroll
        for (int q = 0; q < PER; ++q) {
          const T y = shfl_idx(xp[q], j / PER);
          if (j % PER == q) v = y;
        }
        wex[k] = op_add(v, wex[k]);
      }
      if (!dead) dead = !wait(&sh.ready[p], pp);
      const T prefix = pre[p];
      if (!dead) {
        uint4 *dst = reinterpret_cast<uint4 *>(out + base) + tid;
#pragma unroll
        for (int k = 0; k < CH; ++k) {
          const T off = op_add(prefix, wex[k]);
          if (kInclusive) {
#pragma unroll
            for (int e = 0; e < E; ++e) c[k].e[e] = op_add(off, c[k].e[e]);
          } else {
#pragma unroll
            for (int e = E - 1; e >= 1; --e) c[k].e[e] = op_add(off, c[k].e[e - 1]);
            c[k].e[0] = off;
          }
          const int first = (k * kScanThreads + tid) * E;
          if (first + E <= count) {
            __stcs(dst + k * kScanThreads, c[k].raw);
          } else {
#pragma unroll
            for (int e = 0; e < E; ++e)
              if (first + e < count) out[base + first + e] = c[k].e[e];
          }
        }
      }
      if ((s += kGroups) >= stages) s -= stages, sp ^= 1u;
      if ((p += kGroups) >= 2 * stages) p -= 2 * stages, pp ^= 1u;
    }
  } else if (warp < kScanWarps + kReduceWarps) {
    // ---- reduce: warp r takes steps r, r + kReduceWarps, ...  The stages are a
    // multiple of kReduceWarps, so a buffer always has the same reduce warp
    // and its phases are awaited in order (tiles may land out of order). ----
    for (int64_t i = warp - kScanWarps; i < steps; i += kReduceWarps) {
      const int s = static_cast<int>(i % stages);
      if (!wait(&sh.full[s], static_cast<uint32_t>(i / stages) & 1u)) break;
      const uint32_t flag = kSegmented && meta[s].head ? kFlagHead : kFlagTail;
      const uint4 *src = reinterpret_cast<const uint4 *>(buf(s)) + lane;
      // eight chains of additions, joined pairwise
      T acc[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] = zero_of<T>();
#pragma unroll 2
      for (int k = 0; k < kScanWarps * CH; k += 8) {
        Chunk<T> q[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) q[u].raw = src[(k + u) * 32];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          T v = op_add(q[u].e[0], q[u].e[1]);
          if (E == 4) v = op_add(v, op_add(q[u].e[E - 2], q[u].e[E - 1]));
          acc[u] = op_add(acc[u], v);
        }
      }
#pragma unroll
      for (int d = 4; d >= 1; d >>= 1)
#pragma unroll
        for (int u = 0; u < d; ++u) acc[u] = op_add(acc[u], acc[u + d]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.empty[s]);
      const T v = warp_sum(acc[0]);
      bool known = lane == 0;
      if constexpr (!kSegmented) known = known && i * G + b != tiles.withheld;
      if (known) st.publish(i * G + b, flag, v);
    }
  } else if (warp == kScanWarps + kReduceWarps) {
    // ---- load ----
    int64_t i = 0;
    // kSegmented: lane l looks up step l of the next 32, with the elements past
    // the tile's last whole 16 bytes, so that no step waits for them
    TileAt ahead{};
    T rest[E - 1];
    for (; i < steps; ++i) {
      const int s = static_cast<int>(i % stages);
      if (kSegmented && (i & 31) == 0 && i + lane < steps) {
        ahead = tiles.at((i + lane) * G + b);
        const int rem = ahead.count % E;
#pragma unroll
        for (int e = 0; e < E - 1; ++e)
          rest[e] = e < rem ? in[ahead.base + ahead.count - rem + e] : zero_of<T>();
      }
      TileAt where;
      if (kSegmented) {
        where.base = __shfl_sync(0xffffffffu, ahead.base, static_cast<int>(i & 31));
        where.count = __shfl_sync(0xffffffffu, ahead.count, static_cast<int>(i & 31));
        where.head = __shfl_sync(0xffffffffu, ahead.head, static_cast<int>(i & 31));
      } else {
        where = tiles.at(i * G + b);
      }
      if (i >= stages && !wait(&sh.empty[s], static_cast<uint32_t>(i / stages - 1) & 1u)) break;
      const int64_t base = where.base;
      const int count = where.count;
      const uint32_t bytes = (static_cast<uint32_t>(count) * sizeof(T)) & ~15u;
      if (count < kTile) {  // a last tile: the rest by plain accesses, zeros past the end
        const int whole = count - count % E;
        T v = zero_of<T>();
        if (kSegmented) {
#pragma unroll
          for (int e = 0; e < E - 1; ++e) {
            const T y = shfl_idx(rest[e], static_cast<int>(i & 31));
            if (lane == e) v = y;
          }
        } else if (whole + lane < count) {
          v = in[base + whole + lane];
        }
        if (lane < E) buf(s)[whole + lane] = v;
        uint4 *chunks = reinterpret_cast<uint4 *>(buf(s));
        for (int c = whole / E + 1 + lane; c < kTile / E; c += 32) chunks[c] = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();  // before a later bulk copy into the same bytes
        __syncwarp();
      }
      if (lane == 0) {
        if (kSegmented) meta[s] = where;
        mbar_arrive_expect_tx(&sh.full[s], bytes);
        if (bytes) tma_load_1d(buf(s), in + base, bytes, &sh.full[s]);
      }
    }
    // The copies in flight land before the block's memory goes, also when the
    // last one is out and an abort sends every other role home: nobody else
    // waits for them then.  Not within the call's limit, which may have run out.
    for (int64_t j = max64(0, i - stages); j < i; ++j)
      mbar_wait_bounded(&sh.full[j % stages], static_cast<uint32_t>(j / stages) & 1u,
                        kDefaultWaitNs, fault);
  } else {
    // ---- prefix: warp q takes steps q, q + kPrefixWarps, ..., so the reads of
    // several waves overlap; the sum of the earlier waves passes from warp to
    // warp ----
    const int q = warp - (kScanWarps + kReduceWarps + 1);
    for (int64_t i = q; i < steps; i += kPrefixWarps) {
      const int64_t first = i * G;
      const int words = static_cast<int>(min64(G, num_tiles - first));
      constexpr int kPer = kMaxBlocks / 32;
      T v[kPer];
      uint32_t have = 0;  // bit j: word lane + 32 j has been read
      uint32_t heads = 0;  // kSegmented, bit j: it is a head's
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        v[j] = zero_of<T>();
        if (lane + 32 * j >= words) have |= 1u << j;
      }
      uint64_t t0 = 0;
      bool ok = true;
      while (true) {
#pragma unroll
        for (int j = 0; j < kPer; ++j)
          if (!((have >> j) & 1u)) {
            uint32_t f;
            st.read(first + lane + 32 * j, f, v[j]);
            if (f != kFlagNone) have |= 1u << j;
            if (kSegmented && f == kFlagHead) heads |= 1u << j;
          }
        if (__all_sync(0xffffffffu, have == (1u << kPer) - 1u)) break;
        if (t0 == 0) t0 = globaltimer_ns();
        const bool stop = globaltimer_ns() - t0 > timeout_ns || *s_abort || fault_raised(abort_flag);
        if (__any_sync(0xffffffffu, stop)) {
          if (lane == 0) {
            raise_fault(fault, EDPP_FAULT_TIMEOUT);
            atomicOr(abort_flag, 1u);
            *s_abort = 1;
          }
          ok = false;
          break;
        }
      }
      if (!ok) break;
      // kSegmented: sums start at the last head up to this tile (`from`) and of
      // the wave (`last`); without one (-1), the carry comes in too
      int from = -1, last = -1;
      if (kSegmented) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          const uint32_t m = __ballot_sync(0xffffffffu, (heads >> j) & 1u);
          const uint32_t mb = m & up_to(static_cast<int>(b) - 32 * j);
          if (m) last = 32 * j + 31 - __clz(m);
          if (mb) from = 32 * j + 31 - __clz(mb);
        }
      }
      T before = zero_of<T>(), total = zero_of<T>();
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int at = lane + 32 * j;
        if (at >= last) total = op_add(total, v[j]);
        if (at >= from && at < b) before = op_add(before, v[j]);
      }
      before = warp_sum(before);
      total = warp_sum(total);
      W sum = W(0);
      if (i > 0) {
        if (!wait(&sh.carried[q], static_cast<uint32_t>(q ? i / kPrefixWarps : i / kPrefixWarps - 1) & 1u))
          break;
        sum = carry[q];
      }
      if (lane == 0) {
        const int nq = q + 1 == kPrefixWarps ? 0 : q + 1;
        carry[nq] = op_add(last < 0 ? sum : W(0), W(total));
        mbar_arrive(&sh.carried[nq]);
        const int p = static_cast<int>(i % (2 * stages));
        pre[p] = static_cast<T>(op_add(from < 0 ? sum : W(0), W(before)));
        mbar_arrive(&sh.ready[p]);
      }
      __syncwarp();
    }
  }
}

// One cooperative launch over `tiles`, its state words zeroed by the caller.
template <typename T, bool kInclusive, typename Tiles>
int launch_pipe(const T *in, T *out, Tiles tiles, void *words, unsigned *abort_flag,
                cudaStream_t st, uint64_t timeout_ns, unsigned *fault) {
  constexpr int kSmem = kStages * kTileBytes;
  auto *kernel = scan_pipe_kernel<T, kInclusive, Tiles>;
  LookbackState<T> state;
  state.bind(words, tiles.num_tiles);
  const int64_t blocks = std::min<int64_t>({tiles.num_tiles, device_sm_count(), kMaxBlocks});
  void *args[] = {&in, &out, &tiles, &state, &abort_flag, &timeout_ns, &fault};
  if (cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel),
                                  dim3(static_cast<unsigned>(blocks)), dim3(kThreads), args, kSmem,
                                  st) != cudaSuccess) {
    cudaGetLastError();  // not co-resident: the caller takes another form
    return EDPP_ENOMEM;
  }
  return launch_status();
}

// Whether a block of the kernel fits an SM of this device (checked once).
template <typename T, bool kInclusive, typename Tiles> bool pipe_fits() {
  constexpr int kSmem = kStages * kTileBytes;
  static std::once_flag once[64];
  static bool fits[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  std::call_once(once[dev], [dev] {
    auto *kernel = scan_pipe_kernel<T, kInclusive, Tiles>;
    int per_sm = 0;
    fits[dev] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) ==
                    cudaSuccess &&
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, kSmem) ==
                    cudaSuccess &&
                per_sm > 0;
    if (!fits[dev]) cudaGetLastError();
  });
  return fits[dev];
}

}  // namespace

template <typename T> size_t scan_pipe_state_bytes(int64_t n) {
  const int64_t tile = kTileBytes / static_cast<int64_t>(sizeof(T));
  return LookbackState<T>::bytes((n + tile - 1) / tile);
}

template <typename T, bool kInclusive>
int scan_pipe(const T *in, T *out, int64_t n, char *header, cudaStream_t st, uint64_t timeout_ns,
              unsigned *fault, int64_t withheld) {
  if (!pipe_fits<T, kInclusive, ArrayTiles<T>>()) return EDPP_ENOMEM;
  constexpr int64_t kTile = kTileBytes / sizeof(T);
  const ArrayTiles<T> tiles{n, (n + kTile - 1) / kTile, withheld};
  if (cudaMemsetAsync(header, 0, kHeader + LookbackState<T>::bytes(tiles.num_tiles), st) !=
      cudaSuccess)
    return EDPP_ECUDA;
  return launch_pipe<T, kInclusive>(in, out, tiles, header + kHeader,
                                    reinterpret_cast<unsigned *>(header + 8), st, timeout_ns,
                                    fault);
}

int scan_pipe_tasks(const int32_t *in, int32_t *out, const DevSeg *segs, const DevTask *tasks,
                    int num_segs, int64_t num_tiles, void *words, unsigned *abort_flag,
                    cudaStream_t st, uint64_t timeout_ns, unsigned *fault) {
  if (!pipe_fits<int32_t, false, TaskTiles>()) return EDPP_ENOMEM;
  return launch_pipe<int32_t, false>(in, out, TaskTiles{segs, tasks, num_segs, num_tiles, fault},
                                     words, abort_flag, st, timeout_ns, fault);
}

#define EDPP_PIPE(T)                                                                             \
  template size_t scan_pipe_state_bytes<T>(int64_t);                                             \
  template int scan_pipe<T, false>(const T *, T *, int64_t, char *, cudaStream_t, uint64_t,      \
                                   unsigned *, int64_t);                                         \
  template int scan_pipe<T, true>(const T *, T *, int64_t, char *, cudaStream_t, uint64_t,       \
                                  unsigned *, int64_t);
EDPP_PIPE(int32_t)
EDPP_PIPE(int64_t)
EDPP_PIPE(float)
#undef EDPP_PIPE

}  // namespace edpp
