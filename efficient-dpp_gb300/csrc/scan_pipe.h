// scan_pipe.h — the pipelined one-launch scan (scan_pipe.cu), for scan.cu.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace edpp {

// Workspace after `header` bytes that scan_pipe zeroes and uses: one 8-byte
// word (two for 8-byte types) per 16 KB tile.
template <typename T> size_t scan_pipe_state_bytes(int64_t n);

// Scan of n > 0 elements; in and out 16-byte aligned, in == out allowed.
// `header`: 256 bytes of the workspace, zeroed here with the state after it;
// the abort flag is at header + 8.  EDPP_ENOMEM (nothing launched) when the
// grid cannot be resident together on this device.  `withheld`: a tile whose sum
// is not published, so that the waits for it run out (self-test).
template <typename T, bool kInclusive>
int scan_pipe(const T *in, T *out, int64_t n, char *header, cudaStream_t st, uint64_t timeout_ns,
              unsigned *fault, int64_t withheld = -1);

struct DevSeg;
struct DevTask;

// Exclusive scan of every segment of a batch (batch_plan.h): `tasks` are the
// scan tiles, each segment's in order from tile 0.  Segment offsets multiples of
// 4 elements, in and out 16-byte aligned.  `words`: num_tiles zeroed 8-byte
// words.  EDPP_ENOMEM as above.
int scan_pipe_tasks(const int32_t *in, int32_t *out, const DevSeg *segs, const DevTask *tasks,
                    int num_segs, int64_t num_tiles, void *words, unsigned *abort_flag,
                    cudaStream_t st, uint64_t timeout_ns, unsigned *fault);

}  // namespace edpp
