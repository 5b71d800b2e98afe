// gather_scatter.h — the tiled gather (gather_tiled.cu), for the C entry
// points in gather_scatter_part.cu.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace edpp {

// Workspace of gather_tiled for `n` > 0 elements.
size_t gather_tiled_bytes(int64_t n);

// out[i] = in[loc[i]] for 0 < n <= INT32_MAX; indices outside [0, n) skipped.
int gather_tiled(const int32_t *in, int32_t *out, int64_t n, const int32_t *loc, void *ws,
                 size_t ws_bytes, cudaStream_t st);

}  // namespace edpp
