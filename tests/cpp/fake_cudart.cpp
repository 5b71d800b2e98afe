// fake_cudart.cpp — stands in for the CUDA runtime under the library's host code,
// so that a machine without a GPU can see which kernels a call launches.
//
// Linked with the library's objects into a library of its own.  Launches are
// recorded by kernel name, grid and kind; copies, memsets and queries succeed
// without touching anything; a launch of a refused kind fails as the runtime
// would fail it.  The device: 152 SMs, 129 MB of L2, two blocks of any kernel
// per SM unless fake_blocks_per_sm() says otherwise.
#include <cuda_runtime_api.h>

#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void *, std::string> &kernels() {
  static std::map<const void *, std::string> m;
  return m;
}
std::string g_log;
int g_refuse = 0;  // FakeKind bits
int g_blocks_per_sm = 2;
cudaError_t g_last = cudaSuccess;
dim3 g_grid, g_block;
size_t g_smem;
cudaStream_t g_stream;
alignas(256) unsigned char g_symbol[1 << 20];

enum FakeKind { kCluster = 1, kCooperative = 2, kProgrammatic = 4 };

cudaError_t launch(const void *fn, dim3 grid, int kind) {
  if (kind & g_refuse) return g_last = cudaErrorCooperativeLaunchTooLarge;
  g_log += kernels()[fn] + " " + std::to_string(grid.x) + " " + std::to_string(kind) + "\n";
  return cudaSuccess;
}
}  // namespace

extern "C" {

const char *fake_log() { return g_log.c_str(); }
void fake_reset(int refuse, int blocks_per_sm) {
  g_log.clear();
  g_refuse = refuse;
  g_blocks_per_sm = blocks_per_sm;
  g_last = cudaSuccess;
}

void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *fn, char *, const char *name, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {
  kernels()[fn] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  g_grid = grid, g_block = block, g_smem = smem, g_stream = stream;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
  *grid = g_grid, *block = g_block, *smem = g_smem;
  *static_cast<cudaStream_t *>(stream) = g_stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *kernel, const void *fn) {
  *kernel = reinterpret_cast<cudaKernel_t>(const_cast<void *>(fn));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3 grid, dim3, void **, size_t, cudaStream_t) {
  return launch(kernel, grid, 0);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *fn, void **) {
  int kind = 0;
  for (unsigned i = 0; i < cfg->numAttrs; ++i) {
    if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension) kind |= kCluster;
    if (cfg->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      kind |= kProgrammatic;
  }
  return launch(fn, cfg->gridDim, kind);
}
cudaError_t cudaLaunchCooperativeKernel(const void *fn, dim3 grid, dim3, void **, size_t,
                                        cudaStream_t) {
  return launch(fn, grid, kCooperative);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaGetDevice(int *dev) {
  *dev = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *value, cudaDeviceAttr attr, int) {
  *value = attr == cudaDevAttrMultiProcessorCount ? 152 : attr == cudaDevAttrL2CacheSize ? 129 << 20
                                                                                         : 0;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  *p = g_symbol;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *blocks, const void *, int,
                                                                   size_t, unsigned) {
  *blocks = g_blocks_per_sm;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1;
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t, cudaStream_t) {
  *p = g_symbol;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void *dst, const void *, size_t n, size_t, cudaMemcpyKind) {
  std::memset(dst, 0, n);
  return cudaSuccess;
}

// Never called by what is tested here.
#define UNUSED(name, ...) \
  cudaError_t name(__VA_ARGS__) { return cudaErrorNotSupported; }
UNUSED(cudaDeviceSynchronize)
UNUSED(cudaFree, void *)
UNUSED(cudaFreeHost, void *)
UNUSED(cudaLaunchHostFunc, cudaStream_t, cudaHostFn_t, void *)
UNUSED(cudaMalloc, void **, size_t)
UNUSED(cudaMallocHost, void **, size_t)
UNUSED(cudaMemcpyToSymbol, const void *, const void *, size_t, size_t, cudaMemcpyKind)
UNUSED(cudaSetDevice, int)
UNUSED(cudaStreamCreateWithFlags, cudaStream_t *, unsigned)
UNUSED(cudaStreamDestroy, cudaStream_t)

}  // extern "C"
