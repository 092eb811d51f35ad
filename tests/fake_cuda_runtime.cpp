// A CUDA runtime without a device, for tests of the host side: linked in front of the library's objects (every call
// named here is wrapped), it answers the queries a launch depends on, keeps a record of the launches and runs nothing.
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>

namespace {

constexpr int kGpcs = 8;
const int kGpcSms[kGpcs] = {20, 20, 20, 19, 18, 18, 18, 15};   // 148 SMs; a cluster lives in one GPC

struct Launch {
  const void *kernel;
  unsigned grid, block, cluster, smem;
};
Launch g_launches[256];
int g_count = 0, g_occupancy_calls = 0, g_occupancy_failures = 0, g_refuse_2d_maps = 0, g_memsets = 0;

void record(const void *kernel, dim3 grid, dim3 block, unsigned cluster, size_t smem) {
  if (g_count < 256) g_launches[g_count++] = Launch{kernel, grid.x * grid.y * grid.z, block.x, cluster, static_cast<unsigned>(smem)};
}

unsigned cluster_of(const cudaLaunchConfig_t *cfg) {
  for (unsigned i = 0; i < cfg->numAttrs; ++i)
    if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension) return cfg->attrs[i].val.clusterDim.x;
  return 1;
}

CUresult encode(CUtensorMap *map, CUtensorMapDataType, cuuint32_t rank, void *, const cuuint64_t *, const cuuint64_t *,
                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                CUtensorMapFloatOOBfill) {
  memset(map, 0, sizeof(*map));
  return g_refuse_2d_maps && rank == 2 ? CUDA_ERROR_INVALID_VALUE : CUDA_SUCCESS;
}

}  // namespace

extern "C" {

int fake_launch_count() { return g_count; }
const Launch *fake_launch(int i) { return &g_launches[i]; }
int fake_memsets() { return g_memsets; }
int fake_occupancy_calls() { return g_occupancy_calls; }
void fake_reset() { g_count = g_occupancy_calls = g_memsets = 0; }
void fake_fail_occupancy(int calls) { g_occupancy_failures = calls; }      // the next queries fail
void fake_refuse_2d_maps(int on) { g_refuse_2d_maps = on; }
int fake_clusters(int size) {
  int fit = 0;
  for (int sms : kGpcSms) fit += sms / size;
  return fit;
}

cudaError_t __wrap_cudaGetDevice(int *dev) { *dev = 0; return cudaSuccess; }
cudaError_t __wrap_cudaDeviceGetAttribute(int *v, cudaDeviceAttr attr, int) {
  *v = attr == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t __wrap_cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t __wrap_cudaGetLastError() { return cudaSuccess; }
cudaError_t __wrap_cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long, cudaDriverEntryPointQueryResult *q) {
  *fn = reinterpret_cast<void *>(&encode);
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t __wrap_cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *cfg) {
  ++g_occupancy_calls;
  if (g_occupancy_failures > 0) {
    --g_occupancy_failures;
    return cudaErrorUnknown;
  }
  *n = fake_clusters(static_cast<int>(cluster_of(cfg)));
  return cudaSuccess;
}
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *kernel, void **) {
  record(kernel, cfg->gridDim, cfg->blockDim, cluster_of(cfg), cfg->dynamicSmemBytes);
  return cudaSuccess;
}
cudaError_t __wrap_cudaLaunchKernel(const void *kernel, dim3 grid, dim3 block, void **, size_t smem, cudaStream_t) {
  record(kernel, grid, block, 1, smem);
  return cudaSuccess;
}
cudaError_t __wrap_cudaMemsetAsync(void *, int, size_t, cudaStream_t) { ++g_memsets; return cudaSuccess; }

}  // extern "C"
