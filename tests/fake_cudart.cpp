// A CUDA runtime that runs nothing: it notes what a library asks of it, one line each, so that host code can be tested without a
// GPU. Two devices of 148 multiprocessors; kernels are known by the names they register.
#include <stddef.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <map>
#include <string>

#include <driver_types.h>
#include <vector_types.h>

namespace {
std::map<const void *, std::string> names;
std::map<std::pair<int, const void *>, int> limits;  // dynamic shared memory that a kernel may ask for, per device
int device = 0;
cudaError_t last = cudaSuccess;
std::string notes;
int watched = -1;  // an int argument of every kernel that is launched goes into the notes

const char *name(const void *f) { return names.count(f) ? names[f].c_str() : "?"; }
int limit(const void *f) { return limits.count({device, f}) ? limits[{device, f}] : 48 * 1024; }
void note(const char *what, const void *f, dim3 grid, dim3 block, size_t smem, int cluster) {
  char line[640];
  snprintf(line, sizeof line, "%s %d %s %u %u %u %u %zu %d\n", what, device, name(f), grid.x, grid.y, grid.z, block.x, smem, cluster);
  notes += line;
}
int blocks_of_cluster(const cudaLaunchAttribute *a, unsigned n) {
  for (unsigned i = 0; i < n; ++i)
    if (a[i].id == cudaLaunchAttributeClusterDimension) return (int)(a[i].val.clusterDim.x * a[i].val.clusterDim.y * a[i].val.clusterDim.z);
  return 1;
}
cudaError_t fail(cudaError_t e) { return last = e; }
}  // namespace

extern "C" {
void fake_set_device(int d) { device = d; }
const char *fake_notes() { return notes.c_str(); }
void fake_clear() { notes.clear(); }
void fake_watch(int argument) { watched = argument; }

void **__cudaRegisterFatBinary(void *) { static void *handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *kernel, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
  names[host] = kernel;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }

cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "refused by the test"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v > 227 * 1024) return fail(cudaErrorInvalidValue);
    limits[{device, f}] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  if ((int)c->dynamicSmemBytes > limit(f)) return fail(cudaErrorInvalidValue);  // as the runtime does
  note("launch", f, c->gridDim, c->blockDim, c->dynamicSmemBytes, blocks_of_cluster(c->attrs, c->numAttrs));
  if (watched >= 0) notes.insert(notes.size() - 1, " " + std::to_string(*static_cast<int *>(args[watched])));
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3 block, void **, size_t smem, cudaStream_t) {
  if ((int)smem > limit(f)) return fail(cudaErrorInvalidValue);
  note("launch", f, grid, block, smem, 1);
  return cudaSuccess;
}
// clusters that are resident: by shared memory and 2048 threads, clusters inside groups of 16 multiprocessors
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c) {
  if ((int)c->dynamicSmemBytes > limit(f)) return fail(cudaErrorInvalidValue);
  const int size = blocks_of_cluster(c->attrs, c->numAttrs);
  int per = (int)(2048 / c->blockDim.x);
  const int room = (int)(228 * 1024 / (c->dynamicSmemBytes + 1376));  // (measured: 115344 bytes fit twice, 115648 do not)
  if (room < per) per = room;
  *n = 9 * (16 * per / size) + 4 * per / size;
  note("occupancy", f, c->gridDim, c->blockDim, c->dynamicSmemBytes, size);
  return cudaSuccess;
}

cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int threads, size_t, unsigned) {
  *n = 1280 / threads;
  return cudaSuccess;
}

cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t) { *p = nullptr; return fail(cudaErrorMemoryAllocation); }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) { return fail(cudaErrorNotSupported); }
cudaError_t cudaMemcpyFromSymbol(void *, const void *, size_t, size_t, cudaMemcpyKind) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return fail(cudaErrorNotSupported); }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaIpcCloseMemHandle(void *) { return fail(cudaErrorNotSupported); }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t *, void *) { return fail(cudaErrorNotSupported); }
cudaError_t cudaIpcOpenMemHandle(void **, cudaIpcMemHandle_t, unsigned) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **p, unsigned, unsigned long long, cudaDriverEntryPointQueryResult *) {
  *p = nullptr;
  return fail(cudaErrorNotSupported);
}
}
