// A stand-in for the CUDA runtime that runs nothing: it notes which kernels the library launches, in which
// order, and which of them may begin before the launch ahead of them has completed.  "Device" memory is
// host memory.  Linked with the library's objects by test_launch_order.py.
#include <string.h>

#include <map>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

namespace {
struct Launch {
  std::string kernel;
  bool early;
  unsigned cluster, grid;
};
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> m;
  return m;
}
std::vector<Launch> launches;
int device = 0;
struct { dim3 grid, block; size_t smem; void* stream; } pushed;
}  // namespace

extern "C" {
void recorder_reset() { launches.clear(); }
int recorder_count() { return (int)launches.size(); }
const char* recorder_kernel(int i) { return launches[i].kernel.c_str(); }
int recorder_early(int i) { return launches[i].early; }
int recorder_grid(int i) { return (int)launches[i].grid; }
void recorder_device(int d) { device = d; }   // 0: 148 SMs, 1: 60
int recorder_cluster(int i) { return (int)launches[i].cluster; }

void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
  pushed = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *static_cast<void**>(stream) = pushed.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void**, size_t, cudaStream_t) {
  launches.push_back({names()[f], false, 1, grid.x});
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  Launch l{names()[f], false, 1, c->gridDim.x};
  for (unsigned i = 0; i < c->numAttrs; i++) {
    if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      l.early = c->attrs[i].val.programmaticStreamSerializationAllowed != 0;
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) l.cluster = c->attrs[i].val.clusterDim.x;
  }
  launches.push_back(l);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(dst, src, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* dst, const void*, size_t n, size_t, cudaMemcpyKind) {
  memset(dst, 0, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = nullptr, cudaErrorInvalidSymbol; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "none"; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { *v = d == 0 ? 148 : 60; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
}
