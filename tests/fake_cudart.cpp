// A CUDA runtime without a device: every call succeeds and launches nothing, memory is the
// caller's, except that a launch is refused when its kernel's name contains the string given to
// fake_refuse() or when its dynamic shared memory is above the kernel's ceiling.  Linked with the
// library's own objects, it lets a test see what the host code does with a refused launch and what
// it asks of the runtime.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
struct Kernel {
  std::string name;
  size_t ceiling = 48 << 10, lowest = 1 << 30, largest = 0;  // lowest: of the ceilings that were set
  int launches = 0, cluster = 0, blocks = 0, early = 0;  // the last launch: cluster and grid along x, dependent
};
std::map<const void*, Kernel>& kernels() {
  static auto* k = new std::map<const void*, Kernel>();
  return *k;
}
std::string refuse;
int most = 8;  // CTAs a cluster
cudaError_t last = cudaSuccess;
struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} pushed;
cudaError_t fail(cudaError_t e) { return last = e; }
cudaError_t launched(const void* fn, size_t smem, dim3 grid) {
  Kernel& k = kernels()[fn];
  k.blocks = (int)grid.x;
  ++k.launches;
  if (smem > k.largest) k.largest = smem;
  if (smem > k.ceiling) return fail(cudaErrorInvalidValue);
  if (!refuse.empty() && k.name.find(refuse) != std::string::npos) return fail(cudaErrorLaunchOutOfResources);
  return cudaSuccess;
}
const Kernel* find(const char* part, const Kernel* after) {
  bool on = after == nullptr;
  for (auto& e : kernels()) {
    if (on && e.second.launches && e.second.name.find(part) != std::string::npos) return &e.second;
    if (&e.second == after) on = true;
  }
  return nullptr;
}
}  // namespace

extern "C" {
// ---- the test's side: of the launched kernels whose (mangled) name contains `part`
void fake_refuse(const char* part) { refuse = part; }
void fake_most(int ctas) { most = ctas; }
int fake_launches(const char* part) {
  int n = 0;
  for (const Kernel* k = nullptr; (k = find(part, k));) n += k->launches;
  return n;
}
size_t fake_largest_smem(const char* part) {
  size_t n = 0;
  for (const Kernel* k = nullptr; (k = find(part, k));) n = k->largest > n ? k->largest : n;
  return n;
}
size_t fake_lowest_ceiling(const char* part) {
  size_t n = 1 << 30;
  for (const Kernel* k = nullptr; (k = find(part, k));) n = k->lowest < n ? k->lowest : n;
  return n;
}
int fake_cluster(const char* part) {
  const Kernel* k = find(part, nullptr);
  return k ? k->cluster : 0;
}
int fake_early(const char* part) {
  const Kernel* k = find(part, nullptr);
  return k ? k->early : -1;
}
int fake_blocks(const char* part) {
  const Kernel* k = find(part, nullptr);
  return k ? k->blocks : 0;
}
void fake_forget() {
  for (auto& e : kernels()) e.second.launches = 0, e.second.largest = 0;
}

// ---- the runtime's side
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  kernels()[host].name = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* stream) {
  pushed = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *static_cast<cudaStream_t*>(stream) = pushed.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 grid, dim3, void**, size_t smem, cudaStream_t) {
  return launched(fn, smem, grid);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
  Kernel& k = kernels()[fn];
  for (unsigned i = 0; i < c->numAttrs; ++i) {
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) k.cluster = (int)c->attrs[i].val.clusterDim.x;
    if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) k.early = 1;
  }
  return launched(fn, c->dynamicSmemBytes, c->gridDim);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused by the test"; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  memset(a, 0, sizeof(*a));
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute at, int v) {
  if (at != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  Kernel& k = kernels()[fn];
  k.ceiling = (size_t)v;
  if (k.ceiling < k.lowest) k.lowest = k.ceiling;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
  const int cl = (int)c->attrs[0].val.clusterDim.x;
  if (cl > most) return fail(cudaErrorInvalidClusterSize);
  return *n = 120 / cl, cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 227 << 10, cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { return *lo = *hi = 0, cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = nullptr, cudaErrorInvalidSymbol; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return memmove(d, s, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemset2DAsync(void* d, size_t pitch, int v, size_t w, size_t h, cudaStream_t) {
  for (size_t r = 0; r < h; ++r) memset(static_cast<char*>(d) + r * pitch, v, w);
  return cudaSuccess;
}
}
