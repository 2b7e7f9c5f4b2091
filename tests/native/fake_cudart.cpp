// A CUDA runtime of host memory for tests of libk2j's host side (preloaded in front of the real one): allocations can be
// made to fail, kernels are noted and not run.  The functions are those libk2j.so imports.
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <string>
#include <vector>

namespace {
std::map<uintptr_t, size_t> g_device;             // "device" allocations
std::map<const void*, std::string> g_kernels;     // host stub -> name
std::vector<std::string> g_log;
size_t g_most = ~(size_t)0;                       // larger allocations fail
uint64_t g_pool_total = 0;                        // what the segmentation's first launch reports as the pool's size
uint64_t g_scan_total = 0;                        // what scans report as the (first) column's total, unless 0
std::vector<uint64_t> g_columns;                  // what the scan of the chunks' class counts reports, unless empty
cudaError_t g_last = cudaSuccess;                 // of a call that failed, until it is asked for
uintptr_t g_handle = 0x1000;
thread_local struct { dim3 grid, block; size_t smem; void* stream; } g_conf;

struct PoolJob { uint32_t blocks; uint64_t room; uint64_t* total; };  // as in k2j_kernels.cuh
void note(const char* what, const void* a, uint64_t b = 0) {
  char line[160];
  snprintf(line, sizeof line, "%s %llx %llu", what, (unsigned long long)(uintptr_t)a, (unsigned long long)b);
  g_log.push_back(line);
}
cudaError_t launched(const void* f, dim3 grid, dim3 block, void** args) {
  const std::string& name = g_kernels[f];
  g_log.push_back("launch " + name + " " + std::to_string(grid.x) + " " + std::to_string(block.x));
  if (name.find("k_scan_small") != std::string::npos || name.find("k_scan_apply") != std::string::npos) {
    uint64_t* totals = *static_cast<uint64_t**>(args[name.find("k_scan_small") != std::string::npos ? 2 : 6]);
    if (totals && grid.x == 13 && !g_columns.empty()) std::copy(g_columns.begin(), g_columns.end(), totals);
    else if (totals && g_scan_total) *totals = g_scan_total;
  }
  if (name.find("k_seg_chunks") != std::string::npos) {
    const PoolJob* job = static_cast<const PoolJob*>(args[1]);
    if (job->total) *job->total = g_pool_total;
    if (job->blocks) note("pool", nullptr, job->room);
  }
  return cudaSuccess;
}
bool on_device(const void* p) {
  auto it = g_device.upper_bound((uintptr_t)p);
  return it != g_device.begin() && (--it, (uintptr_t)p < it->first + it->second);
}
}  // namespace

extern "C" {
void fake_most(size_t bytes) { g_most = bytes; }
void fake_pool_total(uint64_t bytes) { g_pool_total = bytes; }
void fake_columns(const uint64_t* of, int n) { g_columns.assign(of, of + n); }
void fake_scan_total(uint64_t total) { g_scan_total = total; }
int fake_log(char* text, int room) {  // what was noted since the last call, a line each
  std::string all;
  for (const auto& l : g_log) all += l + "\n";
  g_log.clear();
  if ((int)all.size() >= room) return -1;
  memcpy(text, all.c_str(), all.size() + 1);
  return (int)all.size();
}

unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) { g_conf = {grid, block, smem, stream}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = g_conf.grid; *block = g_conf.block; *smem = g_conf.smem; *static_cast<void**>(stream) = g_conf.stream;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { g_kernels[stub] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

cudaError_t cudaMalloc(void** p, size_t n) {
  if (n > g_most) { *p = nullptr; return g_last = cudaErrorMemoryAllocation; }
  *p = calloc(1, n ? n : 1);
  g_device[(uintptr_t)*p] = n ? n : 1;
  note("alloc", *p, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) { g_device.erase((uintptr_t)p); free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); note("copy_and_wait", s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof *a);
  a->type = on_device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t, cudaStream_t) { return launched(f, grid, block, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) { return launched(f, c->gridDim, c->blockDim, args); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(g_handle += 16); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { note("wait", e, (uintptr_t)s); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)(g_handle += 16); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { note("record", e, (uintptr_t)s); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 132; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "out of memory"; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return cudaErrorInvalidSymbol; }
}
