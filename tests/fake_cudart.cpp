// A CUDA runtime without a GPU, for tests of the library's host paths: preloaded into a child process it answers the
// runtime calls that the library makes.  Device memory is host memory, copies and memsets take place at once, kernels
// are noted down and (but for the one that finds the largest degree) not run.  Allocations fail on request, and fake_log() tells what was called, one call a line:
//   malloc <bytes> <ok|fail>    free    host_malloc <ok|fail>    device_sync    launch <stream> <kernel>
//   record <event> <stream>     wait <stream> <event>            sync <stream>  memset <stream>    copy <stream>
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>

namespace {
std::recursive_mutex mu;
std::string log_text;
std::map<const void*, std::string> kernels;
std::unordered_map<void*, size_t> device_blocks;
std::map<uintptr_t, size_t> host_blocks;
bool pinned_seen = false;  // whether pinned host memory is reported as such
cudaError_t last_error = cudaSuccess;
long malloc_good = -1, malloc_bad = 0, host_good = -1, host_bad = 0;  // so many succeed, then so many fail
unsigned long long packed_total = 0;
size_t device_total = (size_t)64 << 30, device_used = 0;
bool capturing = false;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local Config config;

void note(const std::string& line) { log_text += line + "\n"; }
std::string hex(const void* p) {
  char b[32];
  snprintf(b, sizeof b, "%p", p);
  return p ? b : "0";
}
bool fails(long& good, long& bad) {
  if (good < 0 || bad <= 0) return false;
  if (good > 0) {
    --good;
    return false;
  }
  --bad;
  return true;
}
cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) last_error = e;
  return e;
}
}  // namespace

extern "C" {

void fake_fail_malloc(long after, long times) {
  malloc_good = after;
  malloc_bad = times;
}
void fake_fail_host_malloc(long after, long times) {
  host_good = after;
  host_bad = times;
}
void fake_memory(size_t total) { device_total = total; }
void fake_packed(unsigned long long cells) { packed_total = cells; }
void fake_register(void* p, size_t bytes) { host_blocks[reinterpret_cast<uintptr_t>(p)] = bytes; }
void fake_pinned(int on) { pinned_seen = on != 0; }
void fake_capture(int on) { capturing = on != 0; }
size_t fake_used() { return device_used; }
void fake_clear_log() { log_text.clear(); }
const char* fake_log() { return log_text.c_str(); }

void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  config = Config{grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *static_cast<cudaStream_t*>(stream) = config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("launch " + hex(s) + " " + kernels[f]);
  if (kernels[f].find("max_degree_kernel") != std::string::npos) {  // the one whose result decides on host paths
    const unsigned* xadj = *static_cast<const unsigned**>(args[0]);
    const unsigned V = *static_cast<unsigned*>(args[1]);
    unsigned* out = *static_cast<unsigned**>(args[2]);
    unsigned* longs = *static_cast<unsigned**>(args[3]);
    for (unsigned v = 0; v < V; ++v) {
      const unsigned d = xadj[v + 1] - xadj[v];
      *out = d > *out ? d : *out;
      out[1] += d == 0;
      *longs += d > 16384 && d <= 65536;
    }
    const unsigned* adjncy = *static_cast<const unsigned**>(args[4]);
    const unsigned long long E = *static_cast<unsigned long long*>(args[5]);
    unsigned* ends = *static_cast<unsigned**>(args[6]);
    for (unsigned i = 0; i < 4096 && E; ++i) *ends += xadj[adjncy[i * E / 4096]] == xadj[adjncy[i * E / 4096] + 1];
  }
  // the number of cells that the packing kernels report, if a test wants some
  if (packed_total && kernels[f].find("pack_rows_kernel") != std::string::npos) **static_cast<unsigned long long**>(args[7]) = packed_total;
  if (packed_total && kernels[f].find("pack_heads_kernel") != std::string::npos) **static_cast<unsigned long long**>(args[8]) = packed_total;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
  std::lock_guard<std::recursive_mutex> l(mu);
  const bool no = fails(malloc_good, malloc_bad) || device_used + bytes > device_total;
  note("malloc " + std::to_string(bytes) + (no ? " fail" : " ok"));
  if (no) return set(cudaErrorMemoryAllocation);
  *p = calloc(1, bytes ? bytes : 1);
  device_blocks[*p] = bytes;
  device_used += bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::recursive_mutex> l(mu);
  if (!p) return cudaSuccess;
  note("free");
  const auto it = device_blocks.find(p);
  if (it == device_blocks.end()) return set(cudaErrorInvalidValue);
  device_used -= it->second;
  device_blocks.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) {
  std::lock_guard<std::recursive_mutex> l(mu);
  const bool no = fails(host_good, host_bad);
  note(std::string("host_malloc ") + (no ? "fail" : "ok"));
  if (no) return set(cudaErrorMemoryAllocation);
  *p = calloc(1, bytes ? bytes : 1);
  host_blocks[reinterpret_cast<uintptr_t>(*p)] = bytes;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { return cudaMallocHost(p, bytes); }
cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("host_free");
  host_blocks.erase(reinterpret_cast<uintptr_t>(p));
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* unused, size_t* total) {
  *unused = device_total - device_used;
  *total = device_total;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("copy " + hex(st));
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("memset " + hex(st));
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof *a);
  const bool device = device_blocks.count(const_cast<void*>(p)) != 0;
  a->type = device ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  auto it = host_blocks.upper_bound(reinterpret_cast<uintptr_t>(p));
  if (pinned_seen && it != host_blocks.begin() && reinterpret_cast<uintptr_t>(p) < (--it)->first + it->second) {
    a->type = cudaMemoryTypeHost;
    a->devicePointer = a->hostPointer = const_cast<void*>(p);
  }
  return cudaSuccess;
}

static CUresult pointer_attribute(void* out, CUpointer_attribute what, CUdeviceptr p) {
  auto it = host_blocks.upper_bound(p);
  if (it == host_blocks.begin() || p >= (--it)->first + it->second) return CUDA_ERROR_INVALID_VALUE;
  if (what == CU_POINTER_ATTRIBUTE_RANGE_START_ADDR) *static_cast<CUdeviceptr*>(out) = it->first;
  else if (what == CU_POINTER_ATTRIBUTE_RANGE_SIZE) *static_cast<size_t*>(out) = it->second;
  else return CUDA_ERROR_INVALID_VALUE;
  return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* found) {
  const bool have = std::string(name) == "cuPointerGetAttribute";
  *f = have ? reinterpret_cast<void*>(&pointer_attribute) : nullptr;
  if (found) *found = have ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrComputeCapabilityMinor ? 0 : 65535;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("device_sync");
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last_error; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  memset(a, 0, sizeof *a);
  a->ptxVersion = a->binaryVersion = 100;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static char room[1 << 22];
  *p = room;
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(calloc(1, 8));
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("sync " + hex(s));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("wait " + hex(s) + " " + hex(e));
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* st) {
  *st = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(calloc(1, 8));
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> l(mu);
  note("record " + hex(e) + " " + hex(s));
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}

}  // extern "C"
