// fake_cudart.cpp -- a CUDA runtime without a GPU for tests of the library's
// host code: the library's own objects are linked against it.  Device memory
// is accounted for, not backed (fake_reset sets its size); kernels and copies
// to the device do nothing; copies to the host give zeros.  Every launch,
// allocation, copy, synchronisation and event goes to a log that a test reads,
// a launch can be made to fail, and a stream can be declared to be captured:
// what CUDA refuses during a capture is then refused and logged.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {

std::map<const void*, std::string> kernels;     // host stub -> device name
std::map<char*, size_t> blocks;
size_t capacity = 0, used = 0;
char* next_address = reinterpret_cast<char*>(size_t(1) << 40);
std::string log_text, fail_name;
int fail_after = -1, next_handle = 0;
cudaStream_t captured = nullptr;
cudaError_t last = cudaSuccess;

void note(const char* what, const void* a = nullptr, const void* b = nullptr) {
  char line[512];
  std::snprintf(line, sizeof line, "%s %zu %zu\n", what, (size_t)a, (size_t)b);
  log_text += line;
}
cudaError_t result(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
void* handle() { return reinterpret_cast<void*>((size_t)++next_handle); }

bool refused(const char* what) {
  if (!captured) return false;
  note((std::string("refused ") + what).c_str());
  return true;
}

cudaError_t allocate(void** p, size_t bytes, const char* what) {
  *p = nullptr;
  if (used + bytes > capacity) {
    note((std::string(what) + " fails").c_str(), (void*)bytes);
    return result(cudaErrorMemoryAllocation);
  }
  *p = next_address;
  next_address += (bytes + 511) / 256 * 256;
  blocks[(char*)*p] = bytes;
  used += bytes;
  note(what, (void*)bytes);
  return cudaSuccess;
}
void give_back(void* p) {
  auto it = blocks.find((char*)p);
  if (it == blocks.end()) {
    if (p) note("bad free", p);
    return;
  }
  used -= it->second;
  blocks.erase(it);
}

cudaError_t launch(const void* f, dim3 g, cudaStream_t st) {
  const std::string& name = kernels[f];
  if (!fail_name.empty() && name.find(fail_name) != std::string::npos && fail_after-- == 0) {
    note(("launch fails " + name).c_str(), st);
    return result(cudaErrorLaunchOutOfResources);
  }
  note(("launch " + name).c_str(), st, (void*)((size_t)g.x * g.y * g.z));
  return cudaSuccess;
}

CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}

struct Config {
  dim3 grid, block;
  size_t smem;
  void* stream;
} config;

}  // namespace

extern "C" {

// ------------------------------------------------------------- for tests --
void fake_reset(size_t bytes) {
  capacity = bytes;
  log_text.clear();
  fail_name.clear();
  fail_after = -1;
  captured = nullptr;
  last = cudaSuccess;
}
size_t fake_used() { return used; }
void fake_capture(void* stream) { captured = static_cast<cudaStream_t>(stream); }
void fake_fail(const char* name, int after) {
  fail_name = name;
  fail_after = after;
}
size_t fake_log(char* out, size_t n) {
  if (out && n > log_text.size()) {
    std::memcpy(out, log_text.c_str(), log_text.size() + 1);
    log_text.clear();
  }
  return log_text.size();
}

// --------------------------------------------------------- registration --
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(&config); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
  config = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = config.grid;
  *b = config.block;
  *smem = config.smem;
  *static_cast<void**>(st) = config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void**, size_t, cudaStream_t st) {
  return launch(k, g, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->stream);
}

// --------------------------------------------------------------- device --
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->multiProcessorCount = 152;
  p->major = 10;
  p->minor = 3;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  if (refused("cudaDeviceSynchronize")) return result(cudaErrorStreamCaptureUnsupported);
  note("sync");
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) { *a = 0; *b = -1; return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory" : "error of the fake runtime";
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = 40;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t,
                                                                   unsigned) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *f = reinterpret_cast<void*>(encode);
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

// --------------------------------------------------------------- memory --
cudaError_t cudaMalloc(void** p, size_t n) {
  if (refused("cudaMalloc")) return result(cudaErrorStreamCaptureUnsupported);
  return allocate(p, n, "malloc");
}
cudaError_t cudaFree(void* p) {
  if (refused("cudaFree")) return result(cudaErrorStreamCaptureUnsupported);
  note("free", p);
  give_back(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return allocate(p, n, "mallocasync"); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t st) {
  note("freeasync", st, p);
  give_back(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  note("memgetinfo");
  *f = capacity > used ? capacity - used : 0;
  *t = capacity;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  note("hostalloc", (void*)n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* dst, const void*, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  if (k == cudaMemcpyDeviceToHost) std::memset(dst, 0, n);
  note("copy", (void*)n, st);
  return cudaSuccess;
}
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return allocate(p, 64 << 20, "symbol"); }

// ---------------------------------------------------- streams and events --
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = static_cast<cudaStream_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) {
  *s = static_cast<cudaStream_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  if (refused("cudaStreamSynchronize")) return result(cudaErrorStreamCaptureUnsupported);
  note("streamsync", st);
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus* s) {
  *s = captured && st == captured ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t st, cudaStreamCaptureMode) {
  captured = st;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  captured = nullptr;
  *g = static_cast<cudaGraph_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = static_cast<cudaGraphExec_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
  note("graph", st);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
  note("wait", st, e);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = static_cast<cudaEvent_t>(handle());
  note("eventcreate", *e);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = static_cast<cudaEvent_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  note("record", e, st);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}

}  // extern "C"
