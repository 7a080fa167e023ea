// A stand-in for the CUDA runtime on a machine without a GPU: device memory is
// host memory, a launch is written down instead of run, and a chosen
// allocation fails.  Linked with the library's objects it shows which kernels
// the host code launches, on which work lists, and what it does when memory
// runs out.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {

struct Launch {
  std::string name;
  dim3 grid, block;
  const int4* items = nullptr;  // ensemble kernels: their work list
};
std::map<const void*, std::string> names;   // host stub -> kernel
std::map<char*, size_t> blocks;             // live allocations
std::vector<std::vector<Launch>> graphs;    // captured launches
std::vector<Launch> captured;
bool capturing = false;
std::string text;
int fail_in = -1;  // the allocation that fails: 0 the next one
float elapsed = 1e6f;
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
void* cfg_stream;

bool live(const void* p, size_t n) {
  auto it = blocks.upper_bound((char*)p);
  if (it == blocks.begin()) return false;
  --it;
  return (const char*)p + n <= it->first + it->second;
}
void emit(const Launch& l) {
  char line[512];
  std::snprintf(line, sizeof(line), "%s %u %u %u x %u %u", l.name.c_str(), l.grid.x, l.grid.y, l.grid.z, l.block.x,
                l.block.y);
  text += line;
  if (l.items) {
    if (!live(l.items, sizeof(int4) * l.grid.x)) {
      text += " list gone";
    } else {
      unsigned long long h = 1469598103934665603ull;
      for (unsigned i = 0; i < l.grid.x; i++)
        for (int v : {l.items[i].x, l.items[i].y, l.items[i].z, l.items[i].w}) h = (h ^ (unsigned)v) * 1099511628211ull;
      std::snprintf(line, sizeof(line), " list %016llx", h);
      text += line;
    }
  }
  text += "\n";
}
cudaError_t launch(const void* f, dim3 grid, dim3 block, void** args) {
  Launch l;
  l.name = names[f];
  l.grid = grid;
  l.block = block;
  // ke_*(boxes, items, ..): the second argument is the work list, one entry a block
  if (l.name.find("ke_sweep") != std::string::npos) l.items = *(const int4**)args[1];
  if (capturing) captured.push_back(l);
  else emit(l);
  return cudaSuccess;
}
cudaError_t allocate(void** p, size_t n) {
  *p = nullptr;
  if (fail_in >= 0 && fail_in-- == 0) return cudaErrorMemoryAllocation;
  *p = std::calloc(1, n ? n : 1);
  blocks[(char*)*p] = n;
  return cudaSuccess;
}
cudaError_t release(void* p) {
  blocks.erase((char*)p);
  std::free(p);
  return cudaSuccess;
}

}  // namespace

extern "C" {

// for the tests
void fake_fail_in(int n) { fail_in = n; }
long long fake_live_bytes() {
  long long n = 0;
  for (auto& b : blocks) n += (long long)b.second;
  return n;
}
const char* fake_launches() {
  static std::string out;
  out.swap(text);
  text.clear();
  return out.c_str();
}

void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*,
                            int*) {
  names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) {
  cfg_grid = g;
  cfg_block = b;
  cfg_smem = smem;
  cfg_stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = cfg_grid;
  *b = cfg_block;
  *smem = cfg_smem;
  *(void**)s = cfg_stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void** args, size_t, cudaStream_t) {
  return launch((const void*)k, g, b, args);
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t, cudaStream_t) {
  return launch(f, g, b, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return launch(f, c->gridDim, c->blockDim, args);
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorInvalidSymbol; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
  return cudaErrorNotSupported;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)1;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = true;
  captured.clear();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capturing = false;
  graphs.push_back(captured);
  *g = (cudaGraph_t)graphs.size();
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  *x = (cudaGraphExec_t)g;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  for (const Launch& l : graphs[(size_t)x - 1]) emit(l);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)1;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)1;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
// every measurement is the best so far
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  elapsed *= 0.99f;
  *ms = elapsed;
  return cudaSuccess;
}

}  // extern "C"
