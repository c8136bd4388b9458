// fake_cuda.cpp -- a recording stand-in for the CUDA runtime: device memory is host memory, kernels do not
// run, copies and memsets happen at once, and every operation that a stream would order is printed as one
// line. Linked with the library's host code instead of libcudart (host_log.cu), so that the order, streams,
// launch attributes and graphs of the API's calls can be checked without a GPU.
//
// TEST INFRASTRUCTURE ONLY.
#include <cuda_runtime_api.h>
#include <cxxabi.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

// the launch arguments worth printing (host_log.cu knows the kernels' parameters)
extern "C" std::string* fake_describe(const char* name, unsigned gridY, void** args);
// the next 4-byte copy to the host reads this value instead, if not 0
extern "C" {
unsigned fake_next_word = 0;
}

namespace {
std::map<const void*, std::string>& kernels() {
  static std::map<const void*, std::string> m;
  return m;
}
std::map<cudaStream_t, int> g_streams{{nullptr, 0}};
int g_nextStream = 1, g_nextGraph = 1;
struct Graph {
  int id;
  std::vector<std::string> ops;
};
Graph* g_capture = nullptr;         // one capture at a time
cudaStream_t g_captureOrigin = nullptr;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_config;

void op(const std::string& s) {
  if (g_capture) {
    g_capture->ops.push_back(s);
  } else {
    std::printf("%s\n", s.c_str());
  }
}
std::string on(cudaStream_t s) {
  auto it = g_streams.find(s);
  return " stream=" + std::to_string(it == g_streams.end() ? -1 : it->second);
}
cudaError_t launched(const void* f, unsigned gridY, void** args, cudaStream_t s, bool pdl) {
  const std::string& name = kernels()[f];
  std::string* d = fake_describe(name.c_str(), gridY, args);
  op("launch " + name.substr(0, name.find('(')) + on(s) + (pdl ? " pdl=1" : " pdl=0") + *d);
  delete d;
  return cudaSuccess;
}
}  // namespace

extern "C" {
// what the compiler's host stubs call
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  int st = 0;
  char* d = abi::__cxa_demangle(name, nullptr, nullptr, &st);
  std::string s = st == 0 ? d : name;
  std::free(d);
  if (s.rfind("void ", 0) == 0) { s = s.substr(5); }
  for (size_t i; (i = s.find("owl::")) != std::string::npos;) { s.erase(i, 5); }
  for (size_t i; (i = s.find(", ")) != std::string::npos;) { s.erase(i + 1, 1); }
  kernels()[host] = s;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  g_config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = g_config.grid;
  *block = g_config.block;
  *smem = g_config.smem;
  *static_cast<cudaStream_t*>(stream) = g_config.stream;
  return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void** args, size_t, cudaStream_t s) {
  return launched(f, grid.y, args, s, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  bool pdl = false;
  for (unsigned i = 0; i < c->numAttrs; ++i) {
    if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) {
      pdl = c->attrs[i].val.programmaticStreamSerializationAllowed != 0;
    }
  }
  return launched(f, c->gridDim.y, args, c->stream, pdl);
}

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  std::memcpy(d, s, n);
  op("copy" + on(st));
  (void)k;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  std::memcpy(d, s, n);
  if (k == cudaMemcpyDeviceToHost && n == 4 && fake_next_word) {
    std::memcpy(d, &fake_next_word, 4);
    fake_next_word = 0;
  }
  op("copy-and-wait stream=0");
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  std::memset(p, v, n);
  op("memset" + on(st));
  return cudaSuccess;
}
// asynchronous with respect to the host on device memory
cudaError_t cudaMemset(void* p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags) {
  *s = static_cast<cudaStream_t>(std::malloc(1));
  g_streams[*s] = g_nextStream++;
  op("stream " + std::to_string(g_streams[*s]) + (flags & cudaStreamNonBlocking ? " non-blocking" : " blocking"));
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  g_streams.erase(s);
  std::free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  op("wait" + on(s));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = static_cast<cudaEvent_t>(std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  g_capture = new Graph{g_nextGraph++, {}};
  g_captureOrigin = s;
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
  *st = g_capture && s == g_captureOrigin ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(g_capture);
  g_capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph*>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
  const Graph* g = reinterpret_cast<const Graph*>(e);
  op("graph " + std::to_string(g->id) + on(s));
  for (const auto& x : g->ops) { op(x + " graph=" + std::to_string(g->id)); }
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<Graph*>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete reinterpret_cast<Graph*>(e);
  return cudaSuccess;
}

cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  return cudaSuccess;
}
cudaError_t cudaDeviceGetPCIBusId(char* s, int n, int) {
  std::snprintf(s, n, "fake");
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}  // extern "C"
