// A CUDA runtime without a GPU, for host-path tests: the library's own objects
// link against it instead of the real one. Device memory is host memory,
// cleared on allocation; copies and fills happen at once; kernels do nothing but
// leave a line in the log, "launch" on a stream and "record" in a capture. Two
// devices. Allocations can be made to fail, and a device that is synchronised
// while one of its streams captures refuses and spoils the capture, as CUDA
// documents it.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

struct CUstream_st {
  int device;
  unsigned long long id;
  bool capturing;
};
struct CUevent_st {
  int device;
};
struct CUmemPoolHandle_st {
  int device;
  size_t held;  // freed and not given back
};

namespace {
struct Block {
  size_t bytes;
  int device;
  cudaMemPool_t pool;
};
std::recursive_mutex lock;
std::map<void*, Block> blocks;
std::map<const void*, std::string> kernels;
std::vector<cudaStream_t> streams;
std::string text;
CUstream_st legacy[2] = {{0, 1, false}, {1, 2, false}};
unsigned long long next_id = 3;
size_t fail_from = ~(size_t)0, fail_to = 0;
int fail_times = 0, fail_after = 0;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local std::vector<Config> configs;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
template <class... A>
void note(const char* format, A... a) {
  char line[512];
  snprintf(line, sizeof line, format, a...);
  text += line;
  text += '\n';
}
cudaStream_t real(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy ? &legacy[device] : s; }
bool capturing(int dev) {
  for (cudaStream_t s : streams)
    if (s->device == dev && s->capturing) return true;
  return false;
}
cudaError_t allocate(void** p, size_t bytes, cudaMemPool_t pool, int dev) {
  *p = nullptr;
  if (fail_times > 0 && bytes >= fail_from && bytes <= fail_to && fail_after-- <= 0) {
    fail_times--;
    note("refuse %zu", bytes);
    return done(cudaErrorMemoryAllocation);
  }
  *p = std::calloc(1, bytes ? bytes : 1);
  blocks[*p] = {bytes, dev, pool};
  note("alloc %p %zu device %d%s", *p, bytes, dev, pool ? " pool" : "");
  return cudaSuccess;
}
cudaError_t launch(const char* name, dim3 g, dim3 b, cudaStream_t s) {
  s = real(s);
  if (s->device != device) return done(cudaErrorInvalidResourceHandle);
  note("%s %s grid %u block %u stream %llu", s->capturing ? "record" : "launch", name, g.x * g.y * g.z, b.x * b.y * b.z,
       s->id);
  return cudaSuccess;
}
}  // namespace

extern "C" {
// What tests steer and read.
const char* fake_log() { return text.c_str(); }
void fake_clear() { text.clear(); }
void fake_fail(size_t from, size_t to, int times, int after) {  // allocations of `from` to `to` bytes
  fail_from = from, fail_to = to, fail_times = times, fail_after = after;
}
size_t fake_live(int pooled) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  size_t n = 0;
  for (auto& b : blocks) n += (b.second.pool != nullptr) == (pooled != 0);
  return n;
}
unsigned long long fake_id(cudaStream_t s) { return real(s)->id; }

void** __cudaRegisterFatBinary(void*) { return (void**)&legacy; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  kernels[host] = name;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = (cudaKernel_t)host;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st* s) {
  configs.push_back({g, b, smem, s});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  const Config c = configs.back();
  configs.pop_back();
  *g = c.grid, *b = c.block, *smem = c.smem, *(cudaStream_t*)s = c.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  return launch(kernels[(const void*)k].c_str(), g, b, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  return launch(kernels[f].c_str(), c->gridDim, c->blockDim, c->stream);
}

cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d < 0 || d > 1 ? done(cudaErrorInvalidDevice) : (device = d, cudaSuccess); }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::recursive_mutex> hold(lock);
  if (capturing(device)) {
    note("spoiled capture on device %d", device);
    return done(cudaErrorStreamCaptureUnsupported);
  }
  note("sync device %d", device);
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = nullptr, done(cudaErrorInvalidSymbol); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int threads, size_t) {
  return *n = threads >= 512 ? 1 : threads >= 256 ? 2 : 4, cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  return allocate(p, bytes, nullptr, device);
}
cudaError_t cudaFree(void* p) {  // finds the owning device itself
  std::lock_guard<std::recursive_mutex> hold(lock);
  if (!p) return cudaSuccess;
  note("free %p device %d", p, blocks.at(p).device);
  blocks.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps* props) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  note("pool device %d", props->location.id);
  return *pool = new CUmemPoolHandle_st{props->location.id, 0}, cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  note("trim device %d", pool->device);
  return pool->held = 0, cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t bytes, cudaMemPool_t pool, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  if (real(s)->device != pool->device) return done(cudaErrorInvalidValue);
  return allocate(p, bytes, pool, pool->device);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  const Block b = blocks.at(p);
  if (!b.pool || real(s)->device != b.device) return done(cudaErrorInvalidValue);
  note("give back %p stream %llu", p, real(s)->id);
  b.pool->held += b.bytes;
  blocks.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind) { return std::memmove(to, from, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t s) {
  if (!real(s)->capturing) std::memmove(to, from, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  if (!real(s)->capturing) std::memset(p, v, n);
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  *s = new CUstream_st{device, next_id++, false};
  streams.push_back(*s);
  note("stream %llu device %d", (*s)->id, device);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  for (size_t k = 0; k < streams.size(); k++)
    if (streams[k] == s) streams.erase(streams.begin() + k--);
  delete s;
  return cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) { return *id = real(s)->id, cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  if (real(s)->capturing) return done(cudaErrorStreamCaptureUnsupported);
  note("sync stream %llu", real(s)->id);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
  *st = real(s)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { return s->capturing = true, cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  s->capturing = false;
  return *g = (cudaGraph_t)std::calloc(1, 8), cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  return *x = (cudaGraphExec_t)std::calloc(1, 8), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  note("replay stream %llu", real(s)->id);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return std::free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return std::free(x), cudaSuccess; }

cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = new CUevent_st{device}, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete e, cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  if (e->device != real(s)->device) return done(cudaErrorInvalidResourceHandle);
  note("event %p stream %llu", (void*)e, real(s)->id);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::recursive_mutex> hold(lock);
  note("wait %p stream %llu", (void*)e, real(s)->id);
  return cudaSuccess;
}
}
