// fake_cudart.cpp -- a CUDA runtime for host-side tests without a GPU, preloaded
// before libgw.so: two devices whose memory is host memory, copies that happen at
// once, and launches that are checked and logged but not run.
//
// Checked:
//  * shared memory: a launch fails (cudaErrorInvalidValue) when its dynamic shared
//    memory exceeds the kernel's limit on the current device, 48 KB until
//    cudaFuncSetAttribute raises it there;
//  * order: work on the legacy default stream (a memset, or a copy from pageable
//    memory, whose last part may still be in flight when the call returns) and
//    work on a non-blocking stream have no order but by a synchronisation; a line
//    "unordered ..." is logged where one starts while the other may be in flight.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <utility>

namespace {
struct Stream {
  bool blocking;
  bool busy;
  std::set<Stream*> joined;  // streams whose work this one has waited for
};
struct Event {
  Stream* stream;
};
constexpr int kDevices = 2;
int optin = 227 * 1024;  // largest shared memory of a block
constexpr int kStatic = 4096;  // what every kernel has of it without asking
std::recursive_mutex mu;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
bool legacy_busy = false;
std::set<Stream*> streams;
std::map<const void*, std::string> names;
std::map<std::pair<int, const void*>, int> limits;
std::string out;

void note(const std::string& s) { out += s + "\n"; }
cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
// work `what` starts on s (null: the legacy stream)
void starts(cudaStream_t s, const std::string& what) {
  Stream* st = (Stream*)s;
  if (!st) {
    for (Stream* o : streams)
      if (!o->blocking && o->busy) {
        note("unordered " + what + " on the legacy stream");
        break;
      }
    legacy_busy = true;
  } else {
    if (!st->blocking && legacy_busy) note("unordered " + what + " on a non-blocking stream");
    st->busy = true;
  }
}
cudaError_t launch(const void* fn, size_t smem, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  const std::string name = names.count(fn) ? names[fn] : "?";
  const auto it = limits.find({device, fn});
  const size_t limit = it == limits.end() ? 48 * 1024 : (size_t)it->second;
  starts(s, "launch of " + name);
  char b[64];
  snprintf(b, sizeof b, " device %d shared %zu", device, smem);
  if (smem > limit) {
    note("refused " + name + b);
    return ret(cudaErrorInvalidValue);
  }
  note("launch " + name + b);
  return cudaSuccess;
}
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
void* cfg_stream;

int encode_tiled(void*, ...) { return 0; }
}  // namespace

extern "C" {
void fake_set_optin(int bytes) { optin = bytes; }

// the log since the last call, cut to n - 1 bytes
void fake_take(char* b, size_t n) {
  std::lock_guard<std::recursive_mutex> g(mu);
  snprintf(b, n, "%s", out.c_str());
  out.clear();
}

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, void*, void*, void*, void*, int*) {
  std::lock_guard<std::recursive_mutex> g(mu);
  names[fn] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
  cfg_grid = grid;
  cfg_block = block;
  cfg_smem = smem;
  cfg_stream = stream;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = cfg_grid;
  *block = cfg_block;
  *smem = cfg_smem;
  *(void**)stream = cfg_stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
  *k = (cudaKernel_t)fn;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t smem, cudaStream_t s) {
  return launch((const void*)k, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
  return launch(fn, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute a, int v) {
  std::lock_guard<std::recursive_mutex> g(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v < 0 || v + kStatic > optin) return ret(cudaErrorInvalidValue);
    limits[{device, fn}] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* fn) {
  std::lock_guard<std::recursive_mutex> g(mu);
  const auto it = limits.find({device, fn});
  memset(a, 0, sizeof *a);
  a->sharedSizeBytes = kStatic;
  a->maxDynamicSharedSizeBytes = it == limits.end() ? 48 * 1024 : it->second;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t smem) {
  *n = smem + kStatic > (size_t)optin ? 0 : 1;
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) {
  *n = kDevices;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= kDevices) return ret(cudaErrorInvalidDevice);
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? optin : 1;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : "error"; }

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = calloc(1, n);
  return *p ? cudaSuccess : ret(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return cudaMalloc(p, 1 << 20); }
cudaError_t cudaMemset(void* p, int v, size_t n) {
  std::lock_guard<std::recursive_mutex> g(mu);
  starts(nullptr, "memset");
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  starts(s, "memset");
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  std::lock_guard<std::recursive_mutex> g(mu);
  starts(nullptr, "copy");
  if (k == cudaMemcpyDeviceToHost) legacy_busy = false;  // synchronous, after all earlier work of the stream
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  starts(s, "copy");
  memcpy(d, src, n);
  return cudaSuccess;
}

static cudaError_t stream_new(cudaStream_t* s, bool blocking) {
  std::lock_guard<std::recursive_mutex> g(mu);
  Stream* st = new Stream{blocking, false, {}};
  streams.insert(st);
  *s = (cudaStream_t)st;
  return cudaSuccess;
}
cudaError_t cudaStreamCreate(cudaStream_t* s) { return stream_new(s, true); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { return stream_new(s, !(f & cudaStreamNonBlocking)); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  streams.erase((Stream*)s);
  delete (Stream*)s;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  if (Stream* st = (Stream*)s) {
    for (Stream* o : st->joined)
      if (streams.count(o)) o->busy = false;
    st->joined.clear();
    st->busy = false;
  } else {
    legacy_busy = false;
  }
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::recursive_mutex> g(mu);
  legacy_busy = false;
  for (Stream* s : streams) s->busy = false;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::recursive_mutex> g(mu);
  if (s && ((Event*)e)->stream) ((Stream*)s)->joined.insert(((Event*)e)->stream);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return ret(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return ret(cudaErrorNotSupported); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return ret(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return ret(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t) new Event{nullptr};
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete (Event*)e;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  ((Event*)e)->stream = (Stream*)s;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *p = (void*)encode_tiled;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}
