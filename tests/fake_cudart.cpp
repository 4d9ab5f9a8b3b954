// A CUDA runtime for tests of the host side: device memory is host memory,
// kernels do not run, and what is enqueued is recorded.
//
// Order.  Every stream carries a vector clock: an operation counts one on its
// stream, an event holds its stream's clock when recorded, a wait merges it,
// and what the host has synchronized with precedes everything enqueued later.
// cudaFreeAsync checks that every operation enqueued so far on any stream
// precedes it, and counts a fault where one does not (it may still use the
// memory).
//
// Failures.  fake_fail_at(k) makes the k-th enqueued operation from now on
// (k = 0: the next one) return an error and do nothing.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

namespace {

typedef std::vector<long long> Clock;

void merge(Clock& a, const Clock& b) {
  if (a.size() < b.size()) a.resize(b.size(), 0);
  for (size_t i = 0; i < b.size(); i++) a[i] = std::max(a[i], b[i]);
}

struct Stream {
  size_t id;
  Clock clock;
  bool capturing = false;
};
struct Event {
  Clock clock;
  bool capturing = false;
};
struct Graph {
  long long kernels = 0;
};

std::recursive_mutex mu;
std::vector<Stream*> streams;
Clock host;
std::vector<dim3> cfg_dims;
size_t cfg_smem = 0;
cudaStream_t cfg_stream = nullptr;
cudaError_t last = cudaSuccess;
long long ops = 0, fail_at = -1, kernels = 0, captured = 0, faults = 0;

Stream* new_stream() {
  Stream* s = new Stream();
  s->id = streams.size();
  streams.push_back(s);
  return s;
}
Stream* of(cudaStream_t h) {
  static Stream* null_stream = new_stream();
  return h ? (Stream*)h : null_stream;
}
// one enqueued operation on s; false where it is to fail
bool enqueue(Stream* s) {
  if (fail_at >= 0 && ops++ == fail_at) {
    last = cudaErrorUnknown;
    return false;
  }
  merge(s->clock, host);
  if (s->clock.size() <= s->id) s->clock.resize(s->id + 1, 0);
  s->clock[s->id]++;
  return true;
}
cudaError_t launched(Stream* s) {
  if (!enqueue(s)) return last;
  (s->capturing ? captured : kernels)++;
  return cudaSuccess;
}

}  // namespace

#define LOCK std::lock_guard<std::recursive_mutex> lock(mu)

extern "C" {

void fake_fail_at(long long k) { LOCK; ops = 0; fail_at = k; last = cudaSuccess; }
long long fake_ops(void) { return ops; }          // enqueued since fake_fail_at
long long fake_kernels(void) { return kernels; }  // kernels run, graphs' replays included
long long fake_faults(void) { return faults; }    // frees that did not wait for all work

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t s) {
  mu.lock();
  cfg_dims = {g, b};
  cfg_smem = sm;
  cfg_stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* s) {
  *g = cfg_dims[0];
  *b = cfg_dims[1];
  *sm = cfg_smem;
  *(cudaStream_t*)s = cfg_stream;
  mu.unlock();
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t s) {
  LOCK; return launched(of(s));
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
  LOCK; return launched(of(c->stream));
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t,
                                                                   unsigned) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = 1ull << 37; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static std::vector<char> image(8 << 20);
  *p = image.data();
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "injected"; }
cudaError_t cudaGetLastError(void) { LOCK; cudaError_t e = last; last = cudaSuccess; return e; }

cudaError_t cudaMalloc(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) {
  LOCK;
  for (Stream* s : streams) merge(host, s->clock);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t s) {
  LOCK;
  if (!enqueue(of(s))) return last;
  *p = calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t h) {
  LOCK;
  Stream* s = of(h);
  merge(s->clock, host);
  bool after_all = true;
  for (Stream* t : streams) {
    const long long done = t->id < s->clock.size() ? s->clock[t->id] : 0;
    if (t->id < t->clock.size() && t->clock[t->id] > done) after_all = false;
  }
  if (!after_all) faults++;
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t h) {
  LOCK;
  if (!enqueue(of(h))) return last;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t h) {
  LOCK;
  if (!enqueue(of(h))) return last;
  memset(d, v, n);
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  LOCK;
  *s = (cudaStream_t)new_stream();
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { LOCK; merge(host, of(s)->clock); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t h, cudaEvent_t e, unsigned) {
  LOCK;
  Stream* s = of(h);
  if (!enqueue(s)) return last;
  merge(s->clock, ((Event*)e)->clock);
  s->capturing |= ((Event*)e)->capturing;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)new Event();
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t h) {
  LOCK;
  Stream* s = of(h);
  if (!enqueue(s)) return last;
  ((Event*)e)->clock = s->clock;
  ((Event*)e)->capturing = s->capturing;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { LOCK; merge(host, ((Event*)e)->clock); return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  LOCK;
  of(s)->capturing = true;
  captured = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  LOCK;
  for (Stream* s : streams) s->capturing = false;
  Graph* n = new Graph();
  n->kernels = captured;
  *g = (cudaGraph_t)n;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  *x = (cudaGraphExec_t) new Graph(*(Graph*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { delete (Graph*)g; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  LOCK;
  if (!enqueue(of(s))) return last;
  kernels += ((Graph*)x)->kernels;
  return cudaSuccess;
}

}  // extern "C"
