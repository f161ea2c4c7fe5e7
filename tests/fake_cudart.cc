// A CUDA runtime for tests of the library's host code on a machine without a
// GPU: device memory is host memory, copies and fills happen at once, kernels
// do nothing.  What it keeps is the order that a real device would be free to
// choose: work queued on a stream stays pending until the host waits for it,
// and a host copy from pageable memory may still be on its way when the call
// returns.  Calls can be made to fail, and a copy or fill outside the
// allocations is recorded instead of done.  A pool keeps up to 1 GB of what was
// freed, as the library asks, until it is trimmed.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {

struct Stream;
struct Wait {
  uint64_t at;
  Stream *other;
  uint64_t pos;
};
struct Stream {
  uint64_t issued = 0, done = 0;
  std::vector<Wait> waits;
};
struct Event {
  Stream *st = nullptr;
  uint64_t pos = 0;
};
struct Alloc {
  size_t size;
  bool pinned;
};
typedef void (*LaunchHook)(const char *kernel, void **args);

struct Fake {
  std::recursive_mutex mu;
  std::map<uintptr_t, Alloc> mem;
  std::map<const void *, std::string> kernels;
  std::map<std::string, uint64_t> launches;
  std::map<const void *, int> smem;   // limits of dynamic shared memory
  std::vector<Stream *> streams;
  Stream legacy;
  std::vector<std::string> faults;
  std::map<size_t, size_t> tails;   // H2D copies by size: bytes of the allocation behind the last one
  std::string fail_fn;
  long fail_at = -1;
  int fail_err = 0;
  cudaError_t last = cudaSuccess;
  uint64_t limit = ~0ull, used = 0, kept = 0;   // kept: by the pool (in used)
  LaunchHook hook = nullptr;
};

// (made before any other object's constructor uses it, never destroyed)
Fake &F() {
  static Fake *f = new Fake();
  return *f;
}

typedef std::lock_guard<std::recursive_mutex> Lock;

Stream *stream_of(cudaStream_t st) {
  return st == nullptr || st == cudaStreamLegacy ? &F().legacy : reinterpret_cast<Stream *>(st);
}

void complete(Stream *s, uint64_t pos) {
  if (pos <= s->done) return;
  s->done = pos;
  for (size_t i = 0; i < s->waits.size(); i++)
    if (s->waits[i].at <= pos) complete(s->waits[i].other, s->waits[i].pos);
}
void complete_all() {
  complete(&F().legacy, F().legacy.issued);
  for (Stream *s : F().streams) complete(s, s->issued);
}

// Whether this call of `fn` is to fail.
cudaError_t fails(const char *fn) {
  Fake &f = F();
  if (f.fail_at >= 0 && (f.fail_fn.empty() || f.fail_fn == fn) && f.fail_at-- == 0)
    return f.last = (cudaError_t)f.fail_err;
  return cudaSuccess;
}

void fault(const char *what) { F().faults.push_back(what); }

std::map<uintptr_t, Alloc>::iterator find(const void *p) {
  auto it = F().mem.upper_bound((uintptr_t)p);
  if (it == F().mem.begin()) return F().mem.end();
  --it;
  return (uintptr_t)p < it->first + it->second.size ? it : F().mem.end();
}
bool device_range(const void *p, size_t n) {
  auto it = find(p);
  return it != F().mem.end() && !it->second.pinned && (uintptr_t)p + n <= it->first + it->second.size;
}
bool is_pinned(const void *p) {
  auto it = find(p);
  return it != F().mem.end() && it->second.pinned;
}

cudaError_t allocate(void **p, size_t n, bool pinned) {
  Fake &f = F();
  *p = nullptr;
  if (!pinned && n > f.limit - f.used) return f.last = cudaErrorMemoryAllocation;
  *p = calloc(1, n);   // (mapped when touched)
  if (!*p) return f.last = cudaErrorMemoryAllocation;
  if (!pinned) f.used += n;
  f.mem[(uintptr_t)*p] = Alloc{n, pinned};
  return cudaSuccess;
}
void release(void *p, const char *who) {
  if (!p) return;
  auto it = F().mem.find((uintptr_t)p);
  if (it == F().mem.end()) return fault(who);
  if (!it->second.pinned) F().used -= it->second.size;
  F().mem.erase(it);
  free(p);
}

bool copy(void *dst, const void *src, size_t n, cudaMemcpyKind kind) {
  if (!n) return true;
  if ((kind != cudaMemcpyDeviceToHost && !device_range(dst, n)) ||
      (kind != cudaMemcpyHostToDevice && !device_range(src, n))) {
    fault("copy outside the allocations");
    return false;
  }
  if (kind == cudaMemcpyHostToDevice) {
    auto it = find(dst);
    F().tails[n] = it->first + it->second.size - ((uintptr_t)dst + n);
  }
  memmove(dst, src, n);
  return true;
}

cudaError_t set(void *p, int v, size_t n, cudaStream_t st) {
  if (n && !device_range(p, n)) fault("fill outside the allocations");
  else memset(p, v, n);
  stream_of(st)->issued++;
  return cudaSuccess;
}

}  // namespace

#define API extern "C" __attribute__((visibility("default")))
#define FAILS(fn)                                      \
  Lock lock(F().mu);                                   \
  {                                                    \
    const cudaError_t e_ = fails(#fn);                 \
    if (e_ != cudaSuccess) return e_;                  \
  }

// ---- what tests ask
API void fake_reset() {
  Lock lock(F().mu);
  F().launches.clear();
  F().faults.clear();
  F().tails.clear();
  F().fail_at = -1;
  F().last = cudaSuccess;
  F().limit = ~0ull;
  F().hook = nullptr;
  complete_all();
}
// The call of fn (any, where empty) after `skip` more fails with err.
API void fake_fail(const char *fn, long skip, int err) {
  F().fail_fn = fn;
  F().fail_at = skip;
  F().fail_err = err;
}
API uint64_t fake_kept() { return F().kept; }
API int fake_failed() { return F().fail_at < 0; }
API void fake_limit(uint64_t bytes) { F().limit = bytes; }
// Device memory held, without what the pool keeps.
API uint64_t fake_used() { return F().used - F().kept; }
API uint64_t fake_pending(void *st) {
  Stream *s = stream_of((cudaStream_t)st);
  return s->issued - s->done;
}
API uint64_t fake_pending_all() {
  uint64_t n = F().legacy.issued - F().legacy.done;
  for (Stream *s : F().streams) n += s->issued - s->done;
  return n;
}
API uint64_t fake_launches(const char *part) {
  uint64_t n = 0;
  for (auto &x : F().launches)
    if (x.first.find(part) != std::string::npos) n += x.second;
  return n;
}
API long fake_faults() { return (long)F().faults.size(); }
API const char *fake_fault(long i) { return F().faults[i].c_str(); }
// Bytes from p to the end of its allocation (-1: none).
API long fake_room(const void *p) {
  auto it = find(p);
  return it == F().mem.end() ? -1 : (long)(it->first + it->second.size - (uintptr_t)p);
}
API long fake_tail_of_copy(size_t bytes) { return F().tails.count(bytes) ? (long)F().tails[bytes] : -1; }
API void fake_hook(LaunchHook h) { F().hook = h; }

// ---- the runtime
API cudaError_t cudaGetLastError() {
  Lock lock(F().mu);
  const cudaError_t e = F().last;
  F().last = cudaSuccess;
  return e;
}
API const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
static thread_local int t_device = 0;
API cudaError_t cudaGetDevice(int *d) { *d = t_device; return cudaSuccess; }
API cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
API cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -5; return cudaSuccess; }
API cudaError_t cudaMemGetInfo(size_t *free_b, size_t *total) { *free_b = *total = 1ull << 38; return cudaSuccess; }
// (one limit a kernel for all threads: lowered by one call, it fails another's launch)
API cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute a, int v) {
  Lock lock(F().mu);
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  if (F().smem.count(fn) && F().smem[fn] > v) fault(("limit of shared memory lowered: " + F().kernels[fn]).c_str());
  F().smem[fn] = v;
  return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 8;
  return cudaSuccess;
}
API cudaError_t cudaGetSymbolAddress(void **p, const void *) { FAILS(cudaGetSymbolAddress) return allocate(p, 16 << 20, false); }

API cudaError_t cudaMalloc(void **p, size_t n) { FAILS(cudaMalloc) return allocate(p, n, false); }
API cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { FAILS(cudaHostAlloc) return allocate(p, n, true); }
API cudaError_t cudaFree(void *p) { Lock lock(F().mu); complete_all(); release(p, "cudaFree of no allocation"); return cudaSuccess; }
API cudaError_t cudaFreeHost(void *p) { Lock lock(F().mu); complete_all(); release(p, "cudaFreeHost of no allocation"); return cudaSuccess; }
API cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { FAILS(cudaMemPoolCreate) *p = (cudaMemPool_t)8; return cudaSuccess; }
API cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
API cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) {
  Lock lock(F().mu);
  F().used -= F().kept;
  F().kept = 0;
  return cudaSuccess;
}
API cudaError_t cudaDeviceSynchronize() { Lock lock(F().mu); complete_all(); return cudaSuccess; }
API cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  FAILS(cudaMallocFromPoolAsync)
  if (!pool) fault("allocation from no pool");
  const uint64_t reused = F().kept < n ? F().kept : n;
  F().kept -= reused;
  F().used -= reused;
  return allocate(p, n, false);
}
API cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
  Lock lock(F().mu);
  const uint64_t before = F().used;
  release(p, "cudaFreeAsync of no allocation");
  const uint64_t size = before - F().used, room = (1ull << 30) - F().kept, keep = size < room ? size : room;
  F().kept += keep;
  F().used += keep;
  return cudaSuccess;
}

API cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  FAILS(cudaMemcpy)
  Stream &l = F().legacy;
  complete(&l, l.issued);
  copy(d, s, n, k);
  if (k == cudaMemcpyHostToDevice && !is_pinned(s)) l.issued++;   // staged: its end is not waited for
  return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  FAILS(cudaMemcpyAsync)
  copy(d, s, n, k);
  Stream *x = stream_of(st);
  x->issued++;
  if (k == cudaMemcpyDeviceToHost && !is_pinned(d)) complete(x, x->issued);
  return cudaSuccess;
}
API cudaError_t cudaMemset(void *p, int v, size_t n) { FAILS(cudaMemset) return set(p, v, n, nullptr); }
API cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t st) { FAILS(cudaMemsetAsync) return set(p, v, n, st); }

static cudaError_t new_stream(cudaStream_t *s) {
  Stream *x = new Stream();
  F().streams.push_back(x);
  *s = reinterpret_cast<cudaStream_t>(x);
  return cudaSuccess;
}
API cudaError_t cudaStreamCreate(cudaStream_t *s) { FAILS(cudaStreamCreate) return new_stream(s); }
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { FAILS(cudaStreamCreateWithFlags) return new_stream(s); }
API cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { FAILS(cudaStreamCreateWithPriority) return new_stream(s); }
API cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }   // (what is pending stays counted)
API cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  FAILS(cudaStreamSynchronize)
  complete(stream_of(st), stream_of(st)->issued);
  return cudaSuccess;
}
API cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t ev, unsigned) {
  FAILS(cudaStreamWaitEvent)
  const Event *e = reinterpret_cast<Event *>(ev);
  Stream *s = stream_of(st);
  if (e->st) s->waits.push_back(Wait{s->issued + 1, e->st, e->pos});
  return cudaSuccess;
}
API cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
API cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = (cudaGraph_t)8; return cudaSuccess; }
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long) { *g = (cudaGraphExec_t)8; return cudaSuccess; }
API cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo *) { return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
API cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
API cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

API cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { FAILS(cudaEventCreateWithFlags) *e = (cudaEvent_t) new Event(); return cudaSuccess; }
API cudaError_t cudaEventCreate(cudaEvent_t *e) { FAILS(cudaEventCreate) *e = (cudaEvent_t) new Event(); return cudaSuccess; }
API cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t st) {
  FAILS(cudaEventRecord)
  Event *e = reinterpret_cast<Event *>(ev);
  e->st = stream_of(st);
  e->pos = e->st->issued;
  return cudaSuccess;
}
API cudaError_t cudaEventSynchronize(cudaEvent_t ev) {
  FAILS(cudaEventSynchronize)
  const Event *e = reinterpret_cast<Event *>(ev);
  if (e->st) complete(e->st, e->pos);
  return cudaSuccess;
}
API cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
API cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

// ---- launches (what the compiler's stubs call)
API void **__cudaRegisterFatBinary(void *) { static void *h = nullptr; return &h; }
API void __cudaRegisterFatBinaryEnd(void **) {}
API void __cudaUnregisterFatBinary(void **) {}
API void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
API void __cudaRegisterFunction(void **, const char *fn, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
  F().kernels[fn] = name;
}
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
};
static thread_local Config t_config;
API unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
  t_config = Config{grid, block, smem, st};
  return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
  *grid = t_config.grid;
  *block = t_config.block;
  *smem = t_config.smem;
  *static_cast<cudaStream_t *>(st) = t_config.st;
  return cudaSuccess;
}
API cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) { *k = (cudaKernel_t)fn; return cudaSuccess; }
API cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t st) {
  FAILS(launch)
  const std::string &name = F().kernels[(const void *)k];
  F().launches[name]++;
  if (!grid.x || !grid.y || !grid.z || !block.x) fault(("empty launch of " + name).c_str());
  const void *fn = (const void *)k;
  if (smem > 48 * 1024 && (!F().smem.count(fn) || (size_t)F().smem[fn] < smem))
    fault(("shared memory above its limit: " + name).c_str());
  stream_of(st)->issued++;
  if (F().hook) F().hook(name.c_str(), args);
  return cudaSuccess;
}
