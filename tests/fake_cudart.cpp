// A stand-in for the CUDA runtime: the calls that libhodlr_b200 makes, on host
// memory, with two devices.  Kernels do nothing, so results mean nothing; what
// it models is what the library's host code has to get right:
//   * a launch stays queued until its stream, an event after it, or the device
//     is waited for;
//   * cudaFree of cudaMalloc memory waits for the device, of stream-ordered
//     memory it does not: such a free while work is queued is counted;
//   * stream-ordered pools keep what is freed up to their release threshold,
//     which no other allocation can use until the pool is trimmed; a device
//     holds `capacity` bytes;
//   * a kernel takes more than 48 KB of dynamic shared memory only on a device
//     where its attribute says so.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>

namespace {

constexpr int kDevices = 2;

struct Pool {
  int dev = 0;
  size_t used = 0, reserved = 0;
  unsigned long long threshold = 0;
};
struct Block {
  int dev;
  size_t bytes;
  Pool *pool;   // null: cudaMalloc
};
struct Event {
  int dev = 0;
  cudaStream_t s = nullptr;
};

std::recursive_mutex mu;
std::map<void *, Block> blocks;
Pool default_pool[kDevices];
std::set<Pool *> pools[kDevices];
size_t capacity = size_t(1) << 32, plain[kDevices];
std::set<cudaStream_t> queued[kDevices];
std::map<std::pair<int, const void *>, int> smem_of;
long long frees_under_work, device_waits, launches_seen;
thread_local int cur;
thread_local cudaError_t last;
thread_local std::set<cudaStream_t> capturing;

using Lock = std::lock_guard<std::recursive_mutex>;

cudaError_t fails(cudaError_t e) {
  last = e;
  return e;
}

size_t mapped(int dev) {
  size_t s = plain[dev] + default_pool[dev].reserved;
  for (Pool *p : pools[dev]) s += p->reserved;
  return s;
}

void enqueue(cudaStream_t s) {
  if (!capturing.count(s)) queued[cur].insert(s);
}

cudaError_t pool_alloc(void **out, size_t bytes, Pool *p) {
  const size_t more = p->used + bytes > p->reserved ? p->used + bytes - p->reserved : 0;
  if (more > capacity || mapped(p->dev) > capacity - more) return fails(cudaErrorMemoryAllocation);
  p->reserved += more;
  p->used += bytes;
  *out = std::calloc(bytes ? bytes : 1, 1);
  blocks[*out] = Block{p->dev, bytes, p};
  return cudaSuccess;
}

void release(void *ptr) {
  const Block b = blocks.at(ptr);
  blocks.erase(ptr);
  if (b.pool) {
    b.pool->used -= b.bytes;
    if (b.pool->reserved > b.pool->threshold)
      b.pool->reserved = b.pool->used > b.pool->threshold ? b.pool->used : b.pool->threshold;
  } else {
    plain[b.dev] -= b.bytes;
  }
  std::free(ptr);
}

cudaError_t launch(const void *f, size_t smem, cudaStream_t s) {
  Lock l(mu);
  ++launches_seen;
  const auto it = smem_of.find({cur, f});
  if (smem > 48 * 1024 && (it == smem_of.end() || (size_t)it->second < smem))
    return fails(cudaErrorInvalidValue);
  enqueue(s);
  return cudaSuccess;
}

struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t s;
};
thread_local Config pushed;

}  // namespace

extern "C" {

// ---- what the tests read and set ------------------------------------------------------
void fake_set_capacity(unsigned long long bytes) { capacity = bytes; }
long long fake_frees_under_work() { return frees_under_work; }
long long fake_device_waits() { return device_waits; }
long long fake_launches() { return launches_seen; }
int fake_set_device(int dev) { return cudaSetDevice(dev); }
// bytes used / mapped: pool 0 the default one, 1 the library's own
unsigned long long fake_pool_bytes(int which, int mapped_too) {
  Lock l(mu);
  Pool *p = which == 0 ? &default_pool[cur] : pools[cur].empty() ? nullptr : *pools[cur].begin();
  return !p ? 0 : mapped_too ? p->reserved : p->used;
}

// ---- devices, errors ------------------------------------------------------------------
cudaError_t cudaGetDevice(int *d) { *d = cur; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= kDevices) return fails(cudaErrorInvalidDevice);
  cur = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) {
  return e == cudaSuccess ? "no error" : e == cudaErrorMemoryAllocation ? "out of memory" : "error";
}
cudaError_t cudaDeviceSynchronize() {
  Lock l(mu);
  ++device_waits;
  queued[cur].clear();
  return cudaSuccess;
}

// ---- memory ---------------------------------------------------------------------------
cudaError_t cudaMalloc(void **p, size_t bytes) {
  Lock l(mu);
  if (bytes > capacity || mapped(cur) > capacity - bytes) return fails(cudaErrorMemoryAllocation);
  plain[cur] += bytes;
  *p = std::calloc(bytes ? bytes : 1, 1);
  blocks[*p] = Block{cur, bytes, nullptr};
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  Lock l(mu);
  if (!p) return cudaSuccess;
  const Block b = blocks.at(p);
  if (!b.pool)
    queued[b.dev].clear();
  else if (!queued[b.dev].empty())
    ++frees_under_work;
  release(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t bytes, cudaStream_t) {
  Lock l(mu);
  return pool_alloc(p, bytes, &default_pool[cur]);
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t) {
  Lock l(mu);
  return pool_alloc(p, bytes, reinterpret_cast<Pool *>(pool));
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
  Lock l(mu);
  if (p) release(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) { *p = std::malloc(bytes); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  Lock l(mu);
  *t = capacity;
  *f = capacity > mapped(cur) ? capacity - mapped(cur) : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int dev) {
  default_pool[dev].dev = dev;
  *p = reinterpret_cast<cudaMemPool_t>(&default_pool[dev]);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const struct cudaMemPoolProps *props) {
  Lock l(mu);
  Pool *q = new Pool;
  q->dev = props->location.id;
  pools[q->dev].insert(q);
  *p = reinterpret_cast<cudaMemPool_t>(q);
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
  Lock l(mu);
  Pool *q = reinterpret_cast<Pool *>(p);
  const size_t floor = q->used > keep ? q->used : keep;
  if (q->reserved > floor) q->reserved = floor;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void *v) {
  if (a == cudaMemPoolAttrReleaseThreshold)
    reinterpret_cast<Pool *>(p)->threshold = *static_cast<unsigned long long *>(v);
  return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void *v) {
  Lock l(mu);
  const Pool *q = reinterpret_cast<Pool *>(p);
  *static_cast<unsigned long long *>(v) =
      a == cudaMemPoolAttrReservedMemCurrent ? q->reserved : q->used;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind, cudaStream_t) {
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                              enum cudaMemcpyKind, cudaStream_t) {
  for (size_t i = 0; i < h; ++i)
    std::memmove((char *)d + i * dp, (const char *)s + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  static char symbol[1 << 20];
  *p = symbol;
  return cudaSuccess;
}

// ---- streams, events, graphs ----------------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(new char);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  Lock l(mu);
  queued[cur].erase(s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new Event);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<Event *>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  *reinterpret_cast<Event *>(e) = Event{cur, s};
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  Lock l(mu);
  const Event *v = reinterpret_cast<Event *>(e);
  queued[v->dev].erase(v->s);
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) {
  *c = capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode) {
  capturing.insert(s);
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
  capturing.erase(s);
  *g = reinterpret_cast<cudaGraph_t>(new char);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(new char);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<char *>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete reinterpret_cast<char *>(e);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  Lock l(mu);
  enqueue(s);
  return cudaSuccess;
}

// ---- kernels --------------------------------------------------------------------------
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
  Lock l(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_of[{cur, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t s) {
  return launch(f, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  return launch(f, c->dynamicSmemBytes, c->stream);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void *s) {
  pushed = Config{grid, block, smem, static_cast<cudaStream_t>(s)};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *static_cast<cudaStream_t *>(s) = pushed.s;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *,
                            void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
