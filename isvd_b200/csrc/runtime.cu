// Device context, errors and stream-ordered allocation for libisvd_gpu_b200.
#include "runtime.h"

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

extern "C" size_t isvd_gpu_memory_limit;  // include/isvd/gpu/env.h
extern "C" size_t isvd_gpu_alloc_limit;   // include/isvd/b200.h

namespace isvdb {

std::atomic<unsigned long long> g_launches{0};

static Runtime g_rt;
static bool g_init = false;
static std::mutex g_init_mu;
static int g_precision = -1;

void fail(int code, const char *fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  throw Error(code, buf);
}

void check_cuda(cudaError_t e, const char *what, const char *file, int line) {
  if (e == cudaSuccess) return;
  int code = (e == cudaErrorMemoryAllocation) ? kErrMemory : kErrCuda;
  fail(code, "CUDA error %s (%s) in %s at %s:%d", cudaGetErrorName(e), cudaGetErrorString(e), what, file, line);
}

bool Runtime::initialised() { return g_init; }

Runtime &Runtime::get() {
  if (g_init) return g_rt;
  std::lock_guard<std::mutex> lk(g_init_mu);
  if (g_init) return g_rt;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  cudaDeviceProp prop;
  CK(cudaGetDeviceProperties(&prop, dev));
  g_rt.device = dev;
  g_rt.num_sms = prop.multiProcessorCount;
  g_rt.cc_major = prop.major;
  g_rt.cc_minor = prop.minor;
  g_rt.smem_optin = prop.sharedMemPerBlockOptin;
  CK(cudaStreamCreateWithFlags(&g_rt.own_stream, cudaStreamNonBlocking));
  g_rt.stream = g_rt.own_stream;
  CK(cudaStreamCreateWithFlags(&g_rt.copy_stream, cudaStreamNonBlocking));
  // Keep freed pool memory cached: repeated solves reuse it without new cudaMalloc calls.
  cudaMemPool_t pool;
  CK(cudaDeviceGetDefaultMemPool(&pool, dev));
  uint64_t thr = UINT64_MAX;
  CK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr));
  CK(cudaMalloc(&g_rt.ctl, 4096));
  CK(cudaMemset(g_rt.ctl, 0, 4096));
  CK(cudaMallocHost(&g_rt.host_pin, 64 * sizeof(double)));
  g_init = true;
  return g_rt;
}

void Runtime::reset() {
  std::lock_guard<std::mutex> lk(g_init_mu);
  if (!g_init) return;
  cudaStreamSynchronize(g_rt.stream);
  cudaFree(g_rt.ctl);
  cudaFreeHost(g_rt.host_pin);
  if (g_rt.stage) {
    cudaStreamSynchronize(g_rt.copy_stream);
    cudaFreeHost(g_rt.stage);
    for (cudaEvent_t e : g_rt.stage_ev) cudaEventDestroy(e);
  }
  cudaStreamDestroy(g_rt.own_stream);
  cudaStreamDestroy(g_rt.copy_stream);
  g_rt = Runtime();
  g_init = false;
}

int default_precision() {
  if (g_precision < 0) {
    const char *e = getenv("ISVD_GPU_PRECISION");
    g_precision = (e && (!strcmp(e, "mixed") || !strcmp(e, "1"))) ? kMixed : kNative;
  }
  return g_precision;
}

void set_default_precision(int p) { g_precision = p; }

Spare *g_spare = nullptr;

static bool capturing() {
  cudaStreamCaptureStatus s;
  CK(cudaStreamIsCapturing(Runtime::get().stream, &s));
  return s != cudaStreamCaptureStatusNone;
}

static cudaError_t try_alloc(void **p, size_t bytes) {
  Runtime &rt = Runtime::get();
  if (isvd_gpu_alloc_limit > 0 && !capturing()) {  // diagnostic: as if the device had no more
    cudaMemPool_t pool;
    unsigned long long used = 0;
    CK(cudaStreamSynchronize(rt.stream));
    CK(cudaDeviceGetDefaultMemPool(&pool, rt.device));
    CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
    if (used + bytes > isvd_gpu_alloc_limit) return cudaErrorMemoryAllocation;
  }
  const cudaError_t e = cudaMallocAsync(p, bytes, rt.stream);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

void trim_pool() {
  Runtime &rt = Runtime::get();
  cudaMemPool_t pool;
  CK(cudaStreamSynchronize(rt.stream));
  CK(cudaDeviceGetDefaultMemPool(&pool, rt.device));
  CK(cudaMemPoolTrimTo(pool, 0));
}

void *dev_alloc(size_t bytes) {
  void *p = nullptr;
  cudaError_t e = try_alloc(&p, bytes);
  if (e != cudaSuccess && g_spare && !capturing() && g_spare->give_back()) {
    trim_pool();
    e = try_alloc(&p, bytes);
  }
  if (e != cudaSuccess)
    fail(kErrMemory, "device allocation of %zu bytes failed (%s)", bytes, cudaGetErrorString(e));
  return p;
}

size_t device_budget() {
  Runtime &rt = Runtime::get();
  size_t free_b = 0, total_b = 0;
  CK(cudaMemGetInfo(&free_b, &total_b));
  // memory the library's pool holds but does not use counts as free (it is reused first)
  cudaMemPool_t pool;
  CK(cudaDeviceGetDefaultMemPool(&pool, rt.device));
  unsigned long long reserved = 0, used = 0;
  CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved));
  CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
  if (reserved > used) free_b += (size_t)(reserved - used);
  const size_t lim = isvd_gpu_memory_limit;
  return lim > 0 ? std::min(free_b, lim) : free_b;
}

long long host_panel_rows(long long m, long long n, size_t resident_bytes, size_t row_bytes, size_t work_bytes,
                          size_t elem) {
  // without a limit, what fits in any device needs no look at the free memory (100 us)
  if (isvd_gpu_memory_limit == 0 && resident_bytes + work_bytes <= ((size_t)128 << 20)) return 0;
  const size_t budget = device_budget();
  if (resident_bytes + work_bytes <= budget) return 0;
  const size_t avail = budget > work_bytes ? budget - work_bytes : 0;
  long long P = (long long)(avail / std::max<size_t>(row_bytes, 1));
  const long long cap = std::max<long long>(128, (long long)((1ll << 30) / ((long long)n * (long long)elem)));
  P = std::min(P, cap);
  if (P >= m) return m;
  P = P / 128 * 128;
  if (P < 128)
    fail(kErrMemory, "not enough GPU memory for a host A streamed in panels of 128 rows (%zu bytes usable, "
                     "%zu needed)", budget, work_bytes + 128 * row_bytes);
  return P;
}

void dev_free(void *p) {
  if (!p || !g_init) return;
  cudaFreeAsync(p, g_rt.stream);
}

bool is_device_pointer(const void *p) {
  if (!p) return false;
  cudaPointerAttributes attr;
  cudaError_t e = cudaPointerGetAttributes(&attr, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
}

namespace {

bool pageable(const void *p) {
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return attr.type == cudaMemoryTypeUnregistered;
}

// The pinned buffers and their events, all or none.
bool stage_ready(Runtime &rt) {
  if (rt.stage) return true;
  void *p = nullptr;
  cudaError_t e = cudaMallocHost(&p, Runtime::kStageSlots * Runtime::kStageBytes);
  int made = 0;
  while (e == cudaSuccess && made < Runtime::kStageSlots) {
    e = cudaEventCreateWithFlags(&rt.stage_ev[made], cudaEventDisableTiming);
    if (e == cudaSuccess) ++made;
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    while (made > 0) cudaEventDestroy(rt.stage_ev[--made]);
    if (p) cudaFreeHost(p);
    return false;
  }
  rt.stage = static_cast<unsigned char *>(p);
  return true;
}

}  // namespace

// The driver copies pageable memory through its own pinned buffer with one thread, about 9 GB/s of the link's
// 55.  Here each of up to eight threads takes 2 MB pieces in turn: waits until its buffer's last copy is
// done, fills it, enqueues the copy: a 12007 x 3001 FP32 solve with A in host memory (144 MB) 22.2 -> 9.9 ms.
// Below 4 MB the threads' start outweighs it.
void copy_to_device(void *dst, size_t dpitch, const void *src, size_t spitch, size_t width, size_t rows,
                    cudaStream_t st) {
  if (width == 0 || rows == 0) return;
  constexpr size_t kBytes = Runtime::kStageBytes;
  Runtime &rt = Runtime::get();
  const int threads = std::min<int>(Runtime::kStageSlots / 2, (int)std::thread::hardware_concurrency() / 2);
  // (cudaStreamPerThread names another stream in each of the threads)
  if (width * rows < (4u << 20) || threads < 2 || st == cudaStreamPerThread || !pageable(src) || !stage_ready(rt)) {
    CK(cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, rows, cudaMemcpyHostToDevice, st));
    return;
  }
  if (width == spitch && width == dpitch) {  // contiguous: one long line
    width *= rows;
    spitch = dpitch = width;
    rows = 1;
  }
  // pieces: whole lines, or stretches of one line when a line is longer than a buffer
  const size_t lines = std::max<size_t>(1, kBytes / width);
  const size_t cut = width > kBytes ? (width + kBytes - 1) / kBytes : 1;
  const size_t pieces = cut > 1 ? rows * cut : (rows + lines - 1) / lines;
  std::atomic<size_t> next{0};
  std::atomic<int> error{(int)cudaSuccess};
  auto work = [&](int t) {
    cudaError_t e = cudaSetDevice(rt.device);
    int turn = 0;
    for (size_t i; e == cudaSuccess && (i = next.fetch_add(1)) < pieces; turn ^= 1) {
      const int slot = 2 * t + turn;
      unsigned char *buf = rt.stage + slot * kBytes;
      if ((e = cudaEventSynchronize(rt.stage_ev[slot])) != cudaSuccess) break;
      size_t r0, n, off = 0, w = width;
      if (cut > 1) {
        r0 = i / cut; n = 1;
        off = (i % cut) * kBytes;
        w = std::min(kBytes, width - off);
      } else {
        r0 = i * lines;
        n = std::min(lines, rows - r0);
      }
      const unsigned char *from = static_cast<const unsigned char *>(src) + r0 * spitch + off;
      for (size_t r = 0; r < n; ++r) memcpy(buf + r * w, from + r * spitch, w);
      e = cudaMemcpy2DAsync(static_cast<unsigned char *>(dst) + r0 * dpitch + off, dpitch, buf, w, w, n,
                            cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaEventRecord(rt.stage_ev[slot], st);
    }
    if (e != cudaSuccess) error.store((int)e);
  };
  std::vector<std::thread> pool;
  const int count = (int)std::min<size_t>(threads, pieces);
  try {
    pool.reserve(count);
    for (int t = 1; t < count; ++t) pool.emplace_back(work, t);
  } catch (const std::exception &) {  // no more threads or memory: the threads that run take all pieces
  }
  work(0);
  for (std::thread &t : pool) t.join();
  CK((cudaError_t)error.load());
}

void sync() { CK(cudaStreamSynchronize(Runtime::get().stream)); }

void inject_timeout(const char *tag, int *status, cudaStream_t st) {
  const char *e = getenv("ISVD_GPU_INJECT_TIMEOUT");
  if (e && !strcmp(e, tag)) CK(cudaMemsetAsync(status, kErrTimeout, 1, st));  // the low byte
}

struct ProfEntry {
  double ms = 0.0, flops = 0.0;
  unsigned long long count = 0;
};
static std::map<std::string, ProfEntry> g_prof;
static std::mutex g_prof_mu;
static bool g_profiling = false;

bool profiling() { return g_profiling; }
void set_profiling(bool on) { g_profiling = on; }

unsigned long long count_kernel_nodes(cudaGraph_t g) {
  size_t n = 0;
  CK(cudaGraphGetNodes(g, nullptr, &n));
  std::vector<cudaGraphNode_t> nodes(n);
  if (n) CK(cudaGraphGetNodes(g, nodes.data(), &n));
  unsigned long long k = 0;
  for (size_t i = 0; i < n; ++i) {
    cudaGraphNodeType t;
    CK(cudaGraphNodeGetType(nodes[i], &t));
    if (t == cudaGraphNodeTypeKernel) ++k;
  }
  return k;
}

GraphPair::GraphPair(cudaStream_t s) : st(s) {
  const char *env = getenv("ISVD_GPU_GRAPHS");
  const bool off = env && env[0] == '0';
  // stream-ordered allocations inside the body go to the library stream: only that one is captured
  usable = !off && s != nullptr && s != cudaStreamLegacy && s != cudaStreamPerThread && !profiling() &&
           s == Runtime::get().stream;
}

GraphPair::~GraphPair() {
  for (int i = 0; i < 2; ++i)
    if (exec[i]) cudaGraphExecDestroy(exec[i]);
}
Collective &collective() {
  static Collective c;
  return c;
}

namespace {
template <class T>
void allreduce_impl(T *p, size_t count, int dtype, cudaStream_t st) {
  Collective &c = collective();
  if (c.nranks <= 1 || !c.fn || count == 0) return;
  if (c.on_device) {
    c.fn(p, count, dtype, st, c.user);
    CK(cudaGetLastError());
    return;
  }
  static void *pin = nullptr;
  static size_t pin_bytes = 0;
  const size_t bytes = count * sizeof(T);
  if (bytes > pin_bytes) {
    if (pin) cudaFreeHost(pin);
    pin = nullptr;
    pin_bytes = 0;
    if (cudaMallocHost(&pin, bytes) != cudaSuccess) fail(kErrMemory, "pinned staging for the AllReduce");
    pin_bytes = bytes;
  }
  CK(cudaMemcpyAsync(pin, p, bytes, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  c.fn(pin, count, dtype, st, c.user);
  CK(cudaMemcpyAsync(p, pin, bytes, cudaMemcpyHostToDevice, st));
  CK(cudaStreamSynchronize(st));  // the staging buffer is reused by the next call
}
}  // namespace

void allreduce_sum(double *p, size_t count, cudaStream_t st) { allreduce_impl(p, count, 1, st); }
void allreduce_sum(float *p, size_t count, cudaStream_t st) { allreduce_impl(p, count, 0, st); }

void profile_add(const char *tag, double ms, double flops) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  ProfEntry &e = g_prof[tag];
  e.ms += ms;
  e.flops += flops;
  e.count += 1;
}
bool profile_get(const char *tag, double *ms, unsigned long long *count, double *flops) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  auto it = g_prof.find(tag);
  if (it == g_prof.end()) return false;
  if (ms) *ms = it->second.ms;
  if (count) *count = it->second.count;
  if (flops) *flops = it->second.flops;
  return true;
}
void profile_reset() {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  g_prof.clear();
}

}  // namespace isvdb
