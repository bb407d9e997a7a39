// Context, device memory and timing entry points.
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "common.cuh"

thread_local std::string g_ruai_global_err;

int ruai_fail(ruai_ctx* ctx, int code, const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (ctx) ctx->err = buf;
  g_ruai_global_err = buf;
  return code;
}

static void ruai_pool_forget(ruai_ctx* c);
static void ruai_pool_contexts(int ordinal, int change);  // the device's last context gives the kept memory back

RUAI_API const char* ruai_version(void) { return "ruai_b200 0.1 (sm_100a)"; }

RUAI_API int ruai_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

RUAI_API const char* ruai_last_error(const ruai_ctx* ctx) { return ctx ? ctx->err.c_str() : g_ruai_global_err.c_str(); }

RUAI_API int ruai_ctx_create(int ordinal, void* stream_or_null, ruai_ctx** out) {
  if (!out) return ruai_fail(nullptr, RUAI_ERR_ARG, "ruai_ctx_create: out is NULL");
  *out = nullptr;
  int n = ruai_device_count();
  if (n <= 0) return ruai_fail(nullptr, RUAI_ERR_CUDA, "no CUDA device: this library has no CPU fallback");
  if (ordinal < 0 || ordinal >= n) return ruai_fail(nullptr, RUAI_ERR_ARG, "device ordinal %d out of range (%d devices)", ordinal, n);
  RUAI_CUDA(nullptr, cudaSetDevice(ordinal));
  cudaDeviceProp prop;
  RUAI_CUDA(nullptr, cudaGetDeviceProperties(&prop, ordinal));
  if (prop.major != 10)
    return ruai_fail(nullptr, RUAI_ERR_UNSUPPORTED, "device %d is sm_%d%d; this library is built for sm_100a only", ordinal, prop.major, prop.minor);
  ruai_ctx* c = new ruai_ctx();
  c->ordinal = ordinal;
  c->sm_count = prop.multiProcessorCount;
  if (stream_or_null) c->stream = (cudaStream_t)stream_or_null;
  else {
    cudaError_t e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) { delete c; return ruai_fail(nullptr, RUAI_ERR_CUDA, "cudaStreamCreate: %s", cudaGetErrorString(e)); }
    c->own_stream = true;
  }
  cudaEventCreate(&c->ev0);
  cudaEventCreate(&c->ev1);
  const char* pdl = getenv("RUAI_B200_PDL");
  if (pdl && pdl[0] == '0') c->use_pdl = false;
  const char* bulk = getenv("RUAI_B200_BULK");
  if (bulk && bulk[0] == '0') c->use_bulk = false;
  const char* tc = getenv("RUAI_B200_TC");
  if (tc && tc[0] == '0') c->use_tc = false;
  if (cudaMalloc(&c->status, sizeof(int)) != cudaSuccess || cudaMemset(c->status, 0, sizeof(int)) != cudaSuccess) {
    delete c;
    return ruai_fail(nullptr, RUAI_ERR_CUDA, "cannot allocate the status word");
  }
  int rc = ruai_ctx_reserve(c, 8u << 20, 4096);
  if (rc != RUAI_OK) { g_ruai_global_err = c->err; delete c; return rc; }
  ruai_pool_contexts(ordinal, 1);
  *out = c;
  return RUAI_OK;
}

RUAI_API int ruai_ctx_destroy(ruai_ctx* c) {
  if (!c) return RUAI_OK;
  DeviceGuard g(c->ordinal);
  cudaStreamSynchronize(c->stream);
  ruai_pool_forget(c);
  cudaFree(c->partial);
  cudaFree(c->counters);
  cudaFree(c->status);
  cudaFree(c->ps_sync);
  cudaFree(c->sample_buf);
  cudaEventDestroy(c->ev0);
  cudaEventDestroy(c->ev1);
  if (c->own_stream) cudaStreamDestroy(c->stream);
  ruai_pool_contexts(c->ordinal, -1);
  delete c;
  return RUAI_OK;
}

int ruai_ctx_reserve(ruai_ctx* c, size_t partial_bytes, size_t counters) {
  DeviceGuard g(c->ordinal);
  if (partial_bytes > c->partial_bytes) {
    RUAI_CUDA(c, cudaStreamSynchronize(c->stream));
    if (c->partial) cudaFree(c->partial);
    c->partial = nullptr;
    c->partial_bytes = 0;
    RUAI_CUDA(c, ruai_device_malloc((void**)&c->partial, partial_bytes));
    c->partial_bytes = partial_bytes;
    c->scratch_epoch++;
  }
  if (counters > c->counters_n) {
    RUAI_CUDA(c, cudaStreamSynchronize(c->stream));
    if (c->counters) cudaFree(c->counters);
    c->counters = nullptr;
    c->counters_n = 0;
    RUAI_CUDA(c, cudaMalloc(&c->counters, counters * sizeof(unsigned)));
    RUAI_CUDA(c, cudaMemset(c->counters, 0, counters * sizeof(unsigned)));
    c->counters_n = counters;
    c->scratch_epoch++;
  }
  return RUAI_OK;
}

int ruai_ctx_check_status(ruai_ctx* c) {
  int st = 0;
  RUAI_CUDA(c, cudaMemcpyAsync(&st, c->status, sizeof st, cudaMemcpyDeviceToHost, c->stream));
  RUAI_CUDA(c, cudaStreamSynchronize(c->stream));
  if (st == 0) return RUAI_OK;
  cudaMemsetAsync(c->status, 0, sizeof(int), c->stream);
  if (c->ps_sync) {  // a persistent launch that gave up leaves its barrier count undefined: start over
    cudaMemsetAsync(c->ps_sync, 0, 64, c->stream);
    c->ps_bar_base = 0;
  }
  if (st == 5) return ruai_fail(c, RUAI_ERR_SHAPE, "a decode step was launched at a position beyond the cache capacity; nothing was written there");
  return ruai_fail(c, RUAI_ERR_TIMEOUT, "a bounded wait inside a kernel ran out (status %d); results of that launch are invalid", st);
}

RUAI_API int ruai_ctx_synchronize(ruai_ctx* c) {
  if (!c) return ruai_fail(nullptr, RUAI_ERR_ARG, "ctx is NULL");
  DeviceGuard g(c->ordinal);
  return ruai_ctx_check_status(c);
}

// ---- ruai_malloc / ruai_free ----------------------------------------------------------------
//
// A program makes a tensor per call and drops it soon after; cudaMalloc and cudaFree between launches cost more than most Linears
// (int8 2048 x 2048, one row: 7 us on the device of 25 a call; 4096 x 14336 results: 0.9 ms of mapping and unmapping).  Freed blocks
// are kept for the next request of their size class.  cudaFree waits for the device, so a block may be freed while a kernel on ANY
// stream still uses it; here it is set aside, and given out only after its context's stream and then the device have been waited for,
// once for all the blocks set aside until then, when so many of the wanted class lie waiting that it pays.
// At most kPoolBytes are kept per device; they are given back when memory runs short and with the device's last context.
namespace {

constexpr size_t kPoolBytes = 512ull << 20;
constexpr int kPoolDevices = 64;

struct Pool {
  std::mutex lock;
  std::unordered_map<void*, size_t> live;         // blocks handed out, by size class
  std::map<size_t, std::vector<void*>> clean;     // nothing on the device uses them
  std::map<ruai_ctx*, std::map<size_t, std::vector<void*>>> aside;  // freed through a context since its last device-wide wait
  size_t bytes = 0;                               // in clean and aside
  int contexts = 0;
};
Pool& pool_of(int ordinal) {
  static Pool* pools = new Pool[kPoolDevices];  // never destroyed: the driver may be gone before static destructors run
  return pools[ordinal];
}
bool pooled(int ordinal) { return ordinal >= 0 && ordinal < kPoolDevices; }

size_t size_class(size_t bytes) {
  if (bytes > (1ull << 20)) return (bytes + (2ull << 20) - 1) / (2ull << 20) * (2ull << 20);
  size_t c = 512;
  while (c < bytes) c *= 2;
  return c;
}
// Waits for the context's stream and the device and makes the blocks set aside through the context before that clean.  The wait is
// cudaFree's, which other threads' captures allow as they allow any cudaFree.
bool pool_settle(ruai_ctx* c, Pool& p) {
  std::map<size_t, std::vector<void*>> moved;
  {
    std::lock_guard<std::mutex> g(p.lock);
    moved.swap(p.aside[c]);
  }
  void* dummy = nullptr;
  const bool ok = cudaStreamSynchronize(c->stream) == cudaSuccess && cudaMalloc(&dummy, 512) == cudaSuccess && cudaFree(dummy) == cudaSuccess;
  if (!ok) (void)cudaGetLastError();
  std::lock_guard<std::mutex> g(p.lock);
  for (auto& kv : moved) {
    std::vector<void*>& to = ok ? p.clean[kv.first] : p.aside[c][kv.first];
    to.insert(to.end(), kv.second.begin(), kv.second.end());
  }
  return ok;
}
void pool_trim(Pool& p) {
  std::vector<void*> out;
  {
    std::lock_guard<std::mutex> g(p.lock);
    auto all = [&](std::map<size_t, std::vector<void*>>& m) {
      for (auto& kv : m) out.insert(out.end(), kv.second.begin(), kv.second.end());
      m.clear();
    };
    all(p.clean);
    for (auto& kv : p.aside) all(kv.second);
    p.bytes = 0;
  }
  for (void* q : out) cudaFree(q);  // waits for the device
}
void* pool_take(Pool& p, size_t cls) {
  std::lock_guard<std::mutex> g(p.lock);
  auto it = p.clean.find(cls);
  if (it == p.clean.end() || it->second.empty()) return nullptr;
  void* q = it->second.back();
  it->second.pop_back();
  p.bytes -= cls;
  p.live[q] = cls;
  return q;
}

}  // namespace

// What was set aside through a context that goes is freed.
static void ruai_pool_forget(ruai_ctx* c) {
  if (!pooled(c->ordinal)) return;
  Pool& p = pool_of(c->ordinal);
  std::map<size_t, std::vector<void*>> moved;
  {
    std::lock_guard<std::mutex> g(p.lock);
    auto it = p.aside.find(c);
    if (it == p.aside.end()) return;
    moved.swap(it->second);
    p.aside.erase(it);
    for (auto& kv : moved) p.bytes -= kv.first * kv.second.size();
  }
  for (auto& kv : moved)
    for (void* q : kv.second) cudaFree(q);
}

static void ruai_pool_contexts(int ordinal, int change) {
  if (!pooled(ordinal)) return;
  Pool& p = pool_of(ordinal);
  bool last;
  {
    std::lock_guard<std::mutex> g(p.lock);
    p.contexts += change;
    last = p.contexts == 0;
  }
  if (last) pool_trim(p);
}

// cudaMalloc on the current device that gives the kept blocks back before it reports that memory has run out.
cudaError_t ruai_device_malloc(void** out, size_t bytes) {
  cudaError_t e = cudaMalloc(out, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  int ordinal = 0;
  if (cudaGetDevice(&ordinal) != cudaSuccess || !pooled(ordinal)) return e;
  Pool& p = pool_of(ordinal);
  {
    std::lock_guard<std::mutex> g(p.lock);
    if (p.bytes == 0) return e;
  }
  (void)cudaGetLastError();
  pool_trim(p);
  return cudaMalloc(out, bytes);
}

RUAI_API int ruai_malloc(ruai_ctx* c, size_t bytes, void** out) {
  if (!c || !out) return ruai_fail(c, RUAI_ERR_ARG, "ruai_malloc: NULL argument");
  DeviceGuard g(c->ordinal);
  *out = nullptr;
  if (!pooled(c->ordinal) || bytes > kPoolBytes / 2) {
    RUAI_CUDA(c, ruai_device_malloc(out, bytes ? bytes : 1));
    return RUAI_OK;
  }
  Pool& p = pool_of(c->ordinal);
  const size_t cls = size_class(bytes);
  if ((*out = pool_take(p, cls)) != nullptr) return RUAI_OK;
  size_t waiting = 0;
  {
    std::lock_guard<std::mutex> l(p.lock);
    auto& mine = p.aside[c];
    auto it = mine.find(cls);
    if (it != mine.end()) waiting = it->second.size();
  }
  // Until then new ones are mapped, which costs hundreds of microseconds for a large block: two of those do.
  if (waiting >= 32 || (waiting * cls >= (4ull << 20) && (waiting >= 2 || cls >= (64ull << 20)))) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &st) != cudaSuccess) (void)cudaGetLastError();
    if (st == cudaStreamCaptureStatusNone && pool_settle(c, p) && (*out = pool_take(p, cls)) != nullptr) return RUAI_OK;
  }
  RUAI_CUDA(c, ruai_device_malloc(out, cls));
  std::lock_guard<std::mutex> l(p.lock);
  p.live[*out] = cls;
  return RUAI_OK;
}

RUAI_API int ruai_free(ruai_ctx* c, void* p) {
  if (!c) return ruai_fail(nullptr, RUAI_ERR_ARG, "ctx is NULL");
  DeviceGuard g(c->ordinal);
  bool kept = false, full = false;
  if (p && pooled(c->ordinal)) {
    Pool& pool = pool_of(c->ordinal);
    std::lock_guard<std::mutex> l(pool.lock);
    auto it = pool.live.find(p);
    if (it != pool.live.end()) {
      const size_t cls = it->second;
      pool.live.erase(it);
      pool.aside[c][cls].push_back(p);
      pool.bytes += cls;
      full = pool.bytes > kPoolBytes;
      kept = true;
    }
  }
  if (kept) {
    if (full) pool_trim(pool_of(c->ordinal));  // of sizes no longer asked for, most of it
    return RUAI_OK;
  }
  RUAI_CUDA(c, cudaStreamSynchronize(c->stream));
  RUAI_CUDA(c, cudaFree(p));
  return RUAI_OK;
}

RUAI_API int ruai_memcpy_h2d(ruai_ctx* c, void* dst, const void* src, size_t bytes) {
  if (!c) return ruai_fail(nullptr, RUAI_ERR_ARG, "ctx is NULL");
  DeviceGuard g(c->ordinal);
  RUAI_CUDA(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->stream));
  RUAI_CUDA(c, cudaStreamSynchronize(c->stream));
  return RUAI_OK;
}

RUAI_API int ruai_memcpy_d2h(ruai_ctx* c, void* dst, const void* src, size_t bytes) {
  if (!c) return ruai_fail(nullptr, RUAI_ERR_ARG, "ctx is NULL");
  DeviceGuard g(c->ordinal);
  RUAI_CUDA(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
  RUAI_CUDA(c, cudaStreamSynchronize(c->stream));
  return RUAI_OK;
}

RUAI_API int ruai_timer_start(ruai_ctx* c) {
  if (!c) return ruai_fail(nullptr, RUAI_ERR_ARG, "ctx is NULL");
  RUAI_CUDA(c, cudaEventRecord(c->ev0, c->stream));
  return RUAI_OK;
}

RUAI_API int ruai_timer_stop_ms(ruai_ctx* c, float* ms) {
  if (!c || !ms) return ruai_fail(c, RUAI_ERR_ARG, "NULL argument");
  RUAI_CUDA(c, cudaEventRecord(c->ev1, c->stream));
  RUAI_CUDA(c, cudaEventSynchronize(c->ev1));
  RUAI_CUDA(c, cudaEventElapsedTime(ms, c->ev0, c->ev1));
  return RUAI_OK;
}

// Tuning knob: the split-k count of the tensor-core GEMVs (0 = the chooser decides).
RUAI_API int ruai_ctx_force_splits(ruai_ctx* c, unsigned splits) {
  if (!c) return ruai_fail(c, RUAI_ERR_ARG, "NULL argument");
  if (splits > 8) return ruai_fail(c, RUAI_ERR_ARG, "splits %u: 0 (automatic) or 1..8", splits);
  c->force_splits = splits;
  return RUAI_OK;
}

// Profiling hooks, present only in builds made with RUAI_B200_TRACE=1 (never in the library as shipped).
#ifdef RUAI_B200_TRACE
RUAI_API int ruai_debug_force_splits(ruai_ctx* c, unsigned splits) {  // also the profiling bits above the count
  c->force_splits = splits;
  return RUAI_OK;
}

RUAI_API int ruai_debug_trace(ruai_ctx* c, void* dev_buf, unsigned slots) {
  c->trace = (unsigned long long*)dev_buf;
  c->trace_slots = slots;
  c->trace_seq = 0;
  return RUAI_OK;
}
#endif
