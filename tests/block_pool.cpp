// Runs block_pool.cuh against a stand-in for the CUDA runtime: addresses without memory behind them, streams that can be capturing,
// and work that goes on until the device is waited for.  One scenario per run; exit status 0: it held.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <future>
#include <set>
#include <string>
#include <vector>

#include <new>

#include "../ruai_b200/csrc/block_pool.cuh"

#define CHECK(c)                                                     \
  do {                                                               \
    if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } \
  } while (0)

// Operator new that can be told to fail.
static bool host_memory_out = false;
void* operator new(size_t n) {
  void* p = host_memory_out ? nullptr : std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

namespace fake {
struct Host {  // the stand-in's own containers are not what fails
  bool was = host_memory_out;
  Host() { host_memory_out = false; }
  ~Host() { host_memory_out = was; }
};
std::mutex lock;
std::map<char*, size_t> memory;      // what the driver has handed out
std::vector<std::pair<char*, size_t>> freed;  // addresses to hand out again, last first
size_t limit = ~(size_t)0, used = 0, waits = 0;
std::set<cudaStream_t> capturing, spoiled;
std::set<void*> busy;                // work that is still going on reads or writes it
std::function<void()> during_wait;
cudaError_t last = cudaSuccess;
char* next = (char*)0x1000000;
void wait() {
  if (!during_wait) return;
  auto f = during_wait;
  during_wait = nullptr;
  f();
}
cudaStream_t stream(int i) { return (cudaStream_t)(size_t)(16 + i); }
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** out, size_t bytes) {
  const fake::Host h;
  std::lock_guard<std::mutex> g(fake::lock);
  if (fake::used + bytes > fake::limit) return cudaErrorMemoryAllocation;
  char* at = fake::next;
  auto same = std::find_if(fake::freed.rbegin(), fake::freed.rend(), [&](auto& f) { return f.second >= bytes; });
  if (same != fake::freed.rend()) { at = same->first; fake::freed.erase(std::next(same).base()); }
  else fake::next += (bytes + 4095) / 4096 * 4096;
  fake::memory[at] = bytes;
  fake::used += bytes;
  *out = at;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {  // may wait for the device, or not
  const fake::Host h;
  std::lock_guard<std::mutex> g(fake::lock);
  if (fake::busy.count(p)) { std::printf("memory in use goes back to the driver\n"); std::exit(1); }
  if (!p) return cudaSuccess;
  auto it = fake::memory.find((char*)p);
  if (it == fake::memory.end()) return fake::last = cudaErrorInvalidValue;
  fake::used -= it->second;
  fake::freed.push_back(*it);
  fake::memory.erase(it);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  fake::wait();
  if (fake::capturing.count(s)) { fake::spoiled.insert(s); return fake::last = cudaErrorStreamCaptureUnsupported; }
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) {
  ++fake::waits;
  fake::wait();
  fake::busy.clear();
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
  *st = fake::capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
}

using namespace block_pool;

struct Context {  // what ctx.cu makes of a ruai_ctx
  int ordinal;
  cudaStream_t stream;
  explicit Context(int i, int ordinal_ = 0) : ordinal(ordinal_), stream(fake::stream(i)) { CHECK(attach(this, ordinal, stream)); }
  ~Context() { detach(this, ordinal); }
  void* get(size_t bytes) {
    void* p = nullptr;
    return allocate(ordinal, bytes, &p) == cudaSuccess ? p : nullptr;
  }
  cudaError_t put(void* p) { return give_back(ordinal, stream, p); }
};
constexpr size_t MB = 1 << 20;

// Requests of this size until one comes from the blocks kept.
void* reused(Context& c, size_t bytes) {
  std::set<void*> seen;
  for (int i = 0; i < 200; ++i) {
    void* p = c.get(bytes);
    CHECK(p);
    if (!seen.insert(p).second) return p;
    c.put(p);
  }
  return nullptr;
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "reuse") {
    Context c(0);
    for (size_t bytes : {size_t(1), size_t(4096), MB, 3 * MB, 200 * MB}) CHECK(reused(c, bytes));
    const size_t used = fake::used;
    CHECK(c.put(c.get(300 * MB)) == cudaSuccess && fake::used == used);  // too large to be kept
  } else if (what == "last context") {
    {
      Context a(0);
      { Context b(1); b.put(b.get(MB)); a.put(a.get(4 * MB)); }
      a.put(a.get(MB));
    }
    CHECK(fake::memory.empty());
  } else if (what == "limit") {
    Context c(0);
    std::vector<void*> all;
    for (int i = 0; i < 40; ++i) all.push_back(c.get(32 * MB));
    for (void* p : all) {
      CHECK(c.put(p) == cudaSuccess);
      size_t kept = 0;
      for (auto& m : fake::memory) kept += m.second;
      size_t out = 0;
      for (void* q : all) out += q > p ? 32 * MB : 0;
      CHECK(kept - out <= kKeptBytes);
    }
  } else if (what == "out of memory") {
    Context c(0);
    fake::limit = 300 * MB;
    std::vector<void*> all;
    for (int i = 0; i < 8; ++i) all.push_back(c.get(32 * MB));
    for (void* p : all) c.put(p);
    CHECK(c.get(250 * MB));                       // what is kept makes room
    CHECK(!c.get(250 * MB));
    void* p = nullptr;
    CHECK(device_malloc(&p, 40 * MB) == cudaSuccess);
  } else if (what == "free in a capture") {       // the graph goes on using the block after the capture
    Context c(0);
    void* p = c.get(4096);
    fake::capturing.insert(c.stream);
    CHECK(c.put(p) != cudaSuccess);
    CHECK(fake::spoiled.count(c.stream) && fake::last == cudaSuccess);  // the error is reported once
    fake::capturing.clear();
    for (int i = 0; i < 100; ++i) {
      void* q = c.get(4096);
      CHECK(q != p && c.put(q) == cudaSuccess);
    }
    CHECK(c.put(p) == cudaSuccess);               // after the capture it is a block like any other
  } else if (what == "capture of another context") {
    Context a(0), b(1);
    void* p = a.get(4096);
    fake::capturing.insert(b.stream);
    CHECK(a.put(p) == cudaSuccess && !fake::memory.count((char*)p));  // to the driver, which may refuse it
    fake::capturing.clear();
    CHECK(a.put(a.get(4096)) == cudaSuccess && !fake::memory.empty());
  } else if (what == "request in a capture") {
    Context c(0);
    std::vector<void*> all;
    for (int i = 0; i < 40; ++i) all.push_back(c.get(4096));
    for (void* q : all) c.put(q);
    c.put(reused(c, 4096));
    const size_t used = fake::used;
    fake::capturing.insert(c.stream);
    CHECK(c.get(4096) && fake::used > used);      // the driver's answer, whatever it is
  } else if (what == "freed twice") {
    Context c(0), d(1);
    void* p = c.get(4096);
    CHECK(c.put(p) == cudaSuccess);
    CHECK(c.put(p) != cudaSuccess && d.put(p) != cudaSuccess && fake::memory.count((char*)p));
    CHECK(reused(c, 4096));                       // the same once it is clean
    std::vector<void*> all;
    for (int i = 0; i < 40; ++i) all.push_back(c.get(4096));
    for (void* q : all) CHECK(c.put(q) == cudaSuccess);
    for (void* q : all) CHECK(c.put(q) != cudaSuccess && fake::memory.count((char*)q));
    CHECK(c.put((void*)0x10) != cudaSuccess && fake::last == cudaSuccess);  // not allocated at all: cudaFree's error
  } else if (what == "freed through another device") {
    Context a(0, 0), b(1, 1);
    void* p = a.get(4096);
    CHECK(b.put(p) == cudaSuccess && !fake::memory.count((char*)p));
    void* q = nullptr;
    CHECK(cudaMalloc(&q, 4096) == cudaSuccess && q == p);  // another owner of the address
    CHECK(a.put(q) == cudaSuccess && !fake::memory.count((char*)q));
  } else if (what == "address of a block that cudaFree took") {
    Context c(0);
    void* p = c.get(4 * MB);
    cudaFree(p);
    fake::freed = {{(char*)p, 300 * MB}};
    void* q = c.get(300 * MB);
    CHECK(q == p && c.put(q) == cudaSuccess && !fake::memory.count((char*)q));
  } else if (what == "trim during a wait" || what == "out of memory during a wait") {
    Context a(0), b(1);
    std::vector<void*> mine, others;
    for (int i = 0; i < 4; ++i) mine.push_back(a.get(4 * MB));
    for (int i = 0; i < 20; ++i) others.push_back(b.get(32 * MB));
    for (void* p : mine) a.put(p);
    std::future<bool> other;
    fake::during_wait = [&] {
      other = std::async(std::launch::async, [&] {
        if (what == "trim during a wait") {
          for (void* p : others) b.put(p);        // beyond the limit
          return true;
        }
        fake::limit = fake::used;
        void* p = nullptr;
        return device_malloc(&p, 4096) == cudaSuccess;  // there is memory kept
      });
      other.wait_for(std::chrono::milliseconds(300));
    };
    void* p = a.get(4 * MB);                      // waits for the device
    CHECK(other.valid() && other.get());
    fake::limit = ~(size_t)0;
    size_t out = p ? 4 * MB : 0;
    if (what != "trim during a wait") out += 20 * 32 * MB + 4096;
    CHECK(of(0).bytes == fake::used - out);
  } else if (what == "used by another stream") {  // nothing but a wait for the whole device ends that use
    Context a(0), b(1);
    for (size_t bytes : {size_t(4096), 4 * MB, 64 * MB}) {
      void* p = a.get(bytes);
      fake::busy.insert(p);
      CHECK(a.put(p) == cudaSuccess);
      for (int i = 0; i < 200; ++i) {
        void* q = (i & 1 ? a : b).get(bytes);
        CHECK(!fake::busy.count(q));
        a.put(q);
      }
      CHECK(fake::busy.empty());
    }
  } else if (what == "limit with work going on") {
    Context c(0);
    std::vector<void*> all;
    for (int i = 0; i < 40; ++i) all.push_back(c.get(32 * MB));
    for (void* p : all) {
      fake::busy.insert(p);
      c.put(p);
    }
  } else if (what == "host memory out") {         // what a C caller could not catch
    Context c(0);
    void *p = c.get(4096), *q = c.get(8192);
    host_memory_out = true;
    void* r = c.get(4096);
    const bool attached = attach(&p, 0, c.stream);
    const cudaError_t first = c.put(p), second = c.put(r);
    host_memory_out = false;
    CHECK(r && !attached && first == cudaSuccess && second == cudaSuccess);
    CHECK(!fake::memory.count((char*)p) && !fake::memory.count((char*)r) && c.put(q) == cudaSuccess);
  } else {
    std::printf("no scenario \"%s\"\n", what.c_str());
    return 2;
  }
  return 0;
}
