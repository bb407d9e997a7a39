// Device memory of ruai_malloc / ruai_free (ctx.cu): blocks given back are kept for later requests of their size.  Host code that needs
// nothing but the CUDA runtime's interface, so that it can be run against a stand-in for it.
//
// A program makes a tensor per call and drops it soon after; cudaMalloc and cudaFree between launches cost more than most Linears
// (int8 2048 x 2048, one row: 7 us on the device of 25 a call; 4096 x 14336 results: 0.9 ms of mapping and unmapping).  Freed blocks
// are kept for the next request of their size class.  A block may be freed while a kernel on ANY stream still uses it, as cudaFree lets a
// caller do; it is set aside, and given out only after a cudaDeviceSynchronize, once for all the blocks set aside until then, when so
// many of the wanted class lie waiting that it pays.  (A cudaFree in its place would do as a wait only by a side effect that CUDA does not
// promise.  Where a capture forbids the wait it forbids the cudaMalloc that a request would come to otherwise.)
// At most kKeptBytes are kept per device; they are given back when memory runs short and with the device's last context.
// While a stream of the device's contexts is being captured, nothing is kept or given out: a graph uses its memory whenever it is
// replayed, which no wait sees, so what is freed then is for the driver to refuse, as cudaFree after a wait for the stream does.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <list>
#include <map>
#include <mutex>
#include <new>
#include <unordered_map>
#include <utility>

namespace block_pool {

constexpr size_t kKeptBytes = 512ull << 20;
constexpr int kDevices = 64;

using Blocks = std::map<size_t, std::list<void*>>;  // by size class

struct Block {
  size_t cls;
  int ordinal;
  bool kept;  // in clean or aside, not with a caller
};
struct Pool {  // of a device
  Blocks clean;                            // nothing on the device uses them
  Blocks aside;                            // freed since the last device-wide wait
  size_t bytes = 0;                        // in clean, in aside and on the way from one to the other
  std::mutex settling;                     // held while blocks are on that way: whoever wants all that is kept waits for them; taken before the lock
  std::map<const void*, cudaStream_t> contexts;
};
struct State {
  std::mutex lock;  // held for bookkeeping, not for a wait or a call that maps or unmaps memory
  // Every block of this file's making that has not gone back to the driver: a block may come back through a context of another device, and
  // one that lies here must not come back a second time (the driver counts it as allocated, so cudaFree would take it).
  std::unordered_map<void*, Block> blocks;
  Pool device[kDevices];
};
inline State& state() {
  static State* s = new State;  // never destroyed: the driver may be gone before static destructors run
  return *s;
}
using Lock = std::lock_guard<std::mutex>;
inline Pool& of(int ordinal) { return state().device[ordinal]; }
inline bool pooled(int ordinal) { return ordinal >= 0 && ordinal < kDevices; }

inline size_t size_class(size_t bytes) {
  if (bytes > (1ull << 20)) return (bytes + (2ull << 20) - 1) / (2ull << 20) * (2ull << 20);
  size_t c = 512;
  while (c < bytes) c *= 2;
  return c;
}

inline void forget(const Blocks& all) {  // the lock is held, the blocks are about to be freed
  for (auto& kv : all)
    for (void* q : kv.second) state().blocks.erase(q);
}

inline void merge(Blocks& to, Blocks& from) {
  while (!from.empty()) {  // of nodes that exist: nothing here can throw
    auto node = from.extract(from.begin());
    auto it = to.find(node.key());
    if (it == to.end()) to.insert(std::move(node));
    else it->second.splice(it->second.end(), node.mapped());
  }
}

// Waits for the device and makes the blocks set aside before that clean.
inline bool settle(Pool& p) {
  Lock way(p.settling);
  Blocks moved;
  {
    Lock l(state().lock);
    moved.swap(p.aside);
  }
  if (moved.empty()) return true;  // another thread has just waited
  const bool ok = cudaDeviceSynchronize() == cudaSuccess;
  if (!ok) (void)cudaGetLastError();
  Lock l(state().lock);
  merge(ok ? p.clean : p.aside, moved);
  return ok;
}

inline void trim(Pool& p) {
  Lock way(p.settling);
  Blocks out;
  {
    Lock l(state().lock);
    merge(out, p.clean);
    merge(out, p.aside);
    for (auto& kv : out) p.bytes -= kv.first * kv.second.size();
    forget(out);
  }
  if (out.empty()) return;
  if (cudaDeviceSynchronize() != cudaSuccess) (void)cudaGetLastError();
  for (auto& kv : out)
    for (void* q : kv.second) cudaFree(q);
}

// Whether a stream of the device's contexts is being captured, or cannot be asked.  The lock is held, so that none of them goes meanwhile.
inline bool capturing(const Pool& p) {
  bool any = false;
  for (auto& kv : p.contexts) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(kv.second, &st) != cudaSuccess) {
      (void)cudaGetLastError();
      any = true;
    }
    any = any || st != cudaStreamCaptureStatusNone;
  }
  return any;
}

inline void* take(Pool& p, size_t cls) {  // the lock is held
  auto it = p.clean.find(cls);
  if (it == p.clean.end() || it->second.empty()) return nullptr;
  void* q = it->second.back();
  it->second.pop_back();
  p.bytes -= cls;
  auto b = state().blocks.find(q);
  if (b == state().blocks.end()) return nullptr;  // a caller gave it to cudaFree after ruai_free
  b->second.kept = false;
  return q;
}

// A context of the device more; the device's last one to go gives the kept memory back.
// false: the host is out of memory.  (Callers of the C interface cannot catch what the containers throw.)
inline bool attach(const void* context, int ordinal, cudaStream_t stream) {
  if (!pooled(ordinal)) return true;
  try {
    Lock l(state().lock);
    of(ordinal).contexts[context] = stream;
  } catch (const std::bad_alloc&) {
    return false;
  }
  return true;
}
inline void detach(const void* context, int ordinal) {
  if (!pooled(ordinal)) return;
  Pool& p = of(ordinal);
  bool last;
  {
    Lock l(state().lock);
    p.contexts.erase(context);
    last = p.contexts.empty();
  }
  if (last) trim(p);
}

// cudaMalloc on the current device that gives the kept blocks back before it reports that memory has run out.
inline cudaError_t device_malloc(void** out, size_t bytes) {
  cudaError_t e = cudaMalloc(out, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  int ordinal = 0;
  if (cudaGetDevice(&ordinal) != cudaSuccess || !pooled(ordinal)) return e;
  Pool& p = of(ordinal);
  {
    Lock l(state().lock);
    if (p.bytes == 0) return e;
  }
  (void)cudaGetLastError();
  trim(p);
  return cudaMalloc(out, bytes);
}

// A block on a device, which is current.
inline cudaError_t allocate(int ordinal, size_t bytes, void** out) {
  if (!pooled(ordinal) || bytes > kKeptBytes / 2) {
    const cudaError_t e = device_malloc(out, bytes ? bytes : 1);
    if (e != cudaSuccess) return e;
    Lock l(state().lock);
    state().blocks.erase(*out);  // left by a caller that gave a block of ours to cudaFree itself
    return cudaSuccess;
  }
  Pool& p = of(ordinal);
  const size_t cls = size_class(bytes);
  size_t waiting = 0;
  {
    Lock l(state().lock);
    if (!capturing(p)) {
      if ((*out = take(p, cls)) != nullptr) return cudaSuccess;
      auto it = p.aside.find(cls);
      if (it != p.aside.end()) waiting = it->second.size();
    }
  }
  // Until then new ones are mapped.  Small blocks: 32, since a wait stops the host's lead over the device (one-row int8 Linear of 2048 x
  // 2048, us a call: 9.5 after 8 blocks, 9.2 after 16, 8.8 after 32, 8.6 after 64; the first 400 calls, which map them, 14 with any of
  // these).  Mapping costs hundreds of microseconds for a large one, so two of 4 MB in all do (results of 11 MB: 46.7 after one, 42.5
  // after two, 40.5 after four, which is twice the memory), and one of 64 MB, of which no more than eight could be kept.
  if (waiting >= 32 || (waiting * cls >= (4ull << 20) && (waiting >= 2 || cls >= (64ull << 20))))
    if (settle(p)) {
      Lock l(state().lock);
      if ((*out = take(p, cls)) != nullptr) return cudaSuccess;
    }
  const cudaError_t e = device_malloc(out, cls);
  if (e != cudaSuccess) return e;
  try {
    Lock l(state().lock);
    state().blocks[*out] = {cls, ordinal, false};
  } catch (const std::bad_alloc&) {  // not in the book: its ruai_free is cudaFree's
  }
  return cudaSuccess;
}

// Frees a block on behalf of a context of a device, which is current, on its stream.
inline cudaError_t give_back(int ordinal, cudaStream_t stream, void* q) {
  bool kept = false, full = false;
  {
    Lock l(state().lock);
    auto it = state().blocks.find(q);
    if (it != state().blocks.end()) {
      if (it->second.kept) return cudaErrorInvalidValue;  // freed already: cudaFree's answer
      if (it->second.ordinal == ordinal && !capturing(of(ordinal))) {
        Pool& p = of(ordinal);
        try {
          p.aside[it->second.cls].push_back(q);
          p.bytes += it->second.cls;
          it->second.kept = kept = true;
          full = p.bytes > kKeptBytes;
        } catch (const std::bad_alloc&) {  // then it goes back to the driver
        }
      }
    }
  }
  if (full) trim(of(ordinal));  // of sizes no longer asked for, most of it
  if (kept) return cudaSuccess;
  cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();  // it is reported here, and not by the next launch's check as well
    return e;
  }
  std::unordered_map<void*, Block>::node_type entry;
  {
    Lock l(state().lock);
    entry = state().blocks.extract(q);  // before another thread can be given the address
  }
  e = cudaFree(q);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    Lock l(state().lock);
    if (entry) state().blocks.insert(std::move(entry));
  }
  return e;
}

}  // namespace block_pool
