// Device memory of the engine: growing buffers, and the pool of the instance
// that the C API drives; and its page-locked host memory.
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>

#include <memory>
#include <utility>
#include <vector>

namespace tb {

// Whether a kernel on device `dev` may work on a caller's array at p: device
// memory of that device, aligned for its elements.  Anything else (another
// GPU's memory, which needs peer access, managed or host memory) is left to
// copies, which reach it without.
inline bool kernel_reaches(const cudaPointerAttributes& a, int dev, const void* p, size_t align) {
  return a.type == cudaMemoryTypeDevice && a.device == dev && reinterpret_cast<uintptr_t>(p) % align == 0;
}
inline bool kernel_reaches(const void* p, int dev, size_t align) {
  cudaPointerAttributes a = {};
  if (!p || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return kernel_reaches(a, dev, p, align);
}

// Whether a host array is page-locked (from its first byte to its last).
inline bool page_locked(const void* p, size_t bytes) {
  for (const char* c : {static_cast<const char*>(p), static_cast<const char*>(p) + (bytes ? bytes - 1 : 0)}) {
    cudaPointerAttributes a = {};
    if (!p || cudaPointerGetAttributes(&a, c) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (a.type != cudaMemoryTypeHost) return false;
  }
  return true;
}

// Device bytes of the engine whose calls this thread is running (the
// serving form's admission accounting); null: not counted.
extern thread_local long long* g_dbuf_account;
// When set, buffers are allocated and freed stream-ordered on this stream
// (cudaMallocAsync / cudaFreeAsync), so engines that run side by side on their
// own streams never wait for each other's frees; null: cudaMalloc / cudaFree.
extern thread_local cudaStream_t g_dbuf_stream;
// With g_dbuf_stream: the pool the stream-ordered allocations come from
// (null: the device's current pool).
extern thread_local cudaMemPool_t g_dbuf_pool;

// Device memory of one engine: a memory pool of its own, for the instance that
// the C API drives.  A new mesh needs about 200 buffers, which cost 90 us each
// with cudaMalloc and 80 us with cudaFree; the pool maps device memory in
// larger pieces (a new mesh of 450 k nodes from registration to its first data
// update and the end of the instance, medians of 30: 53 to 57 ms without a pool,
// 25 to 28 with it).  It is made for the first buffer, as a solver's set-up may
// end before that, keeps up to kKeep bytes that no buffer uses, and goes back to
// the device with the engine's last buffer.
//
// Buffers of kDirect and more come from the device directly: mapping them is
// what they cost, and a pool that gives back what it does not use maps some of
// it again (18.6 M nodes, first preprocess, first call and the instance's end,
// medians: 238 to 292, 18 to 21 and 60 to 63 ms all from the pool, 194 to 220, 16
// and 33 to 42 so; 218 to 228, 24 and 42 to 47 without a pool; with 16 or 256 MB
// as the line 199 to 216 and 38 to 42).
//
// A buffer may be used on any of the streams that the engine's work runs on
// (users).  It goes back to the pool, on the pool's own stream, after
// everything that is on them when it is let go: nothing is handed out again
// while a kernel may still read it, and no other work on the device is waited
// for.  Where that order cannot be had (a user stream is being captured), the
// buffer is held until it can.
struct DevPool {
  static constexpr uint64_t kKeep = 512ull << 20;
  static constexpr size_t kDirect = 64ull << 20;
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;
  cudaEvent_t ev = nullptr;
  int device = -1;
  std::vector<cudaStream_t> users;  // (empty: nothing of the engine is running any more)
  std::vector<void*> held;          // let go, and not back in the pool yet
  bool made = false;
  DevPool() = default;
  void make() {
    made = true;
    if (cudaGetDevice(&device) != cudaSuccess) return;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    uint64_t keep = kKeep;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) pool = nullptr;
    if (pool && (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
                 cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
                 cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess)) {
      if (st) cudaStreamDestroy(st);
      cudaMemPoolDestroy(pool);
      pool = nullptr;
    }
    if (!pool) cudaGetLastError();
  }
  ~DevPool() {
    if (!pool) return;
    give_back();
    cudaStreamSynchronize(st);
    cudaMemPoolDestroy(pool);
    cudaEventDestroy(ev);
    cudaStreamDestroy(st);
  }
  DevPool(const DevPool&) = delete;
  DevPool& operator=(const DevPool&) = delete;
  // false: the caller asks the device directly (which, when the pool had no
  // room, then has what it did not use)
  bool alloc(void** p, size_t bytes) {
    if (bytes >= kDirect) return false;
    if (!made) make();
    int d = -1;
    if (!pool || cudaGetDevice(&d) != cudaSuccess || d != device) return false;
    give_back();
    if (cudaMallocFromPoolAsync(p, bytes, pool, st) == cudaSuccess) {
      if (cudaStreamSynchronize(st) == cudaSuccess) return true;
      cudaFreeAsync(*p, st);
    }
    cudaGetLastError();
    cudaMemPoolTrimTo(pool, 0);
    return false;
  }
  void free(void* p) {
    held.push_back(p);
    give_back();
  }

 private:
  void give_back() {
    if (held.empty() || !after_users()) return;
    for (void* p : held) cudaFreeAsync(p, st);
    held.clear();
  }
  // the pool's stream goes on after everything on the users' streams
  bool after_users() {
    for (cudaStream_t s : users) {
      cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;  // (an event of a capture would draw st into it)
      if (cudaStreamIsCapturing(s, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone ||
          cudaEventRecord(ev, s) != cudaSuccess || cudaStreamWaitEvent(st, ev, 0) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
    }
    return true;
  }
};
// The pool of the instance whose calls this thread makes; empty, or with
// g_dbuf_stream: none.
extern thread_local std::weak_ptr<DevPool> g_dbuf_dev;

template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  long long* acct = nullptr;  // where this allocation is counted
  cudaStream_t st = nullptr;  // stream-ordered allocation: its stream
  bool async = false;
  std::shared_ptr<DevPool> dev;  // or: the pool it comes from
  DBuf() = default;
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept { swap(o); }
  DBuf& operator=(DBuf&& o) noexcept {
    swap(o);
    return *this;
  }
  ~DBuf() { release(); }
  void swap(DBuf& o) {
    std::swap(p, o.p);
    std::swap(n, o.n);
    std::swap(acct, o.acct);
    std::swap(st, o.st);
    std::swap(async, o.async);
    std::swap(dev, o.dev);
  }
  cudaError_t ensure(size_t count) {
    if (count <= n && p) return cudaSuccess;
    // a buffer that has to grow again gets a quarter more, so slowly growing
    // sizes (moving meshes) do not reallocate every call
    const size_t grow = (p && count) ? count / 4 : 0;
    release();
    size_t c = count ? count + grow : 1;
    const size_t bytes = c * sizeof(T);
    async = g_dbuf_stream != nullptr;
    st = g_dbuf_stream;
    if (!async) dev = g_dbuf_dev.lock();
    if (dev && !dev->alloc((void**)&p, bytes)) dev.reset();
    cudaError_t e = dev           ? cudaSuccess
                    : !async      ? cudaMalloc((void**)&p, bytes)
                    : g_dbuf_pool ? cudaMallocFromPoolAsync((void**)&p, bytes, g_dbuf_pool, st)
                                  : cudaMallocAsync((void**)&p, bytes, st);
    if (e == cudaSuccess) {
      n = c;
      acct = g_dbuf_account;
      if (acct) *acct += (long long)bytes;
    } else {
      p = nullptr;
    }
    return e;
  }
  void release() {
    if (p) {
      if (dev) dev->free(p);
      else if (async) cudaFreeAsync(p, st);
      else cudaFree(p);
      if (acct) *acct -= (long long)(n * sizeof(T));
    }
    p = nullptr;
    n = 0;
    acct = nullptr;
    async = false;
    dev.reset();
    st = nullptr;
  }
};

// One page-locked host allocation of an engine, for the small buffers below
// and the data update's slots: an allocation takes 2.4 ms whatever its size up to
// 2 MB, and 0.45 ms to free (three of them were a tenth of a new mesh's way from
// its registration to the end of its instance).
struct PinArena {
  static constexpr size_t kBytes = 2u << 20, kSlots = 3u << 19;  // the slots' share of it at the end
  char* p = nullptr;
  size_t used = 0;
  cudaError_t make() {
    if (p) return cudaSuccess;
    const cudaError_t e = cudaMallocHost((void**)&p, kBytes);
    if (e != cudaSuccess) p = nullptr;
    return e;
  }
  // a piece before the slots, null where none is left
  char* take(size_t bytes) {
    if (bytes > kBytes - kSlots - used || make() != cudaSuccess) return nullptr;
    char* q = p + used;
    used += (bytes + 255) / 256 * 256;
    return q;
  }
  char* slots() { return make() == cudaSuccess ? p + (kBytes - kSlots) : nullptr; }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    used = 0;
  }
};

// Page-locked host memory that grows: copies to and from it do not hold the
// host (a 4-byte read-back into pageable memory costs 14 us, into this 5).
// From the arena while that has room (a piece that was outgrown stays there).
struct PinBuf {
  char* p = nullptr;
  size_t n = 0;
  bool own = false;
  cudaError_t ensure(size_t bytes, PinArena& arena) {
    if (bytes <= n) return cudaSuccess;
    release();
    const size_t c = bytes + bytes / 2 + 4096;
    cudaError_t e = cudaSuccess;
    if (!(p = arena.take(c))) {
      e = cudaMallocHost((void**)&p, c);
      own = e == cudaSuccess;
    }
    if (e == cudaSuccess) n = c;
    else p = nullptr;
    return e;
  }
  void release() {
    if (own) cudaFreeHost(p);
    p = nullptr;
    n = 0;
    own = false;
  }
};

}  // namespace tb
