// DevPool and DBuf (tioga_b200/csrc/devmem.h) over a fake CUDA runtime that
// keeps each stream's order: work is queued on streams and runs only when a
// synchronise asks for it.  Prints "ok" or what went wrong.
#include <stdio.h>
#include <stdlib.h>

#include <functional>
#include <map>
#include <queue>
#include <set>

#include "devmem.h"

namespace tb {
thread_local long long* g_dbuf_account = nullptr;
thread_local cudaStream_t g_dbuf_stream = nullptr;
thread_local cudaMemPool_t g_dbuf_pool = nullptr;
thread_local std::weak_ptr<DevPool> g_dbuf_dev;
}  // namespace tb

namespace {
struct Stream {
  struct Op {
    std::function<bool()> run;  // false: not yet
  };
  std::queue<Op> ops;
  bool capturing = false;
};
struct Event {
  long long recorded = 0, reached = 0;
};
std::set<Stream*> streams;
std::set<void*> in_pool;               // handed back and not handed out again
std::map<void*, int> readers;          // kernels queued that still read a block
int bad = 0, next_block = 1, device_syncs = 0, pools = 0;

void expect(bool ok, const char* what) {
  if (!ok) {
    printf("failed: %s\n", what);
    bad++;
  }
}
bool step(Stream* s) {
  if (s->ops.empty() || !s->ops.front().run()) return false;
  s->ops.pop();
  return true;
}
cudaError_t drain(Stream* want) {  // until want is empty; every stream may go on meanwhile
  while (!want->ops.empty()) {
    bool any = false;
    for (Stream* s : streams) any = step(s) || any;
    if (!any) return cudaErrorUnknown;
  }
  return cudaSuccess;
}
Stream* S(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
// a kernel on s that reads block p
void use(cudaStream_t s, void* p) {
  readers[p]++;
  S(s)->ops.push({[p] {
    expect(!in_pool.count(p), "a block is back in the pool while a queued kernel reads it");
    readers[p]--;
    return true;
  }});
}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) {  // as while some stream of the device is being captured
  device_syncs++;
  return cudaErrorStreamCaptureUnsupported;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  Stream* n = new Stream;
  streams.insert(n);
  *s = reinterpret_cast<cudaStream_t>(n);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  streams.erase(S(s));
  delete S(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return drain(S(s)); }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
  *c = S(s)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new Event);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<Event*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  expect(!S(s)->capturing, "an event is recorded into a capture");
  Event* v = reinterpret_cast<Event*>(e);
  const long long id = ++v->recorded;
  S(s)->ops.push({[v, id] {
    if (v->reached < id) v->reached = id;
    return true;
  }});
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  Event* v = reinterpret_cast<Event*>(e);
  const long long id = v->recorded;
  S(s)->ops.push({[v, id] { return v->reached >= id; }});
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  pools++;
  *p = reinterpret_cast<cudaMemPool_t>(&pools);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { pools--; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t s) {
  // stream-ordered: what is in the pool once the frees queued on s have run
  drain(S(s));
  if (!in_pool.empty()) {
    *p = *in_pool.begin();
    in_pool.erase(in_pool.begin());
    expect(readers[*p] == 0, "a block is handed out while a queued kernel reads it");
  } else {
    *p = reinterpret_cast<void*>((size_t)next_block++ << 20);
  }
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  S(s)->ops.push({[p] {
    in_pool.insert(p);
    return true;
  }});
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t, cudaStream_t) { *p = malloc(1); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) { *p = malloc(1); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
}

int main() {
  const size_t big = 1 << 20;
  cudaStream_t main_st, side;
  cudaStreamCreateWithFlags(&main_st, 0);
  cudaStreamCreateWithFlags(&side, 0);
  auto pool = std::make_shared<tb::DevPool>();
  pool->users = {main_st, side};
  tb::g_dbuf_dev = pool;
  expect(pools == 0 && streams.size() == 2, "the pool is made before there is a buffer");
  {
    // buffers that grow while kernels of either stream still read them
    tb::DBuf<char> a, b, c;
    a.ensure(big);
    b.ensure(big);
    for (int k = 1; k < 6; k++) {
      use(main_st, a.p);
      use(side, b.p);
      a.ensure(a.n + 1);
      b.ensure(b.n + 1);
      c.release();
      c.ensure(big);
    }
    expect(device_syncs == 0, "the whole device is waited for");
    // the side stream is being captured: a buffer let go now stays out of the
    // pool, and goes back once the capture has ended
    drain(S(main_st));
    drain(S(side));
    void* last = c.p;
    use(side, last);
    S(side)->capturing = true;
    c.release();
    a.ensure(a.n + 1);
    expect(a.p != last && !in_pool.count(last), "a buffer let go during a capture is handed out");
    S(side)->capturing = false;
    b.ensure(b.n + 1);
    drain(S(pool->st));
    expect(in_pool.count(last) || b.p == last, "a buffer let go during a capture never goes back");
    drain(S(main_st));
    drain(S(side));
    S(main_st)->capturing = true;
    a.release();
    S(main_st)->capturing = false;
    pool->users.clear();  // as at the engine's end
    // large buffers do not come from the pool
    tb::DBuf<char> large, below;
    large.ensure(tb::DevPool::kDirect);
    below.ensure(tb::DevPool::kDirect - 1);
    expect(!large.dev && below.dev, "which buffers come from the pool");
  }
  pool.reset();
  expect(pools == 0, "the pool outlives its last buffer");
  printf("%s\n", bad ? "bad" : "ok");
  return bad != 0;
}
