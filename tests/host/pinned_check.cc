// PinArena and PinBuf (tioga_b200/csrc/devmem.h) over a fake runtime: one
// page-locked allocation serves an instance's small buffers and slots, pieces
// never overlap, and what outgrows it is allocated and freed by itself.
#include <stdio.h>
#include <stdlib.h>

#include <utility>
#include <vector>

#include "devmem.h"

namespace {
int allocs = 0, live = 0, bad = 0;
bool none_left = false;
void expect(bool ok, const char* what) {
  if (!ok) {
    printf("failed: %s\n", what);
    bad++;
  }
}
}  // namespace

extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (none_left) return cudaErrorMemoryAllocation;
  *p = malloc(n);
  allocs++;
  live++;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  free(p);
  live--;
  return cudaSuccess;
}
}

int main() {
  {
    tb::PinArena arena;
    tb::PinBuf a, b, c;
    expect(a.ensure(1024, arena) == cudaSuccess && b.ensure(300, arena) == cudaSuccess, "small buffers");
    char* slots = arena.slots();
    std::vector<std::pair<char*, size_t>> pieces = {{slots, tb::PinArena::kSlots}, {a.p, a.n}, {b.p, b.n}};
    expect(c.ensure(20000, arena) == cudaSuccess, "a third");
    pieces.push_back({c.p, c.n});
    a.ensure(40000, arena);  // outgrown: another piece
    pieces.push_back({a.p, a.n});
    for (size_t i = 0; i < pieces.size(); i++) {
      const char* p = pieces[i].first;
      expect(p >= arena.p && p + pieces[i].second <= arena.p + tb::PinArena::kBytes, "a piece leaves the arena");
      expect((p - arena.p) % 64 == 0, "a piece is not aligned");
      for (size_t j = 0; j < i; j++)
        expect(p + pieces[i].second <= pieces[j].first || pieces[j].first + pieces[j].second <= p, "pieces overlap");
    }
    expect(allocs == 1, "more than one allocation for an instance's usual buffers");
    char* kept = a.p;
    expect(a.ensure(100, arena) == cudaSuccess && a.p == kept, "a buffer that is large enough moves");
    b.ensure(600000, arena);  // past the arena
    expect(allocs == 2 && b.n >= 600000, "a large buffer has an allocation of its own");
    b.ensure(2000000, arena);
    expect(allocs == 3 && live == 2, "a buffer's own allocation is freed when it grows");
    none_left = true;
    expect(c.ensure(900000, arena) != cudaSuccess && c.n == 0, "an allocation that fails is reported");
    tb::PinArena other;
    expect(!other.slots() && !other.take(10), "an arena that cannot be made gives nothing");
    none_left = false;
    a.release();
    b.release();
    c.release();
    arena.release();
  }
  expect(live == 0, "memory is left");
  printf("%s\n", bad ? "bad" : "ok");
  return bad != 0;
}
