// DonorSlots::at (tioga_b200/csrc/engine.h) on the host: places of good
// indices, -1 for every index that is outside its array.
#include <limits.h>
#include <stdio.h>

#include "engine.h"

int main() {
  // two systems of two and three blocks, K = 3 slots per node
  tb::BlockInfo bi[5] = {};
  for (int b = 0; b < 5; b++) bi[b].sblk0 = b < 2 ? 0 : 2;
  const tb::DonorSlots s{nullptr, 3, 100, 60, bi, 5};
  int bad = 0;
  auto expect = [&](long long got, long long want, const char* what) {
    if (got != want) {
      printf("failed: %s: %lld\n", what, got);
      bad++;
    }
  };
  expect(s.at(0, 0, 0), 0, "first");
  expect(s.at(99, 4, 59), 99 * 3 + 2, "last");
  expect(s.at(7, 1, 3), 7 * 3 + 1, "second block");
  expect(s.at(7, 2, 3), 7 * 3, "first block of the second system");
  for (int g : {-1, 100, INT_MAX, INT_MIN}) expect(s.at(g, 0, 0), -1, "node");
  for (int d : {-1, 5, INT_MAX, INT_MIN}) expect(s.at(0, d, 0), -1, "block");
  for (int c : {-1, 60, INT_MAX, INT_MIN}) expect(s.at(0, 0, c), -1, "cell");
  const tb::DonorSlots few{nullptr, 2, 100, 60, bi, 5};
  expect(few.at(0, 4, 0), -1, "a block past the node's slots");
  bi[1].sblk0 = 2;
  expect(s.at(0, 1, 0), -1, "a block before its system");
  printf("%s\n", bad ? "bad" : "ok");
  return bad != 0;
}
