// kernel_reaches (tioga_b200/csrc/devmem.h): which of a caller's arrays a kernel
// of the instance's device may work on.
#include <stdio.h>

#include "devmem.h"

namespace {
cudaPointerAttributes answer;
cudaError_t status = cudaSuccess;
}  // namespace

extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  *a = answer;
  return status;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}

int main() {
  int bad = 0;
  auto expect = [&](cudaMemoryType type, int device, uintptr_t p, size_t align, bool want, const char* what) {
    answer = {};
    answer.type = type;
    answer.device = device;
    if (tb::kernel_reaches(reinterpret_cast<void*>(p), 1, align) != want) {
      printf("failed: %s\n", what);
      bad++;
    }
  };
  expect(cudaMemoryTypeDevice, 1, 0x1000, 4, true, "this device's memory");
  expect(cudaMemoryTypeDevice, 1, 0x1004, 4, true, "an aligned part of it");
  expect(cudaMemoryTypeDevice, 1, 0x1002, 4, false, "a misaligned part of it");
  expect(cudaMemoryTypeDevice, 1, 0x1004, 8, false, "a misaligned part of it for doubles");
  expect(cudaMemoryTypeDevice, 0, 0x1000, 4, false, "another device's memory");
  expect(cudaMemoryTypeHost, 1, 0x1000, 4, false, "pinned host memory");
  expect(cudaMemoryTypeManaged, 1, 0x1000, 4, false, "managed memory");
  expect(cudaMemoryTypeUnregistered, 1, 0x1000, 4, false, "pageable host memory");
  expect(cudaMemoryTypeDevice, 1, 0, 4, false, "no array");
  status = cudaErrorInvalidValue;
  expect(cudaMemoryTypeDevice, 1, 0x1000, 4, false, "an unknown pointer");
  printf("%s\n", bad ? "bad" : "ok");
  return bad != 0;
}
