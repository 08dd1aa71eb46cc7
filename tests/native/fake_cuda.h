// What a test sees of the fake CUDA runtime (fake_cuda.cpp).
#pragma once
#include <cstdint>

struct Fake {
  uint64_t outputs = 0;    // how many outputs the next runs "find"
  uint64_t overflows = 0;  // how many of the next runs overflow first
  uint64_t dead = 0;       // uses of freed or null buffers so far
  uint64_t allocations = 0;
  uint64_t captures = 0;   // stream captures so far
  uint64_t kernels = 0;    // kernels run so far
  uint64_t marks = 0;      // marking launches so far
  uint64_t d2h = 0;        // bytes copied back by eager runs so far
};

Fake& fake();
// The allocation after the next `skip` ones fails.
void fake_fail_allocation(int64_t skip);
// Run (or record) one kernel that does nothing.
void fake_kernel();
