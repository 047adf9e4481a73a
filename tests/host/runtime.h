// A CUDA runtime without a device, for tests that link the library's own objects: device memory
// is host memory whose 32-bit words are all 1, copies copy, kernels do nothing, and the
// allocation numbered `fail_at` (and, with `fail_on`, every later one) is refused. Functions
// not defined here return success (generated by host_program.py).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <map>

namespace fake {
extern long allocations, fail_at, fail_on;  // of device memory
extern std::map<void*, size_t> live;        // every block in use
extern long syncs;
}  // namespace fake
