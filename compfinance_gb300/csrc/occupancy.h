// Resident blocks per SM of a kernel at a block size and a dynamic shared-memory size.
#pragma once
#include <cstddef>

namespace cf {

// As cudaOccupancyMaxActiveBlocksPerMultiprocessor, after raising the kernel's dynamic shared-memory
// limit to smem where it is lower; returns cudaError_t.  Answers are kept per device, kernel and
// sizes for the life of the process (a few hundred at most: 64 KB), so that a launch asks the
// runtime once and not every time: the two calls took 4 us, and a choice between staging forms
// made up to nine of them.  The limit is only ever raised: callers of any context and thread may
// launch with any size they asked about.
int kernel_occupancy(const void* fn, int threads, size_t smem, int* blocks);

}  // namespace cf
