// A CUDA runtime on the CPU for tests of the host driver: device memory is host memory, and everything
// ordered on a stream is queued in issue order and runs when the host waits, as late as it may.  An
// asynchronous copy reads its source then, as a system does whose devices read pageable memory directly.
// Device memory has a budget; freed blocks of a memory pool count against it until the pool is trimmed.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <functional>

namespace fake {
void enqueue(std::function<void()> op);
extern size_t budget;       // bytes of device memory
size_t used();              // live blocks and what pools hold
extern bool threadsFail;    // pthread_create returns EAGAIN
size_t pending();           // operations that no wait has run yet
extern int failingRecord;   // the event record, counted from now, that fails; 0: none
}  // namespace fake
