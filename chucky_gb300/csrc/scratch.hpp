// Device scratch of one call, stream-ordered, from a bounded pool.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#ifndef CHUCKY_SCRATCH_EMULATED // (the CPU emulation of the kernels has its own)
namespace chucky {

// What the pool keeps between calls at most (more is handed back to the
// device at the next synchronization after its work is done).  Mapping device memory afresh costs a call
// hundreds of microseconds.
constexpr size_t kScratchKept = size_t(256) << 20;

// `bytes` of device memory for work queued on `st` from now on, or nullptr:
// out of memory, the stream is being captured (a graph would own the
// memory), or the context cannot be told from others.  No host wait.
void* scratch_acquire(size_t bytes, cudaStream_t st);
// The memory is free again once the work queued on `st` so far is done.
void scratch_release(void* p, cudaStream_t st);
// Hands the pool's unused memory of the current context back.
void scratch_trim();

// The ID of the calling thread's current context (never reused), 0: unknown.
unsigned long long current_context_id();

} // namespace chucky
#else
namespace chucky {
inline void scratch_trim() {}
} // namespace chucky
#endif
