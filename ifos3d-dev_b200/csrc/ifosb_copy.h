// Copies between pageable host memory (the callers' arrays) and the device.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <functional>

namespace ifosb {

// fn(0) .. fn(parts - 1), each once, on as many threads (the caller's among them).
void run_parts(int parts, const std::function<void(int)> &fn);
// Threads worth starting for `bytes` of host work.
int host_parts(size_t bytes);

// dst <- src in the order of `st`, like cudaMemcpyAsync with cudaMemcpyDefault. A large
// copy from or to pageable memory goes through pinned chunks filled or emptied by a few
// threads, and the call returns when the host side is done (a copy to the host: when it
// has arrived). result: dst is likely an array nobody has touched yet.
cudaError_t host_copy(void *dst, const void *src, size_t bytes, cudaStream_t st, bool result = false);

// The pinned chunks are shared by the process's engines and optimisers: made by the
// first large copy, given back when the last of them goes.
void host_copy_retain();
void host_copy_release();

}  // namespace ifosb
