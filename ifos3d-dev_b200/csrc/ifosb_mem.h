// Device memory of the library's objects, and what some of them hold only for as long as
// no other wants it.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace ifosb {

// Device memory whose owner can do without it, at a price in speed.
struct Spare {
    int device = -1;
    // Frees it; false while the owner's kernels may be using it. Any thread may ask.
    virtual bool give_back() = 0;

protected:
    ~Spare() = default;
};
// Listed from when it holds memory until it has been given back or its owner goes.
void spare_add(Spare *s);
void spare_remove(Spare *s);

// cudaMalloc; while it fails for want of memory, the current device's spares are given back
// one after another.
cudaError_t device_alloc(void **p, size_t bytes);

}  // namespace ifosb
