// See ifosb_mem.h.
#include "ifosb_mem.h"

#include <algorithm>
#include <mutex>
#include <vector>

namespace ifosb {
namespace {

// Held while spares are given back, so that an owner that goes waits for it. An owner may
// list a spare while it keeps it from being given back: give_back() never waits for one.
std::mutex &list_mutex() {
    static std::mutex *m = new std::mutex;  // outlives every owner
    return *m;
}
std::vector<Spare *> &list() {
    static std::vector<Spare *> *l = new std::vector<Spare *>;
    return *l;
}

}  // namespace

void spare_add(Spare *s) {
    std::lock_guard<std::mutex> l(list_mutex());
    list().push_back(s);
}

void spare_remove(Spare *s) {
    std::lock_guard<std::mutex> l(list_mutex());
    list().erase(std::remove(list().begin(), list().end(), s), list().end());
}

cudaError_t device_alloc(void **p, size_t bytes) {
    cudaError_t r = cudaMalloc(p, bytes);
    if (r != cudaErrorMemoryAllocation) return r;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return r;
    std::lock_guard<std::mutex> l(list_mutex());
    std::vector<Spare *> &v = list();
    for (size_t q = 0; r == cudaErrorMemoryAllocation && q < v.size();) {
        if (v[q]->device != dev || !v[q]->give_back()) {
            ++q;
            continue;
        }
        v.erase(v.begin() + q);
        cudaGetLastError();  // of the attempt that failed
        r = cudaMalloc(p, bytes);
    }
    return r;
}

}  // namespace ifosb
