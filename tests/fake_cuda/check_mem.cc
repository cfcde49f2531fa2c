// device_alloc and the spares (ifosb_mem.h) on the fake runtime.
#include "../../ifos3d-dev_b200/csrc/ifosb_mem.h"
#include "fake.h"

#include <mutex>
#include <thread>

using namespace ifosb;

struct Held : Spare {
    void *p = nullptr;
    std::mutex busy;
    int asked = 0;
    Held(int dev, size_t bytes) {
        device = dev;
        if (cudaMalloc(&p, bytes) == cudaSuccess) spare_add(this);
    }
    bool give_back() override {
        ++asked;
        std::unique_lock<std::mutex> l(busy, std::try_to_lock);
        if (!l.owns_lock()) return false;
        cudaFree(p);
        p = nullptr;
        return true;
    }
};

static int run() {
    void *p = nullptr;
    fake().free_bytes = 1000;
    Held a(0, 300), b(0, 300), other(1, 300);
    CHECK(a.p && b.p && other.p);  // 100 left
    // what fits asks nobody
    CHECK(device_alloc(&p, 50) == cudaSuccess && a.asked + b.asked + other.asked == 0);
    cudaFree(p);
    // one spare of this device is enough: the next one keeps its memory
    CHECK(device_alloc(&p, 350) == cudaSuccess && !a.p && b.p && b.asked == 0);
    cudaFree(p);  // 400 free
    // a spare in use is not waited for and stays listed
    {
        std::unique_lock<std::mutex> use(b.busy);
        cudaError_t r = cudaSuccess;
        std::thread([&] { r = device_alloc(&p, 600); }).join();
        CHECK(r == cudaErrorMemoryAllocation && b.p && b.asked == 1);
    }
    CHECK(device_alloc(&p, 600) == cudaSuccess && !b.p && b.asked == 2);
    cudaFree(p);  // 700 free
    // nothing left to ask, another device's spare untouched; one that has gone is not asked
    CHECK(device_alloc(&p, 900) == cudaErrorMemoryAllocation);
    CHECK(a.asked == 1 && b.asked == 2 && other.p && other.asked == 0);
    spare_remove(&other);
    other.device = 0;
    CHECK(device_alloc(&p, 900) == cudaErrorMemoryAllocation && other.asked == 0);
    return 0;
}
int main() { return run(); }
