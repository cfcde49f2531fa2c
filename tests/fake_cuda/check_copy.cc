// host_copy (ifosb_copy.h) on the fake runtime. One argument: what to check.
#include "../../ifos3d-dev_b200/csrc/ifosb_copy.h"
#include "fake.h"

#include <cstring>
#include <string>
#include <thread>

using namespace ifosb;

// enough cores for several threads a copy, whatever the machine has
unsigned std::thread::hardware_concurrency() noexcept { return 16; }

constexpr size_t MB = 1 << 20;

struct Device {
    char *p = nullptr;
    explicit Device(size_t n) { cudaMalloc((void **)&p, n); }
    ~Device() { cudaFree(p); }
};
static std::vector<char> pattern(size_t n, int seed) {
    std::vector<char> v(n);
    unsigned x = 12345u + seed;
    for (char &c : v) c = (char)((x = x * 1664525u + 1013904223u) >> 24);
    return v;
}
static cudaStream_t stream() {
    cudaStream_t s;
    cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    return s;
}

// Up and down at this size: the bytes arrive, through the chunks or not.
static int both_ways(size_t n, cudaStream_t st, bool up_chunks, bool down_chunks, bool result) {
    Device d(n);
    const std::vector<char> in = pattern(n, (int)n);
    fake().chunk_copies = fake().driver_copies = 0;
    CHECK(host_copy(d.p, in.data(), n, st) == cudaSuccess);
    CHECK((fake().chunk_copies > 0) == up_chunks && (fake().driver_copies == 1) == !up_chunks);
    std::vector<char> out(n + 2, 7);  // what comes after `in` on the stream, into an array of its own
    fake().chunk_copies = fake().driver_copies = 0;
    CHECK(host_copy(out.data() + 1, d.p, n, st, result) == cudaSuccess);
    CHECK((fake().chunk_copies > 0) == down_chunks && (fake().driver_copies == 1) == !down_chunks);
    CHECK(std::memcmp(out.data() + 1, in.data(), n) == 0 && out[0] == 7 && out[n + 1] == 7);
    return 0;
}
static int sizes() {
    cudaStream_t st = stream();
    host_copy_retain();
    for (size_t at : {4 * MB, 5 * MB, 8 * MB, 9 * MB, 16 * MB, 17 * MB, 24 * MB, 33 * MB})
        for (long d : {-5, -4, -1, 0, 1, 4, 5}) {
            const size_t n = at + d;
            if (both_ways(n, st, n >= 8 * MB, n >= 8 * MB, false)) return 1;
            if (both_ways(n, st, n >= 8 * MB, n >= 4 * MB, true)) return 1;
        }
    for (size_t n : {(size_t)1, (size_t)4, MB - 4, MB + 4})
        if (both_ways(n, st, false, false, true)) return 1;
    host_copy_release();
    CHECK(fake().pinned.empty());
    return 0;
}

// A partner that is not pageable memory leaves the copy to the driver.
static int partners() {
    cudaStream_t st = stream();
    host_copy_retain();
    const size_t n = 12 * MB;
    Device a(n), b(n);
    char *pin;
    cudaHostAlloc((void **)&pin, n, cudaHostAllocDefault);
    const std::vector<char> in = pattern(n, 3);
    std::memcpy(pin, in.data(), n);
    fake().chunk_copies = fake().driver_copies = 0;
    CHECK(host_copy(a.p, pin, n, st) == cudaSuccess);
    CHECK(host_copy(b.p, a.p, n, st) == cudaSuccess);
    CHECK(cudaStreamSynchronize(st) == cudaSuccess);
    std::memset(pin, 0, n);
    CHECK(host_copy(pin, b.p, n, st, true) == cudaSuccess && cudaStreamSynchronize(st) == cudaSuccess);
    CHECK(fake().chunk_copies == 2 && fake().driver_copies == 0);  // whole copies from and to the pinned array
    CHECK(std::memcmp(pin, in.data(), n) == 0);
    std::vector<char> out(n);
    CHECK(host_copy(out.data(), in.data(), n, st) == cudaSuccess);
    CHECK(fake().driver_copies == 1 && out == in);
    cudaFreeHost(pin);
    host_copy_release();
    return 0;
}

// Two callers: one has the chunks, the other goes the driver's way; both get their bytes.
static int callers() {
    host_copy_retain();
    int bad[2] = {0, 0};
    auto work = [&](int who) {
        cudaStream_t st = stream();
        Device d(20 * MB);
        for (int q = 0; q < 12 && !bad[who]; ++q) {
            const size_t n = 9 * MB + 777 * q + who;
            const std::vector<char> in = pattern(n, 100 * who + q);
            std::vector<char> out(n);
            bad[who] = host_copy(d.p, in.data(), n, st) != cudaSuccess || host_copy(out.data(), d.p, n, st, q & 1) != cudaSuccess ||
                       cudaStreamSynchronize(st) != cudaSuccess || out != in;
        }
    };
    std::thread t(work, 1);
    work(0);
    t.join();
    CHECK(!bad[0] && !bad[1]);
    host_copy_release();
    return 0;
}

// A chunk that cannot be sent: the driver's copy stands in, and what the caller's stream
// does next to the same memory is not undone by chunks that were on their way.
static int failed() {
    cudaStream_t st = stream();
    host_copy_retain();
    const size_t n = 20 * MB;
    for (int chunk = 0; chunk < 20; ++chunk) {
        Device d(n);
        const std::vector<char> in = pattern(n, chunk), next = pattern(MB, 50 + chunk);
        fake().chunk_copies = fake().driver_copies = 0;
        fake().fail_chunk = chunk;
        CHECK(host_copy(d.p, in.data(), n, st) == cudaSuccess);
        fake().fail_chunk = -1;
        CHECK(fake().driver_copies == 1);
        for (size_t q = 0; q < n / MB; ++q)
            CHECK(cudaMemcpyAsync(d.p + q * MB, next.data(), MB, cudaMemcpyDefault, st) == cudaSuccess);
        CHECK(cudaStreamSynchronize(st) == cudaSuccess);
        fake_drain();
        for (size_t q = 0; q < n / MB; ++q) CHECK(std::memcmp(d.p + q * MB, next.data(), MB) == 0);
        // and the other way: the array is whole when the call returns
        std::vector<char> out(n);
        const std::vector<char> want(d.p, d.p + n);
        fake().chunk_copies = 0;
        fake().fail_chunk = chunk;
        CHECK(host_copy(out.data(), d.p, n, st, true) == cudaSuccess);
        fake().fail_chunk = -1;
        fake_drain();
        CHECK(out == want);
        // the chunks still serve
        if (both_ways(n, st, true, true, true)) return 1;
    }
    host_copy_release();
    return 0;
}

// The caller's context stays the calling thread's.
static int context() {
    cudaStream_t st = stream();
    host_copy_retain();
    fake_context = 5;
    if (both_ways(20 * MB, st, true, true, true)) return 1;
    CHECK(fake_context == 5);
    host_copy_release();
    return 0;
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "sizes") return sizes();
    if (what == "partners") return partners();
    if (what == "callers") return callers();
    if (what == "failed") return failed();
    if (what == "context") return context();
    return 2;
}
