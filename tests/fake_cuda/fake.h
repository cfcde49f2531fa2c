// The fake runtime's state, for the checks that use it.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <functional>
#include <map>
#include <mutex>
#include <vector>

struct FakeStream {
    std::vector<std::function<void()>> ops;
    size_t done = 0;
};
struct FakeEvent {
    FakeStream *st = nullptr;  // where it was last recorded
    size_t upto = 0;           // operations of that stream that come before
};

struct Fake {
    std::recursive_mutex m;
    std::map<char *, size_t> device, pinned;
    size_t free_bytes = (size_t)1 << 40;
    // counts and faults
    int driver_copies = 0;   // of pageable memory
    int chunk_copies = 0;    // to or from pinned memory
    int fail_chunk = -1;     // this chunk copy fails (counted from 0)
    int mallocs_failed = 0;
};
Fake &fake();
void fake_drain();                 // runs all that is queued on any stream
extern thread_local int fake_context;  // the thread's: 0 the device's primary, else the caller's own

// in a function that returns 0 when all is well
#define CHECK(c)                                                     \
    do {                                                             \
        if (!(c)) {                                                  \
            std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c); \
            return 1;                                                \
        }                                                            \
    } while (0)
