#include "fake.h"

#include <cstdlib>
#include <cstring>

Fake &fake() {
    static Fake *f = new Fake;
    return *f;
}
thread_local int fake_context = 0;
static std::vector<FakeStream *> &streams() {
    static std::vector<FakeStream *> *v = new std::vector<FakeStream *>;
    return *v;
}
#define LOCK std::lock_guard<std::recursive_mutex> lock(fake().m)

static void run_to(FakeStream *s, size_t upto) {
    while (s->done < upto) {
        const std::function<void()> op = s->ops[s->done];
        s->ops[s->done++] = nullptr;
        op();
    }
}
void fake_drain() {
    LOCK;
    for (FakeStream *s : streams()) run_to(s, s->ops.size());
}

static bool within(const std::map<char *, size_t> &m, const void *p) {
    auto it = m.upper_bound((char *)p);
    if (it == m.begin()) return false;
    --it;
    return (char *)p < it->first + it->second;
}

cudaError_t cudaMalloc(void **p, size_t bytes) {
    LOCK;
    if (bytes > fake().free_bytes) {
        ++fake().mallocs_failed;
        return cudaErrorMemoryAllocation;
    }
    fake().free_bytes -= bytes;
    *p = std::calloc(1, bytes);
    fake().device[(char *)*p] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    LOCK;
    if (!p) return cudaSuccess;
    fake().free_bytes += fake().device[(char *)p];
    fake().device.erase((char *)p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) {
    LOCK;
    *p = std::calloc(1, bytes);
    fake().pinned[(char *)*p] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    LOCK;
    fake().pinned.erase((char *)p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    LOCK;
    *s = new FakeStream;
    streams().push_back(*s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    LOCK;
    run_to(s, s->ops.size());
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    return cudaStreamSynchronize(s);  // the object stays: an event may name it
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = new FakeEvent;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    LOCK;
    e->st = s;
    e->upto = s->ops.size();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    LOCK;
    if (e->st) run_to(e->st, e->upto);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    LOCK;
    FakeStream *of = e->st;
    const size_t upto = e->upto;
    s->ops.push_back([of, upto] {
        if (of) run_to(of, upto);
    });
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t bytes, cudaMemcpyKind, cudaStream_t s) {
    LOCK;
    Fake &f = fake();
    const bool ps = within(f.pinned, src), pd = within(f.pinned, dst);
    const bool hs = !ps && !within(f.device, src), hd = !pd && !within(f.device, dst);
    if (ps || pd) {
        if (f.chunk_copies++ == f.fail_chunk) return cudaErrorUnknown;
    } else if (hs || hd) {
        ++f.driver_copies;
    }
    if (hs) {  // pageable source: staged before the call returns
        std::vector<char> staged((const char *)src, (const char *)src + bytes);
        s->ops.push_back([dst, staged] { std::memcpy(dst, staged.data(), staged.size()); });
    } else {
        s->ops.push_back([dst, src, bytes] { std::memcpy(dst, src, bytes); });
    }
    if (hd) run_to(s, s->ops.size());  // to pageable memory: there when the call returns
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    LOCK;
    a->type = within(fake().device, p) ? cudaMemoryTypeDevice : within(fake().pinned, p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) {
    fake_context = 0;  // makes the device's primary context the thread's
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
